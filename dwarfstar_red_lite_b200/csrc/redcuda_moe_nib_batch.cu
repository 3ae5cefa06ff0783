// Routed experts of a batch in the nibble layout (redcuda_moe_nib.cu): gate/up with SiLU * mul, or down, of the pairs that
// k_group_pairs sorted by expert and cut into work items of at most 8 pairs (wide digits: 6).
//
// Arithmetic as in redcuda_moe_nib.cu: mma.sync m16n8k32 s8, weights as A, activation digits as B, s32 sums per 32-weight group
// times the integer group scale, fp32 scaling by d / 8 per 256-column block.
//
// What bounds it: per SM a record (16 rows x 256 columns, 2208 bytes) takes 96 cycles of HBM time. For a full item it also takes
// 192 cycles of one scheduler's MMA and of its integer multiply pipe each (8 and 2 cycles an instruction, measured). So
//   - a warp works on two records that meet the same digits at a time (the gate and the up tile of the same rows; two
//     neighbouring tiles of down): the digits are read from shared memory once for both, SiLU(gate) * up needs no exchange between
//     warps;
//   - a lane loads its fragments of a record straight into registers, the next step's as soon as this step's are used up: no
//     staging in shared memory, no barrier to poll;
//   - nothing in the main loop waits for another warp. The digits of an item are copied into one of two buffers while the other
//     one is multiplied, and a warp draws its next piece (a pair of tiles over the whole row) from a counter in shared memory when
//     the first records of it are to be requested;
//   - a block takes contiguous runs of pieces, half of its share first, then a quarter, and so on, from a global counter: an
//     item's digits are staged by the few blocks that share it, and blocks that start late (the shared expert runs beside this
//     kernel on another stream) take fewer runs.
// The form before it drew units of 4 tiles per block, staged the digits anew for each and met at two block barriers per unit.
#define RC_PDL_DEFAULT 0
#include "redcuda_nib.cuh"
#include "redcuda_kernels.cuh"

#include <type_traits>

namespace rc {

constexpr uint32_t NBB_WARPS = 12u;               // 168 registers: two records' sums and results for a full item, and a step's fragments; ten of the 24 forms spill 8 to 24 bytes
constexpr uint32_t NBB_COLS = 24u;                // digit columns of an item
// tile pairs of a piece: enough that drawing it is small beside it, few enough that a small batch still reaches every warp
__host__ __device__ constexpr uint32_t nbb_pairs(uint32_t ncols) { return ncols >= 1024u ? 1u : ncols == 512u ? 2u : 4u; }
__host__ __device__ constexpr uint32_t nbb_smem(uint32_t ncols) { return 2u * NBB_COLS * (ncols + 32u); }
constexpr uint32_t NBB_MIN_RUN = 8u;              // pieces of the last, smallest runs

// streamed once: past L1
__device__ __forceinline__ uint4 nbb_ldg(const uint8_t *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 nbb_ldg2(const uint8_t *p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t nbb_ldg1(const uint8_t *p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
// A lane's part of the two records of a step. q[m][h][i]: codes of row g + 8 h, 32-column groups 4 i .. 4 i + 3, of record m; sc[m][i]: the
// scales of these groups, rows g and g + 8; d[m]: d of the two rows. Every piece is loaded again for the next step once it is used up.
struct NbbFrag { uint4 q[2][2][2]; uint2 sc[2][2]; uint32_t d[2]; };
// Half i (four groups) of the two records against NT tiles of digits: the exact s32 products of a group times its integer scale, added up
// in blk[m][n]: rows g (0, 1) and g + 8 (2, 3), columns 2 t and 2 t + 1 of tile n.
template <uint32_t FMT, int NT, uint32_t BPITCH>
__device__ __forceinline__ void nbb_half(const NbbFrag &F, const int i, const int8_t *Bl, const int (&z)[4], int (&blk)[2][NT][4]) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        uint2 bf[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) bf[n] = *reinterpret_cast<const uint2 *>(Bl + (uint32_t)n * 8u * BPITCH + (uint32_t)(4 * i + kk) * 32u);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint4 &qa = F.q[m][0][i], &qb = F.q[m][1][i];
            const uint32_t wa = kk == 0 ? qa.x : kk == 1 ? qa.y : kk == 2 ? qa.z : qa.w, wb = kk == 0 ? qb.x : kk == 1 ? qb.y : kk == 2 ? qb.z : qb.w;
            uint32_t a0, a1, a2, a3;
            nb_expand<FMT>(wa, a0, a2);
            nb_expand<FMT>(wb, a1, a3);
            const int sa = (int)nb_prmt(F.sc[m][i].x, 0u, 0x4440u + (uint32_t)kk);
            const int sb = (int)nb_prmt(F.sc[m][i].y, 0u, 0x4440u + (uint32_t)kk);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                int p[4];
                nb_mma(p, a0, a1, a2, a3, bf[n].x, bf[n].y, z);
                blk[m][n][0] += sa * p[0]; blk[m][n][1] += sa * p[1];
                blk[m][n][2] += sb * p[2]; blk[m][n][3] += sb * p[3];
            }
        }
    }
}

// What the warps of a block share about the item part they work on
struct NbbSeg {
    const uint8_t *rec;        // the expert's first record (gate, or down)
    uint32_t first, count;     // pieces [first, first + count) of the item; count 0: no work is left
    uint32_t nt;               // pairs
    uint32_t row[8];           // their ids
    float sx[8];               // and scales (three digits)
};

// GATEUP: the two records of a step are the same tile of gate and of up. Otherwise they are two neighbouring tiles.
template <uint32_t FMT, bool GATEUP, uint32_t NCOLS>
__global__ void __launch_bounds__(NBB_WARPS * 32u, 1) k_nib_batch(const __grid_constant__ MmaArgs A) {
    pdl_prologue();
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr bool WIDE = FMT != NIB_IQ2;
    constexpr uint32_t BPR = NCOLS / 256u, TPP = nbb_pairs(NCOLS), BPITCH = NCOLS + 32u, ND = WIDE ? 4u : 3u;
    __shared__ NbbSeg s_seg[2];
    __shared__ float s_sxw[2][WIDE ? NIB_WIDE_PAIRS * BPR : 1u];       // wide: scales of the item's pairs and blocks
    __shared__ uint32_t s_taken[2], s_left[2], s_run[2];               // pieces drawn, warps that are through with the buffer; what is left of the block's run
    __shared__ __align__(8) uint64_t s_told[2], s_full[2];             // the part's description is in s_seg; its pairs and digits are there as well
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    int8_t *digits = reinterpret_cast<int8_t *>(smem);
    const uint32_t full_s = nb_smem(&s_full[0]), told_s = nb_smem(&s_told[0]);
    const uint32_t ntile = A.nrows >> 4, npair = GATEUP ? ntile : ntile / 2u, PPI = (npair + TPP - 1u) / TPP;     // tile pairs and pieces of an item
    const uint32_t total = *A.n_items * PPI, share = (total + gridDim.x - 1u) / gridDim.x;
    bool failed = false;

    // run k of the launch: every block's first run is half of its share, the next ones a quarter, an eighth, ...; small shares are not cut
    auto run_of = [&](uint32_t k, uint32_t &lo, uint32_t &hi) {
        uint32_t base = 0u, r = k / gridDim.x, size = share <= 2u * NBB_WARPS ? share : max(share / 2u, NBB_MIN_RUN);
        for (; r; --r) { base += size * gridDim.x; if (base >= total) break; size = max(size / 2u, NBB_MIN_RUN); }
        lo = min(base + (k % gridDim.x) * size, total); hi = min(lo + size, total);
    };
    // Puts the block's next item part into buffer `buf` (all lanes of one warp; nobody else uses the buffer). The pairs that are not
    // there leave their digit columns as they are: a column of the product depends on no other.
    auto fill = [&](uint32_t buf) {
        NbbSeg &S = s_seg[buf];
        uint32_t lo = s_run[0], hi = s_run[1];
        if (lo >= hi && lo < total) {
            uint32_t k = 0u;
            if (lane == 0) k = gridDim.x + atomicAdd(A.work, 1u);
            run_of(__shfl_sync(0xffffffffu, k, 0), lo, hi);
        }
        uint32_t nt = 0u, row = 0u, count = 0u, p0 = 0u;
        if (lo < hi) {
            const uint32_t item = lo / PPI, first = lo - item * PPI, u = A.item_u[item];
            p0 = A.item_p0[item];
            uint32_t e = A.uexp[u] - A.expert_begin;
            nt = min(A.item_tok, A.ustart[u + 1u] - p0);
            if (e >= A.n_local) { if (A.status && lane == 0) A.status[ST_EXPERT_RANGE] = 1u; e = 0u; nt = 0u; }      // never index the arena with a foreign id
            count = min(PPI - first, hi - lo);
            if (lane == 0) { S.rec = A.w0 + (size_t)e * A.mat_bytes; S.first = first; S.nt = nt; }
        }
        __syncwarp();                // every lane has read the run
        // the description first: it lets the warps request weights while the pairs are looked up and their digits copied
        if (lane == 0) {
            S.count = count; s_run[0] = lo + count; s_run[1] = hi; s_taken[buf] = 0u; s_left[buf] = 0u;
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(told_s + 8u * buf) : "memory");
        }
        if (lane < nt) { row = A.sorted[p0 + lane]; S.row[lane] = row; row /= A.x_div; }
        if (!WIDE && lane < nt) S.sx[lane] = A.sx[row];
        if (WIDE)
#pragma unroll
            for (uint32_t i0 = 0u; i0 < NIB_WIDE_PAIRS * BPR; i0 += 32u) {
                const uint32_t i = i0 + lane, r = __shfl_sync(0xffffffffu, row, i / BPR & 31u);
                if (i < NIB_WIDE_PAIRS * BPR) s_sxw[buf][i] = i / BPR < nt ? A.sx[(size_t)r * BPR + i % BPR] : 0.f;
            }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(full_s + 8u * buf), "r"(nt * ND * NCOLS) : "memory");
        __syncwarp();
        const uint32_t j = lane / ND < 8u ? lane / ND : 0u, dg = lane % ND, src_row = __shfl_sync(0xffffffffu, row, j);
        // columns: three digits of one or two pairs per tile (3 * pair + digit) up to four pairs, a tile per digit beyond; wide: 4 * pair + digit
        const uint32_t col = WIDE ? lane : nt <= 4u ? 8u * (j >> 1) + 3u * (j & 1u) + dg : 8u * dg + j;
        if (lane < nt * ND)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         :: "r"(nb_smem(digits) + (buf * NBB_COLS + col) * BPITCH), "l"(A.xq + ((size_t)src_row * ND + dg) * NCOLS), "r"(NCOLS), "r"(full_s + 8u * buf) : "memory");
    };

    if (tid == 0) {
        for (uint32_t i = 0; i < 2u; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(told_s + 8u * i));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(full_s + 8u * i));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        uint32_t lo, hi;
        run_of(blockIdx.x, lo, hi);
        s_run[0] = lo; s_run[1] = hi;
    }
    __syncthreads();
    // ---- the warp's pieces ----
    struct Piece { const uint8_t *rec; uint32_t pair0, steps; };
    const size_t to_up = GATEUP ? (size_t)(A.w1 - A.w0) : 0u;
    uint32_t seg = 0u;                                   // the warp draws from item part seg, seg + 1, ... (buffer seg % 2)
    auto wait_for = [&](uint32_t bars, uint32_t k) {      // part k's description (told_s) or digits (full_s)
        if (!failed) failed = !__all_sync(0xffffffffu, nb_wait(bars + 8u * (k & 1u), (k >> 1) & 1u));
        return !failed;
    };
    // the first two parts; the second by the warp that a small batch has least work for
    if (warp == 0) fill(0u);
    else if (warp == NBB_WARPS - 1u && wait_for(told_s, 0u)) fill(1u);
    __syncwarp();
    auto told = [&](uint32_t k) {                        // is part k's description there already?
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(done) : "r"(told_s + 8u * (k & 1u)), "r"((k >> 1) & 1u) : "memory");
        return __all_sync(0xffffffffu, done != 0u) != 0;
    };
    auto draw = [&](uint32_t k, Piece &P) {              // a piece of part k, or false: the part has none left
        const NbbSeg &S = s_seg[k & 1u];
        uint32_t i = 0u;
        if (lane == 0) i = atomicAdd(&s_taken[k & 1u], 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= S.count) return false;
        P.pair0 = (S.first + i) * TPP;
        P.steps = min(TPP, npair - P.pair0) * BPR;
        P.rec = S.rec + (size_t)P.pair0 * ((GATEUP ? 1u : 2u) * BPR * NIB_REC);
        return true;
    };
    auto leave = [&](uint32_t k) {                       // the last warp to leave a buffer puts the next part into it
        uint32_t n = 0u;
        __syncwarp();
        if (lane == 0) { __threadfence_block(); n = atomicAdd(&s_left[k & 1u], 1u); __threadfence_block(); }
        if (__shfl_sync(0xffffffffu, n, 0) == NBB_WARPS - 1u) fill(k & 1u);
    };
    // this lane's place in the two records of step s of a piece
    auto place = [&](const Piece &P, uint32_t s, const uint8_t *&a, const uint8_t *&b) {
        if (GATEUP) { a = P.rec + (size_t)s * NIB_REC; b = a + to_up; }
        else {
            const uint32_t q = s / BPR;
            a = P.rec + (size_t)(s + q * BPR) * NIB_REC;
            b = a + BPR * NIB_REC;
        }
    };
    const uint32_t lane_code = nib_lane_off(g, t), lane_sc = NIB_SC_OFF + g * 8u, lane_d = NIB_D_OFF + g * 4u;
    NbbFrag F;
    auto load_half = [&](const int i, const uint8_t *a, const uint8_t *b) {
        F.sc[0][i] = nbb_ldg2(a + lane_sc + 64 * i); F.sc[1][i] = nbb_ldg2(b + lane_sc + 64 * i);
        F.q[0][0][i] = nbb_ldg(a + lane_code + 512 * i); F.q[0][1][i] = nbb_ldg(a + lane_code + 1024 + 512 * i);
        F.q[1][0][i] = nbb_ldg(b + lane_code + 512 * i); F.q[1][1][i] = nbb_ldg(b + lane_code + 1024 + 512 * i);
    };
    auto load_d = [&](const uint8_t *a, const uint8_t *b) { F.d[0] = nbb_ldg1(a + lane_d); F.d[1] = nbb_ldg1(b + lane_d); };
    // A fragment is loaded half a step before its use, which a few warps on an SM cannot hide from HBM: where fewer than half of a block's
    // warps get a piece, the piece's records, which lie together, are sent for in L2 at once. us a layer without and with: 2 tokens (5 pieces
    // a block) 49.6 and 48.1, but 3 tokens (7) 44.2 and 45.3, 6 (13) 52.3 and 56.1. (Sent for by the warp that fills the buffer, before the others know of
    // the part, they take the first loads' place: 2 tokens 51.0 against 50.5.)
    auto send_for = [&](const Piece &P) {
        if (lane == 0) {
            const uint32_t bytes = P.steps * NIB_REC;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(P.rec), "r"(GATEUP ? bytes : 2u * bytes) : "memory");
            if (GATEUP) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(P.rec + to_up), "r"(bytes) : "memory");
        }
    };
    int zero[4];                     // opaque to the compiler: four registers that stay zero, the accumulator input of every MMA
    asm volatile("mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;" : "=r"(zero[0]), "=r"(zero[1]), "=r"(zero[2]), "=r"(zero[3]));

    Piece P{}, N{};
    uint32_t digits_of = 0xffffffffu;    // the part whose digits this warp has waited for
    bool have = false, more = true;  // N holds the next piece, whose first step is in F; there may be one
    for (;;) {
        if (have) P = N;
        else {
            for (;;) {
                if (!wait_for(told_s, seg)) break;
                if (s_seg[seg & 1u].count == 0u) { more = false; break; }
                if (draw(seg, P)) break;
                leave(seg); ++seg;
            }
            if (failed || !more) break;
            const uint8_t *a, *b;
            place(P, 0u, a, b);
            load_half(0, a, b); load_half(1, a, b); load_d(a, b);
            if (2u * share < NBB_WARPS) send_for(P);
        }
        have = false;
        if (digits_of != seg) { if (!wait_for(full_s, seg)) break; digits_of = seg; }
        const uint32_t cur = seg, buf = seg & 1u;
        const NbbSeg &S = s_seg[buf];
        const uint32_t nt = S.nt;
        // The next piece is drawn when its first step is due: from this item part or, if the block has it already, from the next
        // (never from the one behind that: its buffer is this part's).
        auto draw_next = [&]() {
            if (!more) return;
            if (seg == cur) {
                if (draw(cur, N)) { have = true; return; }
                seg = cur + 1u;
            }
            if (!told(seg)) return;
            if (s_seg[seg & 1u].count == 0u) more = false; else have = draw(seg, N);
        };
        const int8_t *Bl = digits + (buf * NBB_COLS + g) * BPITCH + 8u * t;
        auto work = [&](auto nt_tag, auto packed_tag) {
            constexpr int NT = decltype(nt_tag)::value;
            constexpr bool PACKED = decltype(packed_tag)::value;
            for (uint32_t q = 0u, s = 0u; s < P.steps; ++q) {
                float out[2][NT][WIDE ? 2 : 4];
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int j = 0; j < (WIDE ? 2 : 4); ++j) out[m][n][j] = 0.f;
#pragma unroll 1
                for (uint32_t c = 0u; c < BPR; ++c, ++s) {
                    if (s + 1u == P.steps) draw_next();
                    const uint8_t *a, *b;            // the step behind this one; where none is known, this piece's first records are read again
                    if (s + 1u < P.steps) place(P, s + 1u, a, b); else if (have) place(N, 0u, a, b); else place(P, 0u, a, b);
                    int blk[2][NT][4];
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int n = 0; n < NT; ++n) blk[m][n][0] = blk[m][n][1] = blk[m][n][2] = blk[m][n][3] = 0;
                    nbb_half<FMT, NT, BPITCH>(F, 0, Bl + c * 256u, zero, blk);
                    load_half(0, a, b);
                    nbb_half<FMT, NT, BPITCH>(F, 1, Bl + c * 256u, zero, blk);
                    load_half(1, a, b);
                    float d[2][2];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const __half2 h = *reinterpret_cast<const __half2 *>(&F.d[m]);
                        d[m][0] = 0.125f * __low2float(h); d[m][1] = 0.125f * __high2float(h);
                    }
                    load_d(a, b);
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            if constexpr (WIDE) {
                                const float w = s_sxw[buf][(2u * n + (t >> 1)) * BPR + c] * (t & 1u ? 65536.0f : 1.0f);      // a power of two: d * w is exact
                                out[m][n][0] += (d[m][0] * w) * fmaf(256.0f, (float)blk[m][n][1], (float)blk[m][n][0]);
                                out[m][n][1] += (d[m][1] * w) * fmaf(256.0f, (float)blk[m][n][3], (float)blk[m][n][2]);
                            } else {
                                out[m][n][0] += d[m][0] * (float)blk[m][n][0]; out[m][n][1] += d[m][0] * (float)blk[m][n][1];
                                out[m][n][2] += d[m][1] * (float)blk[m][n][2]; out[m][n][3] += d[m][1] * (float)blk[m][n][3];
                            }
                        }
                }
                // v0, v1 = the value of pair pr, row r (0 .. 15) of the two tiles
                const uint32_t pair = P.pair0 + q, row0 = (GATEUP ? pair : 2u * pair) << 4;
                auto store = [&](uint32_t pr, uint32_t r, float v0, float v1) {
                    float *o = A.out + (size_t)S.row[pr] * A.out_stride + row0 + r;
                    if (GATEUP) *o = (v0 / (1.0f + expf(-v0))) * v1;
                    else { o[0] = v0; o[16] = v1; }
                };
#pragma unroll
                for (int n = 0; n < (PACKED || WIDE ? NT : 1); ++n) {
                    if constexpr (WIDE) {
                        const float v0 = nib_pair_sum(out[0][n][0], out[0][n][1], t), v1 = nib_pair_sum(out[1][n][0], out[1][n][1], t);
                        const uint32_t pr = 2u * n + (t >> 1);
                        if (pr < nt) store(pr, g + 8u * (t & 1u), v0, v1);
                    } else if constexpr (PACKED) {
                        // columns 3 * pair + digit: t = 0 has two digits of the first pair, t = 2 two of the second, t = 1 the others
                        const uint32_t src = (lane & ~3u) + 1u, pr = 2u * n + (t >> 1);
                        float v[2][2];
#pragma unroll
                        for (int m = 0; m < 2; ++m)
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const float x = __shfl_sync(0xffffffffu, out[m][n][2 * h], src), y = __shfl_sync(0xffffffffu, out[m][n][2 * h + 1], src);
                                v[m][h] = t == 0u ? out[m][n][2 * h] + A.dw1 * out[m][n][2 * h + 1] + A.dw2 * x : y + A.dw1 * out[m][n][2 * h] + A.dw2 * out[m][n][2 * h + 1];
                            }
                        if (!(t & 1u) && pr < nt) {
                            const float sx = S.sx[pr];
                            store(pr, g, v[0][0] * sx, v[1][0] * sx); store(pr, g + 8u, v[0][1] * sx, v[1][1] * sx);
                        }
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 2u; ++j) {
                            const uint32_t pr = 2u * t + j;
                            if (pr >= nt) continue;
                            const float sx = S.sx[pr];
                            float v[2][2];
#pragma unroll
                            for (int m = 0; m < 2; ++m)
#pragma unroll
                                for (int h = 0; h < 2; ++h) v[m][h] = out[m][0][2 * h + j] + A.dw1 * out[m][NT > 1 ? 1 : 0][2 * h + j] + A.dw2 * out[m][NT > 2 ? 2 : 0][2 * h + j];
                            store(pr, g, v[0][0] * sx, v[1][0] * sx); store(pr, g + 8u, v[0][1] * sx, v[1][1] * sx);
                        }
                    }
                }
            }
        };
        using one = std::integral_constant<int, 1>; using two = std::integral_constant<int, 2>; using three = std::integral_constant<int, 3>;
        if (nt <= 2u) work(one{}, std::true_type{});
        else if (nt <= 4u) work(two{}, std::true_type{});
        else work(three{}, std::bool_constant<WIDE>{});
        for (uint32_t k = cur; k < seg; ++k) leave(k);
    }
    // Digits that never came (the status word says so; the launch's results are void): no piece is drawn any more, and what is still on
    // its way to the buffers is given as long again before the block may end.
    if (failed) {
        if (lane == 0 && A.status) A.status[ST_TIMEOUT] = 1u;
        for (uint32_t k = seg; k < seg + 2u; ++k) nb_wait(full_s + 8u * (k & 1u), (k >> 1) & 1u);
    }
}

int launch_nib_batch(MmaArgs &A, uint32_t max_items, cudaStream_t s) {
    const bool gateup = A.w1 != nullptr;
    RC_REQUIRE(nib_shape_ok(A.nrows, A.ncols), "nibble experts: matrix %ux%u is not tileable", A.nrows, A.ncols);
    RC_REQUIRE(gateup || A.nrows % 32u == 0, "nibble experts: %u rows of down are not pairs of tiles", A.nrows);      // (every size the layout takes as columns is)
    RC_REQUIRE(A.work != nullptr && A.item_tok >= 1u && A.item_tok <= (A.fmt == NIB_IQ2 ? 8u : NIB_WIDE_PAIRS), "nibble experts: work counter missing or items of %u pairs", A.item_tok);
    A.act_bits = act_digit_bits(); A.dw1 = (float)(1u << A.act_bits); A.dw2 = A.dw1 * A.dw1;
    static int sm_count = 0;
    if (!sm_count) { int dev = 0; RC_CUDA(cudaGetDevice(&dev)); RC_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev)); }
    const uint32_t tiles = A.nrows / 16u, pairs = gateup ? tiles : tiles / 2u, tpp = nbb_pairs(A.ncols);
    const uint64_t pieces = (uint64_t)max_items * ((pairs + tpp - 1u) / tpp);
    const uint32_t grid = (uint32_t)(pieces < (uint64_t)sm_count ? (pieces ? pieces : 1u) : (uint64_t)sm_count);
    prof_begin(gateup ? "moe_gateup" : "moe_down", s);
    // Down is launched ahead of the end of the kernel before it, the short one that makes its digits, so that its blocks set themselves up beside that.
    // us a layer, plainly and so: 2 tokens 50.6 and 48.4, 6 54.7 and 52.5, 24 105.3 and 103.3, 64 161.1 and 159.4, 300 308.2 and 306.6, 1400 957.9
    // and 957.2. Gate/up, behind an event that another stream records, gains nothing by it: 2 50.6, 24 105.3, 64 161.4.
#define RC_NBB_LAUNCH(GU, NC) do { \
        RC_CUDA(cudaFuncSetAttribute(k_nib_batch<FMT, GU, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nbb_smem(NC))); \
        RC_LAUNCH_PDL_IF(!GU, (k_nib_batch<FMT, GU, NC>), grid, NBB_WARPS * 32u, nbb_smem(NC), s, A); } while (0)
    auto launch = [&](auto fmt) -> int {
        constexpr uint32_t FMT = decltype(fmt)::value;
        if (gateup) {
            if (A.ncols == 2048u) RC_NBB_LAUNCH(true, 2048u); else if (A.ncols == 1024u) RC_NBB_LAUNCH(true, 1024u);
            else if (A.ncols == 512u) RC_NBB_LAUNCH(true, 512u); else RC_NBB_LAUNCH(true, 256u);
        } else {
            if (A.ncols == 2048u) RC_NBB_LAUNCH(false, 2048u); else if (A.ncols == 1024u) RC_NBB_LAUNCH(false, 1024u);
            else if (A.ncols == 512u) RC_NBB_LAUNCH(false, 512u); else RC_NBB_LAUNCH(false, 256u);
        }
        return 1;
    };
    if (!(A.fmt == NIB_IQ2 ? launch(std::integral_constant<uint32_t, NIB_IQ2>{}) : A.fmt == NIB_IQ3 ? launch(std::integral_constant<uint32_t, NIB_IQ3>{})
                           : launch(std::integral_constant<uint32_t, NIB_IQ2W>{}))) return 0;
#undef RC_NBB_LAUNCH
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc
