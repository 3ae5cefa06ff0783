// Routed IQ2_XXS and IQ3_S experts in the "nibble" layout: a load-time re-coding whose decode needs no table in shared memory.
//
// Why: IQ2_XXS stores 8 weights as one codebook index (8 bits) plus 7 sign bits; turning them into tensor-core operands
// costs two dependent shared-memory lookups and ~10 integer instructions per 8 weights, and the expert kernels were
// bound by instruction issue at a sixth of HBM speed (57 M warp instructions per gate/up launch of a 64-token batch).
// Here every weight is re-coded once, at load, as a 4-bit code (bits 1:0 = which of the three codebook magnitudes
// 8 / 25 / 43, bit 2 = sign); a lane then expands 4 weights into an int8 operand register with ONE instruction
// (prmt against an 8-byte table held in two registers). IQ3_S experts take the same layout (NIB_IQ3): their magnitudes are the
// odd numbers 1 .. 15, so a signed weight is 2 n + 1 with n in -8 .. 7 and the code is n itself in two's complement; as the
// high nibble of a byte with 8 below it, it IS the int8 operand 8 (2 n + 1) - one mask-and-or per 4 weights, and the block
// scale d / 8 serves both formats. A layer of IQ3_S experts took 549 us for 24 tokens on the CUDA-core kernel, 104 here.
// Dequantised values are unchanged bit for bit
// (redcuda_nib_dequant_rows against rl_quant_dequant_row, native/redlite_native_quant_cpu.c:166-191). The price is bytes:
// 138 per 256 weights instead of 66 (IQ3_S: 110), i.e. 2.09x (1.25x) the HBM footprint and traffic of the routed experts.
//
// Layout of one expert matrix [nrows][ncols], bpr = ncols / 256 blocks per row: one contiguous RECORD of 2208 bytes per
// (16-row tile, 256-column block), records ordered [tile][block], so that a warp fetches everything it needs for one
// block of its tile with a single bulk copy:
//   codes  @0     per row and 32-column group kg four words t of 8 weights 32 kg + 8 t .. +7 of the block, weight j in bits
//                 4j+3..4j (NIB_IQ3: weights j and j + 4 in the low and high nibble of byte j); placed by nib_code_off so that a
//                 warp's loads of them are contiguous in device memory and free of bank conflicts in shared memory
//   scales @2048  16 rows x 8 B, byte kg = 2 s + 1, s the 4-bit scale of the 32-weight group (nib_sc_off)
//   d      @2176  16 fp16 block scales (nib_d_off)
// Arithmetic is the integer tensor-core scheme of redcuda_moe_mma.cu (mma.sync m16n8k32 s8, activations as three
// balanced digits per value, s32 sums per 32-weight group scaled by the integer 2s+1, fp32 scaling by d/8 per block).
// Layers with IQ3_S matrices take the wide form of the digits (actw_scale in redcuda_moe_mma.cuh): four per value and a scale per
// 256-column block, applied with d / 8. On the CUDA-core kernel they had fp32 rows; relative errors of an expert's output against
// 64-bit sums (hidden 2048, ffn 512, rows from Gaussian to one element of 10000): fp32 rows 1.3e-7 to 2.1e-7, wide digits 0.8e-7
// to 1.2e-7. The fourth digit costs nothing where items hold one or two pairs, which fill one tile either way.
//
// Here: the re-coding and the two kernels of a single token (k_nib_one for gate/up, k_nib_down_tail); batches are in
// redcuda_moe_nib_batch.cu. Every warp streams its 16-row tiles through a private ring of records (one cp.async.bulk and one mbarrier
// each). Waits on the mbarriers are bounded: a warp that gives up raises the status word and the block winds down.
// Column layout of the digits: items of up to four pairs pack two (pair, digit) triples into an 8-column tile (cols 3 * pair + digit);
// larger items use one tile per digit (col = 8 * digit + pair), so a lane holds all three digits of its two pairs and the
// epilogue needs no exchange. Wide form: col = 4 * pair + digit, two pairs a tile and as many tiles as the item's pairs need (one to
// three); the two lanes that hold a pair's digits exchange one sum each at the end of a tile.
#define RC_PDL_DEFAULT 0
#include "redcuda_common.cuh"
#include "redcuda_dot.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_nib.cuh"
#include "redcuda_stage.cuh"
#include "../../include/redcuda.h"

#include <stdlib.h>
#include <type_traits>

namespace rc {

uint64_t nib_matrix_bytes(uint32_t nrows, uint32_t ncols) { return (uint64_t)nrows * (ncols / 256u) * NIB_BLOCK_BYTES; }
bool nib_shape_ok(uint32_t nrows, uint32_t ncols) { return nrows % 16u == 0 && (ncols == 256u || ncols == 512u || ncols == 1024u || ncols == 2048u); }

// ---- GGUF rows of IQ2_XXS / IQ3_S -> nibble layout: one thread per (block, group kg, quarter t). Matrices that follow one
// another in memory are repacked as one (their row counts are multiples of 16): a layer's 512 experts take one launch per
// projection, where a planar repack and a recoding per matrix took 1024 ----
template <uint32_t FMT>
__global__ void k_nib_repack(const uint8_t *__restrict__ raw, uint64_t nb, uint32_t bpr, const RcBooks bk, uint8_t *__restrict__ dst) {
    pdl_prologue();
    const uint64_t total = nb * 32u;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = i >> 5;
        const uint32_t kg = ((uint32_t)i >> 2) & 7u, t = (uint32_t)i & 3u;
        const uint64_t row = b / bpr;
        const uint32_t blk = (uint32_t)(b - row * bpr);
        const uint8_t *bp = raw + b * (FMT == NIB_IQ3 ? 110u : 66u);
        uint32_t word = 0u, s4;
        if (FMT != NIB_IQ3) {
            const unsigned short *q = reinterpret_cast<const unsigned short *>(bp + 2u + kg * 8u);
            const uint32_t auxs = (uint32_t)q[2] | ((uint32_t)q[3] << 16);
            const uint8_t *gv = bk.iq2 + (uint32_t)bp[2u + kg * 8u + t] * 8u;
            const uint32_t s8 = rc_sign8((auxs >> (7u * t)) & 127u);
#pragma unroll
            for (uint32_t j = 0; j < 8u; ++j) {
                const uint32_t m = gv[j] == 0x19u ? 1u : gv[j] == 0x2bu ? 2u : 0u;
                word |= (m | (((s8 >> j) & 1u) << 2)) << (4u * j);
            }
            s4 = auxs >> 28;
        } else {
            const uint8_t *qs = bp + 2u + 8u * kg + 2u * t;
            const uint32_t qh = bp[66u + kg], sg = bp[74u + 4u * kg + t];
            const uint32_t g[2] = {bk.iq3s[qs[0] | ((qh << (8u - 2u * t)) & 256u)], bk.iq3s[qs[1] | ((qh << (7u - 2u * t)) & 256u)]};
#pragma unroll
            for (uint32_t j = 0; j < 8u; ++j) {
                const int m = (int)((g[j >> 2] >> (8u * (j & 3u))) & 255u), v = (sg >> j) & 1u ? -m : m;       // 2 n + 1
                word |= ((uint32_t)((v - 1) >> 1) & 15u) << (8u * (j & 3u) + 4u * (j >> 2));
            }
            s4 = ((uint32_t)bp[106u + (kg >> 1)] >> (4u * (kg & 1u))) & 15u;
        }
        uint8_t *rec = dst + ((row >> 4) * bpr + blk) * NIB_REC;
        const uint32_t rr = (uint32_t)row & 15u;
        *reinterpret_cast<uint32_t *>(rec + nib_code_off(rr, t, kg)) = word;
        if (t == 0u) {
            rec[nib_sc_off(rr, kg)] = (uint8_t)(2u * s4 + 1u);
            if (kg == 0u) *reinterpret_cast<unsigned short *>(rec + nib_d_off(rr)) = *reinterpret_cast<const unsigned short *>(bp);
        }
    }
}

int launch_nib_repack(uint32_t fmt, const uint8_t *raw, uint64_t nrows, uint32_t ncols, uint8_t *dst, cudaStream_t s) {
    RC_REQUIRE(nrows % 16u == 0 && nib_shape_ok(16u, ncols), "nibble layout: %llu rows of %u columns are not tileable (16 rows, 256/512/1024/2048 columns)", (unsigned long long)nrows, ncols);
    RC_REQUIRE(((uintptr_t)dst & 15u) == 0 && ((uintptr_t)raw & 1u) == 0, "nibble layout: unaligned matrix");
    const uint64_t nb = nrows * (ncols / 256u), total = nb * 32u;
    const uint32_t grid = (uint32_t)((total + 255u) / 256u < 148u * 16u ? (total + 255u) / 256u : 148u * 16u);
    prof_begin("nib_repack", s);
    const RcBooks bk{books_iq2(), books_iq3s()};
    // never early: its reads are non-coherent (452 us for a matrix of 512 experts against 462 by the other path)
    if (fmt != NIB_IQ3) RC_LAUNCH_BEHIND_IF(true, (k_nib_repack<NIB_IQ2>), grid ? grid : 1u, 256, 0, s, raw, nb, ncols / 256u, bk, dst);
    else RC_LAUNCH_BEHIND_IF(true, (k_nib_repack<NIB_IQ3>), grid ? grid : 1u, 256, 0, s, raw, nb, ncols / 256u, bk, dst);
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

// ---- nibble layout -> fp32, the float operations of rl_quant_dequant_row in the same order (exact) ----
__global__ void k_nib_dequant(const uint8_t *nib, uint64_t nb, uint32_t nrows, uint32_t bpr, float *__restrict__ out) {
    pdl_prologue();
    const uint64_t total = nb * 32u;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = i >> 5;
        const uint32_t kg = ((uint32_t)i >> 2) & 7u, t = (uint32_t)i & 3u;
        const uint32_t row = (uint32_t)(b / bpr), blk = (uint32_t)(b - (uint64_t)row * bpr);
        const uint8_t *rec = nib + ((uint64_t)(row >> 4) * bpr + blk) * NIB_REC;
        const uint32_t rr = row & 15u;
        const uint32_t word = *reinterpret_cast<const uint32_t *>(rec + nib_code_off(rr, t, kg));
        const uint32_t scb = rec[nib_sc_off(rr, kg)];
        const float d = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rec + nib_d_off(rr))));
        const float db = d * (0.5f + (float)((scb - 1u) >> 1)) * 0.25f;
        float *o = out + ((uint64_t)row * bpr + blk) * 256u + kg * 32u + t * 8u;
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) {
            const uint32_t code = (word >> (4u * j)) & 7u, m = code & 3u;
            const float v = db * (m == 0u ? 8.0f : m == 1u ? 25.0f : 43.0f);
            o[j] = (code & 4u) ? -v : v;
        }
    }
}

constexpr uint32_t NIB_WARPS = 8u;
constexpr uint32_t NIB_STAGES = 8u;       // records in flight per warp: a warp requests its whole tile of 2048 columns at once, one HBM round trip

// A warp's private ring of record slots. Records are requested in stream order: first the rest of the current unit (cur_*), then the
// first ones of the next unit (nxt_*), so the ring never drains at a unit boundary. Between two reads exactly one request is made,
// which keeps NIB_STAGES - 1 records in flight behind the one being read.
struct NibRing {
    uint32_t stage_s, bar_s;           // shared-memory addresses of slot 0 and of its mbarrier
    uint32_t prod, cons, phase;        // next slot to fill / to read; bit s = parity the next read of slot s waits for
    const uint8_t *cur_src, *nxt_src;
    uint32_t cur_rem, nxt_rem, nxt_taken;
    uint32_t timed_out;
};
__device__ __forceinline__ void nib_request(NibRing &R, uint32_t lane) {
    const uint8_t *src;
    if (R.cur_rem) { src = R.cur_src; R.cur_src += NIB_REC; --R.cur_rem; }
    else if (R.nxt_rem) { src = R.nxt_src; R.nxt_src += NIB_REC; --R.nxt_rem; ++R.nxt_taken; }
    else return;
    if (lane == 0) nb_fetch(R.stage_s + R.prod * NIB_REC, src, R.bar_s + 8u * R.prod);
    R.prod = R.prod + 1u == NIB_STAGES ? 0u : R.prod + 1u;
}
// waits for the oldest record; returns its slot. After a wait ran out no further wait is attempted (the results of the
// launch are void: the caller raises the status word).
__device__ __forceinline__ uint32_t nib_acquire(NibRing &R) {
    const uint32_t slot = R.cons;
    if (!R.timed_out && !nb_wait(R.bar_s + 8u * slot, (R.phase >> slot) & 1u)) R.timed_out = 1u;
    return slot;
}
__device__ __forceinline__ void nib_release(NibRing &R) {
    __syncwarp();                      // every lane has read the slot: it may be refilled
    R.phase ^= 1u << R.cons;
    R.cons = R.cons + 1u == NIB_STAGES ? 0u : R.cons + 1u;
}

// A unit's tiles for one warp. vals[ti][0], [1] = rows g and g + 8 on the lanes t == 0 (three digits: times the token's scale sx), or
// vals[ti][0] = row g (t == 0) or g + 8 (t == 1) in the wide form, whose block scales are sxw.
template <uint32_t FMT, uint32_t BPR, uint32_t BPITCH, uint32_t TPW>
__device__ __forceinline__ void nib_tiles(NibRing &R, const uint8_t *my_stage, const int8_t *Bbase, const float *sxw, uint32_t tiles, uint32_t lane, uint32_t g, uint32_t t,
                                          const int (&z)[4], float dw1, float dw2, float sx, float (&vals)[TPW][2]) {
    for (uint32_t ti = 0; ti < tiles; ++ti) {
        float out[3][4], ow[1][2] = {{0.f, 0.f}};
        out[0][0] = out[0][1] = out[0][2] = out[0][3] = 0.f;
        for (uint32_t c = 0; c < BPR; ++c) {
            nib_request(R, lane);
            const uint32_t slot = nib_acquire(R);
            if constexpr (FMT != NIB_IQ2) nib_chunk_wide<FMT, 1, BPITCH, BPR>(my_stage + slot * NIB_REC, Bbase + c * 256u, sxw + c, g, t, z, ow);
            else nib_chunk<FMT, 1, BPITCH>(my_stage + slot * NIB_REC, Bbase + c * 256u, g, t, z, out);
            nib_release(R);
        }
        if (FMT != NIB_IQ2) vals[ti][0] = nib_pair_sum(ow[0][0], ow[0][1], t);
        else {
            const uint32_t src = (lane & ~3u) + 1u;      // digits 0 and 1 are the columns of lane t = 0, digit 2 is lane t = 1's first
            const float x0 = __shfl_sync(0xffffffffu, out[0][0], src), x1 = __shfl_sync(0xffffffffu, out[0][2], src);
            vals[ti][0] = (out[0][0] + dw1 * out[0][1] + dw2 * x0) * sx; vals[ti][1] = (out[0][2] + dw1 * out[0][3] + dw2 * x1) * sx;
        }
    }
}

// Gate/up with SiLU * mul of a single token's experts: blocks of 8 warps take units of 4 x TPW tiles; warps 0-3 the gate rows, warps
// 4-7 the up rows of the same tiles; the up values cross a small shared buffer and the gate warps store SiLU(gate) * up. The token is
// quantised in the kernel, while the first records arrive.
template <uint32_t FMT, uint32_t NCOLS>
__global__ void __launch_bounds__(NIB_WARPS * 32u, 1) k_nib_one(const __grid_constant__ MmaArgs A) {
    pdl_prologue();
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr uint32_t BPR = NCOLS / 256u, TPW = BPR >= 8u ? 1u : 8u / BPR, UNIT_TILES = 4u * TPW, BPITCH = NCOLS + 32u;
    constexpr bool WIDE = FMT != NIB_IQ2;
    __shared__ float s_sxw[WIDE ? BPR : 1u];      // scales of the token's blocks
    __shared__ volatile uint32_t s_fail;
    __shared__ __align__(8) uint64_t s_bar[NIB_WARPS][NIB_STAGES];
    __shared__ float2 s_ex[TPW][4][32];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    uint8_t *my_stage = smem + warp * (NIB_STAGES * NIB_REC);
    int8_t *Bs = reinterpret_cast<int8_t *>(smem + NIB_WARPS * NIB_STAGES * NIB_REC);
    const uint32_t ntile_rows = A.nrows >> 4, U = (ntile_rows + UNIT_TILES - 1u) / UNIT_TILES;
    const uint32_t total = *A.n_items * U;
    const bool is_up = warp >= 4u;
    const uint32_t wslot = warp & 3u;
    const uint8_t *wmat = is_up ? A.w1 : A.w0;
    NibRing R{};
    R.stage_s = nb_smem(my_stage); R.bar_s = nb_smem(&s_bar[warp][0]);

    struct Unit {
        const uint8_t *rec;        // first record of this warp's tiles in the unit (records of a tile, then of the next tile, are contiguous)
        uint32_t item;             // = the pair
        uint32_t tile0, n;         // first 16-row tile of this warp and the number of records it streams in the unit
    };
    auto decode = [&](uint32_t unit, Unit &I) {
        const uint32_t rb = unit % U;
        I.item = unit / U;
        uint32_t e = A.uexp[I.item] - A.expert_begin;
        const bool ok = e < A.n_local;
        if (!ok) { if (A.status && tid == 0) A.status[ST_EXPERT_RANGE] = 1u; e = 0u; }     // never index the arena with a foreign id
        I.tile0 = rb * UNIT_TILES + wslot * TPW;
        const uint32_t tiles = I.tile0 >= ntile_rows ? 0u : min(TPW, ntile_rows - I.tile0);
        I.n = ok ? tiles * BPR : 0u;
        I.rec = wmat + (size_t)e * A.mat_bytes + (size_t)I.tile0 * BPR * NIB_REC;
    };

    // the units are few and equal: block b takes b, b + grid, ...
    if (tid == 0) s_fail = 0u;
    if (lane == 0) {
        for (uint32_t i = 0; i < NIB_STAGES; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(R.bar_s + 8u * i));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    uint32_t cur = blockIdx.x;
    uint32_t ahead = 0u;             // records of the CURRENT unit already requested (while the previous unit was multiplying)
    Unit I{}, N{};
    if (cur < total) decode(cur, I);
    // the first records are on their way while the block quantises the token
    R.cur_src = I.rec; R.cur_rem = I.n;
    while (ahead + 1u < NIB_STAGES && ahead < I.n) { nib_request(R, lane); ++ahead; }
    __shared__ uint32_t s_red[NIB_WARPS];
    float sx = 1.0f;
    if (WIDE) {
        // a warp per block of the row; columns 0..3 of the one tile in use, columns 4..7 zero
        if (warp < BPR) {
            const uint32_t k = warp * 256u + lane * 8u;
            const float4 v0 = *reinterpret_cast<const float4 *>(A.x_raw + k), v1 = *reinterpret_cast<const float4 *>(A.x_raw + k + 4u);
            float up;
            const float scale = actw_scale(__reduce_max_sync(0xffffffffu, max(act_mag4(v0), act_mag4(v1))), up);
            if (lane == 0) s_sxw[warp] = scale;
            const uint32_t w0[4] = {actw_digits(v0.x, up), actw_digits(v0.y, up), actw_digits(v0.z, up), actw_digits(v0.w, up)};
            const uint32_t w1[4] = {actw_digits(v1.x, up), actw_digits(v1.y, up), actw_digits(v1.z, up), actw_digits(v1.w, up)};
            uint32_t p0[4], p1[4];
            actw_planes(w0, p0); actw_planes(w1, p1);
#pragma unroll
            for (uint32_t col = 0u; col < 8u; ++col)
                *reinterpret_cast<uint2 *>(Bs + col * BPITCH + k) = col < 4u ? make_uint2(p0[col & 3u], p1[col & 3u]) : make_uint2(0u, 0u);
        }
    } else {
        // every unit multiplies the same activation row, so the block turns it into digits itself (the arithmetic of
        // k_quant_act): columns 0..2 of the one tile in use, columns 3..7 zero
        uint32_t mx = 0u;
        for (uint32_t k = tid * 4u; k < NCOLS; k += NIB_WARPS * 128u) mx = max(mx, act_mag4(*reinterpret_cast<const float4 *>(A.x_raw + k)));
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) s_red[warp] = mx;
        __syncthreads();
        mx = s_red[0];
        for (uint32_t w = 1; w < NIB_WARPS; ++w) mx = max(mx, s_red[w]);
        const float qmax = act_qmax(A.act_bits), inv = 1.0f / (sx = act_scale(mx, qmax));
        for (uint32_t k = tid * 4u; k < NCOLS; k += NIB_WARPS * 128u) {
            const float4 v = *reinterpret_cast<const float4 *>(A.x_raw + k);
            const float f[4] = {v.x, v.y, v.z, v.w};
            uint32_t p0 = 0, p1 = 0, p2 = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                int d0, d1, d2;
                act_digits(f[i], inv, qmax, A.act_bits, d0, d1, d2);
                p0 |= (uint32_t)(d0 & 255) << (8 * i); p1 |= (uint32_t)(d1 & 255) << (8 * i); p2 |= (uint32_t)(d2 & 255) << (8 * i);
            }
            *reinterpret_cast<uint32_t *>(Bs + k) = p0;
            *reinterpret_cast<uint32_t *>(Bs + BPITCH + k) = p1;
            *reinterpret_cast<uint32_t *>(Bs + 2u * BPITCH + k) = p2;
#pragma unroll
            for (uint32_t col = 3u; col < 8u; ++col) *reinterpret_cast<uint32_t *>(Bs + col * BPITCH + k) = 0u;
        }
    }
    __syncthreads();
    int zero[4];                     // opaque to the compiler: four registers that stay zero, the accumulator input of every MMA
    asm volatile("mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;" : "=r"(zero[0]), "=r"(zero[1]), "=r"(zero[2]), "=r"(zero[3]));
    while (cur < total) {
        const uint32_t nxt = cur + gridDim.x;
        // this unit's stream; NIB_STAGES - 1 of its records are put in flight before the first read
        R.cur_src = I.rec + (size_t)ahead * NIB_REC; R.cur_rem = I.n - ahead; R.nxt_rem = 0u; R.nxt_taken = 0u;
        for (uint32_t i = ahead; i + 1u < NIB_STAGES; ++i) nib_request(R, lane);
        if (nxt < total) { decode(nxt, N); if (I.n + 1u >= NIB_STAGES) { R.nxt_src = N.rec; R.nxt_rem = N.n; } }     // a unit shorter than the ring does not look ahead
        float vals[TPW][2];
        const uint32_t tiles = I.n / BPR;
        nib_tiles<FMT, BPR, BPITCH, TPW>(R, my_stage, Bs + (size_t)g * BPITCH + 8u * t, s_sxw, tiles, lane, g, t, zero, A.dw1, A.dw2, sx, vals);
        if (R.timed_out && lane == 0) { s_fail = 1u; if (A.status) A.status[ST_TIMEOUT] = 1u; }
        if (is_up) for (uint32_t ti = 0; ti < tiles; ++ti) s_ex[ti][wslot][lane] = make_float2(vals[ti][0], vals[ti][1]);
        __syncthreads();             // up values are in s_ex
        const bool fail = s_fail != 0u;
        if (!is_up && t < (WIDE ? 2u : 1u)) {
            for (uint32_t ti = 0; ti < tiles; ++ti) {
                const float2 up = s_ex[ti][wslot][lane];
                float *o = A.out + (size_t)I.item * A.out_stride + ((I.tile0 + ti) << 4) + g;
                const float g0 = vals[ti][0], g1 = vals[ti][1];
                if (WIDE) o[8u * t] = (g0 / (1.0f + expf(-g0))) * up.x;
                else { o[0] = (g0 / (1.0f + expf(-g0))) * up.x; o[8] = (g1 / (1.0f + expf(-g1))) * up.y; }
            }
        }
        if (nxt < total) __syncthreads();      // s_ex and s_fail have been read (the same for every thread of the block)
        if (fail) break;             // some warp's copy never arrived (status word raised): no further unit
        ahead = R.nxt_taken;
        cur = nxt; I = N;
    }
}

// ---- single token: down projection of the selected experts + shared expert's down rows + weighted sum + residual ----
// grid = nrows / 16 (one 16-row tile per block), block = top_k + 2 warps: warp k < top_k takes expert k (its tile's
// records arrive by bulk copy while the warp quantises expert k's activation row), the last two warps take the shared
// expert's 16 rows (Q6_K, CUDA cores). Partial rows meet in shared memory and are summed in router order.
constexpr uint32_t NIB_TAIL_MAX_K = 14u;
// One block an SM is all there is (the second launch bound): with registers for loads further ahead a decode step of 16 layers takes 597 us instead of 609
template <uint32_t FMT, uint32_t NCOLS>
__global__ void __launch_bounds__((NIB_TAIL_MAX_K + 2u) * 32u, 1) k_nib_down_tail(const __grid_constant__ NibTailArgs A) {
    pdl_prologue();
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr uint32_t BPR = NCOLS / 256u, BPITCH = NCOLS + 32u, PER_LANE = NCOLS / 32u, ND = FMT == NIB_IQ2 ? 3u : 4u;      // ND: digits of a value
    __shared__ __align__(8) uint64_t s_bar[NIB_TAIL_MAX_K];
    __shared__ float s_part[NIB_TAIL_MAX_K][16], s_sh[16];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u, K = A.top_k;
    uint8_t *recs = smem;                                                    // [K][BPR] records
    int8_t *digits = reinterpret_cast<int8_t *>(smem + K * BPR * NIB_REC);   // [K][ND][BPITCH]
    int8_t *zrow = digits + K * ND * BPITCH;                                 // one row of zeros: the digit columns from ND on of every tile
    float *xs = reinterpret_cast<float *>(zrow + BPITCH);                    // shared expert's activation, padded rows of redcuda_dot.cuh
    const uint32_t row0 = blockIdx.x * 16u;

    // the warp's records are requested before anything else: the expert's id is the only thing they wait for
    bool live = true;
    uint8_t *my_rec = recs + warp * BPR * NIB_REC;
    const uint32_t bar = nb_smem(&s_bar[warp < K ? warp : 0u]);
    if (warp < K) {
        uint32_t e = A.ids[warp] - A.expert_begin;
        if (e >= A.n_local) { if (A.status && lane == 0) A.status[ST_EXPERT_RANGE] = 1u; e = 0u; live = false; }      // never index the arena with a foreign id
        if (lane == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const uint8_t *src = A.w_down + (size_t)e * A.mat_bytes + (size_t)blockIdx.x * BPR * NIB_REC;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(BPR * NIB_REC) : "memory");
            for (uint32_t c = 0; c < BPR; ++c)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             :: "r"(nb_smem(my_rec + c * NIB_REC)), "l"(src + (size_t)c * NIB_REC), "r"(NIB_REC), "r"(bar) : "memory");
        }
        __syncwarp();
    }
    for (uint32_t k = tid * 4u; k < BPITCH; k += blockDim.x * 4u) *reinterpret_cast<uint32_t *>(zrow + k) = 0u;
    if (A.sh_down) for (uint32_t k = tid * 4u; k < NCOLS; k += blockDim.x * 4u) *reinterpret_cast<float4 *>(xs + xi(k)) = *reinterpret_cast<const float4 *>(A.sh_act + k);
    if (tid < 16u) s_sh[tid] = 0.f;
    __syncthreads();
    if (warp < K) {
        // this expert's activation row -> digits (the arithmetic of k_quant_act), while the records are in flight
        const float *ar = A.act + (size_t)warp * A.act_stride;
        float v[PER_LANE];
        uint32_t mx = 0u, mxb[BPR];        // of the row, of its blocks
#pragma unroll
        for (uint32_t c = 0; c < BPR; ++c) mxb[c] = 0u;
#pragma unroll
        for (uint32_t i = 0; i < PER_LANE / 4u; ++i) {
            const float4 q = *reinterpret_cast<const float4 *>(ar + lane * 4u + 128u * i);
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
            mx = max(mx, act_mag4(q)); mxb[i / 2u] = max(mxb[i / 2u], act_mag4(q));
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        const float qmax = act_qmax(A.bits), sx = act_scale(mx, qmax), inv = 1.0f / sx;
        int8_t *mine = digits + warp * ND * BPITCH;
        float sxb[BPR];
        if (ND == 4u) {
#pragma unroll
            for (uint32_t i = 0; i < PER_LANE / 4u; ++i) {
                float up;
                sxb[i / 2u] = actw_scale(i & 1u ? mxb[i / 2u] : (mxb[i / 2u] = __reduce_max_sync(0xffffffffu, mxb[i / 2u])), up);
                const uint32_t w[4] = {actw_digits(v[4 * i], up), actw_digits(v[4 * i + 1], up), actw_digits(v[4 * i + 2], up), actw_digits(v[4 * i + 3], up)};
                uint32_t pl[4];
                actw_planes(w, pl);
#pragma unroll
                for (uint32_t dg = 0; dg < 4u; ++dg) *reinterpret_cast<uint32_t *>(mine + dg * BPITCH + lane * 4u + 128u * i) = pl[dg];
            }
        } else
#pragma unroll
        for (uint32_t i = 0; i < PER_LANE / 4u; ++i) {
            uint32_t p0 = 0, p1 = 0, p2 = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int d0, d1, d2;
                act_digits(v[4 * i + j], inv, qmax, A.bits, d0, d1, d2);
                p0 |= (uint32_t)(d0 & 255) << (8 * j); p1 |= (uint32_t)(d1 & 255) << (8 * j); p2 |= (uint32_t)(d2 & 255) << (8 * j);
            }
            const uint32_t k = lane * 4u + 128u * i;
            *reinterpret_cast<uint32_t *>(mine + k) = p0;
            *reinterpret_cast<uint32_t *>(mine + BPITCH + k) = p1;
            *reinterpret_cast<uint32_t *>(mine + 2u * BPITCH + k) = p2;
        }
        __syncwarp();
        if (!__all_sync(0xffffffffu, nb_wait(bar, 0u))) { live = false; if (A.status && lane == 0) A.status[ST_TIMEOUT] = 1u; }
        float out[3][4];
#pragma unroll
        for (int n = 0; n < 3; ++n) { out[n][0] = out[n][1] = out[n][2] = out[n][3] = 0.f; }
        int zero[4];
        asm volatile("mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;" : "=r"(zero[0]), "=r"(zero[1]), "=r"(zero[2]), "=r"(zero[3]));
        const int8_t *Bl = (g < ND ? mine + g * BPITCH : zrow) + 8u * t;       // columns 0 .. ND - 1 = the pair's digits, the rest of the tile is zero
        if constexpr (ND == 4u) {
            float ow[1][2] = {{0.f, 0.f}};
            if (live)
#pragma unroll
                for (uint32_t c = 0; c < BPR; ++c) nib_chunk_wide<FMT, 1, BPITCH, 0u>(my_rec + c * NIB_REC, Bl + c * 256u, &sxb[c], g, t, zero, ow);
            const float r = nib_pair_sum(ow[0][0], ow[0][1], t);
            if (t < 2u) s_part[warp][g + 8u * t] = r;
        } else {
        if (live) for (uint32_t c = 0; c < BPR; ++c) nib_chunk<FMT, 1, BPITCH>(my_rec + c * NIB_REC, Bl + c * 256u, g, t, zero, out);
        const uint32_t src = (lane & ~3u) + 1u;
        const float x0 = __shfl_sync(0xffffffffu, out[0][0], src), x1 = __shfl_sync(0xffffffffu, out[0][2], src);
        if (t == 0u) {
            s_part[warp][g] = (out[0][0] + A.dw1 * out[0][1] + A.dw2 * x0) * sx;
            s_part[warp][g + 8u] = (out[0][2] + A.dw1 * out[0][3] + A.dw2 * x1) * sx;
        }
        }
    } else if (A.sh_down) {
        const uint32_t sw = warp - K;                                       // 0 or 1: rows 8 sw .. 8 sw + 7 of the tile
        uint32_t lpr = 32u;
        while (lpr > (NCOLS >> 6)) lpr >>= 1;
        const uint32_t rw = 32u / lpr, slot = lane / lpr, sub = lane % lpr;
        const SBooks sb{nullptr, nullptr};
        for (uint32_t r = 0; r < 8u; r += rw) {
            const uint32_t rr = 8u * sw + r + slot;                         // rw <= 8 for every row length from 256 up
            float a[1];
            row_dot<RC_Q6_K, 1>(A.sh_down, A.sh_nb, (uint64_t)(row0 + rr), NCOLS, lpr, sub, xs, x_padded(NCOLS), sb, a);
            if (sub == 0u) s_sh[rr] = a[0];
        }
    }
    __syncthreads();
    if (tid < 16u) {
        const uint32_t row = row0 + tid;
        float acc = 0.f;
        for (uint32_t k = 0; k < K; ++k) { const float wk = A.wk[k]; if (wk != 0.f) acc += wk * s_part[k][tid]; }
        if (A.sh_down) acc += s_sh[tid] * (A.scalar ? A.scalar[0] : 1.0f);
        if (A.resid) acc += A.resid[row];
        A.out[row] = acc;
    }
}

bool nib_tail_ok(uint32_t top_k, uint32_t nrows, uint32_t ncols) {
    return top_k >= 1u && top_k <= NIB_TAIL_MAX_K && nrows % 16u == 0 && (ncols == 256u || ncols == 512u || ncols == 1024u);
}

int launch_nib_down_tail(NibTailArgs &A, cudaStream_t s) {
    RC_REQUIRE(nib_tail_ok(A.top_k, A.nrows, A.ncols), "nibble down tail: top_k %u, %ux%u is not a shape it serves", A.top_k, A.nrows, A.ncols);
    A.bits = act_digit_bits(); A.dw1 = (float)(1u << A.bits); A.dw2 = A.dw1 * A.dw1;
    const uint32_t bpr = A.ncols / 256u, bpitch = A.ncols + 32u;
    const size_t smem = (size_t)A.top_k * bpr * NIB_REC + (size_t)A.top_k * (A.fmt == NIB_IQ2 ? 3u : 4u) * bpitch + bpitch + (size_t)x_padded(A.ncols) * 4u + 16u;
    const uint32_t threads = (A.top_k + 2u) * 32u, grid = A.nrows / 16u;
    // launched plainly: ahead of time its blocks would gather on the SMs that the 80 gate / up blocks of a top-10 layer leave free
    // (28.9 against 26.7 us a layer, measured when it took that long; 24.5 now)
    prof_begin("moe_down_tail", s);
#define RC_TAIL_LAUNCH(NC) do { \
        RC_CUDA(cudaFuncSetAttribute(k_nib_down_tail<FMT, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        RC_LAUNCH((k_nib_down_tail<FMT, NC>), grid, threads, smem, s, A); } while (0)
    auto launch = [&](auto fmt) -> int {
        constexpr uint32_t FMT = decltype(fmt)::value;
        if (A.ncols == 256u) RC_TAIL_LAUNCH(256u); else if (A.ncols == 512u) RC_TAIL_LAUNCH(512u); else RC_TAIL_LAUNCH(1024u);
        return 1;
    };
    if (!(A.fmt == NIB_IQ2 ? launch(std::integral_constant<uint32_t, NIB_IQ2>{}) : A.fmt == NIB_IQ3 ? launch(std::integral_constant<uint32_t, NIB_IQ3>{})
                           : launch(std::integral_constant<uint32_t, NIB_IQ2W>{}))) return 0;
#undef RC_TAIL_LAUNCH
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

// A.w0 / A.w1: nibble-layout gate and up matrices of the experts, A.x_raw the token's row
int launch_nib_one(MmaArgs &A, uint32_t top_k, cudaStream_t s) {
    RC_REQUIRE(nib_shape_ok(A.nrows, A.ncols), "nibble experts: matrix %ux%u is not tileable", A.nrows, A.ncols);
    RC_REQUIRE(A.x_raw && A.w1 && A.item_tok == 1u, "nibble experts: in-kernel quantisation serves the gate/up of a single token");
    A.act_bits = act_digit_bits(); A.dw1 = (float)(1u << A.act_bits); A.dw2 = A.dw1 * A.dw1;
    static int sm_count = 0;
    if (!sm_count) { int dev = 0; RC_CUDA(cudaGetDevice(&dev)); RC_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev)); }
    const uint32_t bpr = A.ncols / 256u, unit_tiles = 4u * (bpr >= 8u ? 1u : 8u / bpr);
    const uint64_t units = (uint64_t)top_k * ((A.nrows / 16u + unit_tiles - 1u) / unit_tiles);
    const uint32_t grid = (uint32_t)(units < (uint64_t)sm_count ? (units ? units : 1u) : (uint64_t)sm_count);
    const size_t smem = (size_t)NIB_WARPS * NIB_STAGES * NIB_REC + 8u * (size_t)(A.ncols + 32u);
    prof_begin("moe_gateup", s);
    // launched ahead of the previous kernel's end
#define RC_NIB_LAUNCH(NC) do { \
        RC_CUDA(cudaFuncSetAttribute(k_nib_one<FMT, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        RC_LAUNCH_PDL((k_nib_one<FMT, NC>), grid, NIB_WARPS * 32u, smem, s, A); } while (0)
    auto launch = [&](auto fmt) -> int {
        constexpr uint32_t FMT = decltype(fmt)::value;
        if (A.ncols == 2048u) RC_NIB_LAUNCH(2048u); else if (A.ncols == 1024u) RC_NIB_LAUNCH(1024u); else if (A.ncols == 512u) RC_NIB_LAUNCH(512u); else RC_NIB_LAUNCH(256u);
        return 1;
    };
    if (!(A.fmt == NIB_IQ2 ? launch(std::integral_constant<uint32_t, NIB_IQ2>{}) : A.fmt == NIB_IQ3 ? launch(std::integral_constant<uint32_t, NIB_IQ3>{})
                           : launch(std::integral_constant<uint32_t, NIB_IQ2W>{}))) return 0;
#undef RC_NIB_LAUNCH
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc

using namespace rc;

// Host-buffer check of the layout: raw IQ2_XXS GGUF rows -> nibble layout -> fp32. Must equal
// redcuda_quant_dequant_rows (and rl_quant_dequant_row) bit for bit.
extern "C" int redcuda_nib_dequant_rows(const uint8_t *rows, uint32_t nrows, uint32_t ncols, float *out) {
    if (!require_device() || !require_books(RC_IQ2_XXS)) return 0;
    RC_REQUIRE(rows && out, "nib dequant: null argument");
    RC_REQUIRE(nib_shape_ok(nrows, ncols), "nib dequant: matrix %ux%u is not tileable (16 rows, 256/512/1024/2048 columns)", nrows, ncols);
    const uint64_t bytes = rc_matrix_bytes(RC_IQ2_XXS, nrows, ncols), nb = (uint64_t)nrows * (ncols / 256u);
    const size_t ob = (size_t)nrows * ncols * 4u, nibb = nib_matrix_bytes(nrows, ncols);
    Stage st;
    if (!st.open(Stage::pad(bytes) + Stage::pad(nibb) + Stage::pad(ob))) return 0;
    uint8_t *raw = st.take(bytes), *nib = st.take(nibb);
    float *o = st.take<float>(ob);
    cudaStream_t s = st.stream();
    if (!st.upload(raw, rows, bytes) || !launch_nib_repack(NIB_IQ2, raw, nrows, ncols, nib, s)) return 0;
    const uint64_t total = nb * 32u;
    RC_LAUNCH((k_nib_dequant), (unsigned)((total + 255u) / 256u < 4096u ? (total + 255u) / 256u : 4096u), 256, 0, s, nib, nb, nrows, ncols / 256u, o);
    RC_LAUNCHED();
    return st.download(out, o, ob) && st.finish();
}
