// Routed experts of a prefill chunk on the 5th-generation tensor cores (tcgen05): for every work item (up to TCX_TN pairs of
// one expert) and every 128-row tile of the expert's matrix, out[pair][row] = sum_k W_e[row][k] * x[pair][k].
//
// The batched form of the expert GEMV (rl_quant_row_dot per row, native/redlite_native_quant_cpu.c:247-266, called per
// selected expert by the MoE layer, native/redlite_native_moe.c); the reference's chunked prefill groups the chunk's
// tokens by expert and runs one matrix product per expert (native/redmetal_engine_prefill.m:889-909).
//
// Operands. The experts are held in the nibble layout (redcuda_moe_mma.cuh): a weight is d/8 * (2s+1) * (+-8|25|43) with
// d the fp16 scale of its 256-block and s the 4-bit scale of its 32-group. The integer (2s+1) * (+-m) is at most 1333, so
// it is ONE exact fp16 value: the weight operand needs a single digit, built with two byte permutes and one half2 FMA
// per pair of weights, and d/8 multiplies the fp32 sums of each 256-column block when they are drained. Activations are two
// fp16 digits (hi + lo, 22 significant bits, power-of-two scale per row), prepared once per row by k_tc_prep_rows; the
// digit rows of an item's pairs are gathered straight into the MMA's swizzled operand tile with 16-byte cp.async pieces, so
// a token that goes to ten experts is stored once.
// The tensor core adds into fp32 without rounding to nearest, so an accumulator covers 64 columns only and the sums of
// the accumulators are taken in fp32 registers.
//
// Every wait is bounded: on a timeout the role raises a flag that stops the other roles at their next wait; the CTA waits
// (bounded) for its own copies, frees its tensor memory, raises the launch's flag and the sticky status word, and returns.
#define RC_PDL_DEFAULT 0
#include "redcuda_common.cuh"
#include "redcuda_dot.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_moe_mma.cuh"
#include "redcuda_tc_gemm.cuh"

#include <cuda_fp16.h>
#include <stdlib.h>

namespace rc {

constexpr uint32_t TCX_KS = 128u, TCX_SUBS = TCX_KS / TC_KS, TCX_SPB = 256u / TCX_KS;      // stage width, 64-column tiles per stage, stages per 256-column block
constexpr uint32_t TCX_RAW = 8u * NIB_REC;                // records of one 256-column block of a 128-row tile
// biased byte tables of the 4-bit codes: 128 + (8, 25, 43, 0) and 128 - (8, 25, 43, 0)
constexpr uint32_t TCX_TAB_POS = 0x80ab9988u, TCX_TAB_NEG = 0x80556778u;

__device__ __forceinline__ uint32_t tcx_prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

__device__ __forceinline__ __half2 tcx_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }

// 8 codes (one word) times the group's integer scale hs -> 8 exact fp16 values. A code selects a biased byte u = 128 + w;
// 0x6400 | u is the fp16 number 1024 + u, and (1024 + u) * sc - 1152 * sc = w * sc with one rounding of an exact integer (hb = -1152 sc).
__device__ __forceinline__ void tcx_decode8(uint32_t word, __half2 hs, __half2 hb, uint32_t *h) {
    const uint32_t b0 = tcx_prmt(TCX_TAB_POS, TCX_TAB_NEG, word), b1 = tcx_prmt(TCX_TAB_POS, TCX_TAB_NEG, word >> 16);
    h[0] = tcx_prmt(b0, 0x64646464u, 0x5140u); h[1] = tcx_prmt(b0, 0x64646464u, 0x5342u);
    h[2] = tcx_prmt(b1, 0x64646464u, 0x5140u); h[3] = tcx_prmt(b1, 0x64646464u, 0x5342u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 v = __hfma2(tcx_h2(h[j]), hs, hb);
        h[j] = *reinterpret_cast<const uint32_t *>(&v);
    }
}

// v[r][k] = b ? SiLU(a) * b : a -> two fp16 digits per value, rows kept row-major, a stage's two digits side by side: xd[r][ncols / 128][digit][128]; x_inv[r]
// undoes the row's power-of-two scale. A warp per row, the row in its registers (8 values a lane and step of 256 columns):
// the memory is what bounds it, and a block per row (two passes, 64 of 256 threads busy in the second) took 58 us where
// 20480 rows of 512 move 126 MB. grid = rows / 8, block = 256; ncols a multiple of 256, at most 256 NCH
template <uint32_t NCH>
__global__ void __launch_bounds__(256) k_tc_prep_rows(const float *a, const float *b, uint32_t stride, uint32_t nrows, uint32_t ncols,
                                                      __half *__restrict__ xd, float *__restrict__ x_inv) {
    pdl_prologue();
    const uint32_t r = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (r >= nrows) return;
    const float *ar = a + (size_t)r * stride, *br = b ? b + (size_t)r * stride : nullptr;
    float v[NCH][8];
    float mx = 0.f;
    const bool vec = ((size_t)ar & 15u) == 0u;       // a caller's rows may begin at any float (their stride is a multiple of four)
#pragma unroll
    for (uint32_t i = 0; i < NCH; ++i) {
        const uint32_t k = i * 256u + lane * 8u;
        if (k >= ncols) break;
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
            const float *q = ar + k + 4u * h;
            const float4 p = vec ? *reinterpret_cast<const float4 *>(q) : make_float4(q[0], q[1], q[2], q[3]);
            v[i][4 * h] = p.x; v[i][4 * h + 1] = p.y; v[i][4 * h + 2] = p.z; v[i][4 * h + 3] = p.w;
        }
        if (br)
#pragma unroll
            for (uint32_t h = 0; h < 2u; ++h) {
                const float4 q = *reinterpret_cast<const float4 *>(br + k + 4u * h);
                v[i][4 * h] = silu_mul(v[i][4 * h], q.x); v[i][4 * h + 1] = silu_mul(v[i][4 * h + 1], q.y);
                v[i][4 * h + 2] = silu_mul(v[i][4 * h + 2], q.z); v[i][4 * h + 3] = silu_mul(v[i][4 * h + 3], q.w);
            }
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) mx = fmaxf(mx, fabsf(v[i][j]));
    }
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    int e = 0;
    if (mx > 0.f && mx < INFINITY) { int ex; frexpf(mx, &ex); e = 14 - ex; }     // max |v| * 2^e in [2^13, 2^14)
    e = e > 100 ? 100 : e < -100 ? -100 : e;
    const float sc = exp2f((float)e);
    if (lane == 0) x_inv[r] = exp2f((float)-e);
    __half *hi = xd + (size_t)r * 2u * ncols;
#pragma unroll
    for (uint32_t i = 0; i < NCH; ++i) {
        const uint32_t k = i * 256u + lane * 8u;
        if (k >= ncols) break;
        __half h[8], l[8];
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) {
            const float s = v[i][j] * sc;
            h[j] = __float2half_rn(s);
            l[j] = __float2half_rn(s - __half2float(h[j]));
        }
        __half *o = hi + (k / TCX_KS) * 2u * TCX_KS + k % TCX_KS;
        *reinterpret_cast<uint4 *>(o) = *reinterpret_cast<const uint4 *>(h);
        *reinterpret_cast<uint4 *>(o + TCX_KS) = *reinterpret_cast<const uint4 *>(l);
    }
}

// shared-memory matrix descriptor, K-major rows of 128 bytes (64 halves) with the 128-byte swizzle: the 16-byte chunk c of
// row r sits at r * 128 + ((c ^ (r % 8)) * 16) of a 1024-byte aligned tile; 8-row groups are 1024 bytes apart. A k-step
// of 16 halves is addressed by advancing the start address by 32 bytes.
__device__ __forceinline__ uint64_t tcx_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint32_t tcx_sw128(uint32_t r, uint32_t c) { return r * 128u + ((c ^ (r & 7u)) << 4); }

// D[tmem] (+)= A[tmem] * B[smem], kind::f16: row i of A in lane i, two halves a column, 8 columns a k-step of 16. Issued by the lane
// whose `leader` is set; the warp stays converged, so that addresses and descriptors live in uniform registers (in code of one lane they do
// not, and moving them there for every MMA took longer than the MMA)
__device__ __forceinline__ void tcx_mma_ts(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// one poll, without being put to sleep until the barrier moves on
__device__ __forceinline__ uint32_t tcx_test(uint32_t mbar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
    return done;
}

constexpr uint32_t TCX_NB = 6u, TCX_NRAW = 4u, TCX_NI = 4u;                                // buffers: activation stages, records of a block, units
constexpr uint32_t TCX_W_RAW = 2u, TCX_W_GATHER = 3u, TCX_W_DECODE = 4u, TCX_N_DECODE = 8u, TCX_W_DRAIN = 12u, TCX_N_DRAIN = 8u;
constexpr uint32_t TCX_THREADS = 32u * (TCX_W_DRAIN + TCX_N_DRAIN);
constexpr uint32_t TCX_T = 2u;                                                               // 128-row tiles of a group
constexpr uint32_t TCX_B_DIGIT = TCX_TN * TC_KS * 2u, TCX_B_SUB = 2u * TCX_B_DIGIT, TCX_B_BUF = TCX_SUBS * TCX_B_SUB;      // rows of 64 columns: hi, then lo; of a stage
constexpr uint32_t TCX_NA = 5u, TCX_A_COLS = TCX_KS / 2u, TCX_TM_A = TCX_T * TCX_SUBS * TCX_TN, TCX_TM_COLS = 512u;    // tensor memory: accumulators of TN columns, one per 64 columns of a stage and tile, then stages of decoded weights
static_assert(TCX_SPB == 2u && TCX_SUBS == 2u && TCX_NB % TCX_SPB == 0u && TCX_TN % 16u == 0u && TCX_TN <= 64u, "the stages of a block lie side by side; the workers' chunks");
static_assert(TCX_TM_A + TCX_NA * TCX_A_COLS <= TCX_TM_COLS, "tensor memory of a CTA");

struct TcxUnit { uint32_t live, expert, group0, ntok, ncol, pad[3]; uint32_t row[TCX_TN], pair[TCX_TN]; float xinv[TCX_TN]; };     // ncol: accumulator columns, ntok rounded up to 16

// A persistent CTA per SM; its warps are roles that meet on mbarriers, without a block barrier between set-up and end. A group is two 128-row
// tiles (the gate and the up tile of the same rows, or two tiles of down) for one item (up to TN pairs of an expert), so the activations of a
// stage are brought in once for both; a unit of work is A.upg groups of one item, some sixteen blocks of 256 columns, so that looking it up
// (a chain of five loads) stays hidden.
//   warps 0-1     issue the MMAs of the first and of the second tile (one lane each) and commit their completion to the barriers of what they
//                 have read: while one polls barriers the other's MMAs run
//   warp 2        draws units from a counter and publishes their pairs, one ahead; requests the records of block after block (cp.async.bulk)
//   warp 3        gathers the activation digits of stage after stage (16-byte cp.async pieces into the swizzled operand tile)
//   warps 4-11    decode the records: a thread owns a row and writes its fp16 values to tensor memory, from where the MMA reads its A operand
//                 (warps 4-7 the first stage of a block, 8-11 the second)
//   warps 12-19   read a stage's accumulators (12-15 those of the first tile, 16-19 of the second), add them, scaled by d / 8, to fp32
//                 register sums, and store these at the end of a group
// What bounds it is the decode warps' chain (two barriers, the record out of shared memory, 190 instructions, four stores and an arrival, some 1500
// cycles a block where the MMAs of 48 pairs take 770 and HBM delivers a block to every SM in 770), and with full items the MMAs' wait for the drain.
// How it came here, us for gate/up and down of 2048 tokens (40 pairs an expert): decoded weights in shared memory, one CTA per item and up to 32
// blocks, items of 64 pairs, 128-column stages: 463 and 304, bound by shared memory (operand A written and read, 64 KB a stage of the 128
// bytes a cycle that it moves, beside 64 KB of B) and by an issuing lane outside converged code, whose addresses have to be brought to
// uniform registers for every MMA. Operand A in tensor memory, persistent, two tiles a gather: 391 and 208; MMAs issued from converged code: 272 and 167;
// waits of a dozen instructions instead of loops inlined twenty times (120 KB of code: five programs share an instruction cache): 240 and 136
// with accumulators of 256 columns. Accumulators of 64 columns cost 20 us of each launch and take the error from 8.6e-7 to 3.0e-7. Records requested from
// converged code (eight lanes with an address each are served one after the other) and barriers polled ahead of their use: 254 and 153 for
// 2048 tokens, 700 tokens 207 and 112 -> 179 and 104. Taken back: decode and drain by the same eight warps (322 and 196), items of 64 pairs with four stages
// of activations instead of six (260 and 152 against 240 and 136), a decode warp per tile instead of per stage (the same time, and barrier phases can
// be passed unseen).
__global__ void __launch_bounds__(TCX_THREADS, 1) k_tc_experts(const __grid_constant__ TcxArgs A) {
    pdl_prologue();
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t a_full[TCX_NA], a_empty[TCX_NA], acc_full[TCX_T], acc_empty[TCX_T], b_full[TCX_NB], b_empty[TCX_NB], raw_full[TCX_NRAW], raw_empty[TCX_NRAW],
        unit_full[TCX_NI], unit_empty[TCX_NI];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t fail;               // a bounded wait ran out: every role stops at its next wait
    __shared__ __align__(16) TcxUnit s_unit[TCX_NI];
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31u;
    const uint32_t bpr = A.ncols >> 8, ncb = bpr * A.upg;            // 256-column blocks of a row; of a unit, one after the other for its groups
    const uint32_t gtiles = TCX_T / A.nmat;                          // row tiles of a matrix in a group
    uint8_t *b_base = smem, *raw_base = smem + TCX_NB * TCX_B_BUF;
    if (tid == 0) {
        fail = 0u;
        auto init = [](uint64_t *bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count)); };
        for (uint32_t i = 0; i < TCX_NA; ++i) { init(&a_full[i], TCX_N_DECODE / TCX_SPB); init(&a_empty[i], 1u); }
        for (uint32_t i = 0; i < TCX_T; ++i) { init(&acc_full[i], 1u); init(&acc_empty[i], TCX_N_DRAIN / TCX_T); }
        for (uint32_t i = 0; i < TCX_NB; ++i) { init(&b_full[i], 1u); init(&b_empty[i], TCX_T); }
        for (uint32_t i = 0; i < TCX_NRAW; ++i) { init(&raw_full[i], 1u); init(&raw_empty[i], TCX_N_DECODE); }
        for (uint32_t i = 0; i < TCX_NI; ++i) { init(&unit_full[i], 1u); init(&unit_empty[i], TCX_T + 1u + TCX_N_DECODE + TCX_N_DRAIN); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0u) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_slot)), "r"(TCX_TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    const uint32_t fail_at = smem_u32(const_cast<uint32_t *>(&fail));
    auto wait = [&](uint64_t *bar, uint32_t parity) { return tc_wait(smem_u32(bar), parity, fail_at); };
    // a poll ahead of the place where its answer is needed (a barrier's answer takes some hundred cycles, a role's turn has two or three), and the wait there
    auto poll = [&](uint64_t *bar, uint32_t parity) { return tcx_test(smem_u32(bar), parity); };
    auto wait_polled = [&](uint32_t polled, uint64_t *bar, uint32_t parity) { return __all_sync(0xffffffffu, polled) || wait(bar, parity); };
    auto unit_wait = [&](uint32_t n) { return wait(&unit_full[n % TCX_NI], (n / TCX_NI) & 1u); };
    auto unit_done = [&](uint32_t n) { __syncwarp(); if (lane == 0) tc_arrive(smem_u32(&unit_empty[n % TCX_NI])); };

    if (warp < TCX_T) {
        // ------------------------------------------------------------------ MMA issue
        const uint32_t leader = tc_elect();
        const uint64_t desc0 = tcx_desc_sw128(smem_u32(b_base));
        uint32_t ka = 0u, b = 0u, bph = 0u, a = warp * TCX_SPB, aph = 0u;       // accumulations of this tile so far; activation and weight stage buffers and their phases
        bool ok = true;
        for (uint32_t n = 0; ok && (ok = unit_wait(n)); ++n) {
            const TcxUnit &U = s_unit[n % TCX_NI];
            const uint32_t live = __shfl_sync(0xffffffffu, U.live, 0), ncol = __shfl_sync(0xffffffffu, U.ncol, 0);
            unit_done(n);
            if (!live) break;
            const uint32_t idesc = tc_idesc(ncol);
#pragma unroll 1
            for (uint32_t i = 0; i < ncb && ok; ++i) {
#pragma unroll 1
                for (uint32_t h = 0; h < TCX_SPB && ok; ++h, ++ka) {
                    const uint32_t b_there = poll(&b_full[b], bph), a_there = poll(&a_full[a], aph), d_free = ka ? poll(&acc_empty[warp], (ka - 1u) & 1u) : 1u;
                    if (!(ok = wait_polled(b_there, &b_full[b], bph) && wait_polled(a_there, &a_full[a], aph) && wait_polled(d_free, &acc_empty[warp], (ka - 1u) & 1u))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // An accumulator covers 64 columns, the lo digits first: the adder truncates, so what is lost grows with the steps that meet large
                    // sums. Relative error of an expert's output against 64-bit sums (rows of 2048 Gaussian values): 8.6e-7 with accumulators of 256 columns
                    // (whether the lo digits share them or not), 4.7e-7 of 128, 3.0e-7 of 64, where the fp32 sums of the drain are as much.
#pragma unroll
                    for (uint32_t j = 0; j < TCX_SUBS; ++j)
#pragma unroll
                        for (uint32_t kk = 0; kk < 8u; ++kk)         // + 32 bytes per k-step; the first MMA overwrites
                            tcx_mma_ts(leader, tmem + (warp * TCX_SUBS + j) * TCX_TN, tmem + TCX_TM_A + a * TCX_A_COLS + 32u * j + 8u * (kk & 3u),
                                       desc0 + b * (TCX_B_BUF >> 4) + j * (TCX_B_SUB >> 4) + (kk < 4u ? TCX_B_DIGIT >> 4 : 0u) + 2u * (kk & 3u), idesc, kk ? 1u : 0u);
                    tc_commit_if(leader, smem_u32(&acc_full[warp]));
                    tc_commit_if(leader, smem_u32(&b_empty[b]));
                    tc_commit_if(leader, smem_u32(&a_empty[a]));
                    if (++b == TCX_NB) { b = 0u; bph ^= 1u; }
                    if ((a += h == TCX_SPB - 1u ? TCX_SPB * (TCX_T - 1u) + 1u : 1u) >= TCX_NA) { a -= TCX_NA; aph ^= 1u; }      // behind a block, over the other tile's
                }
            }
        }
    } else if (warp == TCX_W_RAW) {
        // ------------------------------------------------------------------ units and weight records
        const uint32_t upi = A.nrows / TC_M / gtiles / A.upg, n_units = *A.n_items * upi;      // units of an item
        // The next unit is looked up in steps, one behind each request of this one's records, so that no step waits for the loads of the
        // step before it
        uint32_t f_u = 0u, f_x = 0u, f_p0 = 0u, f_e = 0u, f_nt = 0u, f_live = 0u, f_pair[2] = {0u, 0u}, f_row[2] = {0u, 0u};
        float f_inv[2] = {0.f, 0.f};
        bool ok = true;
        auto look = [&](uint32_t step, uint32_t n) {
            switch (step) {
                case 0: if (lane == 0) f_u = atomicAdd(A.work, 1u); break;
                case 1:
                    f_u = __shfl_sync(0xffffffffu, f_u, 0);
                    f_live = f_u < n_units ? 1u : 0u;
                    if (f_live) { f_x = A.item_u[f_u / upi]; f_p0 = A.item_p0[f_u / upi]; }
                    break;
                case 2: if (f_live) { f_e = A.uexp[f_x] - A.expert_begin; f_nt = A.ustart[f_x + 1u]; } break;
                case 3:
                    f_nt = f_live ? min(f_nt - f_p0, TCX_TN) : 0u;
                    if (f_live && f_e >= A.n_local) {     // cannot happen with k_group_pairs' output; never an address
                        if (lane == 0 && A.status) A.status[ST_EXPERT_RANGE] = 1u;
                        f_e = 0u; f_nt = 0u;
                    }
#pragma unroll
                    for (uint32_t i = 0; i < 2u; ++i) f_pair[i] = lane + 32u * i < f_nt ? A.sorted[f_p0 + lane + 32u * i] : 0u;
                    break;
                case 4:
#pragma unroll
                    for (uint32_t i = 0; i < 2u; ++i) { f_row[i] = f_pair[i] / A.x_div; f_inv[i] = lane + 32u * i < f_nt ? A.x_inv[f_row[i]] : 0.f; }
                    break;
                default: {
                    if (n >= TCX_NI && !(ok = wait(&unit_empty[n % TCX_NI], ((n / TCX_NI) - 1u) & 1u))) return;
                    TcxUnit &U = s_unit[n % TCX_NI];
                    if (lane == 0) { U.live = f_live; U.expert = f_e; U.group0 = (f_u % upi) * A.upg; U.ntok = f_nt; U.ncol = f_nt ? (f_nt + 15u) & ~15u : 16u; }
#pragma unroll
                    for (uint32_t i = 0; i < 2u; ++i)
                        if (lane + 32u * i < TCX_TN) { U.row[lane + 32u * i] = f_row[i]; U.pair[lane + 32u * i] = f_pair[i]; U.xinv[lane + 32u * i] = f_inv[i]; }
                    __syncwarp();
                    if (lane == 0) tc_arrive(smem_u32(&unit_full[n % TCX_NI]));
                }
            }
        };
        const uint32_t leader = tc_elect();
        const uint64_t tile_step = (uint64_t)bpr * NIB_REC;      // from a 16-row tile to the next
        uint32_t kb = 0u, step = 0u;
#pragma unroll 1
        while (step < 6u) look(step++, 0u);
        for (uint32_t n = 0; ok && f_live; ++n) {
            const uint32_t e = __shfl_sync(0xffffffffu, f_e, 0), group0 = __shfl_sync(0xffffffffu, (f_u % upi) * A.upg, 0);
            step = 0u;
            const uint64_t base = (uint64_t)e * A.mat_bytes + (uint64_t)(group0 * gtiles * 8u) * tile_step;      // record (16-row tile j, block c) of a matrix at (j * bpr + c) * NIB_REC
            const uint8_t *src0 = A.w[0] + base, *src1 = A.nmat == 2u ? A.w[1] + base : src0 + 8u * tile_step;
            uint32_t c = 0u;
#pragma unroll 1
            for (uint32_t i = 0; i < ncb * TCX_T && ok; ++i, ++kb) {
                const uint32_t k = kb % TCX_NRAW;
                if (kb >= TCX_NRAW && !(ok = wait(&raw_empty[k], ((kb / TCX_NRAW) - 1u) & 1u))) break;
                const uint32_t bar = smem_u32(&raw_full[k]), dst = smem_u32(raw_base + k * TCX_RAW);
                asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}\n" :: "r"(bar), "r"(TCX_RAW), "r"(leader) : "memory");
                // by one lane of a converged warp, its addresses uniform: eight lanes with an address each are served one after the other
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j)
                    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}\n"
                                 :: "r"(dst + j * NIB_REC), "l"(src0 + (uint64_t)j * tile_step), "r"(NIB_REC), "r"(bar), "r"(leader) : "memory");
                const uint8_t *other = src1;              // the other tile's turn; after both, the next block of the row or the next group
                src1 = src0;
                if (i & 1u) {
                    const bool row_end = ++c == bpr;
                    const uint64_t step_bytes = (uint64_t)(row_end ? (gtiles * 8u - 1u) * bpr + 1u : 1u) * NIB_REC;
                    if (row_end) c = 0u;
                    src1 += step_bytes;
                    src0 = other + step_bytes;
                } else src0 = other;
                if (step < 6u) look(step++, n + 1u);
            }
#pragma unroll 1
            while (ok && step < 6u) look(step++, n + 1u);
        }
        // copies that nobody waited for may still be writing into this CTA's shared memory: wait for the last ones (bounded)
        if (lane == 0)
            for (uint32_t k = kb > TCX_NRAW ? kb - TCX_NRAW : 0u; k < kb; ++k) mbar_wait(smem_u32(&raw_full[k % TCX_NRAW]), (k / TCX_NRAW) & 1u);
    } else if (warp == TCX_W_GATHER) {
        // ------------------------------------------------------------------ activation gather
        // lane: k chunk lane % 8 of the token slots lane / 8 + 4 m, both digits, both 64-column tiles of a stage
        constexpr uint32_t M = TCX_TN / 4u;
        const uint32_t kc = lane & 7u, ttb = lane >> 3;
        const uint32_t dst0 = smem_u32(b_base) + tcx_sw128(ttb, kc), dst1 = smem_u32(b_base) + tcx_sw128(ttb + 4u, kc);      // 8 slots further: the same swizzle phase, 1024 bytes
        uint32_t ks = 0u, given = 0u, b = 0u, bph = 1u, gb = 0u;         // stages requested, stages handed over; their buffers, and the phase that must have ended before one is filled again
        bool ok = true;
        auto hand = [&]() {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(smem_u32(&b_full[gb]));
            ++given;
            gb = gb + 1u == TCX_NB ? 0u : gb + 1u;
        };
        for (uint32_t n = 0; ok && (ok = unit_wait(n)); ++n) {
            const TcxUnit &U = s_unit[n % TCX_NI];
            const uint32_t live = U.live, ncol = U.ncol;
            const __half *src[M];
#pragma unroll
            for (uint32_t m = 0; m < M; ++m) src[m] = A.xd + (size_t)U.row[ttb + 4u * m] * 2u * A.ncols + kc * 8u;     // slots beyond the item's pairs read row 0: their columns are not stored
            unit_done(n);
            if (!live) break;
            for (uint32_t s = 0, col = 0; s < ncb * TCX_SPB && ok; ++s, ++ks) {
                if (ks >= TCX_NB && !__all_sync(0xffffffffu, tcx_test(smem_u32(&b_empty[b]), bph))) {      // no room yet: what is on its way can be waited for
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    while (given < ks) hand();
                    if (!(ok = wait(&b_empty[b], bph))) break;
                }
                const uint32_t bb[2] = {dst0 + b * TCX_B_BUF, dst1 + b * TCX_B_BUF};
#pragma unroll
                for (uint32_t m = 0; m < M; ++m) {
                    if (4u * m >= ncol) break;
                    const __half *sp = src[m] + col;
#pragma unroll
                    for (uint32_t i = 0; i < 2u * TCX_SUBS; ++i)      // digit i / 2, 64-column tile i % 2
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(bb[m & 1u] + (i & 1u) * TCX_B_SUB + (i >> 1) * TCX_B_DIGIT + (m >> 1) * 1024u), "l"(sp + i * TC_KS) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (given + 2u < ks + 1u) {          // two stages may be on their way while the next is requested
                    asm volatile("cp.async.wait_group 2;" ::: "memory");
                    hand();
                }
                col += 2u * TCX_KS;
                if (col == 2u * A.ncols) col = 0u;
                if (++b == TCX_NB) { b = 0u; bph ^= 1u; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        while (ok && given < ks) hand();
    } else if (warp < TCX_W_DRAIN) {
        // ------------------------------------------------------------------ weight decode (256 threads)
        const uint32_t half = (warp - TCX_W_DECODE) >> 2, row = (warp & 3u) * 32u + lane, rr = row & 15u, kg0 = 4u * half;
        const uint32_t ta0 = tmem + (((warp & 3u) * 32u) << 16) + TCX_TM_A;
        const uint8_t *raw0 = raw_base + (row >> 4) * NIB_REC;
        uint4 wd[4];                                      // piece t: code words of the columns 32 kg + 8 t .. + 7, kg = kg0 .. kg0 + 3, of the next block
        uint32_t sc4 = 0u, kl = 0u, a = half, aph = 1u;   // their four scales; blocks read from shared memory; weight stage buffer, and the phase that must have ended before it is filled (at first, the one before the barrier's first)
        bool ok = true;
        auto load = [&](uint32_t polled) -> bool {
            const uint32_t k = kl % TCX_NRAW;
            if (!wait_polled(polled, &raw_full[k], (kl / TCX_NRAW) & 1u)) return false;
            const uint8_t *raw = raw0 + k * TCX_RAW;
#pragma unroll
            for (uint32_t t = 0; t < 4u; ++t) wd[t] = *reinterpret_cast<const uint4 *>(raw + nib_code_off(rr, t, kg0));
            sc4 = *reinterpret_cast<const uint32_t *>(raw + nib_sc_off(rr, kg0));
            __syncwarp();
            if (lane == 0) tc_arrive(smem_u32(&raw_empty[k]));
            ++kl;
            return true;
        };
        for (uint32_t n = 0; ok && (ok = unit_wait(n)); ++n) {
            const uint32_t live = s_unit[n % TCX_NI].live;
            unit_done(n);
            if (!live || !(ok = load(0u))) break;
#pragma unroll 1
            for (uint32_t i = 0; i < ncb * TCX_T; ++i) {
                const uint32_t raw_there = poll(&raw_full[kl % TCX_NRAW], (kl / TCX_NRAW) & 1u), a_free = poll(&a_empty[a], aph);
                uint32_t h[4][16];                        // all of them before the first store: a register that a store still has to read cannot be written
#pragma unroll
                for (uint32_t kg = 0; kg < 4u; ++kg) {
                    const __half2 hs = __hsub2(tcx_h2(tcx_prmt(sc4, 0x64646464u, 0x4040u + 0x0101u * kg)), __float2half2_rn(1024.0f)), hb = __hmul2(hs, __float2half2_rn(-1152.0f));
#pragma unroll
                    for (uint32_t t = 0; t < 4u; ++t) tcx_decode8(kg == 0u ? wd[t].x : kg == 1u ? wd[t].y : kg == 2u ? wd[t].z : wd[t].w, hs, hb, h[kg] + 4u * t);
                }
                if (i + 1u < ncb * TCX_T && !(ok = load(raw_there))) break;        // on its way while this block is stored
                if (!(ok = wait_polled(a_free, &a_empty[a], aph))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (uint32_t kg = 0; kg < 4u; ++kg)
                    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                                 :: "r"(ta0 + a * TCX_A_COLS + kg * 16u), "r"(h[kg][0]), "r"(h[kg][1]), "r"(h[kg][2]), "r"(h[kg][3]), "r"(h[kg][4]), "r"(h[kg][5]), "r"(h[kg][6]), "r"(h[kg][7]),
                                    "r"(h[kg][8]), "r"(h[kg][9]), "r"(h[kg][10]), "r"(h[kg][11]), "r"(h[kg][12]), "r"(h[kg][13]), "r"(h[kg][14]), "r"(h[kg][15]) : "memory");
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc_arrive(smem_u32(&a_full[a]));
                if ((a += TCX_SPB) >= TCX_NA) { a -= TCX_NA; aph ^= 1u; }
            }
        }
    } else {
        // ------------------------------------------------------------------ accumulator drain and epilogue (256 threads)
        const uint32_t half = (warp - TCX_W_DRAIN) >> 2, row = (warp & 3u) * 32u + lane, tlane = tmem + (((warp & 3u) * 32u) << 16);
        const uint32_t mat = A.nmat == 2u ? half : 0u, tile_of = A.nmat == 2u ? 0u : half;      // this warp's tile of a group
        float2 acc[TCX_TN / 2u];
        uint32_t ka = 0u;                                 // accumulations drained
        bool ok = true;
        for (uint32_t n = 0; ok && (ok = unit_wait(n)); ++n) {
            const TcxUnit &U = s_unit[n % TCX_NI];
            if (!U.live) break;
            const uint32_t ncol = U.ncol, ntok = U.ntok;
            uint32_t tile = U.group0 * gtiles + tile_of;
            const uint8_t *dptr = A.w[mat] + (uint64_t)U.expert * A.mat_bytes + (uint64_t)((tile * 8u + (row >> 4)) * bpr) * NIB_REC + nib_d_off(row & 15u);
            unsigned short dnext = __ldg(reinterpret_cast<const unsigned short *>(dptr));        // d of this thread's row, requested a block ahead
            uint32_t c = 0u;
#pragma unroll 1
            for (uint32_t i = 0; i < ncb && ok; ++i) {
                if (c == 0u)
#pragma unroll
                    for (uint32_t j = 0; j < TCX_TN / 2u; ++j) acc[j] = make_float2(0.f, 0.f);
                const float d = 0.125f * __half2float(__ushort_as_half(dnext));
                const bool last = ++c == bpr;             // of the group
                dptr += (uint64_t)(last ? (gtiles * 8u - 1u) * bpr + 1u : 1u) * NIB_REC;        // records from the last block of a row to the first of the next group's
                if (i + 1u < ncb) dnext = __ldg(reinterpret_cast<const unsigned short *>(dptr));
#pragma unroll 1
                for (uint32_t h = 0; h < TCX_SPB; ++h, ++ka) {
                    if (!(ok = wait(&acc_full[half], ka & 1u))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (uint32_t t = 0; t < TCX_TN; t += 16u) {
                        if (t >= ncol) break;
                        uint32_t m[TCX_SUBS][16];
#pragma unroll
                        for (uint32_t j = 0; j < TCX_SUBS; ++j)
                            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                                         : "=r"(m[j][0]), "=r"(m[j][1]), "=r"(m[j][2]), "=r"(m[j][3]), "=r"(m[j][4]), "=r"(m[j][5]), "=r"(m[j][6]), "=r"(m[j][7]),
                                           "=r"(m[j][8]), "=r"(m[j][9]), "=r"(m[j][10]), "=r"(m[j][11]), "=r"(m[j][12]), "=r"(m[j][13]), "=r"(m[j][14]), "=r"(m[j][15])
                                         : "r"(tlane + (half * TCX_SUBS + j) * TCX_TN + t));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (uint32_t j = 0; j < 16u; j += 2u)
                            acc[(t + j) / 2u] = __ffma2_rn(make_float2(d, d), __fadd2_rn(make_float2(__uint_as_float(m[0][j]), __uint_as_float(m[0][j + 1u])),
                                                           make_float2(__uint_as_float(m[1][j]), __uint_as_float(m[1][j + 1u]))), acc[(t + j) / 2u]);
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc_arrive(smem_u32(&acc_empty[half]));
                }
                if (!ok) break;
                if (last) {                               // store the group's results
                    c = 0u;
                    float *o = A.out[mat] + tile * TC_M + row;
                    tile += gtiles;
#pragma unroll
                    for (uint32_t t0 = 0; t0 < TCX_TN; t0 += 4u) {
                        if (t0 >= ntok) break;
                        const uint4 pair = *reinterpret_cast<const uint4 *>(U.pair + t0);
                        const float4 inv = *reinterpret_cast<const float4 *>(U.xinv + t0);
                        const float2 s0 = acc[t0 / 2u], s1 = acc[t0 / 2u + 1u];
                        o[(size_t)pair.x * A.out_stride] = s0.x * inv.x;
                        if (t0 + 1u < ntok) o[(size_t)pair.y * A.out_stride] = s0.y * inv.y;
                        if (t0 + 2u < ntok) o[(size_t)pair.z * A.out_stride] = s1.x * inv.z;
                        if (t0 + 3u < ntok) o[(size_t)pair.w * A.out_stride] = s1.y * inv.w;
                    }
                }
            }
            unit_done(n);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (fail && tid == 0) {
        atomicExch(A.err, 1u);
        if (A.status) A.status[ST_TIMEOUT] = 1u;
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TCX_TM_COLS) : "memory");
}

bool tcx_shape_ok(uint32_t nrows, uint32_t ncols) { return nrows % TC_M == 0 && nrows && (ncols == 256u || ncols == 512u || ncols == 1024u || ncols == 2048u); }

int launch_tc_prep_rows(const float *a, const float *b, uint32_t stride, uint32_t nrows, uint32_t ncols, __half *xd, float *x_inv, cudaStream_t s) {
    RC_REQUIRE(ncols % 256u == 0 && ncols && ncols <= 2048u && stride % 4u == 0 && nrows, "tc experts: rows of %u columns (stride %u) are not tileable, or no rows", ncols, stride);
    prof_begin(b ? "tcx_prep_act" : "tcx_prep_x", s);
    const uint32_t grid = (nrows + 7u) / 8u;
    if (ncols <= 512u) RC_LAUNCH((k_tc_prep_rows<2>), grid, 256, 0, s, a, b, stride, nrows, ncols, xd, x_inv);
    else RC_LAUNCH((k_tc_prep_rows<8>), grid, 256, 0, s, a, b, stride, nrows, ncols, xd, x_inv);
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

int launch_tc_experts(TcxArgs &A, uint32_t max_items, const char *tag, cudaStream_t s) {
    RC_REQUIRE(tcx_shape_ok(A.nrows, A.ncols), "tc experts: matrix %ux%u is not tileable (128 rows, 256/512/1024/2048 columns)", A.nrows, A.ncols);
    RC_REQUIRE((A.nmat == 1u || A.nmat == 2u) && A.w[0] && (A.nmat == 1u || A.w[1]) && max_items && A.x_div && A.work, "tc experts: bad matrix count or empty launch");
    RC_REQUIRE((uint64_t)max_items * (A.nrows / TC_M * A.nmat / TCX_T) <= 0x7fffffffu, "tc experts: %u work items are too many", max_items);
    const size_t smem = (size_t)TCX_NB * TCX_B_BUF + (size_t)TCX_NRAW * TCX_RAW;
    // groups of a unit: some sixteen blocks, fewer where that would leave SMs without work
    const uint32_t groups = A.nrows / TC_M * A.nmat / TCX_T;
    for (A.upg = groups; A.upg > 1u && (A.upg * (A.ncols >> 8) * TCX_T > 16u || (uint64_t)max_items * (groups / A.upg) < 148u * 4u);) A.upg >>= 1;
    const uint64_t units = (uint64_t)max_items * (groups / A.upg);
    const uint32_t grid = units < 148u ? (uint32_t)units : 148u;
    prof_begin(tag, s);
    RC_CUDA(cudaFuncSetAttribute(k_tc_experts, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    RC_LAUNCH((k_tc_experts), grid, TCX_THREADS, smem, s, A);
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc
