// Q6_K matrix x many activation rows on the integer tensor-core path (mma.sync m16n8k16, s8 x s8 -> s32).
//
// Used when one Q6_K matrix meets a batch of tokens (the shared expert of a ragged decode batch): the CUDA-core GEMV
// re-decodes the weights for every four tokens, whereas here a lane rebuilds two operand registers (4 weights of rows
// g and g+8) per 16-column scale group with ~14 integer instructions and then serves 8 tokens per three MMAs.
//
//   weight      w = d * sc * q,  q = 6-bit value - 32 in [-32, 31] (one int8), sc the int8 scale of the 16-group
//   activation  x = sx * (65536*q2 + 256*q1 + q0), balanced 8-bit digits (k_quant_act)
//   per group   the three digit products of a (row, token) are exact s32 (|.| <= 2^16); digits 1 and 2 are recombined
//               exactly in s32 (|.| < 2^25), the result and digit 0 converted to fp32 and accumulated with the fp32
//               scale d*sc
//
// Block = 8 warps = MS matrices x KS column splits x TGB groups of 8 tokens, for one tile of 16 rows. Weights and digits of a panel of
// columns are staged in shared memory by bulk copies, a row each, at pitches that keep the fragment loads free of bank conflicts.
// (Loaded straight from global memory, 4 bytes a lane from eight rows 1024 bytes apart, the kernel was bound by the L1 tag rate: 88
// cycles an SM for every 16 columns of 8 tokens. Shared expert of 64 tokens: 26 + 13 us then.)
// Partial sums meet in shared memory, where the epilogue (plain store or SiLU(gate)*up) is applied.
#define RC_PDL_DEFAULT 0
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_nib.cuh"
#include "redcuda_q6k_panels.cuh"

namespace rc {

// z: a quad of registers holding zero for the whole kernel (a literal 0 costs four moves in front of every MMA)
__device__ __forceinline__ void mma_s8_k16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, const int (&z)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};\n"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(z[0]), "r"(z[1]), "r"(z[2]), "r"(z[3]));
}

struct Q6Args {
    const uint8_t *w[2];
    uint64_t nb;
    uint32_t nrows, ncols, ntok;
    const int8_t *xq; const float *sx;      // digits [ntok][3][ncols], scale per token
    float *out; uint32_t out_stride;        // out[token * out_stride + row]
    uint32_t *status;
    uint32_t MS, KS, panel;                 // matrices and column splits per block (8 % (MS * KS) == 0), columns staged at a time
    uint32_t bits; float dw1;               // digit width and 2^bits
};
// the steps of q6m_panels, as the kernel's lambdas
template <class S, class W, class M> struct Q6Panels { S send; W arrived; M multiply; };
template <class S, class W, class M> Q6Panels(S, W, M) -> Q6Panels<S, W, M>;

__global__ void __launch_bounds__(256, 2) k_q6k_mma(const __grid_constant__ Q6Args A) {
    pdl_prologue();
    extern __shared__ __align__(16) uint8_t q6m_smem[];
    __shared__ float part[8][16][8];        // per warp: 16 rows x 8 tokens
    __shared__ float s_d[2][16][Q6M_PANEL / 256u];
    __shared__ __align__(8) uint64_t s_bar;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t MS = A.MS, KS = A.KS, TGB = 8u / (MS * KS);
    const uint32_t mat = warp % MS, ks = (warp / MS) % KS, tgl = warp / (MS * KS);
    const uint32_t tg = blockIdx.y * TGB + tgl;                 // group of 8 tokens
    const uint32_t row0 = blockIdx.x * 16u, bpr = A.ncols >> 8;
    const uint32_t tok_first = blockIdx.y * TGB * 8u, ntok_b = min(TGB * 8u, A.ntok - tok_first);     // the block's tokens
    const uint32_t u_begin = ks * (2u * bpr / KS), u_end = u_begin + 2u * bpr / KS;                   // the warp's runs of 128 columns
    const uint32_t pcmax = A.panel, a_bytes = q6m_a_bytes(pcmax);
    const uint32_t ql_pitch = pcmax / 2u + 16u, qh_pitch = pcmax / 4u + 16u, sc_pitch = pcmax / 16u + 16u, b_pitch = pcmax + 16u;
    uint8_t *b_base = q6m_smem + MS * a_bytes;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_bar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    float out[4] = {0.f, 0.f, 0.f, 0.f};
    int z[4];
    asm volatile("mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;" : "=r"(z[0]), "=r"(z[1]), "=r"(z[2]), "=r"(z[3]));
    auto send = [&](uint32_t blk0, uint32_t nblk) {
        const uint32_t pc = nblk * 256u;
        __syncthreads();                     // the barrier is ready; the panel before this one has been read
        if (tid == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(MS * 16u * (pc / 2u + pc / 4u + pc / 16u) + ntok_b * 3u * pc) : "memory");
        __syncthreads();
        for (uint32_t i = tid; i < MS * 48u + ntok_b * 3u; i += 256u) {
            const uint8_t *src;
            uint8_t *dst;
            uint32_t n;
            if (i < MS * 48u) {
                const uint32_t m = i / 48u, j = i - m * 48u, plane = j >> 4, r = j & 15u;
                const uint64_t blk = (uint64_t)(row0 + r) * bpr + blk0;
                uint8_t *am = q6m_smem + m * a_bytes;
                if (plane == 0u) { src = A.w[m] + blk * 128u; dst = am + r * ql_pitch; n = pc / 2u; }
                else if (plane == 1u) { src = A.w[m] + rc_q6_qh(A.nb) + blk * 64u; dst = am + 16u * ql_pitch + r * qh_pitch; n = pc / 4u; }
                else { src = A.w[m] + rc_q6_sc(A.nb) + blk * 16u; dst = am + 16u * (ql_pitch + qh_pitch) + r * sc_pitch; n = pc / 16u; }
            } else {                         // tokens beyond the batch leave their columns as they are: a column of the product depends on no other
                const uint32_t j = i - MS * 48u;
                src = reinterpret_cast<const uint8_t *>(A.xq) + ((size_t)tok_first * 3u + j) * A.ncols + blk0 * 256u; dst = b_base + j * b_pitch; n = pc;
            }
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n), "r"(bar) : "memory");
        }
        for (uint32_t i = tid; i < MS * 16u * nblk; i += 256u) {
            const uint32_t m = i / (16u * nblk), j = i - m * 16u * nblk, r = j / nblk, c = j - r * nblk;
            s_d[m][r][c] = __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short *>(A.w[m] + rc_q6_d(A.nb)) + (uint64_t)(row0 + r) * bpr + blk0 + c)));
        }
    };
    auto arrived = [&](uint32_t parity) { return __syncthreads_and(nb_wait(bar, parity)) != 0; };      // its block barrier also publishes s_d
    auto multiply = [&](uint32_t blk0, uint32_t nblk) {
        if (tg * 8u >= A.ntok) return;
        const uint8_t *xb = b_base + (tgl * 8u + g) * 3u * b_pitch + 4u * t, *am = q6m_smem + mat * a_bytes;
        for (uint32_t u = max(u_begin, 2u * blk0); u < min(u_end, 2u * (blk0 + nblk)); ++u) {
            const uint32_t b = (u >> 1) - blk0, h = u & 1u;
            uint32_t ql[2][2][2], qh[2][2];       // [row g / g + 8][columns 0..15 / 16..31 of a run of 32][runs 0, 2 / 1, 3]
            float d[2];
            uint2 sc[2];
#pragma unroll
            for (uint32_t hr = 0; hr < 2u; ++hr) {
                const uint32_t r = g + 8u * hr;
#pragma unroll
                for (uint32_t i = 0; i < 2u; ++i) {
                    const uint8_t *lp = am + r * ql_pitch + b * 128u + 64u * h + 16u * i + 4u * t;
                    ql[hr][i][0] = *reinterpret_cast<const uint32_t *>(lp); ql[hr][i][1] = *reinterpret_cast<const uint32_t *>(lp + 32u);
                    qh[hr][i] = *reinterpret_cast<const uint32_t *>(am + 16u * ql_pitch + r * qh_pitch + b * 64u + 32u * h + 16u * i + 4u * t);
                }
                sc[hr] = *reinterpret_cast<const uint2 *>(am + 16u * (ql_pitch + qh_pitch) + r * sc_pitch + b * 16u + 8u * h);
                d[hr] = s_d[mat][r][b];
            }
#pragma unroll
            for (uint32_t q = 0; q < 4u; ++q)
#pragma unroll
                for (uint32_t i = 0; i < 2u; ++i) {
                    const uint8_t *xp = xb + b * 256u + h * 128u + 32u * q + 16u * i;
                    uint32_t a[2];
                    float scl[2];
#pragma unroll
                    for (uint32_t hr = 0; hr < 2u; ++hr) {
                        const uint32_t v = ((ql[hr][i][q & 1u] >> (4u * (q >> 1))) & 0x0F0F0F0Fu) | (((qh[hr][i] >> (2u * q)) & 0x03030303u) << 4);
                        const uint32_t x = v ^ 0x20202020u;            // 6-bit two's complement of (value - 32)
                        a[hr] = x + (x & 0x20202020u) * 6u;             // sign-extend every byte to 8 bits (bits 6,7 were clear: no carry)
                        scl[hr] = d[hr] * (float)(int)(signed char)((q < 2u ? sc[hr].x : sc[hr].y) >> (16u * (q & 1u) + 8u * i));
                    }
                    int d0[4], d1[4], d2[4];
                    mma_s8_k16(d0, a[0], a[1], *reinterpret_cast<const uint32_t *>(xp), z);
                    mma_s8_k16(d1, a[0], a[1], *reinterpret_cast<const uint32_t *>(xp + b_pitch), z);
                    mma_s8_k16(d2, a[0], a[1], *reinterpret_cast<const uint32_t *>(xp + 2u * b_pitch), z);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int hi = d1[c] + (d2[c] << A.bits);                 // 8-bit digits: the full recombination would leave s32
                        out[c] += scl[c >> 1] * fmaf(A.dw1, (float)hi, (float)d0[c]);
                    }
                }
        }
    };
    Q6Panels steps{send, arrived, multiply};
    const bool ok = q6m_panels(steps, bpr, pcmax / 256u);
    // accumulator columns 2t, 2t+1 of this lane are tokens tg*8 + 2t, +1
    const uint32_t tk0 = tg * 8u + 2u * t;
    const float s0 = tk0 < A.ntok ? A.sx[tk0] : 0.f, s1 = tk0 + 1u < A.ntok ? A.sx[tk0 + 1u] : 0.f;
    part[warp][g][2u * t] = out[0] * s0; part[warp][g][2u * t + 1u] = out[1] * s1;
    part[warp][g + 8u][2u * t] = out[2] * s0; part[warp][g + 8u][2u * t + 1u] = out[3] * s1;
    if (!ok && tid == 0 && A.status) A.status[ST_TIMEOUT] = 1u;      // a copy never came: the results are void
    __syncthreads();
    // epilogue: TGB token groups x 16 rows x 8 tokens
    for (uint32_t idx = tid; idx < TGB * 128u; idx += 256u) {
        const uint32_t tl = idx >> 7, row = (idx >> 3) & 15u, c = idx & 7u;
        const uint32_t tkn = (blockIdx.y * TGB + tl) * 8u + c;
        if (tkn >= A.ntok || row0 + row >= A.nrows) continue;
        float val[2] = {0.f, 0.f};
        for (uint32_t m = 0; m < MS; ++m)
            for (uint32_t k = 0; k < KS; ++k) val[m] += part[(tl * KS + k) * MS + m][row][c];
        float v = val[0];
        if (MS == 2u) v = (val[0] / (1.0f + expf(-val[0]))) * val[1];
        A.out[(size_t)tkn * A.out_stride + row0 + row] = v;
    }
}

// Once per layer or engine, on its device: a launch may then take what shared memory it needs. (Asked for at every launch it cost the host
// about half a microsecond, twice a layer, where the host's queueing is what a small batch waits for.)
int q6k_mma_init() {
    RC_CUDA(cudaFuncSetAttribute(k_q6k_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Q6M_SMEM));
    return 1;
}

// out[t][r] = W0[r].x[t]   or   SiLU(W0[r].x[t]) * (W1[r].x[t]) for Q6_K matrices and activations already in digit form.
int launch_q6k_mma(const uint8_t *w0, const uint8_t *w1, uint64_t nb, uint32_t nrows, uint32_t ncols, uint32_t ntok,
                   const int8_t *xq, const float *sx, float *out, uint32_t out_stride, const char *tag, cudaStream_t s) {
    RC_REQUIRE(nrows % 16u == 0 && ncols % 256u == 0, "q6k mma: matrix %ux%u must be a multiple of 16 rows x 256 columns", nrows, ncols);
    if (!ntok) return 1;
    Q6Args A{};
    A.w[0] = w0; A.w[1] = w1 ? w1 : w0; A.nb = nb; A.nrows = nrows; A.ncols = ncols; A.ntok = ntok; A.xq = xq; A.sx = sx;
    A.out = out; A.out_stride = out_stride; A.status = status_words();
    A.bits = act_digit_bits(); A.dw1 = (float)(1u << A.bits);
    const Q6Plan P = q6m_plan(w1 != nullptr, nrows, ncols, ntok);
    A.MS = P.MS; A.KS = P.KS; A.panel = P.panel;
    const uint32_t tok_block = 8u * (8u / (P.MS * P.KS));
    const dim3 grid(nrows / 16u, (ntok + tok_block - 1u) / tok_block);
    prof_begin(tag, s);
    RC_LAUNCH((k_q6k_mma), grid, 256, P.smem, s, A);
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc
