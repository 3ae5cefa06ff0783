// Router logits of a chunk as integer products on the 5th-generation tensor cores (tcgen05, kind::i8), and in double where these do not give the sum.
//
// The logits loop of the reference (native/redlite_native_engine_cpu.c:347-355) sums in double, and so does k_router_logits, whose fp64 tensor
// instructions run at 64 FMA per SM and clock: 133 us for 2048 tokens x 512 experts x 2048 columns, 119 of them the instructions themselves. Here a
// row of x and a row of W are fixed point, five balanced 8-bit digits d_i with a power-of-two scale per row: v 2^e = sum_i d_i 2^(8 (4 - i)), in steps of
// a quantum q that is at most 2^-37 of the row's largest magnitude (and more than 2^-38): an element of 2^-14 of the largest or more is exact, a smaller one
// off by at most q / 2. The products of two digits and their sums over a row are exact in 32 bits (5 x 8192 x 2^14 < 2^31), so that digits with the same
// i + j = s share an accumulator. s up to 5 is kept (19 of 25 products); the six sums are added in double, scaled by powers of two and rounded once.
// With r the sum of what a row's elements are off by, in quanta, a sum of n columns lacks at most
//     E = q_x q_w (2^38 (r_x + r_w) + 3.1 2^30 n)
// (no element exceeds 2^38 quanta; left out are three products of two digits of s = 6, at most 2^14 in units of 2^16 q_x q_w, and less below them). A logit with
// E <= 2^-24 |logit| stands: its sum is right to the rounding of fp32, and nearly always by far more, since errors of both signs meet. Every other is
// summed again in double (k_rt_exact): those that nearly cancel (eight in ten thousand with Gaussian rows of 2048), those of rows whose largest element stands out by so
// much that the others lose digits, and the rows that are not finite, whose scale is NaN.
//
// k_rt_digits_x / _w   fp32 rows -> digits in the layout that a stage reads: [tile][stage of 64 columns][digit, 16-byte chunk, row], K-major core matrices; and a
//                      row's (q, r)
// k_rt_logits<TOK>     one CTA = 128 experts x TOK tokens x all columns: a producer warp (two bulk copies a stage), an MMA warp (two k-steps of 32 columns
//                      a stage, seven MMAs each: digit i of W against as many digits of x as keep s <= 5, side by side in N), four drain warps at the end.
//                      The MMAs of a k-step take 608 cycles for 64 tokens and the operands 30 KB from L2, which delivers some 43 bytes a cycle to an SM: 700.
//                      These also set the bit of a logit whose E is too large.
// k_rt_exact           the logits with their bit set, in double: a block per eight tokens, a warp per logit
#define RC_PDL_DEFAULT 0
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_tc_gemm.cuh"

#include <math.h>

namespace rc {

constexpr uint32_t RT_D = 5u, RT_S = 6u, RT_KS = 64u, RT_CH = RT_KS / 16u, RT_NS = 3u;      // digits, sums kept, columns of a stage, its 16-byte chunks, stages in flight
constexpr uint32_t RT_A_DIGIT = RT_CH * 128u * 16u, RT_A_BUF = RT_D * RT_A_DIGIT;            // 8 KB, 40 KB
constexpr uint32_t RT_THREADS = 192u;

// v 2^(38 - e) as a rounded integer, e the exponent of the row's largest magnitude (mx = f 2^e, f in [0.5, 1)), in two parts of 32 bits: a holds digits 0 to 2
// (|v 2^(22 - e)| < 2^22), b the two below. Adding 1.5 2^23 leaves a float's rounded value in its mantissa; every difference here is exact.
// Conversions to and from double are served at a few values a cycle, and 64-bit shifts are three instructions each.
// Returned: what that is off by, in quanta.
__device__ __forceinline__ float rt_fixed(float v, float up0, float up1, uint32_t &a, uint32_t &b) {
    const float magic = 12582912.0f, t = (v * up0) * up1, ta = t + magic, r = (t - (ta - magic)) * 65536.0f, rb = r + magic;
    int ia = __float_as_int(ta) - __float_as_int(magic), ib = __float_as_int(rb) - __float_as_int(magic);
    if (ib > 32639) { ib -= 65536; ++ia; }                           // what two balanced digits do not hold
    // adding 128 to every digit makes all bytes non-negative, so that the carries resolve themselves; digit 0 stays within 64
    a = ((uint32_t)ia + 0x808080u) ^ 0x808080u; b = ((uint32_t)ib + 0x8080u) ^ 0x8080u;
    return fabsf(r - (rb - magic));
}

// Eight rows of ncols values (those from `live` on are zeros) -> digits at out + [stage][digit * dstride + chunk * cstride + row * 16], a chunk of 16 values a
// thread and step: neighbouring lanes take neighbouring rows, whose chunks lie side by side. block = 512
__device__ __forceinline__ void rt_digits_rows(const float *rows, uint32_t stride, uint32_t live, uint32_t ncols, uint8_t *out, size_t stage_bytes, uint32_t dstride, uint32_t cstride,
                                               double2 *row_out) {
    __shared__ uint32_t s_mag[16];
    __shared__ float s_off[16][8];
    __shared__ float2 s_up[8];                                       // the multiplier 2^(22 - e) of a row as two factors; zero where every digit is to be zero
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    auto load4 = [&](uint32_t r, uint32_t k) {
        if (r >= live) return make_float4(0.f, 0.f, 0.f, 0.f);
        const float *p = rows + (size_t)r * stride + k;              // a caller's rows may begin at any float
        return ((size_t)p & 15u) == 0u ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
    };
    uint32_t mag = 0u;                                               // |v| as bits: NaN above infinity above every number
#pragma unroll 8
    for (uint32_t k = (warp & 1u) * 128u + lane * 4u; k < ncols; k += 256u) {
        const float4 v = load4(warp >> 1, k);
        mag = max(mag, max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu), max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu)));
    }
    mag = __reduce_max_sync(0xffffffffu, mag);
    if (lane == 0) s_mag[warp] = mag;
    __syncthreads();
    if (threadIdx.x < 8u) {
        // a zero row has scale 0, one that is not finite NaN
        mag = max(s_mag[2u * threadIdx.x], s_mag[2u * threadIdx.x + 1u]);
        int e = (int)(mag >> 23) - 126;
        if (mag < 0x00800000u) frexpf(__uint_as_float(mag), &e);     // subnormal
        row_out[threadIdx.x].x = mag >= 0x7f800000u ? (double)NAN : mag ? __hiloint2double((e - 38 + 1023) << 20, 0) : 0.0;
        const int h = (22 - e) / 2;
        auto pow2 = [](int x) { return __int_as_float((x + 127) << 23); };
        s_up[threadIdx.x] = mag && mag < 0x7f800000u ? make_float2(pow2(h), pow2(22 - e - h)) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const uint32_t r = threadIdx.x & 7u;
    const float2 up = s_up[r];
    float off = 0.f;
#pragma unroll 1
    for (uint32_t ch = threadIdx.x >> 3; ch < ncols / 16u; ch += 64u) {
        float4 v[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) v[q] = load4(r, ch * 16u + q * 4u);
        uint32_t d[RT_D][4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            const float f[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
            uint32_t a[4], b[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) off += rt_fixed(up.x == 0.f ? 0.f : f[j], up.x, up.y, a[j], b[j]);
            // byte i of the four values side by side
            const uint32_t a01 = __byte_perm(a[0], a[1], 0x5140), a23 = __byte_perm(a[2], a[3], 0x5140), b01 = __byte_perm(b[0], b[1], 0x5140), b23 = __byte_perm(b[2], b[3], 0x5140);
            d[4][q] = __byte_perm(b01, b23, 0x5410); d[3][q] = __byte_perm(b01, b23, 0x7632); d[2][q] = __byte_perm(a01, a23, 0x5410); d[1][q] = __byte_perm(a01, a23, 0x7632);
            d[0][q] = __byte_perm(__byte_perm(a[0], a[1], 0x0062), __byte_perm(a[2], a[3], 0x0062), 0x5410);
        }
        uint8_t *o = out + (size_t)(ch / RT_CH) * stage_bytes + (ch % RT_CH) * cstride + r * 16u;
#pragma unroll
        for (uint32_t i = 0; i < RT_D; ++i) *reinterpret_cast<uint4 *>(o + (size_t)i * dstride) = make_uint4(d[i][0], d[i][1], d[i][2], d[i][3]);
    }
    off += __shfl_xor_sync(0xffffffffu, off, 8);                     // the lanes of a row
    off += __shfl_xor_sync(0xffffffffu, off, 16);
    if (lane < 8u) s_off[warp][lane] = off;
    __syncthreads();
    if (threadIdx.x < 8u) {
        float sum = 0.f;
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) sum += s_off[i][threadIdx.x];
        row_out[threadIdx.x].y = (double)sum;
    }
}

// grid = rows rounded up to the token tile / 8 (rows beyond ntok become zeros)
__global__ void __launch_bounds__(512) k_rt_digits_x(const float *x, uint32_t x_stride, uint32_t ntok, uint32_t ncols, uint32_t tok, uint8_t *__restrict__ xq, double2 *__restrict__ xs) {
    pdl_prologue();
    const uint32_t t = blockIdx.x * 8u, tile = t / tok, tt = t - tile * tok;
    const size_t stage = (size_t)RT_D * RT_KS * tok;
    rt_digits_rows(x + (size_t)t * x_stride, x_stride, t < ntok ? ntok - t : 0u, ncols, xq + (size_t)tile * (ncols / RT_KS) * stage + tt * 16u, stage, tok * 16u, RT_D * tok * 16u, xs + t);
}
// grid = experts / 8
__global__ void __launch_bounds__(512) k_rt_digits_w(const float *w, uint32_t ncols, uint8_t *__restrict__ wq, double2 *__restrict__ ws) {
    pdl_prologue();
    const uint32_t e = blockIdx.x * 8u, tile = e / 128u, r = e % 128u;
    rt_digits_rows(w + (size_t)e * ncols, ncols, 8u, ncols, wq + (size_t)tile * (ncols / RT_KS) * RT_A_BUF + r * 16u, RT_A_BUF, RT_A_DIGIT, 128u * 16u, ws + e);
}

// instruction descriptor, kind::i8: D = s32, A and B signed 8-bit, both K-major, M = 128
__device__ __forceinline__ uint32_t rt_idesc(uint32_t n) { return (2u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
__device__ __forceinline__ void rt_mma_if(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n"
        :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}

struct RtArgs { const uint8_t *wq, *xq; const double2 *ws, *xs; float *logits; uint32_t *again; uint32_t ntok, n_expert, ncols; uint32_t *err, *status; };

template <uint32_t TOK>
__global__ void __launch_bounds__(RT_THREADS, 1) k_rt_logits(const __grid_constant__ RtArgs A) {
    pdl_prologue();
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr uint32_t B_BUF = RT_D * RT_KS * TOK, STAGE = RT_A_BUF + B_BUF, TMEM_COLS = TOK >= 64u ? 512u : 256u;
    static_assert(RT_S * TOK <= TMEM_COLS && 4u * TOK <= 256u, "six accumulators in tensor memory, four digits of x in one MMA");
    __shared__ __align__(8) uint64_t full[RT_NS], empty[RT_NS], done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t fail;               // a bounded wait ran out
    __shared__ __align__(16) double2 s_xs[TOK];
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31u;
    const uint32_t nstage = A.ncols / RT_KS, t0 = blockIdx.x * TOK;
    const uint8_t *wq = A.wq + (size_t)blockIdx.y * nstage * RT_A_BUF, *xq = A.xq + (size_t)blockIdx.x * nstage * B_BUF;
    if (tid == 0) {
        fail = 0u;
        auto init = [](uint64_t *bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(bar))); };
        for (uint32_t i = 0; i < RT_NS; ++i) { init(&full[i]); init(&empty[i]); }
        init(&done);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid >= RT_THREADS - TOK) s_xs[tid - (RT_THREADS - TOK)] = A.xs[t0 + tid - (RT_THREADS - TOK)];       // rows beyond the tokens are there, as zeros
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0), fail_at = smem_u32(const_cast<uint32_t *>(&fail));
    auto wait = [&](uint64_t *bar, uint32_t parity) { return tc_wait(smem_u32(bar), parity, fail_at); };

    if (warp == 0) {
        // ------------------------------------------------------------------ producer
        uint32_t s = 0u;
        for (; s < nstage; ++s) {
            const uint32_t j = s % RT_NS;
            if (s >= RT_NS && !wait(&empty[j], ((s / RT_NS) - 1u) & 1u)) break;
            if (lane == 0) {
                const uint32_t bar = smem_u32(&full[j]), dst = smem_u32(smem + j * STAGE);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(STAGE) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             :: "r"(dst), "l"(wq + (size_t)s * RT_A_BUF), "r"(RT_A_BUF), "r"(bar) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             :: "r"(dst + RT_A_BUF), "l"(xq + (size_t)s * B_BUF), "r"(B_BUF), "r"(bar) : "memory");
            }
            __syncwarp();
        }
        // after a timeout elsewhere, copies that nobody waits for may still be writing into this CTA's shared memory
        if (fail && lane == 0) for (uint32_t k = s >= RT_NS ? s - RT_NS : 0u; k < s; ++k) mbar_wait(smem_u32(&full[k % RT_NS]), (k / RT_NS) & 1u);
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issue
        const uint32_t leader = tc_elect();
        constexpr uint32_t A_LBO = 128u * 16u, B_LBO = RT_D * TOK * 16u;
        const uint64_t da0 = tc_smem_desc(smem_u32(smem), A_LBO, 128u), db0 = tc_smem_desc(smem_u32(smem) + RT_A_BUF, B_LBO, 128u);
        const uint32_t id1 = rt_idesc(TOK), id2 = rt_idesc(2u * TOK), id3 = rt_idesc(3u * TOK), id4 = rt_idesc(4u * TOK);
        bool ok = true;
#pragma unroll 1
        for (uint32_t s = 0; s < nstage; ++s) {
            const uint32_t j = s % RT_NS;
            if (!(ok = wait(&full[j], (s / RT_NS) & 1u))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t kk = 0; kk < RT_KS / 32u; ++kk) {
                const uint64_t da = da0 + j * (STAGE >> 4) + kk * (2u * A_LBO >> 4), db = db0 + j * (STAGE >> 4) + kk * (2u * B_LBO >> 4);
                const uint32_t more = s | kk;            // the first k-step overwrites: sums 0..3, 4 and 5 are first met in this order
                auto dig = [&](uint32_t i) { return da + i * (RT_A_DIGIT >> 4); };
                const uint64_t db4 = db + 4u * TOK;      // digit 4 of x: TOK rows of 16 bytes a digit
                rt_mma_if(leader, tmem, dig(0u), db, id4, more);
                rt_mma_if(leader, tmem + 4u * TOK, dig(0u), db4, id1, more);
                rt_mma_if(leader, tmem + TOK, dig(1u), db, id4, 1u);
                rt_mma_if(leader, tmem + 5u * TOK, dig(1u), db4, id1, more);
                rt_mma_if(leader, tmem + 2u * TOK, dig(2u), db, id4, 1u);
                rt_mma_if(leader, tmem + 3u * TOK, dig(3u), db, id3, 1u);
                rt_mma_if(leader, tmem + 4u * TOK, dig(4u), db, id2, 1u);
            }
            tc_commit_if(leader, smem_u32(&empty[j]));
        }
        if (ok) tc_commit_if(leader, smem_u32(&done));
    } else if (wait(&done, 0u)) {
        // ------------------------------------------------------------------ drain (128 threads): a thread owns an expert
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t qlane = (warp & 3u) * 32u, e = blockIdx.y * 128u + qlane + lane;
        const double2 W = A.ws[e];
        const double lacks = 0x1p38 * W.y + 3.1 * 0x1p30 * (double)A.ncols;
#pragma unroll 1
        for (uint32_t c = 0; c < TOK && t0 + c < A.ntok; c += 8u) {
            uint32_t m[RT_S][8];
#pragma unroll
            for (uint32_t s = 0; s < RT_S; ++s)
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(m[s][0]), "=r"(m[s][1]), "=r"(m[s][2]), "=r"(m[s][3]), "=r"(m[s][4]), "=r"(m[s][5]), "=r"(m[s][6]), "=r"(m[s][7])
                             : "r"(tmem + (qlane << 16) + s * TOK + c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                const uint32_t t = t0 + c + i;
                if (t >= A.ntok) break;
                double v = (double)(int)m[RT_S - 1u][i], p = 256.0;      // in units of 2^24 of the scaled values' product
#pragma unroll
                for (int s = (int)RT_S - 2; s >= 0; --s) { v = fma((double)(int)m[s][i], p, v); p *= 256.0; }
                const double2 X = s_xs[c + i];
                const double q = W.x * X.x;
                v *= 0x1p24;
                A.logits[(size_t)t * A.n_expert + e] = (float)(v * q);
                const uint32_t again = __ballot_sync(0xffffffffu, !((lacks + 0x1p38 * X.y) * q <= fabs(0x1p-24 * v * q)));
                if (lane == 0) A.again[((size_t)t * A.n_expert + e) >> 5] = again;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (fail && tid == 0) {
        atomicExch(A.err, 1u);
        if (A.status) A.status[ST_TIMEOUT] = 1u;
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TMEM_COLS) : "memory");
}

// The logits that the integer sums do not settle, in double: a block lists those of its eight tokens, its warps take them in turn (each its own token's: the token with the
// most of them made the others wait, 13.5 us for 2048 tokens where this takes 10.5; 23 with an element of 100 in every row, 263 if all are listed). grid = tokens / 8,
// block = 256. The chain of a few rows' loads bounds it while they are few, conversions to double when they are many
__global__ void __launch_bounds__(256, 2) k_rt_exact(const float *w, const float *x, uint32_t x_stride, uint32_t ntok, uint32_t n_expert, uint32_t ncols, const uint32_t *again, float *logits) {
    pdl_prologue();
    __shared__ uint16_t s_list[8192];                // token of the block, expert of the turn's 1024
    __shared__ uint32_t s_n;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, words = n_expert >> 5, t0 = blockIdx.x * 8u;
    for (uint32_t w0 = 0; w0 < words; w0 += 32u) {
        if (threadIdx.x == 0) s_n = 0u;
        __syncthreads();
        uint32_t bits = t0 + warp < ntok && w0 + lane < words ? again[(size_t)(t0 + warp) * words + w0 + lane] : 0u;
        uint32_t at = bits ? atomicAdd(&s_n, __popc(bits)) : 0u;
        for (; bits; bits &= bits - 1u) s_list[at++] = (uint16_t)(warp << 10 | lane << 5 | ((uint32_t)__ffs((int)bits) - 1u));
        __syncthreads();
        const uint32_t n = s_n;
        for (uint32_t k = warp; k < n; k += 8u) {
            const uint32_t item = s_list[k], t = t0 + (item >> 10), e = w0 * 32u + (item & 1023u);
            const float *wr = w + (size_t)e * ncols, *xr = x + (size_t)t * x_stride;
            auto sum = [&](auto load) {
                double a0 = 0.0, a1 = 0.0;
#pragma unroll 8
                for (uint32_t c = lane * 4u; c < ncols; c += 128u) {
                    const float4 b = __ldg(reinterpret_cast<const float4 *>(wr + c)), a = load(xr + c);
                    a0 = fma((double)a.x, (double)b.x, a0); a1 = fma((double)a.y, (double)b.y, a1);
                    a0 = fma((double)a.z, (double)b.z, a0); a1 = fma((double)a.w, (double)b.w, a1);
                }
                return a0 + a1;
            };
            double v;                                // a caller's rows may begin at any float
            if (((size_t)xr & 15u) == 0u) v = sum([](const float *p) { return *reinterpret_cast<const float4 *>(p); });
            else v = sum([](const float *p) { return make_float4(p[0], p[1], p[2], p[3]); });
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) logits[(size_t)t * n_expert + e] = (float)v;
        }
        __syncthreads();
    }
}

bool rt_shape_ok(uint32_t n_expert, uint32_t ncols) { return n_expert % 128u == 0 && n_expert && ncols % RT_KS == 0 && ncols && ncols <= 8192u; }
size_t rt_wq_bytes(uint32_t n_expert, uint32_t ncols) { return (size_t)n_expert * ncols * RT_D; }
static uint32_t rt_tok(uint32_t ntok, uint32_t n_expert) { return (ntok + 31u) / 32u * (n_expert / 128u) <= 148u ? 32u : 64u; }
size_t rt_xq_bytes(uint32_t ntok, uint32_t ncols) { return (size_t)((ntok + 63u) / 64u) * 64u * ncols * RT_D; }
size_t rt_rows(uint32_t ntok) { return (size_t)((ntok + 63u) / 64u) * 64u; }

static size_t rt_smem(uint32_t tok) { return (size_t)RT_NS * (RT_A_BUF + RT_D * RT_KS * tok); }
// before the first launch on a device
int rt_init() {
    RC_CUDA(cudaFuncSetAttribute(k_rt_logits<32u>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rt_smem(32u)));
    RC_CUDA(cudaFuncSetAttribute(k_rt_logits<64u>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rt_smem(64u)));
    return 1;
}

int launch_rt_digits_w(const float *w, uint32_t n_expert, uint32_t ncols, uint8_t *wq, double2 *ws, cudaStream_t s) {
    RC_REQUIRE(rt_shape_ok(n_expert, ncols), "router digits: %u experts of %u columns are not tileable", n_expert, ncols);
    RC_LAUNCH((k_rt_digits_w), n_expert / 8u, 512, 0, s, w, ncols, wq, ws);
    RC_LAUNCHED();
    return 1;
}

int launch_rt_logits(const float *w, const uint8_t *wq, const double2 *ws, const float *x, uint32_t x_stride, uint32_t ntok, uint32_t n_expert, uint32_t ncols, uint8_t *xq, double2 *xs, uint32_t *again,
                     float *logits, uint32_t *err, cudaStream_t s) {
    RC_REQUIRE(rt_shape_ok(n_expert, ncols) && ntok && w && wq && xq, "router logits: %u experts of %u columns are not tileable, or no tokens", n_expert, ncols);
    const uint32_t tok = rt_tok(ntok, n_expert), tiles = (ntok + tok - 1u) / tok;
    prof_begin("moe_router_digits", s);
    RC_LAUNCH((k_rt_digits_x), tiles * tok / 8u, 512, 0, s, x, x_stride, ntok, ncols, tok, xq, xs);
    prof_end(s);
    RC_LAUNCHED();
    const RtArgs A{wq, xq, ws, xs, logits, again, ntok, n_expert, ncols, err, status_words()};
    const dim3 grid(tiles, n_expert / 128u);
    prof_begin("moe_router_logits", s);
    if (tok == 64u) RC_LAUNCH((k_rt_logits<64u>), grid, RT_THREADS, rt_smem(64u), s, A);
    else RC_LAUNCH((k_rt_logits<32u>), grid, RT_THREADS, rt_smem(32u), s, A);
    prof_end(s);
    RC_LAUNCHED();
    prof_begin("moe_router_exact", s);
    RC_LAUNCH_PDL((k_rt_exact), (ntok + 7u) / 8u, 256, 0, s, w, x, x_stride, ntok, n_expert, ncols, (const uint32_t *)again, logits);
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc
