// Single-token matrix-vector products (F32 / F16 / Q6_K rows): the dense projections, the LM head, the router logits with
// the shared expert's gate / up and scalar gate of a decode step.
//
// What bounds it: HBM for the large matrices, the length of the dependent chain for the small ones. The general GEMV
// (redcuda_core.cu) staged x in shared memory behind a barrier and read it back 16 bytes per four weights, turned every
// 6-bit weight into a float with a conversion, and began a row's loads only after the previous row's sums. Here
//   - a warp takes two rows of a 2048-column slice at a time, so that every 16 bytes of x read from shared memory serve both
//     (x in registers instead, one row at a time, left 16 warps an SM: 80 us for a 151936 x 2048 matrix);
//   - a 6-bit weight becomes a float by a byte permute into the mantissa of 2^23 and a packed subtraction, and two
//     weights are multiplied by one packed FMA: 2.7 instructions a weight instead of about 5;
//   - the first rows of resident weights are requested before the wait for the previous kernel (they do not depend on it);
//   - rows wider than a slice are cut over the warps of the block, partial sums meet in shared memory in a fixed order.
// Plain rows (router, scalar gate) are accumulated in double, as everywhere: they decide discrete outcomes.
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_moe_mma.cuh"
#include "redcuda_route.cuh"

namespace rc {

namespace {
constexpr uint32_t G1_WARPS = 8u, G1_QCOLS = 2048u, G1_PCOLS = 512u;      // columns of one warp's slice: Q6_K, plain
__host__ __device__ inline uint32_t g1_slices(uint32_t type, uint32_t ncols) { const uint32_t c = type == RC_Q6_K ? G1_QCOLS : G1_PCOLS; return (ncols + c - 1u) / c; }
// warps that take different slices of the same rows; a slice count that does not divide the warps is walked by every warp
__host__ __device__ inline uint32_t g1_slice_warps(uint32_t slices) { return slices <= G1_WARPS && G1_WARPS % slices == 0u ? slices : 1u; }
// lanes per Q6_K row: the chunks of 64 columns of a short row, rounded up to a power of two
__host__ __device__ inline uint32_t g1_lanes(uint32_t type, uint32_t ncols) {
    if (type != RC_Q6_K) return 32u;
    uint32_t l = 4u;
    while (l < 32u && l < (ncols >> 6)) l <<= 1;
    return l;
}
}  // namespace

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ uint64_t f2_pack(uint32_t lo, uint32_t hi) { return (uint64_t)lo | ((uint64_t)hi << 32); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }

struct Q6Frag { uint4 a, b, h; uint2 sc; unsigned short d; };
struct G1Tile { uint32_t row0, nvr, pair; bool resident; };      // nvr: rows of the tile, counted twice (w0, w1 in turn) for a gate / up pair

// where column k of x sits in shared memory: eight lanes that read their 16 bytes of neighbouring chunks (k = 0, 16, 128, 144 of
// two blocks) hit eight different bank groups
__host__ __device__ __forceinline__ uint32_t g1_xi(uint32_t k) { return (k >> 8) * 268u + ((k >> 7) & 1u) * 136u + (k & 127u); }

// x into shared memory, by every thread of the block; with a norm, normalised on the way. A kernel of its own for it (one block) took 4.6 us
// of a decoding step's chain twice a layer; here it is about one, most of it while the first weights arrive. ncols at most G1_NCOLS then.
constexpr uint32_t G1_NCOLS = 2048u;
template <bool NORM>
__device__ __forceinline__ void gemv1_stage(const GemvArgs &A, uint32_t ncols, float *xs) {
    if (!NORM) {
        for (uint32_t k = threadIdx.x * 4u; k < ncols; k += G1_WARPS * 128u) *reinterpret_cast<float4 *>(xs + g1_xi(k)) = *reinterpret_cast<const float4 *>(A.x + k);
        return;
    }
    // the row waits in shared memory for its sum: the first weights hold the registers
    __shared__ double red[G1_WARPS];
    double ss = 0.0;
    for (uint32_t k = threadIdx.x * 4u; k < ncols; k += G1_WARPS * 128u) {
        float4 v = *reinterpret_cast<const float4 *>(A.x + k);
        if (A.norm.branch) {
            const float4 b = *reinterpret_cast<const float4 *>(A.norm.branch + k);
            v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
        }
        *reinterpret_cast<float4 *>(xs + g1_xi(k)) = v;
        if (blockIdx.x == 0u && A.norm.resid) *reinterpret_cast<float4 *>(A.norm.resid + k) = v;
        ss += (double)v.x * (double)v.x + (double)v.y * (double)v.y + (double)v.z * (double)v.z + (double)v.w * (double)v.w;
    }
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31u) == 0u) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    double tot = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < G1_WARPS; ++i) tot += red[i];
    const double inv = 1.0 / sqrt(tot / (double)ncols + (double)A.norm.eps);
    for (uint32_t k = threadIdx.x * 4u; k < ncols; k += G1_WARPS * 128u) {
        const float4 v = *reinterpret_cast<const float4 *>(xs + g1_xi(k)), w = __ldg(reinterpret_cast<const float4 *>(A.norm.w + k));
        const float4 n = make_float4((float)((double)v.x * inv * (double)w.x), (float)((double)v.y * inv * (double)w.y),
                                     (float)((double)v.z * inv * (double)w.z), (float)((double)v.w * inv * (double)w.w));
        *reinterpret_cast<float4 *>(xs + g1_xi(k)) = n;
        if (blockIdx.x == 0u) *reinterpret_cast<float4 *>(A.norm.normed + k) = n;
    }
}

template <bool NORM, bool STAGED = false>          // STAGED: x is in shared memory
__device__ __forceinline__ void gemv1_q6k(const GemvArgs &A, const GemvJob &J, const G1Tile &T, double *part, float *xs) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t cpr = J.ncols >> 6, bpr = J.ncols >> 8, S = g1_slices(RC_Q6_K, J.ncols), ws = g1_slice_warps(S), lpr = g1_lanes(RC_Q6_K, J.ncols), rw = 32u / lpr;
    const uint32_t slot = lane / lpr, sub = lane % lpr, step = (G1_WARPS / ws) * rw, first = (warp / ws) * rw;
    const uint64_t o_h = rc_q6_qh(J.nb), o_s = rc_q6_sc(J.nb), o_d = rc_q6_d(J.nb);
    const uint64_t bias = f2_pack(__float_as_uint(-8388640.0f), __float_as_uint(-8388640.0f));      // 2^23 + 32
    bool staged = STAGED;
    for (uint32_t sl = warp % ws; sl < S; sl += ws) {
        const uint32_t c = sl * (G1_QCOLS / 64u) + sub;
        const bool on = c < cpr;                                  // lanes past the row's end repeat its last chunk and add nothing
        const uint32_t cc = on ? c : cpr - 1u, bcol = cc >> 2, half = (cc >> 1) & 1u, l0 = (cc & 1u) * 16u;
        auto load = [&](uint32_t vr) {
            vr = min(vr, T.nvr - 1u);
            const uint8_t *w = T.pair && (vr & 1u) ? J.w1 : J.w0;
            const uint64_t blk = (uint64_t)(T.row0 + (vr >> T.pair)) * bpr + bcol;
            const uint8_t *wl = w + blk * 128u + half * 64u + l0;
            Q6Frag f;
            f.a = __ldg(reinterpret_cast<const uint4 *>(wl));
            f.b = __ldg(reinterpret_cast<const uint4 *>(wl + 32u));
            f.h = __ldg(reinterpret_cast<const uint4 *>(w + o_h + blk * 64u + half * 32u + l0));
            f.sc = __ldg(reinterpret_cast<const uint2 *>(w + o_s + blk * 16u + half * 8u));
            f.d = __ldg(reinterpret_cast<const unsigned short *>(w + o_d) + blk);
            return f;
        };
        // two rows at a time: each 16 bytes of x read from shared memory serve both
        Q6Frag f[2];
        if (T.resident || staged) { f[0] = load(first + slot); f[1] = load(first + step + slot); }
        if (!staged) {
            staged = true;
            pdl_wait();
            gemv1_stage<NORM>(A, J.ncols, xs);
            if (!T.resident) { f[0] = load(first + slot); f[1] = load(first + step + slot); }
            __syncthreads();
        }
        const float *xl = xs + bcol * 268u + half * 136u + l0;
        for (uint32_t base = first; base < T.nvr; base += 2u * step) {
            uint64_t s[2][4] = {{0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                uint32_t v[2][4];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t a = w == 0 ? f[r].a.x : w == 1 ? f[r].a.y : w == 2 ? f[r].a.z : f[r].a.w, b = w == 0 ? f[r].b.x : w == 1 ? f[r].b.y : w == 2 ? f[r].b.z : f[r].b.w;
                    const uint32_t h = w == 0 ? f[r].h.x : w == 1 ? f[r].h.y : w == 2 ? f[r].h.z : f[r].h.w;
                    v[r][0] = (a & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u); v[r][1] = (b & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u);
                    v[r][2] = ((a >> 4) & 0x0F0F0F0Fu) | (h & 0x30303030u); v[r][3] = ((b >> 4) & 0x0F0F0F0Fu) | ((h >> 2) & 0x30303030u);
                }
#pragma unroll
                for (int qd = 0; qd < 4; ++qd) {
                    const uint32_t m = 0x4B000000u;
                    const ulonglong2 xv = *reinterpret_cast<const ulonglong2 *>(xl + 32u * qd + 4u * w);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint64_t w01 = f2_add(f2_pack(__byte_perm(v[r][qd], m, 0x7540), __byte_perm(v[r][qd], m, 0x7541)), bias);
                        const uint64_t w23 = f2_add(f2_pack(__byte_perm(v[r][qd], m, 0x7542), __byte_perm(v[r][qd], m, 0x7543)), bias);
                        s[r][qd] = f2_fma(w01, xv.x, s[r][qd]);
                        s[r][qd] = f2_fma(w23, xv.y, s[r][qd]);
                    }
                }
            }
            float acc[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float d = __half2float(__ushort_as_half(f[r].d));
                // the four scales of this lane's runs of 16 sit in every other byte of its half block
                const uint32_t q = l0 ? 8u : 0u;
                const int sc[4] = {(int)(signed char)(f[r].sc.x >> q), (int)(signed char)(f[r].sc.x >> (q + 16u)), (int)(signed char)(f[r].sc.y >> q), (int)(signed char)(f[r].sc.y >> (q + 16u))};
                acc[r] = 0.f;
#pragma unroll
                for (int qd = 0; qd < 4; ++qd) acc[r] += (d * (float)sc[qd]) * (__uint_as_float((uint32_t)s[r][qd]) + __uint_as_float((uint32_t)(s[r][qd] >> 32)));
                if (!on) acc[r] = 0.f;
            }
            if (base + 2u * step < T.nvr) { f[0] = load(base + 2u * step + slot); f[1] = load(base + 3u * step + slot); }      // on the way during the reduction
            for (uint32_t o = lpr >> 1; o; o >>= 1) { acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o); acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], o); }
            if (sub == 0u) {
                if (base + slot < T.nvr) part[(base + slot) * S + sl] = (double)acc[0];
                if (base + step + slot < T.nvr) part[(base + step + slot) * S + sl] = (double)acc[1];
            }
        }
    }
}

template <bool NORM, bool HALF>
__device__ __forceinline__ void gemv1_plain(const GemvArgs &A, const GemvJob &J, const G1Tile &T, double *part, float *xs) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t S = g1_slices(RC_F32, J.ncols), ws = g1_slice_warps(S), step = G1_WARPS / ws;
    bool waited = false;
    for (uint32_t sl = warp % ws; sl < S; sl += ws) {
        const uint32_t k0 = sl * G1_PCOLS + lane * 4u;
        float4 w[4], xv[4];
        auto load = [&](uint32_t vr) {
            const uint8_t *m = T.pair && (vr & 1u) ? J.w1 : J.w0;
            const size_t row = (size_t)(T.row0 + (vr >> T.pair)) * J.ncols;
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                const uint32_t k = k0 + 128u * i;
                if (k >= J.ncols) { w[i] = make_float4(0.f, 0.f, 0.f, 0.f); continue; }
                if (HALF) {
                    const uint2 r = __ldg(reinterpret_cast<const uint2 *>(m + (row + k) * 2u));
                    const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&r.x)), hi = __half22float2(*reinterpret_cast<const __half2 *>(&r.y));
                    w[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
                } else w[i] = __ldg(reinterpret_cast<const float4 *>(m + (row + k) * 4u));
            }
        };
        uint32_t vr = warp / ws;
        if (T.resident && vr < T.nvr) load(vr);
        if (!waited) {
            pdl_wait();
            waited = true;
            if (NORM) { gemv1_stage<NORM>(A, J.ncols, xs); __syncthreads(); }      // every warp has a slice, so all of them come here
        }
        if (!T.resident && vr < T.nvr) load(vr);
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
            const uint32_t k = k0 + 128u * i;
            xv[i] = k < J.ncols ? *reinterpret_cast<const float4 *>(NORM ? xs + g1_xi(k) : A.x + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (; vr < T.nvr; vr += step) {
            double a0 = 0.0, a1 = 0.0;                    // two chains: the double FMA's latency is what a short row waits for
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                a0 = fma((double)w[i].x, (double)xv[i].x, a0); a1 = fma((double)w[i].y, (double)xv[i].y, a1);
                a0 = fma((double)w[i].z, (double)xv[i].z, a0); a1 = fma((double)w[i].w, (double)xv[i].w, a1);
            }
            if (vr + step < T.nvr) load(vr + step);
            double acc = a0 + a1;
            for (uint32_t o = 16u; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0u) part[vr * S + sl] = acc;
        }
    }
    if (!waited) pdl_wait();
}

template <bool NORM>
__global__ void __launch_bounds__(G1_WARPS * 32u, 3) k_gemv1(const __grid_constant__ GemvArgs A) {
    pdl_trigger();
    extern __shared__ __align__(16) double g1_part[];      // [row of the tile (x 2 for a pair)][slice], behind it x
    uint32_t j = 0;
    while (j + 1u < A.njobs && blockIdx.x >= A.job[j + 1u].tile_begin) ++j;
    const GemvJob &J = A.job[j];
    const uint32_t row0 = (blockIdx.x - J.tile_begin) * J.rows_per_tile, nrow = min(J.rows_per_tile, J.nrows - row0), pair = J.epi == GEMV_PAIR_SILU ? 1u : 0u;
    const G1Tile T{row0, nrow << pair, pair, A.resident != 0u};
    float *xs = reinterpret_cast<float *>(g1_part + A.part_doubles);
    if (J.type == RC_Q6_K) gemv1_q6k<NORM>(A, J, T, g1_part, xs);
    else if (J.type == RC_F32) gemv1_plain<NORM, false>(A, J, T, g1_part, xs);
    else gemv1_plain<NORM, true>(A, J, T, g1_part, xs);
    __syncthreads();
    const uint32_t S = g1_slices(J.type, J.ncols);
    for (uint32_t r = threadIdx.x; r < nrow; r += G1_WARPS * 32u) {
        const double *p = g1_part + (size_t)(r << pair) * S;
        double s0 = 0.0, s1 = 0.0;
        for (uint32_t i = 0; i < S; ++i) { s0 += p[i]; if (pair) s1 += p[S + i]; }
        float v = (float)s0;
        if (pair) v = (v / (1.0f + expf(-v))) * (float)s1;
        else if (J.epi == GEMV_SIGMOID) v = 1.0f / (1.0f + expf(-v));
        J.out[row0 + r] = v;
    }
    if (A.tail.ticket) route_tail(A.tail);
}

// ---- one large Q6_K matrix (the LM head) -------------------------------------------------------------------------------
// Instruction issue bounds the products of a matrix of that size in floats: a byte permute per weight to make it one. Here x is four 8-bit digits with a
// power-of-two scale per 256 columns (actw_digits), and a word of four 6-bit weights meets them in four dp4a: the
// sums of 16 columns are exact. The weights stay unsigned (q + 32), an accumulator begins with -32 times its digits' sum. Lanes, rows and loads as in
// gemv1_q6k. 151936 x 2048: 61 us (floats: 72; 255 MB take 39 at the copy rate). What bounds it now are waits for the digit words out of shared memory (half of
// what a warp waits for); 57 % of the issue slots are taken.
//
// The digits hold a value to 2^-30 of the largest of its 256, which is less than fp32 does for the small ones. So a row takes this form only if in each 256
//   - at least 32 values lie within 2^-6 of the largest: these are exact, and what the others lack comes to less than the rounding of the fp32 sums that replace it
//     (2^-23.3 of the block's product in the worst case, in the 2-norm over weights that do not follow the row). One value that stands out, which may meet a zero,
//     is not enough;
//   - the largest is at least 2^-60, so that neither the scale (2^-126 is the least) nor its product with d lose bits, and not above every number.
// Every block sees the whole row and decides alike; a row that does not fit is multiplied as floats.
__device__ __forceinline__ bool g1_digits_fit(const float4 &a, const float4 &b, uint32_t mx) {
    if (mx == 0u) return true;
    if (mx < (127u - 60u) << 23 || mx >= 0x7f800000u) return false;
    const uint32_t least = mx - (6u << 23);
    const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t n = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) n += act_mag(f[i]) >= least ? 1u : 0u;
    return __reduce_add_sync(0xffffffffu, n) >= 32u;
}
// Rows from which a matrix is taken here; below, every block's digits of x cost what they save. us a decode step of 8 layers by rows of its LM head, floats -> digits: 4096
// 496.2 -> 497.0, 8192 505.5 -> 505.1, 16384 514 -> 510, 32768 525 -> 520, 65536 547 -> 545, 151936 611 -> 597 (the kernel alone, with some 5 us of events: 76.3 -> 66.7)
constexpr uint32_t G1_DIGIT_ROWS = 16384u;
__device__ __forceinline__ int g1_dp4a(uint32_t q, uint32_t x, int c) { int d; asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(q), "r"(x), "r"(c)); return d; }

template <bool NORM>
__global__ void __launch_bounds__(G1_WARPS * 32u, 3) k_gemv1_digits(const __grid_constant__ GemvArgs A) {
    pdl_trigger();
    extern __shared__ __align__(16) double g1_part[];      // as in k_gemv1: results of a row that is multiplied as floats; behind them x, its digit words, and -32 times the digit sums of every 16 columns
    float *g1_xs = reinterpret_cast<float *>(g1_part + A.part_doubles);
    __shared__ float s_scale[G1_NCOLS / 256u];
    const GemvJob &J = A.job[0];
    const uint32_t row0 = blockIdx.x * J.rows_per_tile, nrow = min(J.rows_per_tile, J.nrows - row0);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, cpr = J.ncols >> 6, bpr = J.ncols >> 8;
    const uint32_t lpr = g1_lanes(RC_Q6_K, J.ncols), rw = 32u / lpr, slot = lane / lpr, sub = lane % lpr, step = G1_WARPS * rw, first = warp * rw;
    const uint64_t o_h = rc_q6_qh(J.nb), o_s = rc_q6_sc(J.nb), o_d = rc_q6_d(J.nb);
    const bool on = sub < cpr;                              // lanes past the row's end repeat its last chunk and add nothing
    const uint32_t cc = on ? sub : cpr - 1u, bcol = cc >> 2, half = (cc >> 1) & 1u, l0 = (cc & 1u) * 16u;
    float *g1_xd = g1_xs + g1_xi(J.ncols);
    int4 *corr = reinterpret_cast<int4 *>(g1_xd + g1_xi(J.ncols));
    auto load = [&](uint32_t vr) {
        vr = min(vr, nrow - 1u);
        const uint64_t blk = (uint64_t)(row0 + vr) * bpr + bcol;
        const uint8_t *wl = J.w0 + blk * 128u + half * 64u + l0;
        Q6Frag f;
        f.a = __ldg(reinterpret_cast<const uint4 *>(wl));
        f.b = __ldg(reinterpret_cast<const uint4 *>(wl + 32u));
        f.h = __ldg(reinterpret_cast<const uint4 *>(J.w0 + o_h + blk * 64u + half * 32u + l0));
        f.sc = __ldg(reinterpret_cast<const uint2 *>(J.w0 + o_s + blk * 16u + half * 8u));
        f.d = __ldg(reinterpret_cast<const unsigned short *>(J.w0 + o_d) + blk);
        return f;
    };
    Q6Frag f[2];
    if (A.resident) { f[0] = load(first + slot); f[1] = load(first + step + slot); }
    pdl_wait();
    gemv1_stage<NORM>(A, J.ncols, g1_xs);
    if (!A.resident) { f[0] = load(first + slot); f[1] = load(first + step + slot); }
    __syncthreads();
    static_assert(G1_NCOLS / 256u <= G1_WARPS, "a warp per 256 columns, eight neighbouring values a lane");
    bool fit = true;
    if (warp < bpr) {
        const uint32_t at = g1_xi(warp * 256u + lane * 8u);
        const float4 *p = reinterpret_cast<const float4 *>(g1_xs + at);
        const float4 v0 = p[0], v1 = p[1];
        const uint32_t mx = __reduce_max_sync(0xffffffffu, max(act_mag4(v0), act_mag4(v1)));
        fit = g1_digits_fit(v0, v1, mx);
        float up;
        const float scale = actw_scale(mx, up);
        if (lane == 0) s_scale[warp] = scale;
        const uint32_t w0[4] = {actw_digits(v0.x, up), actw_digits(v0.y, up), actw_digits(v0.z, up), actw_digits(v0.w, up)};
        const uint32_t w1[4] = {actw_digits(v1.x, up), actw_digits(v1.y, up), actw_digits(v1.z, up), actw_digits(v1.w, up)};
        uint32_t p0[4], p1[4];
        actw_planes(w0, p0); actw_planes(w1, p1);
        uint4 *o = reinterpret_cast<uint4 *>(g1_xd + at);
        o[0] = make_uint4(p0[0], p0[1], p0[2], p0[3]); o[1] = make_uint4(p1[0], p1[1], p1[2], p1[3]);
        int c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            c[i] = __dp4a((int)p0[i], 0x01010101, __dp4a((int)p1[i], 0x01010101, 0));
            c[i] = -32 * (c[i] + __shfl_xor_sync(0xffffffffu, c[i], 1));
        }
        if (!(lane & 1u)) corr[warp * 16u + (lane >> 1)] = make_int4(c[0], c[1], c[2], c[3]);
    }
    if (!__syncthreads_and(fit)) {
        gemv1_q6k<false, true>(A, J, G1Tile{row0, nrow, 0u, true}, g1_part, g1_xs);
        __syncthreads();
        for (uint32_t r = threadIdx.x; r < nrow; r += G1_WARPS * 32u) J.out[row0 + r] = (float)g1_part[r];
        return;
    }
    const uint4 *xl = reinterpret_cast<const uint4 *>(g1_xd + bcol * 268u + half * 136u + l0);
    const int4 *cl = corr + (bcol * 256u + half * 128u + l0) / 16u;
    const float xscale = s_scale[bcol];
    for (uint32_t base = first; base < nrow; base += 2u * step) {
        float acc[2] = {0.f, 0.f};
        const uint32_t sq = l0 ? 8u : 0u;                   // the four scales of this lane's runs of 16 sit in every other byte of its half block
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            const int4 c0 = cl[2 * qd];
            int s[2][4] = {{c0.x, c0.y, c0.z, c0.w}, {c0.x, c0.y, c0.z, c0.w}};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const uint4 xd = xl[8 * qd + w];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t a = w == 0 ? f[r].a.x : w == 1 ? f[r].a.y : w == 2 ? f[r].a.z : f[r].a.w, b = w == 0 ? f[r].b.x : w == 1 ? f[r].b.y : w == 2 ? f[r].b.z : f[r].b.w;
                    const uint32_t h = w == 0 ? f[r].h.x : w == 1 ? f[r].h.y : w == 2 ? f[r].h.z : f[r].h.w;
                    const uint32_t v = qd == 0 ? (a & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u) : qd == 1 ? (b & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u)
                                     : qd == 2 ? ((a >> 4) & 0x0F0F0F0Fu) | (h & 0x30303030u) : ((b >> 4) & 0x0F0F0F0Fu) | ((h >> 2) & 0x30303030u);
                    s[r][0] = g1_dp4a(v, xd.x, s[r][0]); s[r][1] = g1_dp4a(v, xd.y, s[r][1]); s[r][2] = g1_dp4a(v, xd.z, s[r][2]); s[r][3] = g1_dp4a(v, xd.w, s[r][3]);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {                   // |digit sum| < 2^18: the upper and the lower two are exact as integers, the lower as a float too
                const uint32_t word = qd < 2 ? f[r].sc.x : f[r].sc.y;
                const float sc = (float)(int)(signed char)(word >> (sq + 16u * (qd & 1)));
                acc[r] = fmaf(sc, fmaf(65536.0f, (float)(256 * s[r][3] + s[r][2]), (float)(256 * s[r][1] + s[r][0])), acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) acc[r] = on ? acc[r] * (__half2float(__ushort_as_half(f[r].d)) * xscale) : 0.f;
        if (base + 2u * step < nrow) { f[0] = load(base + 2u * step + slot); f[1] = load(base + 3u * step + slot); }      // on the way during the reduction
        for (uint32_t o = lpr >> 1; o; o >>= 1) { acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o); acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], o); }
        if (sub == 0u) {
            if (base + slot < nrow) J.out[row0 + base + slot] = acc[0];
            if (base + step + slot < nrow) J.out[row0 + base + step + slot] = acc[1];
        }
    }
}
static bool gemv1_digits_ok(const GemvArgs &A) {
    const GemvJob &J = A.job[0];
    return A.njobs == 1u && J.type == RC_Q6_K && J.epi == GEMV_STORE && J.ncols <= G1_NCOLS && J.nrows >= G1_DIGIT_ROWS && !A.tail.ticket;
}

// One token and rows that k_gemv1 holds; the other block types stay with the general kernel.
bool gemv1_ok(const GemvArgs &A) {
    if (A.ntok != 1u || ((uintptr_t)A.x & 15u)) return false;
    for (uint32_t j = 0; j < A.njobs; ++j) {
        const uint32_t t = A.job[j].type;
        if (t != RC_F32 && t != RC_F16 && t != RC_Q6_K) return false;
        if (A.job[j].ncols > 8192u) return false;          // x in shared memory without the opt-in size
    }
    return true;
}

bool gemv1_norm_ok(const GemvArgs &A) {
    for (uint32_t j = 0; j < A.njobs; ++j) if (A.job[j].ncols != A.job[0].ncols || A.job[j].ncols % 4u) return false;
    auto al = [](const void *p) { return ((uintptr_t)p & 15u) == 0u; };
    // one block writes normed and resid while the others still read x, branch and w
    const uintptr_t bytes = (uintptr_t)A.job[0].ncols * sizeof(float);
    auto apart = [&](const float *p, const float *q) { return !p || !q || (uintptr_t)p + bytes <= (uintptr_t)q || (uintptr_t)q + bytes <= (uintptr_t)p; };
    for (const float *o : {A.norm.normed, A.norm.resid})
        if (!apart(o, A.x) || !apart(o, A.norm.branch) || !apart(o, A.norm.w)) return false;
    if (!apart(A.norm.normed, A.norm.resid)) return false;
    return gemv1_ok(A) && A.job[0].ncols <= G1_NCOLS && A.norm.normed && al(A.norm.w) && al(A.norm.branch) && al(A.norm.resid) && al(A.norm.normed);
}

int launch_gemv1(GemvArgs &A, cudaStream_t stream) {
    RC_REQUIRE(!A.norm.w || gemv1_norm_ok(A), "gemv: this input cannot be normalised on the way");
    // Tiles of about equal bytes, three per SM (what the registers let reside), so that a launch is one wave whatever its jobs;
    // at least one row per warp of the block, at most what 8 KB of partial sums hold.
    uint64_t total = 0;
    for (uint32_t j = 0; j < A.njobs; ++j) total += rc_matrix_bytes(A.job[j].type, A.job[j].nrows, A.job[j].ncols) << (A.job[j].epi == GEMV_PAIR_SILU ? 1 : 0);
    const uint64_t target = (total + 443u) / 444u;
    uint32_t tiles = 0;
    size_t smem = 16u;
    bool q6 = false;
    for (uint32_t j = 0; j < A.njobs; ++j) {
        GemvJob &J = A.job[j];
        const uint32_t pair = J.epi == GEMV_PAIR_SILU ? 1u : 0u, S = g1_slices(J.type, J.ncols);
        const uint32_t pass = G1_WARPS / g1_slice_warps(S) * (32u / g1_lanes(J.type, J.ncols)), grain = pass >> pair ? pass >> pair : 1u;
        const uint64_t row = rc_row_bytes(J.type, J.ncols) << pair;
        uint64_t rows = ((target + row - 1u) / row + grain - 1u) / grain * grain;
        const uint32_t cap = 1024u / (S << pair);
        if (rows > cap) rows = cap;
        J.rows_per_tile = (uint32_t)rows;
        J.tile_begin = tiles;
        tiles += (J.nrows + J.rows_per_tile - 1u) / J.rows_per_tile;
        const size_t need = (size_t)(J.rows_per_tile < J.nrows ? J.rows_per_tile : J.nrows) * (S << pair) * sizeof(double);
        if (need > smem) smem = (need + 15u) / 16u * 16u;
        q6 = q6 || J.type == RC_Q6_K;
    }
    A.part_doubles = (uint32_t)(smem / sizeof(double));
    if (q6 || A.norm.w) smem += (size_t)g1_xi(A.job[0].ncols) * sizeof(float) + 16u;
    prof_begin(A.tag ? A.tag : "gemv", stream);
    if (gemv1_digits_ok(A)) {
        smem += (size_t)g1_xi(A.job[0].ncols) * sizeof(float) + (size_t)(A.job[0].ncols / 16u) * sizeof(int4);
        if (A.norm.w) RC_LAUNCH_BEHIND_IF(!A.resident, (k_gemv1_digits<true>), tiles, G1_WARPS * 32u, smem, stream, A);
        else RC_LAUNCH_BEHIND_IF(!A.resident, (k_gemv1_digits<false>), tiles, G1_WARPS * 32u, smem, stream, A);
        prof_end(stream);
        RC_LAUNCHED();
        return 1;
    }
    // weights that a kernel before this one has just laid out are read by the non-coherent path like others: then behind that kernel's end
    if (A.norm.w) RC_LAUNCH_BEHIND_IF(!A.resident, (k_gemv1<true>), tiles, G1_WARPS * 32u, smem, stream, A);
    else RC_LAUNCH_BEHIND_IF(!A.resident, (k_gemv1<false>), tiles, G1_WARPS * 32u, smem, stream, A);
    prof_end(stream);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc
