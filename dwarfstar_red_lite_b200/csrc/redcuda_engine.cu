// rl_engine_* on CUDA: the persistent Qwen3-Next decode engine (every weight and every routed expert resident in HBM).
//
// One token (rl_engine_cpu_step, native/redlite_native_engine_cpu.c:390-441, is the arithmetic being reproduced):
//   embedding row -> 48 x { RMSNorm -> Gated DeltaNet or gated GQA attention -> residual + RMSNorm -> MoE FFN + residual }
//   -> final RMSNorm -> LM head.
// Everything runs on one stream without a host round trip; the host mirrors the reference keeps for parity checks
// (embedding, per-layer outputs, final norm, router ids, native/redlite_native_engine_internal.h:35-47) are copied back
// at the end of the step together with the logits.
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_kquants.cuh"
#include "redcuda_moe_mma.cuh"
#include "redcuda_tc_gemm.cuh"
#include "redcuda_gguf.h"
#include "../../include/redcuda.h"
#include "../../include/rl_engine.h"

#include <math.h>
#include <stdlib.h>
#include <algorithm>
#include <chrono>
#include <new>
#include <vector>

namespace rc {

const uint32_t *moe_last_ids_device(const redcuda_moe *m);   // redcuda_moe.cu
int moe_forward_norm1(redcuda_moe *m, const float *x, const GemvNorm &N, const float *resid, float *out, cudaStream_t s);      // see redcuda_moe.cu
void moe_set_ids_mirror(redcuda_moe *m, uint32_t *dev_ptr);   // a single token's router ids are also written to dev_ptr
size_t moe_workspace_bytes(const redcuda_moe_desc *d);
// expert parallelism: which contiguous share of every layer's experts the engines opened next will hold
static thread_local int g_shard_rank = 0, g_shard_world = 1;
redcuda_moe *moe_create_shared(const redcuda_moe_desc *d, void *workspace);   // workspace shared by layers that run on one stream

static double now_ms() { return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count(); }

// ---- small kernels ----
// out[b] = dequantised embedding row of token[b] (grid = tokens, block = 256 threads)
__global__ void k_embed_row(const uint8_t *__restrict__ base, uint32_t type, uint64_t nb, uint32_t ncols, uint32_t nrows, const uint32_t *token,
                            const uint8_t *iq2, const uint32_t *iq3s, float *__restrict__ out, uint32_t *__restrict__ status) {
    pdl_prologue();
    uint64_t row = token[blockIdx.x];
    if (row >= nrows) { row = 0; if (status && threadIdx.x == 0) status[ST_TOKEN_RANGE] = 1u; }   // never index the table with an id the argmax could not form
    out += (size_t)blockIdx.x * ncols;
    if (type == RC_F32) { for (uint32_t i = threadIdx.x; i < ncols; i += blockDim.x) out[i] = reinterpret_cast<const float *>(base)[row * ncols + i]; return; }
    if (type == RC_F16) { for (uint32_t i = threadIdx.x; i < ncols; i += blockDim.x) out[i] = __half2float(__ushort_as_half(reinterpret_cast<const unsigned short *>(base)[row * ncols + i])); return; }
    if (rc_is_file_layout_quant(type)) {
        const uint8_t *rp = base + row * rc_row_bytes(type, ncols);
        for (uint32_t i = threadIdx.x; i < ncols; i += blockDim.x) out[i] = kq_row_value(type, rp, i);
        return;
    }
    const RcBooks bk{iq2, iq3s};
    const uint32_t bpr = ncols >> 8;
    for (uint32_t g = threadIdx.x; g < bpr * 32u; g += blockDim.x) {
        float v[8];
        rc_decode8(type, base, nb, row * bpr + (g >> 5), g & 31u, bk, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) out[g * 8u + j] = v[j];
    }
}

__device__ __forceinline__ double block_sum_d(double v, double *red) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (uint32_t w = 0; w < (blockDim.x + 31u) / 32u; ++w) t += red[w];
    __syncthreads();
    return t;
}

// normed = RMSNorm(x [+ branch]) * w (engine_cpu.c:96-101, 418-424); resid_out (optional) = x + branch. One block of THREADS per token: 1024 where the token is
// alone, its row is the chain; 256 for the rows of a chunk whose length k_rmsnorm_rows is not built for (it is for the lengths of the engine's models, 1024 and 2048).
template <uint32_t THREADS>
__global__ void __launch_bounds__(THREADS) k_rmsnorm(const float *x, const float *branch, const float *__restrict__ w,
                                                  uint32_t n, float eps, float *__restrict__ resid_out, float *__restrict__ normed) {
    pdl_prologue();
    __shared__ double red[32];
    const size_t tok_off = (size_t)blockIdx.x * n;
    x += tok_off; normed += tok_off;
    if (branch) branch += tok_off;
    if (resid_out) resid_out += tok_off;
    // a row of up to 4096 values stays in registers between the sum and the scaling, and the weights are on their way with it
    constexpr uint32_t KEEP = 4096u / THREADS;
    float keep[KEEP], wk[KEEP];
    double ss = 0.0;
#pragma unroll
    for (uint32_t j = 0; j < KEEP; ++j) {
        const uint32_t i = threadIdx.x + j * THREADS;
        if (i < n) { keep[j] = x[i]; if (branch) keep[j] = keep[j] + branch[i]; wk[j] = w[i]; }
    }
#pragma unroll
    for (uint32_t j = 0; j < KEEP; ++j) {
        const uint32_t i = threadIdx.x + j * THREADS;
        if (i < n) { if (resid_out) resid_out[i] = keep[j]; ss += (double)keep[j] * (double)keep[j]; }
    }
    for (uint32_t i = threadIdx.x + KEEP * THREADS; i < n; i += THREADS) {
        float v = x[i];
        if (branch) v = v + branch[i];
        if (resid_out) resid_out[i] = v;
        ss += (double)v * (double)v;
    }
    const double tot = block_sum_d(ss, red);
    const double inv = 1.0 / sqrt(tot / (double)n + (double)eps);
#pragma unroll
    for (uint32_t j = 0; j < KEEP; ++j) {
        const uint32_t i = threadIdx.x + j * THREADS;
        if (i < n) normed[i] = (float)((double)keep[j] * inv * (double)wk[j]);
    }
    for (uint32_t i = threadIdx.x + KEEP * THREADS; i < n; i += THREADS) {
        float v = x[i];
        if (branch) v = v + branch[i];
        normed[i] = (float)((double)v * inv * (double)w[i]);
    }
}

// The same for the rows of a chunk, a warp each: its loads go out together and no barrier is met. grid = tokens / 4, rows of NV * 128 values, 16-byte aligned.
// 2048 rows of 2048 values, with and without a branch: 11 and 7 us, a block of 256 threads per row 30 and 21
template <uint32_t NV>
__global__ void __launch_bounds__(128) k_rmsnorm_rows(const float *x, const float *branch, const float *w, uint32_t rows, float eps,
                                                      float *__restrict__ resid_out, float *__restrict__ normed) {
    pdl_prologue();
    const uint32_t r = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (r >= rows) return;
    const size_t off = (size_t)r * (NV * 128u) + lane * 4u;
    float4 v[NV];
#pragma unroll
    for (uint32_t i = 0; i < NV; ++i) v[i] = *reinterpret_cast<const float4 *>(x + off + i * 128u);
    if (branch)
#pragma unroll
        for (uint32_t i = 0; i < NV; ++i) {
            const float4 b = *reinterpret_cast<const float4 *>(branch + off + i * 128u);
            v[i].x += b.x; v[i].y += b.y; v[i].z += b.z; v[i].w += b.w;
        }
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < NV; ++i) {
        if (resid_out) *reinterpret_cast<float4 *>(resid_out + off + i * 128u) = v[i];
        s0 = fma((double)v[i].x, (double)v[i].x, s0); s1 = fma((double)v[i].y, (double)v[i].y, s1);
        s0 = fma((double)v[i].z, (double)v[i].z, s0); s1 = fma((double)v[i].w, (double)v[i].w, s1);
    }
    double ss = s0 + s1;
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const double inv = 1.0 / sqrt(ss / (double)(NV * 128u) + (double)eps);
#pragma unroll
    for (uint32_t i = 0; i < NV; ++i) {
        const float4 k = __ldg(reinterpret_cast<const float4 *>(w + lane * 4u + i * 128u));
        *reinterpret_cast<float4 *>(normed + off + i * 128u) = make_float4((float)((double)v[i].x * inv * (double)k.x), (float)((double)v[i].y * inv * (double)k.y),
                                                                             (float)((double)v[i].z * inv * (double)k.z), (float)((double)v[i].w * inv * (double)k.w));
    }
}

template <typename KV> __device__ __forceinline__ KV to_kv(float v);
template <> __device__ __forceinline__ float to_kv<float>(float v) { return v; }
template <> __device__ __forceinline__ __half to_kv<__half>(float v) { return __float2half_rn(v); }
__device__ __forceinline__ float from_kv(float v) { return v; }
__device__ __forceinline__ float from_kv(__half v) { return __half2float(v); }

// Per-head RMSNorm of q and k, NeoX RoPE on the first rope_dims, K/V rows appended to the cache (engine_cpu.c:277-296).
// grid = (n_head + 2 * n_kv, tokens) blocks of head_dim threads; token z sits at position pos_p[z].
template <typename KV>
__global__ void k_attn_prep(const float *qg, const float *kraw, const float *vraw,
                            const float *__restrict__ qn, const float *__restrict__ kn, uint32_t n_head, uint32_t n_kv, uint32_t hd,
                            uint32_t rope_dims, float freq_base, float eps, const uint32_t *pos_p, float *__restrict__ query, float *__restrict__ gate,
                            KV *__restrict__ kcache, KV *__restrict__ vcache) {
    pdl_prologue();
    extern __shared__ float sh[];
    __shared__ double red[32];
    const uint32_t b = blockIdx.x, tid = threadIdx.x, z = blockIdx.y, pos = pos_p[z];   // the position lives in device memory: a captured graph replays for every token
    qg += (size_t)z * n_head * 2u * hd; kraw += (size_t)z * n_kv * hd; vraw += (size_t)z * n_kv * hd;
    query += (size_t)z * n_head * hd; gate += (size_t)z * n_head * hd;
    if (b >= n_head + n_kv) {      // value head: plain append
        const uint32_t kh = b - n_head - n_kv;
        vcache[((size_t)pos * n_kv + kh) * hd + tid] = to_kv<KV>(vraw[(size_t)kh * hd + tid]);
        return;
    }
    const bool is_q = b < n_head;
    const uint32_t h = is_q ? b : b - n_head;
    const float src = is_q ? qg[(size_t)h * 2u * hd + tid] : kraw[(size_t)h * hd + tid];
    if (is_q) gate[(size_t)h * hd + tid] = qg[(size_t)h * 2u * hd + hd + tid];
    const double tot = block_sum_d((double)src * (double)src, red);
    const double inv = 1.0 / sqrt(tot / (double)hd + (double)eps);
    const float val = (float)((double)src * inv * (double)(is_q ? qn[tid] : kn[tid]));
    sh[tid] = val;
    __syncthreads();
    float outv = val;
    if (tid < rope_dims) {
        const uint32_t half = rope_dims >> 1, i = tid < half ? tid : tid - half;
        const float fr = (float)pow((double)freq_base, (double)(-2.0f * (float)i / (float)rope_dims));
        const float theta = __fmul_rn((float)pos, fr);
        const float c = (float)cos((double)theta), s = (float)sin((double)theta);
        const float x0 = sh[i], x1 = sh[half + i];
        outv = tid < half ? __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)) : __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
    }
    if (is_q) query[(size_t)h * hd + tid] = outv;
    else kcache[((size_t)pos * n_kv + h) * hd + tid] = to_kv<KV>(outv);
}

// The same for the tokens of a chunk (a block each, heads over its warps): the angles are computed once per token instead of by every head, which
// made the double-precision pow, cos and sin most of the kernel (2048 tokens x 20 heads of 256: 84 us, now 53). hd = 32 VPL, rope_dims <= hd
template <typename KV, uint32_t VPL>
__global__ void __launch_bounds__(256) k_attn_prep_rows(const float *qg, const float *kraw, const float *vraw, const float *qn, const float *kn,
                                                        uint32_t n_head, uint32_t n_kv, uint32_t rope_dims, float freq_base, float eps, const uint32_t *pos_p,
                                                        float *__restrict__ query, float *__restrict__ gate, KV *__restrict__ kcache, KV *__restrict__ vcache) {
    pdl_prologue();
    constexpr uint32_t hd = VPL * 32u;
    __shared__ float s_cos[hd / 2u], s_sin[hd / 2u], s_row[8][hd];
    const uint32_t z = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, pos = pos_p[z], half = rope_dims >> 1;
    qg += (size_t)z * n_head * 2u * hd; kraw += (size_t)z * n_kv * hd; vraw += (size_t)z * n_kv * hd;
    query += (size_t)z * n_head * hd; gate += (size_t)z * n_head * hd;
    if (tid < half) {
        const float fr = (float)pow((double)freq_base, (double)(-2.0f * (float)tid / (float)rope_dims));
        const float theta = __fmul_rn((float)pos, fr);
        s_cos[tid] = (float)cos((double)theta); s_sin[tid] = (float)sin((double)theta);
    }
    __syncthreads();
    for (uint32_t b = warp; b < n_head + 2u * n_kv; b += 8u) {
        if (b >= n_head + n_kv) {      // value head: plain append
            const uint32_t h = b - n_head - n_kv;
#pragma unroll
            for (uint32_t i = 0; i < VPL; ++i) vcache[((size_t)pos * n_kv + h) * hd + lane + 32u * i] = to_kv<KV>(vraw[(size_t)h * hd + lane + 32u * i]);
            continue;
        }
        const bool is_q = b < n_head;
        const uint32_t h = is_q ? b : b - n_head;
        const float *src = is_q ? qg + (size_t)h * 2u * hd : kraw + (size_t)h * hd, *nw = is_q ? qn : kn;
        float v[VPL];
        double ss = 0.0;
#pragma unroll
        for (uint32_t i = 0; i < VPL; ++i) {
            v[i] = src[lane + 32u * i];
            if (is_q) gate[(size_t)h * hd + lane + 32u * i] = src[hd + lane + 32u * i];
        }
#pragma unroll
        for (uint32_t i = 0; i < VPL; ++i) ss = fma((double)v[i], (double)v[i], ss);
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const double inv = 1.0 / sqrt(ss / (double)hd + (double)eps);
        __syncwarp();                  // the row of the head before has been read
#pragma unroll
        for (uint32_t i = 0; i < VPL; ++i) { v[i] = (float)((double)v[i] * inv * (double)__ldg(nw + lane + 32u * i)); s_row[warp][lane + 32u * i] = v[i]; }
        __syncwarp();
#pragma unroll
        for (uint32_t i = 0; i < VPL; ++i) {
            const uint32_t d = lane + 32u * i;
            if (d < rope_dims) {
                const uint32_t j = d < half ? d : d - half;
                const float c = s_cos[j], sn = s_sin[j], x0 = s_row[warp][j], x1 = s_row[warp][half + j];
                v[i] = d < half ? __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, sn)) : __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, c));
            }
            if (is_q) query[(size_t)h * hd + d] = v[i];
            else kcache[((size_t)pos * n_kv + h) * hd + d] = to_kv<KV>(v[i]);
        }
    }
}

// VPL consecutive cache values of a lane, requested as one to two vector loads (their address is a multiple of their size)
template <typename KV, int VPL>
struct KvRaw {
    static constexpr int BYTES = VPL * (int)sizeof(KV);
    uint32_t w[BYTES / 4];
    __device__ __forceinline__ void load(const KV *p) {
        if constexpr (BYTES % 16 == 0) {
#pragma unroll
            for (int i = 0; i < BYTES / 16; ++i) { const uint4 v = reinterpret_cast<const uint4 *>(p)[i]; w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w; }
        } else if constexpr (BYTES == 8) { const uint2 v = *reinterpret_cast<const uint2 *>(p); w[0] = v.x; w[1] = v.y; }
        else w[0] = *reinterpret_cast<const uint32_t *>(p);
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < BYTES / 4; ++i) w[i] = 0u;
    }
    __device__ __forceinline__ void floats(float (&f)[VPL]) const {
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            if constexpr (sizeof(KV) == 4) f[i] = __uint_as_float(w[i]);
            else f[i] = __half2float(__ushort_as_half((unsigned short)(w[i / 2] >> (16 * (i & 1)))));
        }
    }
};

// Split-K decode attention. grid = (n_kv, nsplit, tokens), block = 256 (8 warps); token z attends to positions <= pos_p[z] (the K/V rows of a whole prefill
// chunk are appended before this runs, so the mask is the sequence length alone). Every block serves the G query heads of one K/V head over a slice of
// positions (K and V rows are read once for all G heads); a warp takes every eighth group of ATTN_POS positions, a lane VPL = head_dim/32 consecutive
// dimensions; online softmax per head. Partials: m, l and the accumulator.
// The instructions of a warp bound it (two groups at 3500 positions): the G x 4 dot products of a group are summed over the lanes together, each exchange
// halving the values that a lane still carries, so that a lane ends with one score of one head, and takes the exponentials of that one only; position by
// position every lane reduced and exponentiated all G. The rows of the next group are requested before the current one is worked on. 3500 positions, 8 heads of 256
// each on 2 K/V heads: 15.8 -> 13.2 us with the events that time it (some 5 of them); a decode step 618 -> 616.
constexpr uint32_t ATTN_POS = 4u;
template <typename KV, int VPL, int G>
__global__ void __launch_bounds__(256, 1) k_attn_decode(const float *query, const KV *kcache, const KV *vcache,
                                                        uint32_t n_kv, const uint32_t *pos_p, uint32_t nsplit, float scale,
                                                        float *__restrict__ part_m, float *__restrict__ part_l, float *__restrict__ part_acc) {
    pdl_prologue();
    extern __shared__ float sm[];            // [8][G][hd] accumulators, then [8][G] each of m, l and the warps' weights
    constexpr uint32_t hd = VPL * 32u, P = ATTN_POS, NV = P * G, R = 32u / NV;      // NV scores of a group, R lanes that end with the same one
    static_assert(NV <= 32u && (NV & (NV - 1u)) == 0u, "scores of a group");
    const uint32_t kvh = blockIdx.x, split = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t n_head = n_kv * G;
    const uint32_t seq_len = pos_p[blockIdx.z] + 1u;
    query += (size_t)blockIdx.z * n_head * hd;
    part_m += (size_t)blockIdx.z * n_head * nsplit; part_l += (size_t)blockIdx.z * n_head * nsplit; part_acc += (size_t)blockIdx.z * n_head * nsplit * hd;
    // slices of at least 32 positions; at short sequences the trailing blocks find an empty slice and report m = -inf
    const uint32_t per = max((seq_len + nsplit - 1u) / nsplit, 32u), p_begin = min(split * per, seq_len), p_end = min(seq_len, p_begin + per);
    const size_t lane_off = (size_t)kvh * hd + lane * VPL, row = (size_t)n_kv * hd;
    KvRaw<KV, VPL> kr[P], vr[P];
    auto fetch = [&](KvRaw<KV, VPL> &to, const KV *cache, uint32_t p) {
        if (p < p_end) to.load(cache + p * row + lane_off); else to.zero();
    };
    uint32_t p0 = p_begin + warp * P;
    if (p0 < p_end)
#pragma unroll
        for (uint32_t j = 0; j < P; ++j) { fetch(kr[j], kcache, p0 + j); fetch(vr[j], vcache, p0 + j); }
    float q[G][VPL], acc[G][VPL], m = -INFINITY, l = 0.f;          // m, l: of the score that this lane ends with, head lane / (P R), position lane / R % P
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < VPL; ++i) { q[g][i] = query[((size_t)kvh * G + g) * hd + lane * VPL + i] * scale; acc[g][i] = 0.f; }
    for (; p0 < p_end; p0 += 8u * P) {
        float v[NV];
#pragma unroll
        for (uint32_t j = 0; j < P; ++j) {
            float kx[VPL];
            kr[j].floats(kx);
            if (p0 + 8u * P < p_end) fetch(kr[j], kcache, p0 + 8u * P + j);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float d = 0.f;
#pragma unroll
                for (int i = 0; i < VPL; ++i) d += q[g][i] * kx[i];
                v[g * P + j] = d;
            }
        }
#pragma unroll
        for (uint32_t o = 16u; o >= R; o >>= 1) {
            const uint32_t half = o / R;                            // values that stay with a lane
            const bool hi = lane & o;
#pragma unroll
            for (uint32_t i = 0; i < half; ++i) {
                const float keep = hi ? v[half + i] : v[i], send = hi ? v[i] : v[half + i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, (int)o);
            }
        }
#pragma unroll
        for (uint32_t o = R / 2u; o; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], (int)o);
        const float s = p0 + lane / R % P < p_end ? v[0] : -INFINITY;
        float mn = fmaxf(m, s);
#pragma unroll
        for (uint32_t o = R; o < P * R; o <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, (int)o));
        const float c = expf(m - mn), pe = expf(s - mn);
        l = l * c + pe;
        m = mn;
        if (!__all_sync(0xffffffffu, c == 1.f)) {                   // no head's maximum rose: nothing to rescale
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float cg = __shfl_sync(0xffffffffu, c, (int)(g * P * R));
#pragma unroll
                for (int i = 0; i < VPL; ++i) acc[g][i] *= cg;
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < P; ++j) {
            float vx[VPL];
            vr[j].floats(vx);
            if (p0 + 8u * P < p_end) fetch(vr[j], vcache, p0 + 8u * P + j);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float w = __shfl_sync(0xffffffffu, pe, (int)((g * P + j) * R));
#pragma unroll
                for (int i = 0; i < VPL; ++i) acc[g][i] += w * vx[i];
            }
        }
    }
#pragma unroll
    for (uint32_t o = R; o < P * R; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, (int)o);
    float *s_acc = sm, *s_m = sm + 8u * G * hd, *s_l = s_m + 8u * G, *s_e = s_l + 8u * G;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        float *to = s_acc + ((size_t)warp * G + g) * hd + lane * VPL;
        if constexpr (VPL % 4 == 0) {
#pragma unroll
            for (int i = 0; i < VPL; i += 4) *reinterpret_cast<float4 *>(to + i) = make_float4(acc[g][i], acc[g][i + 1], acc[g][i + 2], acc[g][i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < VPL; ++i) to[i] = acc[g][i];
        }
    }
    if (lane % (P * R) == 0u) { s_m[warp * G + lane / (P * R)] = m; s_l[warp * G + lane / (P * R)] = l; }
    __syncthreads();
    if (tid < 8u * G) {                                             // thread (w, g): warp w's weight for head g
        const uint32_t g = tid % G;
        float M = -INFINITY, L = 0.f;
        for (uint32_t w = 0; w < 8u; ++w) M = fmaxf(M, s_m[w * G + g]);
        s_e[tid] = M > -INFINITY ? expf(s_m[tid] - M) : 0.f;
        if (tid < (uint32_t)G) {
            if (M > -INFINITY) for (uint32_t w = 0; w < 8u; ++w) L += s_l[w * G + g] * expf(s_m[w * G + g] - M);
            const size_t head = (size_t)kvh * G + g;
            part_m[head * nsplit + split] = M; part_l[head * nsplit + split] = L;
        }
    }
    __syncthreads();
    for (uint32_t idx = tid; idx < G * hd; idx += 256u) {
        const uint32_t g = idx / hd, d = idx - g * hd;
        float A = 0.f;
#pragma unroll
        for (uint32_t w = 0; w < 8u; ++w) A += s_acc[((size_t)w * G + g) * hd + d] * s_e[w * G + g];
        part_acc[(((size_t)kvh * G + g) * nsplit + split) * hd + d] = A;
    }
}

// merge the split partials, normalise, apply the sigmoid output gate (engine_cpu.c:312-317). grid = (n_head, tokens), block = hd
__global__ void k_attn_merge(const float *part_m, const float *part_l, const float *part_acc,
                             const float *gate, uint32_t nsplit, uint32_t hd, float *__restrict__ gated) {
    pdl_prologue();
    const uint32_t h = blockIdx.x, d = threadIdx.x;
    const size_t zoff = (size_t)blockIdx.y * gridDim.x;
    part_m += zoff * nsplit; part_l += zoff * nsplit; part_acc += zoff * nsplit * hd; gate += zoff * hd; gated += zoff * hd;
    // every warp finds the maximum and the normaliser from all slices at once (a slice per lane), the slices' weights go to
    // shared memory, and a thread's values are then independent loads: with 64 slices the serial form took 22 us, all of it
    // the chain of load, exponential and add per slice
    extern __shared__ float s_e[];            // [nsplit], 0 = empty slice
    const uint32_t lane = d & 31u;
    const float *pm = part_m + (size_t)h * nsplit, *pl = part_l + (size_t)h * nsplit, *pa = part_acc + (size_t)h * nsplit * hd + d;
    float M = -INFINITY, L = 0.f, A = 0.f;
    for (uint32_t s = lane; s < nsplit; s += 32u) M = fmaxf(M, pm[s]);
    for (int o = 16; o; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    for (uint32_t s = lane; s < nsplit; s += 32u) {
        const float m = pm[s], e = m == -INFINITY ? 0.f : expf(m - M);
        if (m != -INFINITY) L += pl[s] * e;   // an empty slice wrote its maximum only
        if (d < 32u) s_e[s] = e;
    }
    for (int o = 16; o; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    __syncthreads();
#pragma unroll 8
    for (uint32_t s = 0; s < nsplit; ++s) {   // no branch around the load (it would be waited for slice by slice): an empty slice's row is read and not used
        const float e = s_e[s], v = pa[(size_t)s * hd];
        A += e != 0.f ? v * e : 0.f;
    }
    const double o = (double)A / (double)L;
    gated[(size_t)h * hd + d] = (float)(o / (1.0 + exp(-(double)gate[(size_t)h * hd + d])));
}

// argmax of n floats, ties to the lowest index; one block of 1024
__global__ void k_advance(uint32_t *pos) {
    pdl_prologue(); if (threadIdx.x == 0 && blockIdx.x == 0) *pos += 1u; }

// gen_log / gen_count (optional): the chosen id is also appended to gen_log[*gen_count]
__global__ void __launch_bounds__(1024) k_argmax(const float *v, uint32_t n, uint32_t *__restrict__ out, uint32_t *__restrict__ gen_log,
                                                 uint32_t *__restrict__ gen_count, uint32_t *__restrict__ status) {
    pdl_prologue();
    __shared__ float bv[32];
    __shared__ uint32_t bi[32];
    float best = -INFINITY; uint32_t idx = 0xffffffffu;
    for (uint32_t i = threadIdx.x; i < n; i += 1024u) { const float x = v[i]; if (x > best || (x == best && i < idx)) { best = x; idx = i; } }
    for (int o = 16; o; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o); const uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
    }
    if ((threadIdx.x & 31u) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) if (bv[w] > best || (bv[w] == best && bi[w] < idx)) { best = bv[w]; idx = bi[w]; }
        if (idx >= n) { idx = 0; if (status) status[ST_TOKEN_RANGE] = 1u; }      // every logit NaN: nothing compared greater
        *out = idx;
        if (gen_log) { gen_log[*gen_count] = idx; *gen_count += 1u; }
    }
}

struct EngLayer {
    bool recurrent = false;
    uint32_t ridx = 0, aidx = 0;
    const float *attn_norm = nullptr, *post_norm = nullptr;
    DMat qkv, z, ba, ssm_out, q, k, v, o;
    const float *conv_k = nullptr, *dt = nullptr, *a = nullptr, *ssm_norm = nullptr, *q_norm = nullptr, *k_norm = nullptr;
    redcuda_moe *moe = nullptr;
};

}  // namespace rc

using namespace rc;

struct rl_engine {
    rl_engine_config cfg;
    rl_engine_info info;
    GgufFile gguf;
    std::vector<EngLayer> layers;
    DMat tok_embd, output;
    const float *output_norm = nullptr;
    int ep_rank = 0, ep_world = 1;       // expert shard of this engine (contiguous: experts [rank * E / world, (rank + 1) * E / world))
    redcuda_ep *ep = nullptr;            // attached exchange context (not owned); required before the first step when ep_world > 1
    DevMem dense, state, scratch, moe_ws;      // moe_ws: the expert workspace shared by every layer
    bool kv_half = false;
    uint32_t position = 0, ffn = 0, ffn_sh = 0;
    uint64_t expert_bytes = 0, dense_step_bytes = 0;
    double preload_ms = 0.0;
    // state
    float *conv = nullptr, *rec = nullptr;
    void *kcache = nullptr, *vcache = nullptr;
    // scratch (device)
    float *x0 = nullptr, *normed = nullptr, *branch = nullptr, *resid = nullptr, *qkv = nullptr, *z = nullptr, *ba = nullptr, *ng = nullptr;
    float *dn_qk = nullptr, *dn_v = nullptr, *dn_beta = nullptr, *dn_gate = nullptr, *dn_core = nullptr;
    float *qg = nullptr, *kraw = nullptr, *vraw = nullptr, *query = nullptr, *gate = nullptr, *gated = nullptr, *part_m = nullptr, *part_l = nullptr, *part_acc = nullptr;
    float *embed_d = nullptr, *layer_out_d = nullptr, *final_norm_d = nullptr, *logits_d = nullptr;
    uint32_t *router_ids_d = nullptr, *token_d = nullptr, *gen_tokens_d = nullptr, *pos_d = nullptr, *gen_count_d = nullptr;
    cudaGraphExec_t graph_greedy = nullptr;      // one greedy token (step + LM head + argmax), captured after the first eager token
    bool graph_failed = false;
    uint64_t graph_launches = 0;
    uint32_t max_split = 64, pf_split = 8;
    uint32_t pb = 1;                             // tokens per prefill chunk; every per-token scratch buffer holds pb rows
    float *bx[2] = {nullptr, nullptr};           // layer input / output of a chunk (ping-pong)
    int8_t *xq = nullptr; float *sx = nullptr;   // chunk activations as digit planes for the Q6_K tensor-core projections
    uint32_t *tok_chunk_d = nullptr, *pos_chunk_d = nullptr;
    float *dn_pd = nullptr;          // DeltaNet prefill: the 16 pair products of every group of four tokens and key head
    __half *tc_xs = nullptr; float *tc_xinv = nullptr; uint32_t *tc_err = nullptr;   // tcgen05 GEMM: activation digits, per-token inverse scales, timeout flag
    uint8_t *tc_wd = nullptr; float *tc_winv = nullptr; size_t tc_wd_cap = 0;        // and the weight digits of one launch (widest projection group)
    // host mirrors
    std::vector<float> embed_h, layer_out_h, final_norm_h;
    std::vector<uint32_t> router_ids_h;
    uint32_t *token_pin = nullptr;
    cudaStream_t stream = nullptr;
    int device = 0;
};

static void eng_err(char *error, size_t cap, const char *msg) { if (error && cap) snprintf(error, cap, "%s", msg ? msg : "unknown engine error"); }
#define ENG_FAIL(...) do { char b_[512]; snprintf(b_, sizeof(b_), __VA_ARGS__); eng_err(error, cap, b_); return 0; } while (0)
#define ENG_RC(call) do { if (!(call)) { eng_err(error, cap, redcuda_last_error()); return 0; } } while (0)
#define ENG_CUDA(expr) do { cudaError_t e_ = (expr); if (e_ != cudaSuccess) { ENG_FAIL("%s failed: %s", #expr, cudaGetErrorString(e_)); } } while (0)

static void eng_rmsnorm(rl_engine *e, uint32_t ntok, const float *x, const GemvNorm &N) {
    bool aligned = true;
    for (const void *p : {(const void *)x, (const void *)N.branch, (const void *)N.w, (const void *)N.resid, (const void *)N.normed}) aligned = aligned && ((uintptr_t)p & 15u) == 0u;
    prof_begin(N.branch ? "resid_rmsnorm" : "rmsnorm", e->stream);
    if (ntok < 148u) RC_LAUNCH((k_rmsnorm<1024u>), ntok, 1024, 0, e->stream, x, N.branch, N.w, e->info.hidden, N.eps, N.resid, N.normed);
    else if (e->info.hidden == 2048u && aligned) RC_LAUNCH((k_rmsnorm_rows<16u>), (ntok + 3u) / 4u, 128, 0, e->stream, x, N.branch, N.w, ntok, N.eps, N.resid, N.normed);
    else if (e->info.hidden == 1024u && aligned) RC_LAUNCH((k_rmsnorm_rows<8u>), (ntok + 3u) / 4u, 128, 0, e->stream, x, N.branch, N.w, ntok, N.eps, N.resid, N.normed);
    else RC_LAUNCH((k_rmsnorm<256u>), ntok, 256, 0, e->stream, x, N.branch, N.w, e->info.hidden, N.eps, N.resid, N.normed);
    prof_end(e->stream);
    g_launches.fetch_add(1);
}

// norm (may be null): the input is RMSNorm(x [+ branch]) * w, computed by the GEMV where it can be and by a kernel before it where not
static int eng_gemv(rl_engine *e, const DMat *mats, float *const *outs, uint32_t n, const float *x, const char *tag, const GemvNorm *norm = nullptr) {
    GemvArgs A{};
    A.njobs = n; A.ntok = 1; A.x = x; A.x_stride = mats[0].ncols; A.tag = tag; A.resident = 1u;
    for (uint32_t j = 0; j < n; ++j) {
        GemvJob &J = A.job[j];
        J.w0 = mats[j].base; J.w1 = nullptr; J.out = outs[j]; J.nb = mats[j].nb; J.type = mats[j].type; J.nrows = mats[j].nrows; J.ncols = mats[j].ncols;
        J.out_stride = mats[j].nrows; J.epi = GEMV_STORE;
    }
    if (norm) {
        A.norm = *norm;
        if (!gemv1_norm_ok(A)) { A.norm = GemvNorm{}; A.x = norm->normed; eng_rmsnorm(e, 1u, x, *norm); }
    }
    return launch_gemv(A, e->stream);
}

// ntok tokens at positions pos[0..ntok): decode passes e->pos_d (one token), a prefill chunk its position list
template <typename KV>
static int eng_attention(rl_engine *e, const EngLayer &L, uint32_t ntok, const uint32_t *pos, char *error, size_t cap) {
    const rl_engine_info &in = e->info;
    const uint32_t hd = in.head_dim, nq = in.n_head, nkv = in.n_head_kv, G = nq / nkv;
    const size_t kv_layer = (size_t)in.context * nkv * hd;
    KV *kc = (KV *)e->kcache + kv_layer * L.aidx, *vc = (KV *)e->vcache + kv_layer * L.aidx;
    cudaStream_t s = e->stream;
    prof_begin("attn_prep", s);
#define ENG_PREP(VPL_) RC_LAUNCH((k_attn_prep_rows<KV, VPL_>), ntok, 256, 0, s, e->qg, e->kraw, e->vraw, L.q_norm, L.k_norm, nq, nkv, in.rope_dims, in.rope_freq_base, \
                                 in.rms_eps, pos, e->query, e->gate, kc, vc)
    // few tokens: a block per head, so that the chip is not left to a few of them
    const bool rows = ntok >= 148u && in.rope_dims <= hd;
    if (rows && hd == 256u) ENG_PREP(8u);
    else if (rows && hd == 128u) ENG_PREP(4u);
    else if (rows && hd == 64u) ENG_PREP(2u);
    else RC_LAUNCH((k_attn_prep<KV>), dim3(nq + 2u * nkv, ntok), hd, hd * sizeof(float), s, e->qg, e->kraw, e->vraw, L.q_norm, L.k_norm, nq, nkv, hd, in.rope_dims, in.rope_freq_base,
                                                                      in.rms_eps, pos, e->query, e->gate, kc, vc);
#undef ENG_PREP
    prof_end(s);
    const float scale = (float)(1.0 / sqrt((double)hd));
    {   // a chunk of tokens: the tiled tensor-core kernel (RC_ATTN_CHUNK=0 keeps the per-token kernel, for A/B runs)
        static const bool want = !(getenv("RC_ATTN_CHUNK") && atoi(getenv("RC_ATTN_CHUNK")) == 0);
        if (want && ntok >= 8u && attn_chunk_ok<KV>(hd, G)) {
            ENG_RC(launch_attn_chunk<KV>(e->query, kc, vc, nkv, G, hd, pos, ntok, scale, e->gate, e->gated, s));
            g_launches.fetch_add(1);
            return 1;
        }
    }
    uint32_t nsplit = (in.context + 31u) / 32u;                 // fixed per engine (graph replay): enough slices for a full context
    nsplit = nsplit < 1u ? 1u : nsplit > e->max_split ? e->max_split : nsplit;
    if (ntok > 1u && nsplit > e->pf_split) nsplit = e->pf_split;     // a chunk brings its own parallelism (and the partials are per token)
    const size_t smem = (size_t)(8u * G * hd + 24u * G) * sizeof(float);
    const dim3 grid(nkv, nsplit, ntok);
    prof_begin("attn_decode", s);
#define ENG_ATTN(VPL_, G_) do { \
        if (smem > 48u * 1024u) ENG_CUDA(cudaFuncSetAttribute(k_attn_decode<KV, VPL_, G_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        RC_LAUNCH((k_attn_decode<KV, VPL_, G_>), grid, 256, smem, s, e->query, kc, vc, nkv, pos, nsplit, scale, e->part_m, e->part_l, e->part_acc); } while (0)
    if (hd == 256u && G == 8u) ENG_ATTN(8, 8);
    else if (hd == 128u && G == 8u) ENG_ATTN(4, 8);
    else if (hd == 128u && G == 4u) ENG_ATTN(4, 4);
    else if (hd == 64u && G == 2u) ENG_ATTN(2, 2);
    else if (hd == 64u && G == 4u) ENG_ATTN(2, 4);
    else if (hd == 256u && G == 4u) ENG_ATTN(8, 4);
    else ENG_FAIL("attention shape head_dim %u with %u query heads per KV head is not built", hd, G);
#undef ENG_ATTN
    prof_end(s);
    prof_begin("attn_merge", s);
    RC_LAUNCH((k_attn_merge), dim3(nq, ntok), hd, nsplit * sizeof(float), s, e->part_m, e->part_l, e->part_acc, e->gate, nsplit, hd, e->gated);
    prof_end(s);
    g_launches.fetch_add(3);
    ENG_CUDA(cudaGetLastError());
    return 1;
}

// One token on the device; the token id is already in e->token_d. want_logits: run the LM head.
static int eng_step_device(rl_engine *e, bool want_logits, char *error, size_t cap) {
    const rl_engine_info &in = e->info;
    cudaStream_t s = e->stream;
    if (e->ep_world > 1 && !e->ep) ENG_FAIL("this engine holds an expert shard: attach the exchange context first (redcuda_engine_attach_ep)");
    if (e->position >= in.context) ENG_FAIL("context of %u positions is full", in.context);
    prof_begin("embed", s);
    RC_LAUNCH((k_embed_row), 1, 256, 0, s, e->tok_embd.base, e->tok_embd.type, e->tok_embd.nb, in.hidden, in.vocab, e->token_d, books_iq2(), books_iq3s(), e->embed_d, status_words());
    prof_end(s);
    g_launches.fetch_add(1);
    const float *x = e->embed_d;
    const DnDims D{in.d_conv, in.d_state, in.n_group, in.dt_rank, in.d_inner, in.channels, in.rms_eps};
    for (uint32_t l = 0; l < in.n_layer; ++l) {
        const EngLayer &L = e->layers[l];
        const GemvNorm attn_norm{L.attn_norm, nullptr, in.rms_eps, nullptr, e->normed}, post_norm{L.post_norm, e->branch, in.rms_eps, e->resid, e->normed};
        if (L.recurrent) {
            const DMat mats[3] = {L.qkv, L.z, L.ba};
            float *outs[3] = {e->qkv, e->z, e->ba};
            ENG_RC(eng_gemv(e, mats, outs, 3, x, "dn_proj_gemv", &attn_norm));
            ENG_RC(launch_deltanet(D, 1u, L.conv_k, L.dt, L.a, L.ssm_norm, e->qkv, e->z, e->ba, e->conv + (size_t)L.ridx * (in.d_conv - 1u) * in.channels,
                                   e->rec + (size_t)L.ridx * in.dt_rank * in.d_state * in.d_state, e->dn_qk, e->dn_v, e->dn_beta, e->dn_gate, e->dn_core, e->ng, s));
            float *o1[1] = {e->branch};
            ENG_RC(eng_gemv(e, &L.ssm_out, o1, 1, e->ng, "dn_out_gemv"));
        } else {
            const DMat mats[3] = {L.q, L.k, L.v};
            float *outs[3] = {e->qg, e->kraw, e->vraw};
            ENG_RC(eng_gemv(e, mats, outs, 3, x, "attn_proj_gemv", &attn_norm));
            if (e->kv_half) { if (!eng_attention<__half>(e, L, 1u, e->pos_d, error, cap)) return 0; }
            else { if (!eng_attention<float>(e, L, 1u, e->pos_d, error, cap)) return 0; }
            float *o1[1] = {e->branch};
            ENG_RC(eng_gemv(e, &L.o, o1, 1, e->gated, "attn_out_gemv"));
        }
        float *xo = e->layer_out_d + (size_t)l * in.hidden;
        if (e->ep_world > 1) {
            eng_rmsnorm(e, 1u, x, post_norm);
            ENG_RC(redcuda_ep_layer_forward_n(e->ep, L.moe, 1u, e->normed, nullptr, e->resid, xo, s));
            ENG_CUDA(cudaMemcpyAsync(e->router_ids_d + (size_t)l * RL_ENGINE_MAX_TOPK, redcuda_ep_last_ids_device(e->ep), in.top_k * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        } else {                                             // its router kernel also fills router_ids_d (mirror set at open)
            const int done = moe_forward_norm1(L.moe, x, post_norm, e->resid, xo, s);
            ENG_RC(done);
            if (done < 0) {
                eng_rmsnorm(e, 1u, x, post_norm);
                ENG_RC(redcuda_moe_forward_device(L.moe, 1u, e->normed, nullptr, e->resid, xo, s));
            }
        }
        if (e->ep_world == 1 && in.n_expert > 1024u) ENG_CUDA(cudaMemcpyAsync(e->router_ids_d + (size_t)l * RL_ENGINE_MAX_TOPK, moe_last_ids_device(L.moe), in.top_k * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        x = xo;
    }
    const GemvNorm output_norm{e->output_norm, nullptr, in.rms_eps, nullptr, e->final_norm_d};
    if (want_logits) {
        float *o1[1] = {e->logits_d};
        ENG_RC(eng_gemv(e, &e->output, o1, 1, x, "lm_head_gemv", &output_norm));
    } else eng_rmsnorm(e, 1u, x, output_norm);
    RC_LAUNCH((k_advance), 1, 32, 0, s, e->pos_d);
    g_launches.fetch_add(1);
    ENG_CUDA(cudaGetLastError());
    e->position++;
    return 1;
}

// Projections of a chunk. From 8 tokens on, block-quantised matrices run on the tcgen05 GEMM (the matrices of one call
// share the input, so its fp16 digits are prepared once and one launch covers them all); below that, or with
// RL_PREFILL_TC=0, Q6_K matrices with >= 3 tokens take the mma.sync kernel on int8 digit planes and the rest the GEMV.
static int eng_proj(rl_engine *e, const DMat *mats, float *const *outs, uint32_t n, const float *x, uint32_t ntok, const char *tag) {
    static const bool want_mma = !(getenv("RC_MOE_PATH") && getenv("RC_MOE_PATH")[0] == 'c');
    static const bool want_tc = !(getenv("RL_PREFILL_TC") && atoi(getenv("RL_PREFILL_TC")) == 0);
    bool all_quant = true;
    for (uint32_t i = 0; i < n; ++i) all_quant = all_quant && rc_is_quant(mats[i].type) && mats[i].ncols == mats[0].ncols;
    if (want_tc && all_quant && ntok >= 8u && n <= TC_MAX_JOBS && mats[0].ncols % 256u == 0) {
        uint32_t row_tiles = 0;
        for (uint32_t i = 0; i < n; ++i) row_tiles += tc_row_tiles(mats[i].nrows);
        const uint32_t tn = tc_token_tile(ntok, row_tiles);
        if (!launch_tc_prep_x(x, nullptr, mats[0].ncols, ntok, mats[0].ncols, tn, e->tc_xs, e->tc_xinv, e->stream)) return 0;
        TcArgs A{};
        A.njobs = n; A.ncols = mats[0].ncols; A.ntok = ntok; A.xs = e->tc_xs; A.x_inv = e->tc_xinv; A.err = e->tc_err;
        A.wd = e->tc_wd; A.w_inv = e->tc_winv;
        RC_REQUIRE(tc_wd_bytes(row_tiles, mats[0].ncols) <= e->tc_wd_cap, "projection group %s: %u row tiles x %u columns exceed the weight-digit scratch", tag, row_tiles, mats[0].ncols);
        for (uint32_t i = 0; i < n; ++i) A.job[i] = TcJob{mats[i].base, mats[i].nb, mats[i].type, mats[i].nrows, outs[i], mats[i].nrows, 0u};
        return launch_tc_gemm(A, tn, tag, e->stream);
    }
    GemvArgs A{};
    A.ntok = ntok; A.x = x; A.x_stride = mats[0].ncols; A.tag = tag; A.resident = 1u;
    uint32_t j = 0;
    bool quantised = false;
    for (uint32_t i = 0; i < n; ++i) {
        const DMat &M = mats[i];
        if (want_mma && ntok >= 3u && M.type == RC_Q6_K && M.nrows % 16u == 0 && M.ncols % 256u == 0) {
            if (!quantised) { if (!launch_quant_act(x, M.ncols, ntok, M.ncols, e->xq, e->sx, e->stream)) return 0; quantised = true; }
            if (!launch_q6k_mma(M.base, nullptr, M.nb, M.nrows, M.ncols, ntok, e->xq, e->sx, outs[i], M.nrows, tag, e->stream)) return 0;
            continue;
        }
        GemvJob &J = A.job[j++];
        J.w0 = M.base; J.w1 = nullptr; J.out = outs[i]; J.nb = M.nb; J.type = M.type; J.nrows = M.nrows; J.ncols = M.ncols; J.out_stride = M.nrows; J.epi = GEMV_STORE;
    }
    if (!j) return 1;
    A.njobs = j;
    return launch_gemv(A, e->stream);
}

// A chunk of n consecutive tokens (ids in e->tok_chunk_d, positions in e->pos_chunk_d) through every layer at once:
// projections, router and experts see the n tokens as a batch (each weight byte is read once per chunk); the DeltaNet
// recurrence runs over the tokens inside one kernel with the state in registers; attention appends the chunk's K/V
// rows and masks by position. The mirrors are left holding the last token's rows, as after n single steps
// (the reference's chunked prefill, native/redlite_native_engine.c:600-640).
static int eng_prefill_chunk(rl_engine *e, uint32_t n, bool want_logits, char *error, size_t cap) {
    if (e->ep_world > 1 && !e->ep) ENG_FAIL("this engine holds an expert shard: attach the exchange context first (redcuda_engine_attach_ep)");
    const rl_engine_info &in = e->info;
    cudaStream_t s = e->stream;
    if (e->position + n > in.context) ENG_FAIL("context of %u positions is full", in.context);
    const DnDims D{in.d_conv, in.d_state, in.n_group, in.dt_rank, in.d_inner, in.channels, in.rms_eps};
    const size_t last = (size_t)(n - 1u);
    prof_begin("embed", s);
    RC_LAUNCH((k_embed_row), n, 256, 0, s, e->tok_embd.base, e->tok_embd.type, e->tok_embd.nb, in.hidden, in.vocab, e->tok_chunk_d, books_iq2(), books_iq3s(), e->bx[0], status_words());
    prof_end(s);
    g_launches.fetch_add(1);
    ENG_CUDA(cudaMemcpyAsync(e->embed_d, e->bx[0] + last * in.hidden, in.hidden * 4u, cudaMemcpyDeviceToDevice, s));
    const float *x = e->bx[0];
    for (uint32_t l = 0; l < in.n_layer; ++l) {
        const EngLayer &L = e->layers[l];
        eng_rmsnorm(e, n, x, GemvNorm{L.attn_norm, nullptr, in.rms_eps, nullptr, e->normed});
        if (L.recurrent) {
            const DMat mats[3] = {L.qkv, L.z, L.ba};
            float *outs[3] = {e->qkv, e->z, e->ba};
            ENG_RC(eng_proj(e, mats, outs, 3, e->normed, n, "dn_proj"));
            ENG_RC(launch_deltanet_seq(D, n, L.conv_k, L.dt, L.a, L.ssm_norm, e->qkv, e->z, e->ba, e->conv + (size_t)L.ridx * (in.d_conv - 1u) * in.channels,
                                       e->rec + (size_t)L.ridx * in.dt_rank * in.d_state * in.d_state, e->dn_qk, e->dn_v, e->dn_beta, e->dn_gate, e->dn_core, e->ng, e->dn_pd, s));
            float *o1[1] = {e->branch};
            ENG_RC(eng_proj(e, &L.ssm_out, o1, 1, e->ng, n, "dn_out"));
        } else {
            const DMat mats[3] = {L.q, L.k, L.v};
            float *outs[3] = {e->qg, e->kraw, e->vraw};
            ENG_RC(eng_proj(e, mats, outs, 3, e->normed, n, "attn_proj"));
            if (e->kv_half) { if (!eng_attention<__half>(e, L, n, e->pos_chunk_d, error, cap)) return 0; }
            else { if (!eng_attention<float>(e, L, n, e->pos_chunk_d, error, cap)) return 0; }
            float *o1[1] = {e->branch};
            ENG_RC(eng_proj(e, &L.o, o1, 1, e->gated, n, "attn_out"));
        }
        eng_rmsnorm(e, n, x, GemvNorm{L.post_norm, e->branch, in.rms_eps, e->resid, e->normed});
        float *xo = e->bx[(l + 1u) & 1u];
        if (e->ep_world > 1) ENG_RC(redcuda_ep_layer_forward_n(e->ep, L.moe, n, e->normed, nullptr, e->resid, xo, s));
        else ENG_RC(redcuda_moe_forward_device(L.moe, n, e->normed, nullptr, e->resid, xo, s));
        ENG_CUDA(cudaMemcpyAsync(e->router_ids_d + (size_t)l * RL_ENGINE_MAX_TOPK, (e->ep_world > 1 ? redcuda_ep_last_ids_device(e->ep) : moe_last_ids_device(L.moe)) + last * in.top_k, in.top_k * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        ENG_CUDA(cudaMemcpyAsync(e->layer_out_d + (size_t)l * in.hidden, xo + last * in.hidden, in.hidden * 4u, cudaMemcpyDeviceToDevice, s));
        x = xo;
    }
    const GemvNorm output_norm{e->output_norm, nullptr, in.rms_eps, nullptr, e->final_norm_d};
    if (want_logits) {
        float *o1[1] = {e->logits_d};
        ENG_RC(eng_gemv(e, &e->output, o1, 1, x + last * in.hidden, "lm_head_gemv", &output_norm));
    } else eng_rmsnorm(e, 1u, x + last * in.hidden, output_norm);
    ENG_CUDA(cudaGetLastError());
    e->position += n;
    return 1;
}

static int eng_set_position(rl_engine *e, uint32_t position, char *error, size_t cap) {
    ENG_CUDA(cudaStreamSynchronize(e->stream));
    e->token_pin[2] = position;
    ENG_CUDA(cudaMemcpyAsync(e->pos_d, e->token_pin + 2, 4, cudaMemcpyHostToDevice, e->stream));
    ENG_CUDA(cudaStreamSynchronize(e->stream));
    e->position = position;
    return 1;
}

static int eng_copy_mirrors(rl_engine *e, float *logits, char *error, size_t cap) {
    const rl_engine_info &in = e->info;
    cudaStream_t s = e->stream;
    ENG_CUDA(cudaMemcpyAsync(e->embed_h.data(), e->embed_d, in.hidden * 4u, cudaMemcpyDeviceToHost, s));
    ENG_CUDA(cudaMemcpyAsync(e->layer_out_h.data(), e->layer_out_d, (size_t)in.n_layer * in.hidden * 4u, cudaMemcpyDeviceToHost, s));
    ENG_CUDA(cudaMemcpyAsync(e->final_norm_h.data(), e->final_norm_d, in.hidden * 4u, cudaMemcpyDeviceToHost, s));
    ENG_CUDA(cudaMemcpyAsync(e->router_ids_h.data(), e->router_ids_d, (size_t)in.n_layer * RL_ENGINE_MAX_TOPK * 4u, cudaMemcpyDeviceToHost, s));
    if (logits) ENG_CUDA(cudaMemcpyAsync(logits, e->logits_d, (size_t)in.vocab * 4u, cudaMemcpyDeviceToHost, s));
    ENG_CUDA(cudaStreamSynchronize(s));
    if (status_failed()) ENG_FAIL("%s", redcuda_last_error());
    return 1;
}

static int eng_reset_state(rl_engine *e, char *error, size_t cap) {
    ENG_CUDA(cudaMemsetAsync(e->state.p, 0, e->state.bytes, e->stream));
    if (e->tc_err) ENG_CUDA(cudaMemsetAsync(e->tc_err, 0, 4, e->stream));
    ENG_CUDA(cudaStreamSynchronize(e->stream));
    return eng_set_position(e, 0u, error, cap);
}

// upload one dense GGUF matrix [ncols = shape[0], nrows = shape[1]] into the arena at *off
static int eng_upload(rl_engine *e, const GgufTensor *t, const char *name, uint8_t *arena, size_t *off, uint8_t *scratch, DMat *out, char *error, size_t cap) {
    if (!t) ENG_FAIL("missing tensor %s", name);
    if (t->n_dims != 2u || !t->bytes) ENG_FAIL("tensor %s has an unsupported type (%u) or rank (%u)", name, t->type, t->n_dims);
    const uint32_t ncols = (uint32_t)t->shape[0], nrows = (uint32_t)t->shape[1];
    uint8_t *dst = arena + *off;
    ENG_RC(upload_matrix(t->type, nrows, ncols, e->gguf.data(t), false, dst, scratch, e->stream));
    *out = DMat{dst, t->type, nrows, ncols, rc_is_quant(t->type) ? (uint64_t)nrows * (ncols / 256u) : 0u};
    *off += (t->bytes + 255u) / 256u * 256u;
    return 1;
}

static int eng_upload_f32(rl_engine *e, const GgufTensor *t, const char *name, uint64_t count, uint8_t *arena, size_t *off, const float **out, char *error, size_t cap) {
    if (!t) ENG_FAIL("missing tensor %s", name);
    uint64_t n = 1;
    for (uint32_t d = 0; d < t->n_dims; ++d) n *= t->shape[d];
    if (t->type != 0u || n != count) ENG_FAIL("tensor %s must be F32 with %llu values", name, (unsigned long long)count);
    ENG_CUDA(cudaMemcpyAsync(arena + *off, e->gguf.data(t), count * 4u, cudaMemcpyHostToDevice, e->stream));
    *out = (const float *)(arena + *off);
    *off += (count * 4u + 255u) / 256u * 256u;
    return 1;
}

static int eng_open(rl_engine *e, const char *path, char *error, size_t cap) {
    const double t_open = now_ms();
    if (!require_device()) ENG_FAIL("%s", redcuda_last_error());
    if (!e->gguf.open_file(path)) ENG_FAIL("%s", e->gguf.error.c_str());
    const GgufFile &g = e->gguf;
    if (g.architecture != "qwen3next") ENG_FAIL("GGUF architecture is not qwen3next");
    rl_engine_info &in = e->info;
    memset(&in, 0, sizeof(in));
    in.n_layer = g.u32("qwen3next.block_count"); in.hidden = g.u32("qwen3next.embedding_length"); in.vocab = (uint32_t)g.vocab;
    in.n_expert = g.u32("qwen3next.expert_count"); in.top_k = e->cfg.top_k ? e->cfg.top_k : g.u32("qwen3next.expert_used_count");
    in.context = e->cfg.context ? e->cfg.context : 4096u;
    in.d_conv = g.u32("qwen3next.ssm.conv_kernel"); in.d_inner = g.u32("qwen3next.ssm.inner_size"); in.d_state = g.u32("qwen3next.ssm.state_size");
    in.n_group = g.u32("qwen3next.ssm.group_count"); in.dt_rank = g.u32("qwen3next.ssm.time_step_rank");
    in.n_head = g.u32("qwen3next.attention.head_count"); in.n_head_kv = g.u32("qwen3next.attention.head_count_kv");
    in.head_dim = g.u32("qwen3next.attention.key_length"); in.rope_dims = g.u32("qwen3next.rope.dimension_count");
    in.rope_freq_base = g.f32("qwen3next.rope.freq_base"); in.rms_eps = g.f32("qwen3next.attention.layer_norm_rms_epsilon");
    e->ffn_sh = g.u32("qwen3next.expert_shared_feed_forward_length");
    // the same consistency checks as the reference applies (native/redlite_native_engine.c:213-243)
    if (!in.n_layer || !in.hidden || !in.n_head || !in.n_head_kv || !in.head_dim || !in.rope_dims || !in.n_expert || !in.top_k || in.d_conv < 2u ||
        !in.d_state || !in.n_group || !in.dt_rank || !in.d_inner || !e->ffn_sh || in.rms_eps <= 0.f || in.rope_freq_base <= 0.f ||
        in.head_dim != g.u32("qwen3next.attention.value_length") || in.n_head % in.n_head_kv || in.dt_rank % in.n_group || in.d_inner % in.dt_rank || !in.vocab)
        ENG_FAIL("incomplete or inconsistent qwen3next metadata");
    in.head_v = in.d_inner / in.dt_rank;
    in.channels = 2u * in.d_state * in.n_group + in.d_inner;
    if (in.head_v != in.d_state) ENG_FAIL("DeltaNet head_v != state size");
    if (in.top_k > RL_ENGINE_MAX_TOPK || in.top_k > in.n_expert) ENG_FAIL("top-k out of range");
    if (in.rope_dims > in.head_dim || in.rope_dims % 2u) ENG_FAIL("unsupported RoPE dims");
    if (in.head_dim > 1024u || in.head_dim % 32u) ENG_FAIL("unsupported head_dim %u", in.head_dim);
    {
        const char *v = getenv("RL_KV_F16");      // same switch as the reference (native/redlite_native_engine.c:43-47)
        e->kv_half = v && atoi(v) != 0;
    }
    ENG_CUDA(cudaGetDevice(&e->device));
    ENG_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
    // Prefill chunk: the reference defaults to 2048 tokens per batched dispatch (native/redlite_native_engine.h:37), and so
    // does this engine (2048 is also the ceiling). The chunk sizes the expert workspace (about 0.5 GB at 2048), which all
    // layers share: they run one after the other on the engine's stream. 1 = token by token.
    e->pb = e->cfg.prefill_batch ? std::min(e->cfg.prefill_batch, 2048u) : 2048u;
    e->ep_rank = g_shard_rank; e->ep_world = g_shard_world;
    if (e->ep_world > 1 && in.n_expert % (uint32_t)e->ep_world) ENG_FAIL("%u experts do not divide over %d ranks", in.n_expert, e->ep_world);
    if (e->pb > in.context) e->pb = in.context;

    // ---- layer kinds from tensor names (native/redlite_native_layer_map.c:114-124), sizes of the dense arena
    e->layers.resize(in.n_layer);
    size_t dense_total = 0, scratch_max = 0;
    auto account = [&](const GgufTensor *t) { if (t) { dense_total += (t->bytes + 255u) / 256u * 256u + 256u; if (t->bytes > scratch_max) scratch_max = t->bytes; } };
    const char *rec_names[] = {"attn_qkv.weight", "attn_gate.weight", "ssm_ba.weight", "ssm_conv1d.weight", "ssm_dt.bias", "ssm_a", "ssm_norm.weight", "ssm_out.weight"};
    const char *att_names[] = {"attn_q.weight", "attn_k.weight", "attn_v.weight", "attn_q_norm.weight", "attn_k_norm.weight", "attn_output.weight"};
    const char *common[] = {"attn_norm.weight", "post_attention_norm.weight", "ffn_gate_inp.weight", "ffn_gate_inp_shexp.weight"};
    for (uint32_t l = 0; l < in.n_layer; ++l) {
        bool rec = false, att = false;
        for (const char *n : rec_names) { const GgufTensor *t = g.find_layer(l, n); if (t) { rec = true; account(t); } }
        for (const char *n : att_names) { const GgufTensor *t = g.find_layer(l, n); if (t) { att = true; account(t); } }
        for (const char *n : common) account(g.find_layer(l, n));
        if (rec == att) ENG_FAIL("layer %u has an unknown/mixed structure", l);
        e->layers[l].recurrent = rec;
        if (rec) e->layers[l].ridx = in.n_recurrent++; else e->layers[l].aidx = in.n_attention++;
    }
    const GgufTensor *t_embd = g.find("token_embd.weight"), *t_onorm = g.find("output_norm.weight"), *t_out = g.find("output.weight");
    if (!t_out) t_out = t_embd;      // tied embeddings (native/redlite_native_engine.c:253)
    account(t_embd); account(t_onorm); if (t_out != t_embd) account(t_out);
    if (!e->dense.alloc(dense_total + 4096u)) ENG_FAIL("%s", redcuda_last_error());
    DevMem up_scratch;
    if (!up_scratch.alloc(scratch_max + 256u)) ENG_FAIL("%s", redcuda_last_error());
    uint8_t *arena = e->dense.as<uint8_t>(), *sc = up_scratch.as<uint8_t>();
    size_t off = 0;
    if (!eng_upload(e, t_embd, "token_embd.weight", arena, &off, sc, &e->tok_embd, error, cap)) return 0;
    if (e->tok_embd.ncols != in.hidden || e->tok_embd.nrows != in.vocab) ENG_FAIL("token_embd.weight shape does not match (hidden, vocab)");
    if (t_out != t_embd) { if (!eng_upload(e, t_out, "output.weight", arena, &off, sc, &e->output, error, cap)) return 0; }
    else e->output = e->tok_embd;
    if (e->output.ncols != in.hidden || e->output.nrows != in.vocab) ENG_FAIL("output.weight shape does not match (hidden, vocab)");
    if (!eng_upload_f32(e, t_onorm, "output_norm.weight", in.hidden, arena, &off, &e->output_norm, error, cap)) return 0;
    in.dense_bytes = 0;

    for (uint32_t l = 0; l < in.n_layer; ++l) {
        EngLayer &L = e->layers[l];
        auto T = [&](const char *n) { return g.find_layer(l, n); };
        if (!eng_upload_f32(e, T("attn_norm.weight"), "attn_norm", in.hidden, arena, &off, &L.attn_norm, error, cap) ||
            !eng_upload_f32(e, T("post_attention_norm.weight"), "post_attention_norm", in.hidden, arena, &off, &L.post_norm, error, cap)) return 0;
        if (L.recurrent) {
            if (!eng_upload(e, T("attn_qkv.weight"), "attn_qkv", arena, &off, sc, &L.qkv, error, cap) || !eng_upload(e, T("attn_gate.weight"), "attn_gate", arena, &off, sc, &L.z, error, cap) ||
                !eng_upload(e, T("ssm_ba.weight"), "ssm_ba", arena, &off, sc, &L.ba, error, cap) || !eng_upload(e, T("ssm_out.weight"), "ssm_out", arena, &off, sc, &L.ssm_out, error, cap) ||
                !eng_upload_f32(e, T("ssm_conv1d.weight"), "ssm_conv1d", (uint64_t)in.d_conv * in.channels, arena, &off, &L.conv_k, error, cap) ||
                !eng_upload_f32(e, T("ssm_dt.bias"), "ssm_dt", in.dt_rank, arena, &off, &L.dt, error, cap) || !eng_upload_f32(e, T("ssm_a"), "ssm_a", in.dt_rank, arena, &off, &L.a, error, cap) ||
                !eng_upload_f32(e, T("ssm_norm.weight"), "ssm_norm", in.head_v, arena, &off, &L.ssm_norm, error, cap)) return 0;
            if (L.qkv.ncols != in.hidden || L.qkv.nrows != in.channels || L.z.nrows != in.d_inner || L.ba.nrows != 2u * in.dt_rank || L.ssm_out.ncols != in.d_inner || L.ssm_out.nrows != in.hidden)
                ENG_FAIL("layer %u: DeltaNet tensor shapes do not match the metadata", l);
            e->dense_step_bytes += rc_matrix_bytes(L.qkv.type, L.qkv.nrows, L.qkv.ncols) + rc_matrix_bytes(L.z.type, L.z.nrows, L.z.ncols) +
                                   rc_matrix_bytes(L.ba.type, L.ba.nrows, L.ba.ncols) + rc_matrix_bytes(L.ssm_out.type, L.ssm_out.nrows, L.ssm_out.ncols);
        } else {
            const uint32_t qc = in.n_head * in.head_dim, kvc = in.n_head_kv * in.head_dim;
            if (!eng_upload(e, T("attn_q.weight"), "attn_q", arena, &off, sc, &L.q, error, cap) || !eng_upload(e, T("attn_k.weight"), "attn_k", arena, &off, sc, &L.k, error, cap) ||
                !eng_upload(e, T("attn_v.weight"), "attn_v", arena, &off, sc, &L.v, error, cap) || !eng_upload(e, T("attn_output.weight"), "attn_output", arena, &off, sc, &L.o, error, cap) ||
                !eng_upload_f32(e, T("attn_q_norm.weight"), "attn_q_norm", in.head_dim, arena, &off, &L.q_norm, error, cap) ||
                !eng_upload_f32(e, T("attn_k_norm.weight"), "attn_k_norm", in.head_dim, arena, &off, &L.k_norm, error, cap)) return 0;
            if (L.q.nrows != 2u * qc || L.k.nrows != kvc || L.v.nrows != kvc || L.o.ncols != qc || L.o.nrows != in.hidden) ENG_FAIL("layer %u: attention tensor shapes do not match the metadata", l);
            e->dense_step_bytes += rc_matrix_bytes(L.q.type, L.q.nrows, L.q.ncols) + 2u * rc_matrix_bytes(L.k.type, L.k.nrows, L.k.ncols) + rc_matrix_bytes(L.o.type, L.o.nrows, L.o.ncols);
        }
        // ---- MoE: router, shared expert, every routed expert of the layer
        const GgufTensor *tr = T("ffn_gate_inp.weight"), *tg = T("ffn_gate_inp_shexp.weight"), *sg = T("ffn_gate_shexp.weight"), *su = T("ffn_up_shexp.weight"),
                         *sd = T("ffn_down_shexp.weight"), *ge = T("ffn_gate_exps.weight"), *ue = T("ffn_up_exps.weight"), *de = T("ffn_down_exps.weight");
        if (!tr || !tg || !sg || !su || !sd || !ge || !ue || !de) ENG_FAIL("layer %u: missing MoE tensor", l);
        if (tr->type != 0u || tg->type != 0u || ge->n_dims != 3u || ue->n_dims != 3u || de->n_dims != 3u || ge->shape[2] != in.n_expert || de->shape[2] != in.n_expert ||
            ge->shape[0] != in.hidden || de->shape[1] != in.hidden || ge->type != ue->type || sg->type != su->type || sg->type != sd->type || !ge->bytes || !de->bytes || !sg->bytes)
            ENG_FAIL("layer %u: MoE tensor types or shapes are not supported", l);
        redcuda_moe_desc d;
        memset(&d, 0, sizeof(d));
        d.hidden = in.hidden; d.n_expert = in.n_expert; d.top_k = in.top_k; d.ffn = (uint32_t)ge->shape[1]; d.ffn_sh = (uint32_t)sg->shape[1];
        d.type_gu = ge->type; d.type_down = de->type; d.type_sh = sg->type; d.weights_on_device = 0;
        // under expert parallelism the engine holds a contiguous share of the experts and sees the tokens of every rank
        const uint32_t ec = in.n_expert / (uint32_t)e->ep_world, eb = (uint32_t)e->ep_rank * ec;
        d.expert_begin = eb; d.expert_count = ec; d.max_tokens = e->pb * (uint32_t)e->ep_world;
        d.router = (const float *)g.data(tr);
        d.gate_exps = g.data(ge) + (size_t)eb * (ge->bytes / in.n_expert); d.up_exps = g.data(ue) + (size_t)eb * (ue->bytes / in.n_expert);
        d.down_exps = g.data(de) + (size_t)eb * (de->bytes / in.n_expert);
        d.sh_gate_inp = (const float *)g.data(tg); d.sh_gate = g.data(sg); d.sh_up = g.data(su); d.sh_down = g.data(sd);
        e->ffn = d.ffn;
        {
            const size_t need = moe_workspace_bytes(&d);
            if (!e->moe_ws.p && !e->moe_ws.alloc(need)) ENG_FAIL("%s", redcuda_last_error());
            L.moe = need <= e->moe_ws.bytes ? moe_create_shared(&d, e->moe_ws.p) : redcuda_moe_create(&d);
        }
        if (!L.moe) ENG_FAIL("layer %u: %s", l, redcuda_last_error());
        e->expert_bytes += ge->bytes + ue->bytes + de->bytes;
        e->dense_step_bytes += tr->bytes + tg->bytes + sg->bytes + su->bytes + sd->bytes;
    }
    e->dense_step_bytes += rc_matrix_bytes(e->output.type, e->output.nrows, e->output.ncols);
    in.dense_bytes = off;
    ENG_CUDA(cudaStreamSynchronize(e->stream));
    up_scratch.release();

    // ---- state: conv windows, recurrent states, KV cache (one allocation so that reset is one memset)
    const size_t conv_b = (size_t)(in.d_conv - 1u) * in.channels * in.n_recurrent * 4u, rec_b = (size_t)in.dt_rank * in.d_state * in.d_state * in.n_recurrent * 4u;
    const size_t kv_b = (size_t)in.context * in.n_head_kv * in.head_dim * in.n_attention * (e->kv_half ? 2u : 4u);
    const size_t o_conv = 0, o_rec = (conv_b + 255u) / 256u * 256u, o_k = o_rec + (rec_b + 255u) / 256u * 256u, o_v = o_k + (kv_b + 255u) / 256u * 256u;
    if (!e->state.alloc(o_v + kv_b + 256u)) ENG_FAIL("%s", redcuda_last_error());
    uint8_t *S = e->state.as<uint8_t>();
    e->conv = (float *)(S + o_conv); e->rec = (float *)(S + o_rec); e->kcache = S + o_k; e->vcache = S + o_v;
    in.state_bytes = conv_b + rec_b + 2u * kv_b;

    // ---- scratch
    size_t w = 0;
    auto take = [&](size_t bytes) { const size_t o = w; w = (w + bytes + 255u) / 256u * 256u; return o; };
    const uint32_t qc = in.n_head * in.head_dim, kvc = in.n_head_kv * in.head_dim;
    const size_t T = e->pb;          // rows of every per-token buffer (decode uses row 0)
    const size_t parts = std::max<size_t>(e->max_split, T * e->pf_split);
    const uint32_t widest = std::max(std::max(in.hidden, in.d_inner), qc);
    // weight digits of the widest projection group that the tcgen05 GEMM may be given (4 bytes per weight, rows in tiles of 128)
    size_t wd_bytes = 0, wd_tiles = 0;
    for (uint32_t l = 0; l < in.n_layer; ++l) {
        const EngLayer &L = e->layers[l];
        const DMat *groups[2][3] = {{L.recurrent ? &L.qkv : &L.q, L.recurrent ? &L.z : &L.k, L.recurrent ? &L.ba : &L.v}, {L.recurrent ? &L.ssm_out : &L.o, nullptr, nullptr}};
        for (auto &g : groups) {
            uint32_t tiles = 0;
            for (const DMat *m : g) if (m) tiles += tc_row_tiles(m->nrows);
            wd_bytes = std::max(wd_bytes, tc_wd_bytes(tiles, g[0]->ncols));
            wd_tiles = std::max<size_t>(wd_tiles, tiles);
        }
    }
    const size_t o_twd = take(wd_bytes), o_twi = take(wd_tiles * 4u);
    const size_t o_norm = take(T * in.hidden * 4u), o_br = take(T * in.hidden * 4u), o_res = take(T * in.hidden * 4u), o_qkv = take(T * in.channels * 4u), o_z = take(T * in.d_inner * 4u),
                 o_ba = take(T * 2u * in.dt_rank * 4u), o_ng = take(T * in.d_inner * 4u), o_dqk = take(T * 2u * in.n_group * in.d_state * 4u), o_dv = take(T * in.d_inner * 4u),
                 o_db = take(T * in.dt_rank * 4u), o_dg = take(T * in.dt_rank * 4u), o_dc = take(T * in.d_inner * 4u), o_qg = take(T * 2u * qc * 4u), o_kr = take(T * kvc * 4u), o_vr = take(T * kvc * 4u),
                 o_qu = take(T * qc * 4u), o_ga = take(T * qc * 4u), o_gd = take(T * qc * 4u), o_pm = take((size_t)in.n_head * parts * 4u), o_pl = take((size_t)in.n_head * parts * 4u),
                 o_pa = take((size_t)in.n_head * parts * in.head_dim * 4u), o_em = take(in.hidden * 4u), o_lo = take((size_t)in.n_layer * in.hidden * 4u),
                 o_fn = take(in.hidden * 4u), o_lg = take((size_t)in.vocab * 4u), o_ri = take((size_t)in.n_layer * RL_ENGINE_MAX_TOPK * 4u), o_tk = take(16), o_gt = take(4096u * 4u),
                 o_bx0 = take(T * in.hidden * 4u), o_bx1 = take(T * in.hidden * 4u), o_xq = take(T * 3u * widest), o_sx = take(T * 4u), o_tc = take(T * 4u), o_pc = take(T * 4u),
                 o_txs = take(tc_xs_halves((uint32_t)T, widest, 128u) * 2u), o_txi = take((T + 128u) * 4u), o_ter = take(16),
                 o_pd = take((T + 4u) * in.n_group * 4u * 4u);
    if (!e->scratch.alloc(w)) ENG_FAIL("%s", redcuda_last_error());
    uint8_t *B = e->scratch.as<uint8_t>();
    ENG_CUDA(cudaMemsetAsync(B, 0, w, e->stream));
    e->normed = (float *)(B + o_norm); e->branch = (float *)(B + o_br); e->resid = (float *)(B + o_res); e->qkv = (float *)(B + o_qkv); e->z = (float *)(B + o_z);
    e->ba = (float *)(B + o_ba); e->ng = (float *)(B + o_ng); e->dn_qk = (float *)(B + o_dqk); e->dn_v = (float *)(B + o_dv); e->dn_beta = (float *)(B + o_db);
    e->dn_gate = (float *)(B + o_dg); e->dn_core = (float *)(B + o_dc); e->qg = (float *)(B + o_qg); e->kraw = (float *)(B + o_kr); e->vraw = (float *)(B + o_vr);
    e->query = (float *)(B + o_qu); e->gate = (float *)(B + o_ga); e->gated = (float *)(B + o_gd); e->part_m = (float *)(B + o_pm); e->part_l = (float *)(B + o_pl);
    e->part_acc = (float *)(B + o_pa); e->embed_d = (float *)(B + o_em); e->layer_out_d = (float *)(B + o_lo); e->final_norm_d = (float *)(B + o_fn);
    e->logits_d = (float *)(B + o_lg); e->router_ids_d = (uint32_t *)(B + o_ri); e->token_d = (uint32_t *)(B + o_tk); e->gen_tokens_d = (uint32_t *)(B + o_gt);
    e->pos_d = e->token_d + 2; e->gen_count_d = e->token_d + 3;
    e->bx[0] = (float *)(B + o_bx0); e->bx[1] = (float *)(B + o_bx1); e->xq = (int8_t *)(B + o_xq); e->sx = (float *)(B + o_sx);
    e->tok_chunk_d = (uint32_t *)(B + o_tc); e->pos_chunk_d = (uint32_t *)(B + o_pc);
    for (uint32_t l = 0; l < in.n_layer; ++l) moe_set_ids_mirror(e->layers[l].moe, e->router_ids_d + (size_t)l * RL_ENGINE_MAX_TOPK);
    e->tc_xs = (__half *)(B + o_txs); e->tc_xinv = (float *)(B + o_txi); e->tc_err = (uint32_t *)(B + o_ter);
    e->dn_pd = (float *)(B + o_pd);
    e->tc_wd = B + o_twd; e->tc_winv = (float *)(B + o_twi); e->tc_wd_cap = wd_bytes;
    e->embed_h.assign(in.hidden, 0.f); e->layer_out_h.assign((size_t)in.n_layer * in.hidden, 0.f); e->final_norm_h.assign(in.hidden, 0.f);
    e->router_ids_h.assign((size_t)in.n_layer * RL_ENGINE_MAX_TOPK, 0u);
    ENG_CUDA(cudaMallocHost((void **)&e->token_pin, 64u + 2u * T * 4u));      // [16 words][chunk tokens][chunk positions]
    if (!eng_reset_state(e, error, cap)) return 0;
    e->preload_ms = now_ms() - t_open;
    return 1;
}

extern "C" {

void rl_engine_config_default(rl_engine_config *cfg) {
    if (!cfg) return;
    memset(cfg, 0, sizeof(*cfg));
    cfg->context = 4096u; cfg->cache_mib = 4096u; cfg->enable_gpu = 1;
}

rl_engine *rl_engine_open(const char *model_path, const rl_engine_config *cfg, char *error, size_t cap) {
    if (!model_path) { eng_err(error, cap, "model path required"); return nullptr; }
    rl_engine *e = new (std::nothrow) rl_engine();
    if (!e) { eng_err(error, cap, "engine allocation failed"); return nullptr; }
    if (cfg) e->cfg = *cfg; else rl_engine_config_default(&e->cfg);
    if (e->cfg.enable_cpu) { eng_err(error, cap, "this library has no CPU backend (enable_cpu must be 0)"); delete e; return nullptr; }
    if (e->cfg.mtp_path && e->cfg.mtp_path[0]) { eng_err(error, cap, "multi-token prediction is not part of the CUDA backend"); delete e; return nullptr; }
    if (!eng_open(e, model_path, error, cap)) { rl_engine_close(e); return nullptr; }
    if (error && cap) error[0] = '\0';
    return e;
}

void rl_engine_close(rl_engine *e) {
    if (!e) return;
    if (e->stream) cudaStreamSynchronize(e->stream);
    if (e->graph_greedy) cudaGraphExecDestroy(e->graph_greedy);
    for (auto &L : e->layers) if (L.moe) redcuda_moe_destroy(L.moe);
    if (e->token_pin) cudaFreeHost(e->token_pin);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
}

const rl_engine_info *rl_engine_info_get(const rl_engine *e) { return e ? &e->info : nullptr; }

int rl_engine_reset(rl_engine *e, rl_engine_backend backend, char *error, size_t cap) {
    if (!e || backend != RL_BACKEND_GPU) { eng_err(error, cap, "backend not enabled"); return 0; }
    return eng_reset_state(e, error, cap);
}

uint32_t rl_engine_position(const rl_engine *e, rl_engine_backend backend) { return e && backend == RL_BACKEND_GPU ? e->position : 0u; }

int rl_engine_bench_set_position(rl_engine *e, rl_engine_backend backend, uint32_t position, char *error, size_t cap) {
    if (!e || backend != RL_BACKEND_GPU) { eng_err(error, cap, "backend not enabled"); return 0; }
    if (position >= e->info.context) { eng_err(error, cap, "position beyond the context"); return 0; }
    return eng_set_position(e, position, error, cap);
}

int rl_engine_step(rl_engine *e, rl_engine_backend backend, uint32_t token, float *logits, rl_engine_step_stats *stats, char *error, size_t cap) {
    if (!e) { eng_err(error, cap, "null engine"); return 0; }
    if (backend != RL_BACKEND_GPU) { eng_err(error, cap, "the CPU backend is not part of this library"); return 0; }
    if (token >= e->info.vocab) { eng_err(error, cap, "token id out of range"); return 0; }
    if (e->ep_world > 1) { eng_err(error, cap, "greedy generation on the device is not served under expert parallelism (the exchange's step counter cannot live in a replayed graph); use rl_engine_step"); return 0; }
    const double t0 = now_ms();
    if (stats) memset(stats, 0, sizeof(*stats));
    ENG_CUDA(cudaSetDevice(e->device));
    e->token_pin[0] = token;
    ENG_CUDA(cudaMemcpyAsync(e->token_d, e->token_pin, 4, cudaMemcpyHostToDevice, e->stream));
    if (!eng_step_device(e, logits != nullptr, error, cap)) return 0;
    if (!eng_copy_mirrors(e, logits, error, cap)) return 0;
    if (stats) { stats->total_ms = now_ms() - t0; stats->gpu_ms = stats->total_ms; stats->speculative = 1; stats->resident_slots = stats->slot_capacity = e->info.n_layer * e->info.n_expert; }
    if (error && cap) error[0] = '\0';
    return 1;
}

int rl_engine_prefill(rl_engine *e, rl_engine_backend backend, const uint32_t *tokens, uint32_t count, float *logits, rl_engine_step_stats *stats,
                      char *error, size_t cap) {
    // chunks of prefill_batch tokens (native/redlite_native_engine.c:600-640); a chunk of one token, and prefill_batch = 1,
    // take the single-token path. Only the last token runs the LM head.
    if (!e || !tokens || !count) { eng_err(error, cap, "invalid prefill arguments"); return 0; }
    if (backend != RL_BACKEND_GPU) { eng_err(error, cap, "the CPU backend is not part of this library"); return 0; }
    const double t0 = now_ms();
    if (stats) memset(stats, 0, sizeof(*stats));
    ENG_CUDA(cudaSetDevice(e->device));
    for (uint32_t i = 0; i < count; ++i) if (tokens[i] >= e->info.vocab) { eng_err(error, cap, "token id out of range"); return 0; }
    if (e->position + (uint64_t)count > e->info.context) { eng_err(error, cap, "prompt does not fit the context"); return 0; }
    uint32_t *tok_pin = e->token_pin + 16, *pos_pin = tok_pin + e->pb;
    ENG_CUDA(cudaMemsetAsync(e->tc_err, 0, 4, e->stream));     // a timeout of an earlier call must not fail this one
    for (uint32_t i = 0; i < count;) {
        const uint32_t n = std::min(e->pb, count - i);
        const bool last = i + n == count;
        ENG_CUDA(cudaStreamSynchronize(e->stream));      // the pinned staging words are reused
        if (n == 1u) {
            e->token_pin[0] = tokens[i];
            ENG_CUDA(cudaMemcpyAsync(e->token_d, e->token_pin, 4, cudaMemcpyHostToDevice, e->stream));
            if (!eng_step_device(e, logits != nullptr && last, error, cap)) return 0;
        } else {
            for (uint32_t t = 0; t < n; ++t) { tok_pin[t] = tokens[i + t]; pos_pin[t] = e->position + t; }
            e->token_pin[2] = e->position + n;
            ENG_CUDA(cudaMemcpyAsync(e->tok_chunk_d, tok_pin, n * 4u, cudaMemcpyHostToDevice, e->stream));
            ENG_CUDA(cudaMemcpyAsync(e->pos_chunk_d, pos_pin, n * 4u, cudaMemcpyHostToDevice, e->stream));
            if (!eng_prefill_chunk(e, n, logits != nullptr && last, error, cap)) return 0;
            ENG_CUDA(cudaMemcpyAsync(e->pos_d, e->token_pin + 2, 4, cudaMemcpyHostToDevice, e->stream));
        }
        i += n;
    }
    ENG_CUDA(cudaMemcpyAsync(e->token_pin + 3, e->tc_err, 4, cudaMemcpyDeviceToHost, e->stream));
    if (!eng_copy_mirrors(e, logits, error, cap)) return 0;
    if (e->token_pin[3]) ENG_FAIL("prefill: a tensor-core stage never signalled completion (bounded wait ran out); the engine state holds partial results: call rl_engine_reset before the next use");
    if (stats) { stats->total_ms = now_ms() - t0; stats->gpu_ms = stats->total_ms; }
    if (error && cap) error[0] = '\0';
    return 1;
}

uint32_t rl_engine_prefill_batch(const rl_engine *e) { return e ? e->pb : 0u; }

int redcuda_engine_shard(int rank, int world) {
    if (world < 1 || rank < 0 || rank >= world) { set_error("engine shard: rank %d of %d", rank, world); return 0; }
    g_shard_rank = rank; g_shard_world = world;
    return 1;
}

int redcuda_engine_attach_ep(rl_engine *e, redcuda_ep *ep) {
    if (!e || !ep) { set_error("engine attach: null argument"); return 0; }
    e->ep = ep;
    return 1;
}

int rl_engine_generate_greedy(rl_engine *e, uint32_t token, uint32_t n_new, uint32_t *out_tokens, rl_engine_step_stats *stats, char *error, size_t cap) {
    if (!e || !out_tokens || !n_new || n_new > 4096u) { eng_err(error, cap, "invalid generate arguments (1..4096 new tokens)"); return 0; }
    if (token >= e->info.vocab) { eng_err(error, cap, "token id out of range"); return 0; }
    const double t0 = now_ms();
    if (stats) memset(stats, 0, sizeof(*stats));
    ENG_CUDA(cudaSetDevice(e->device));
    e->token_pin[0] = token;
    ENG_CUDA(cudaMemcpyAsync(e->token_d, e->token_pin, 4, cudaMemcpyHostToDevice, e->stream));
    if (e->position + n_new > e->info.context) { eng_err(error, cap, "not enough context left for the requested tokens"); return 0; }
    ENG_CUDA(cudaMemsetAsync(e->gen_count_d, 0, 4, e->stream));
    auto one_token = [&]() -> int {
        if (!eng_step_device(e, true, error, cap)) return 0;
        RC_LAUNCH((k_argmax), 1, 1024, 0, e->stream, e->logits_d, e->info.vocab, e->token_d, e->gen_tokens_d, e->gen_count_d, status_words());
        g_launches.fetch_add(1);
        return 1;
    };
    for (uint32_t i = 0; i < n_new; ++i) {
        // The first token of an engine runs eagerly (it also sets every kernel attribute); then one token is captured
        // into a CUDA graph — position, token and output slot are read from device memory, so the same graph serves
        // every later token. RL_CUDA_GRAPH=0 keeps everything eager.
        static const bool want_graph = !(getenv("RL_CUDA_GRAPH") && atoi(getenv("RL_CUDA_GRAPH")) == 0);
        if (e->graph_greedy) {
            const uint64_t per_token = e->graph_launches;
            ENG_CUDA(cudaGraphLaunch(e->graph_greedy, e->stream));
            g_launches.fetch_add(per_token);
            e->position++;
            continue;
        }
        if (i >= 1u && want_graph && !e->graph_failed) {
            cudaGraph_t g = nullptr;
            const uint64_t before = g_launches.load();
            const uint32_t pos_before = e->position;
            bool ok = cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
            if (ok) {
                const int rc_ = one_token();
                const cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
                ok = rc_ && ce == cudaSuccess && g;
                e->position = pos_before;                     // capturing ran nothing
            }
            if (ok) ok = cudaGraphInstantiate(&e->graph_greedy, g, 0) == cudaSuccess;
            if (g) cudaGraphDestroy(g);
            if (!ok) { cudaGetLastError(); e->graph_failed = true; e->graph_greedy = nullptr; g_launches.store(before); }
            else { e->graph_launches = g_launches.load() - before; g_launches.store(before); --i; continue; }
        }
        if (!one_token()) return 0;
    }
    ENG_CUDA(cudaMemcpyAsync(out_tokens, e->gen_tokens_d, (size_t)n_new * 4u, cudaMemcpyDeviceToHost, e->stream));
    if (!eng_copy_mirrors(e, nullptr, error, cap)) return 0;
    if (stats) { stats->total_ms = now_ms() - t0; stats->gpu_ms = stats->total_ms; }
    if (error && cap) error[0] = '\0';
    return 1;
}

const float *rl_engine_last_embedding(const rl_engine *e, rl_engine_backend b) { return e && b == RL_BACKEND_GPU ? e->embed_h.data() : nullptr; }
const float *rl_engine_last_layer_output(const rl_engine *e, rl_engine_backend b, uint32_t layer) {
    return e && b == RL_BACKEND_GPU && layer < e->info.n_layer ? e->layer_out_h.data() + (size_t)layer * e->info.hidden : nullptr;
}
const float *rl_engine_last_final_norm(const rl_engine *e, rl_engine_backend b) { return e && b == RL_BACKEND_GPU ? e->final_norm_h.data() : nullptr; }
const uint32_t *rl_engine_last_router_ids(const rl_engine *e, rl_engine_backend b, uint32_t layer) {
    return e && b == RL_BACKEND_GPU && layer < e->info.n_layer ? e->router_ids_h.data() + (size_t)layer * RL_ENGINE_MAX_TOPK : nullptr;
}
int rl_engine_experts_preloaded(const rl_engine *e, double *preload_ms) { if (!e) return 0; if (preload_ms) *preload_ms = e->preload_ms; return 1; }
uint64_t rl_engine_full_residency_mib(const rl_engine *e) { return e ? (e->expert_bytes + (1u << 20) - 1u) >> 20 : 0u; }

int rl_engine_embed_token(const rl_engine *ce, uint32_t token, float *out, char *error, size_t cap) {
    rl_engine *e = const_cast<rl_engine *>(ce);
    if (!e || !out) { eng_err(error, cap, "invalid embed arguments"); return 0; }
    if (token >= e->info.vocab) { eng_err(error, cap, "token id out of range"); return 0; }
    ENG_CUDA(cudaStreamSynchronize(e->stream));
    e->token_pin[1] = token;
    ENG_CUDA(cudaMemcpyAsync(e->token_d + 1, e->token_pin + 1, 4, cudaMemcpyHostToDevice, e->stream));
    RC_LAUNCH((k_embed_row), 1, 256, 0, e->stream, e->tok_embd.base, e->tok_embd.type, e->tok_embd.nb, e->info.hidden, e->info.vocab, e->token_d + 1, books_iq2(), books_iq3s(), e->normed, status_words());
    g_launches.fetch_add(1);
    ENG_CUDA(cudaMemcpyAsync(out, e->normed, e->info.hidden * 4u, cudaMemcpyDeviceToHost, e->stream));
    ENG_CUDA(cudaStreamSynchronize(e->stream));
    return 1;
}

uint64_t rl_engine_step_bytes(const rl_engine *e) {
    if (!e) return 0;
    const rl_engine_info &in = e->info;
    const uint64_t per_expert = e->expert_bytes / ((uint64_t)in.n_layer * in.n_expert);
    const uint64_t states = 2ull * ((uint64_t)in.dt_rank * in.d_state * in.d_state + (uint64_t)(in.d_conv - 1u) * in.channels) * 4u * in.n_recurrent;
    const uint64_t kv = 2ull * (uint64_t)(e->position + 1u) * in.n_head_kv * in.head_dim * (e->kv_half ? 2u : 4u) * in.n_attention;
    return e->dense_step_bytes + per_expert * in.top_k * in.n_layer + states + kv + (uint64_t)in.hidden * rc_row_bytes(e->tok_embd.type, in.hidden) / in.hidden;
}

}  // extern "C"
