// Gated DeltaNet decode step between the projections (deltanet_branch, native/redlite_native_engine_cpu.c:148-230).
//
//   k_dn_prep   beta = sigmoid(b), gate = softplus(a + dt_bias) * A; causal depthwise conv over [conv state, new
//               sample] + SiLU; conv window shifted in place; q and k L2-normalised per key head (fp64 for the small
//               reductions, as the CPU path)
//   k_dn_state  the fp32 delta rule, one warp per state row: the row (d_state floats) is loaded once into the warp's
//               registers, decayed, corrected and read out, then stored — one read and one write of the state,
//               where the CPU path sweeps it four times
//   k_dn_tail   per value head RMSNorm(core) * w * SiLU(z)
//   k_dn_step   all three in one launch, the usual form: the kernels above serve state sizes and head ratios beyond it
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_silu.cuh"
#include "redcuda_stage.cuh"
#include "../../include/redcuda.h"

#include <stdlib.h>
#include <mutex>
#include <new>
#include <type_traits>

namespace rc {

__device__ __forceinline__ double sigmoid_stable(double x) { if (x >= 0.0) { const double z = exp(-x); return 1.0 / (1.0 + z); } const double z = exp(x); return z / (1.0 + z); }
__device__ __forceinline__ double softplus_stable(double x) { if (x > 20.0) return x; if (x < -20.0) return exp(x); return log1p(exp(x)); }

// grid.x = 2*groups (q/k heads) + d_inner/S (v runs) + 1 (beta/gate); grid.y = batch; block = S threads
__global__ void k_dn_prep(DnDims D, const float *__restrict__ conv_kernel, const float *__restrict__ dt_bias, const float *__restrict__ ssm_a,
                          const float *qkv, const float *ba, float *__restrict__ conv_state,
                          float *__restrict__ qk, float *__restrict__ v, float *__restrict__ beta, float *__restrict__ gate) {
    pdl_prologue();
    __shared__ double red[32];
    const uint32_t seq = blockIdx.y, tid = threadIdx.x, S = D.S, ns = D.d_conv - 1u;
    const uint32_t n_qk = 2u * D.groups, n_v = D.d_inner / S;
    if (blockIdx.x == n_qk + n_v) {   // beta / gate of every value head
        const uint32_t width = D.rank / D.groups, stride = 2u * width;
        for (uint32_t h = tid; h < D.rank; h += blockDim.x) {
            const uint32_t g = h / width, l = h - g * width;
            const float *b = ba + (size_t)seq * 2u * D.rank;
            beta[(size_t)seq * D.rank + h] = (float)sigmoid_stable((double)b[g * stride + l]);
            gate[(size_t)seq * D.rank + h] = (float)(softplus_stable((double)b[g * stride + width + l] + (double)dt_bias[h]) * (double)ssm_a[h]);
        }
        return;
    }
    const uint32_t c = blockIdx.x * S + tid;          // channel: q heads, then k heads, then v
    float *cs = conv_state + ((size_t)seq * D.channels + c) * ns;
    const float *kr = conv_kernel + (size_t)c * D.d_conv;
    const float xnew = qkv[(size_t)seq * D.channels + c];
    double acc = 0.0;
    for (uint32_t j = 0; j < ns; ++j) acc += (double)cs[j] * (double)kr[j];
    acc += (double)xnew * (double)kr[ns];
    for (uint32_t j = 0; j + 1u < ns; ++j) cs[j] = cs[j + 1u];
    cs[ns - 1u] = xnew;
    const float y = (float)(acc / (1.0 + exp(-acc)));
    if (blockIdx.x >= n_qk) { v[(size_t)seq * D.d_inner + (c - n_qk * S)] = y; return; }
    // L2 normalisation over the head (block)
    double ss = (double)y * (double)y;
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31u) == 0) red[tid >> 5] = ss;
    __syncthreads();
    double tot = 0.0;
    for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) tot += red[w];
    const double inv = 1.0 / fmax(sqrt(tot), (double)D.eps);
    qk[(size_t)seq * n_qk * S + c] = (float)((double)y * inv);
}

// one warp per (seq, value head, state row); VPL = S / 32 values per lane, element i = lane + 32 * v
template <int VPL>
__global__ void __launch_bounds__(256) k_dn_state(DnDims D, uint32_t batch, const float *qk, const float *v,
                                                  const float *beta, const float *gate,
                                                  float *__restrict__ state, float *__restrict__ core) {
    pdl_prologue();
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint32_t S = D.S;
    const uint64_t rows = (uint64_t)batch * D.rank * S;
    if (gw >= rows) return;
    const uint32_t j = (uint32_t)(gw % S), h = (uint32_t)((gw / S) % D.rank), seq = (uint32_t)(gw / ((uint64_t)S * D.rank));
    const uint32_t kh = h / (D.rank / D.groups);
    const float *q = qk + ((size_t)seq * 2u * D.groups + kh) * S;
    const float *k = qk + ((size_t)seq * 2u * D.groups + D.groups + kh) * S;
    float *row = state + (((size_t)seq * D.rank + h) * S + j) * S;
    const float decay = expf(gate[(size_t)seq * D.rank + h]);
    float m[VPL], kv[VPL];
    float sum = 0.f;
#pragma unroll
    for (int t = 0; t < VPL; ++t) { kv[t] = k[lane + 32 * t]; m[t] = row[lane + 32 * t] * decay; sum += m[t] * kv[t]; }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float delta = (v[(size_t)seq * D.d_inner + (size_t)h * S + j] - sum) * beta[(size_t)seq * D.rank + h];
    float o_acc = 0.f;
#pragma unroll
    for (int t = 0; t < VPL; ++t) { m[t] += kv[t] * delta; o_acc += m[t] * q[lane + 32 * t]; row[lane + 32 * t] = m[t]; }
    for (int o = 16; o; o >>= 1) o_acc += __shfl_xor_sync(0xffffffffu, o_acc, o);
    if (lane == 0) core[(size_t)seq * D.d_inner + (size_t)h * S + j] = o_acc * (1.0f / sqrtf((float)S));
}

// grid (rank, batch), block S threads
__global__ void k_dn_tail(DnDims D, const float *core, const float *z, const float *__restrict__ norm_w, float *__restrict__ out) {
    pdl_prologue();
    __shared__ double red[32];
    const uint32_t h = blockIdx.x, seq = blockIdx.y, i = threadIdx.x, S = D.S;
    const size_t idx = (size_t)seq * D.d_inner + (size_t)h * S + i;
    const float x = core[idx], g = z[idx];
    double ss = (double)x * (double)x;
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((i & 31u) == 0) red[i >> 5] = ss;
    __syncthreads();
    double tot = 0.0;
    for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) tot += red[w];
    const float inv = 1.0f / sqrtf((float)(tot / (double)S) + D.eps);
    const float silu = g / (1.0f + expf(-g));
    out[idx] = x * inv * norm_w[i] * silu;
}

// The whole step in one launch: SPLIT blocks per value head, 8 warps each, a warp owns consecutive state rows. What bounds it is the
// state: one read and one write of 4 S^2 bytes per head (33.5 MB for 8 sequences of 32 heads of 128: 5.1 us at the copy rate). As
// separate kernels, preparation and state update took 13.7 us for them, because the state was requested only after the
// preparation had ended. Here every lane first requests its conv windows and its state rows (RING of them a warp: with one block
// per head of 128 that is 64 registers and the block's whole 64 KB in flight), and the preparation (conv + SiLU, L2 norms, beta and
// gate: the arithmetic of k_dn_prep) runs while they arrive.
// The value heads of one key head all need its q and k. Their blocks form a cluster: each computes q and k for itself, and
// the first one moves the conv windows of the q / k channels on after all of them have read the old ones (cluster barrier).
// One block per head leaves most of the chip idle for a few sequences (a single one: 32 blocks). There 2 or 4 blocks share a
// head's rows and pass each other their parts of the norm's sum; launch_deltanet has the rule and its times.
// DC: conv taps known at compile time (0: D.d_conv); MINB: blocks per SM that the registers allow
template <int VPL, uint32_t DC, uint32_t SPLIT, int MINB, uint32_t RING>
__global__ void __launch_bounds__(256, MINB) k_dn_step(DnDims D, const float *__restrict__ conv_kernel, const float *__restrict__ dt_bias, const float *__restrict__ ssm_a,
                                                    const float *qkv, const float *ba, float *conv_state, float *__restrict__ state,
                                                    const float *z, const float *__restrict__ norm_w, float *__restrict__ out) {
    pdl_prologue();
    constexpr uint32_t S = VPL * 32u, SB = S / SPLIT, RPW = SB / 8u, TAPS = DC ? DC : 1u;        // SB: state rows of this block
    __shared__ float s_q[S], s_k[S], s_v[SB], s_core[SB], s_beta, s_gate;
    __shared__ double red[8], red2[8];
    const uint32_t h = blockIdx.x / SPLIT, part = blockIdx.x % SPLIT, seq = blockIdx.y, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t width = D.rank / D.groups, kh = h / width, first = h - kh * width == 0u && part == 0u, taps = DC ? DC : D.d_conv, ns = taps - 1u;
    // conv channels of this thread: threads 0 .. S-1 the q channels, S .. 2S-1 the k channels of the key head; then 0 .. SB-1 the v channels of the block's rows
    const bool has_qk = tid < 2u * S, has_v = tid < SB;
    const uint32_t c_qk = (tid < S ? kh * S + tid : (D.groups + kh) * S + tid - S), c_v = 2u * D.groups * S + h * S + part * SB + tid;
    float *const cs_base = conv_state + (size_t)seq * D.channels * ns;
    const float *const x_base = qkv + (size_t)seq * D.channels;
    float wq[TAPS], kq[TAPS], wv[TAPS], kv_[TAPS];                 // window + new sample, and the taps
    auto window = [&](uint32_t c, float (&w)[TAPS], float (&k)[TAPS]) {
#pragma unroll
        for (uint32_t j = 0; j < TAPS; ++j) { w[j] = j + 1u < TAPS ? cs_base[(size_t)c * ns + j] : x_base[c]; k[j] = conv_kernel[(size_t)c * taps + j]; }
    };
    if (DC && has_qk) window(c_qk, wq, kq);
    if (DC && has_v) window(c_v, wv, kv_);
    float *rows = state + (((size_t)seq * D.rank + h) * S + part * SB + (size_t)warp * RPW) * S;
    float m[RING][VPL];
    // volatile asm keeps these loads where they are written: all of them are issued before the first row is worked on
    // (left to itself the compiler fetches each row just before its use, with one row in flight per warp)
#pragma unroll
    for (uint32_t r = 0; r < RING; ++r)
#pragma unroll
        for (int t = 0; t < VPL; ++t) asm volatile("ld.global.f32 %0, [%1];" : "=f"(m[r][t]) : "l"(rows + (size_t)r * S + lane + 32 * t));
    __syncwarp();                      // a fixed point between the requests above and the shuffles below
    auto conv_silu = [&](uint32_t c, const float (&w)[TAPS], const float (&k)[TAPS]) {
        double acc = 0.0;
        if (DC) {
#pragma unroll
            for (uint32_t j = 0; j < TAPS; ++j) acc += (double)w[j] * (double)k[j];
        } else {
            for (uint32_t j = 0; j < ns; ++j) acc += (double)cs_base[(size_t)c * ns + j] * (double)conv_kernel[(size_t)c * taps + j];
            acc += (double)x_base[c] * (double)conv_kernel[(size_t)c * taps + ns];
        }
        return (float)(acc / (1.0 + exp(-acc)));
    };
    auto roll = [&](uint32_t c) {
        float *cs = cs_base + (size_t)c * ns;
        const float newest = x_base[c];
        for (uint32_t j = 0; j + 1u < ns; ++j) cs[j] = cs[j + 1u];
        cs[ns - 1u] = newest;
    };
    // used at the end: on its way with the rest
    const size_t idx = (size_t)seq * D.d_inner + (size_t)h * S + part * SB + tid;
    const float g = tid < SB ? z[idx] : 0.f;
    const float y = has_qk ? conv_silu(c_qk, wq, kq) : 0.f;
    __syncwarp();
    if (SPLIT > 1u || width > 1u) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");       // this block has read the key head's windows
    double ss = (double)y * (double)y;
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    if (has_v) { s_v[tid] = conv_silu(c_v, wv, kv_); roll(c_v); }
    else if (tid == S || tid == S + 32u) {          // beta and gate: one thread each, in warps that have no v channels
        const float *b = ba + (size_t)seq * 2u * D.rank + kh * 2u * width + (h - kh * width);
        if (tid == S) s_beta = (float)sigmoid_stable((double)b[0]);
        else s_gate = (float)(softplus_stable((double)b[width] + (double)dt_bias[h]) * (double)ssm_a[h]);
    }
    __syncthreads();
    if (has_qk) {
        const uint32_t w0 = tid < S ? 0u : S / 32u;
        double tot = 0.0;
        for (uint32_t w = 0; w < S / 32u; ++w) tot += red[w0 + w];
        const double inv = 1.0 / fmax(sqrt(tot), (double)D.eps);
        (tid < S ? s_q : s_k)[tid < S ? tid : tid - S] = (float)((double)y * inv);
    }
    __syncwarp();
    if (SPLIT > 1u || width > 1u) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (first && has_qk) roll(c_qk);
    __syncthreads();
    float qv[VPL], kv[VPL];
#pragma unroll
    for (int t = 0; t < VPL; ++t) { qv[t] = s_q[lane + 32 * t]; kv[t] = s_k[lane + 32 * t]; }
    const float decay = expf(s_gate), bh = s_beta, scale = 1.0f / sqrtf((float)S);
#pragma unroll
    for (uint32_t r = 0; r < RPW; ++r) {
        float sum = 0.f;
#pragma unroll
        for (int t = 0; t < VPL; ++t) { m[r % RING][t] = m[r % RING][t] * decay; sum += m[r % RING][t] * kv[t]; }
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float delta = (s_v[warp * RPW + r] - sum) * bh;
        float o_acc = 0.f;
#pragma unroll
        for (int t = 0; t < VPL; ++t) { m[r % RING][t] += kv[t] * delta; o_acc += m[r % RING][t] * qv[t]; rows[(size_t)r * S + lane + 32 * t] = m[r % RING][t]; }
        if (r + RING < RPW) {
#pragma unroll
            for (int t = 0; t < VPL; ++t) asm volatile("ld.global.f32 %0, [%1];" : "=f"(m[r % RING][t]) : "l"(rows + (size_t)(r + RING) * S + lane + 32 * t));
        }
        for (int o = 16; o; o >>= 1) o_acc += __shfl_xor_sync(0xffffffffu, o_acc, o);
        if (lane == 0) s_core[warp * RPW + r] = o_acc * scale;
    }
    __syncthreads();
    // gated RMSNorm over the head (the arithmetic of k_dn_tail)
    float x = 0.f;
    ss = 0.0;
    if (tid < SB) { x = s_core[tid]; ss = (double)x * (double)x; }
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (SPLIT == 1u) {
        if (lane == 0) red2[warp] = ss;
        __syncthreads();
    } else {
        // the head's sum of squares from all of its blocks: each hands its warps' parts to every block of the head
        if (lane == 0 && warp < SB / 32u) {
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(&red2[part * (SB / 32u) + warp]), rank0 = (h - kh * width) * SPLIT;
#pragma unroll
            for (uint32_t p = 0; p < SPLIT; ++p) {
                uint32_t peer;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(rank0 + p));
                asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(peer), "d"(ss) : "memory");
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (tid < SB) {
        double tot = 0.0;
        for (uint32_t w = 0; w < S / 32u; ++w) tot += red2[w];
        const float inv = 1.0f / sqrtf((float)(tot / (double)S) + D.eps);
        const float silu = g / (1.0f + expf(-g));
        out[idx] = x * inv * norm_w[part * SB + tid] * silu;
    }
}

// ---- sequence form: T consecutive tokens of ONE sequence (a prefill chunk) ----
// k_dn_prep_seq   grid (2*groups + d_inner/S + 1, T / 8): token t's conv window is the d_conv-1 samples before it (the conv
//                 state for times before the chunk, chunk rows after); the state itself is rolled by k_dn_conv_roll
// k_dn_state_seq  the delta rule over the T tokens with the state row held in registers: one read and one write of
//                 the state per chunk instead of per token; the next token's q/k/v/beta/gate are fetched while the
//                 current one is reduced
// A block serves DN_PREP_TOK consecutive tokens of its channel group: a thread keeps its channel's samples and results of all of them, so that a sample is
// read once and the eight L2 norms are reduced together, their roots taken by one thread each. Instruction issue bounds it (74 % of the slots, and three
// cycles of waiting for a result between two instructions of a warp; a quarter of them are of doubles, some 30 a value. With exp() and a division of doubles for every
// value, a root and a division in every thread and a barrier per token that was 65, and 119 us for 2048 tokens where this takes 66).
constexpr uint32_t DN_PREP_TOK = 8u;

__global__ void __launch_bounds__(256) k_dn_prep_seq(DnDims D, uint32_t T, const float *__restrict__ conv_kernel, const float *__restrict__ dt_bias, const float *__restrict__ ssm_a,
                                                     const float *qkv, const float *ba, const float *conv_state,
                                                     float *__restrict__ qk, float *__restrict__ v, float *__restrict__ beta, float *__restrict__ gate) {
    pdl_prologue();
    __shared__ double red[8][DN_PREP_TOK], s_inv[DN_PREP_TOK];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, S = D.S, ns = D.d_conv - 1u;
    const uint32_t n_qk = 2u * D.groups, n_v = D.d_inner / S;
    const uint32_t t_begin = blockIdx.y * DN_PREP_TOK, n = min(DN_PREP_TOK, T - t_begin);
    if (blockIdx.x == n_qk + n_v) {
        const uint32_t width = D.rank / D.groups, stride = 2u * width;
        for (uint32_t i = tid; i < n * D.rank; i += blockDim.x) {
            const uint32_t ti = t_begin + i / D.rank, h = i % D.rank, g = h / width, l = h - g * width;
            const float *b = ba + (size_t)ti * 2u * D.rank;
            beta[(size_t)ti * D.rank + h] = (float)sigmoid_stable((double)b[g * stride + l]);
            gate[(size_t)ti * D.rank + h] = (float)(softplus_stable((double)b[g * stride + width + l] + (double)dt_bias[h]) * (double)ssm_a[h]);
        }
        return;
    }
    const uint32_t c = blockIdx.x * S + tid;
    const float *cs = conv_state + (size_t)c * ns;
    const float *kr = conv_kernel + (size_t)c * D.d_conv;
    auto sample = [&](int tau) { return tau < 0 ? cs[(int)ns + tau] : qkv[(size_t)tau * D.channels + c]; };        // tau: time relative to the chunk start
    float y[DN_PREP_TOK];
    if (D.d_conv == 4u) {                                  // the window slides over registers
        float x[DN_PREP_TOK + 3u];
#pragma unroll
        for (uint32_t i = 0; i < DN_PREP_TOK + 3u; ++i) x[i] = i < n + 3u ? sample((int)(t_begin + i) - 3) : 0.f;
        const double k0 = (double)kr[0], k1 = (double)kr[1], k2 = (double)kr[2], k3 = (double)kr[3];
#pragma unroll
        for (uint32_t i = 0; i < DN_PREP_TOK; ++i) y[i] = (float)silu_d(fma((double)x[i + 3u], k3, fma((double)x[i + 2u], k2, fma((double)x[i + 1u], k1, (double)x[i] * k0))));
    } else {
#pragma unroll
        for (uint32_t i = 0; i < DN_PREP_TOK; ++i) {
            double acc = 0.0;
            if (i < n) for (uint32_t j = 0; j <= ns; ++j) acc = fma((double)sample((int)(t_begin + i + j) - (int)ns), (double)kr[j], acc);
            y[i] = (float)silu_d(acc);
        }
    }
    if (blockIdx.x >= n_qk) {
#pragma unroll
        for (uint32_t i = 0; i < DN_PREP_TOK; ++i) if (i < n) v[(size_t)(t_begin + i) * D.d_inner + (c - n_qk * S)] = y[i];
        return;
    }
    // the sums of the eight tokens over the warp: while a lane carries more than one, each exchange halves them
    double a4[4], a2[2], a1;
    const bool hi4 = lane & 16u, hi3 = lane & 8u, hi2 = lane & 4u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double lo = (double)y[i] * (double)y[i], hi = (double)y[i + 4] * (double)y[i + 4];
        a4[i] = (hi4 ? hi : lo) + __shfl_xor_sync(0xffffffffu, hi4 ? lo : hi, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) a2[i] = (hi3 ? a4[i + 2] : a4[i]) + __shfl_xor_sync(0xffffffffu, hi3 ? a4[i] : a4[i + 2], 8);
    a1 = (hi2 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, hi2 ? a2[0] : a2[1], 4);
    a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
    a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
    if ((lane & 3u) == 0u) red[tid >> 5][((lane >> 4) & 1u) * 4u + ((lane >> 3) & 1u) * 2u + ((lane >> 2) & 1u)] = a1;
    __syncthreads();
    if (tid < DN_PREP_TOK) {
        double tot = 0.0;
        for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) tot += red[w][tid];
        s_inv[tid] = 1.0 / fmax(sqrt(tot), (double)D.eps);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < DN_PREP_TOK; ++i) if (i < n) qk[(size_t)(t_begin + i) * n_qk * S + c] = (float)((double)y[i] * s_inv[i]);
}

// the gated RMSNorm of a chunk (the arithmetic of k_dn_tail): a warp per token and value head, VPL values a lane. grid = tokens * heads / 8; the rows are the
// engine's, so aligned. A block of S threads per row with a barrier in it was bound by the scheduling of its blocks: 59 us for 2048 tokens, now 15
template <uint32_t VPL>
__global__ void __launch_bounds__(256) k_dn_tail_seq(DnDims D, uint32_t rows, const float *core, const float *z, const float *norm_w, float *__restrict__ out) {
    pdl_prologue();
    const uint32_t r = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (r >= rows) return;
    const size_t idx = (size_t)r * (VPL * 32u) + lane * VPL;
    struct __align__(VPL > 4u ? 16u : VPL * 4u) Vec { float f[VPL]; };
    const Vec x = *reinterpret_cast<const Vec *>(core + idx), g = *reinterpret_cast<const Vec *>(z + idx);
    double ss = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < VPL; ++i) ss = fma((double)x.f[i], (double)x.f[i], ss);
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.0f / sqrtf((float)(ss / (double)(VPL * 32u)) + D.eps);
    Vec o;
#pragma unroll
    for (uint32_t i = 0; i < VPL; ++i) o.f[i] = x.f[i] * inv * __ldg(norm_w + lane * VPL + i) * (g.f[i] / (1.0f + expf(-g.f[i])));
    *reinterpret_cast<Vec *>(out + idx) = o;
}

// conv state <- the last d_conv-1 samples of [state, chunk]; one thread per channel
__global__ void k_dn_conv_roll(DnDims D, uint32_t T, const float *qkv, float *__restrict__ conv_state) {
    pdl_prologue();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x, ns = D.d_conv - 1u;
    if (c >= D.channels) return;
    float *cs = conv_state + (size_t)c * ns;
    for (uint32_t j = 0; j < ns; ++j) {                     // ascending: a kept sample moves down, so its source is still intact
        const int tau = (int)T + (int)j - (int)ns;
        cs[j] = tau < 0 ? cs[(int)ns + tau] : qkv[(size_t)tau * D.channels + c];
    }
}

// Block = 8 warps = 8 consecutive state rows of ONE value head, so the eight warps need the same q / k rows and the same
// beta / gate of every token: they are staged in shared memory TB tokens at a time by cp.async, one token block ahead
// of the one being applied (a warp that fetched them itself waited for L2 on every token of its sequential chain).
constexpr uint32_t DN_TB = 8u;          // tokens per staged block
template <int VPL>
__global__ void __launch_bounds__(256) k_dn_state_seq(DnDims D, uint32_t T, const float *qk, const float *v,
                                                      const float *beta, const float *gate,
                                                      float *__restrict__ state, float *__restrict__ core) {
    pdl_prologue();
    constexpr uint32_t S = VPL * 32u;
    __shared__ __align__(16) float s_q[2][DN_TB][S], s_k[2][DN_TB][S];
    __shared__ __align__(16) float s_v[2][DN_TB][8];
    __shared__ float s_b[2][DN_TB], s_g[2][DN_TB];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t row0 = blockIdx.x * 8u;                       // first of the block's 8 rows, counted over (head, j)
    const uint32_t h = row0 / S, j0 = row0 - h * S, j = j0 + warp;
    const uint32_t kh = h / (D.rank / D.groups);
    const size_t tok_qk = (size_t)2u * D.groups * S;
    const float *q = qk + (size_t)kh * S, *k = qk + (size_t)(D.groups + kh) * S;
    float *row = state + ((size_t)h * S + j) * S;
    const float scale = 1.0f / sqrtf((float)S);

    auto stage = [&](uint32_t tb, uint32_t buf) {               // tokens [tb * DN_TB, ...) -> buffer buf
        const uint32_t t0 = tb * DN_TB, n = min(DN_TB, T - t0);
        constexpr uint32_t V4 = S / 4u;                          // float4 per q or k row
        for (uint32_t i = tid; i < 2u * n * V4; i += 256u) {
            const uint32_t which = i / (n * V4), r = i - which * n * V4, tt = r / V4, c = (r - tt * V4) * 4u;
            const float *src = (which ? k : q) + (size_t)(t0 + tt) * tok_qk + c;
            float *dst = (which ? &s_k[buf][tt][0] : &s_q[buf][tt][0]) + c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
        }
        for (uint32_t i = tid; i < n * 2u; i += 256u) {          // v of the block's 8 rows: 32 bytes per token
            const uint32_t tt = i >> 1, c = (i & 1u) * 4u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(&s_v[buf][tt][c])),
                         "l"(v + (size_t)(t0 + tt) * D.d_inner + (size_t)h * S + j0 + c) : "memory");
        }
        for (uint32_t i = tid; i < n * 2u; i += 256u) {
            const uint32_t tt = i >> 1;
            const float *src = (i & 1u ? gate : beta) + (size_t)(t0 + tt) * D.rank + h;
            float *dst = i & 1u ? &s_g[buf][tt] : &s_b[buf][tt];
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float m[VPL];
#pragma unroll
    for (int t = 0; t < VPL; ++t) m[t] = row[lane + 32 * t];
    const uint32_t nblk = (T + DN_TB - 1u) / DN_TB;
    stage(0u, 0u);
    for (uint32_t tb = 0; tb < nblk; ++tb) {
        const uint32_t buf = tb & 1u, n = min(DN_TB, T - tb * DN_TB);
        if (tb + 1u < nblk) stage(tb + 1u, buf ^ 1u); else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                         // block tb has landed for every warp
        // Off the token-to-token dependency chain: the block's eight decays are computed once (lane l holds token l % 8's) and
        // the output dot products are only reduced after the eight tokens, all together.
        const float dec_l = expf(s_g[buf][lane & (DN_TB - 1u)]);
        float op[DN_TB];
#pragma unroll
        for (uint32_t tt = 0; tt < DN_TB; ++tt) {
            op[tt] = 0.f;
            if (tt < n) {
                const float decay = __shfl_sync(0xffffffffu, dec_l, (int)tt);
                float kc[VPL];
                float sum = 0.f;
#pragma unroll
                for (int t = 0; t < VPL; ++t) { kc[t] = s_k[buf][tt][lane + 32 * t]; m[t] = m[t] * decay; sum += m[t] * kc[t]; }
                for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                const float delta = (s_v[buf][tt][warp] - sum) * s_b[buf][tt];
                float o_acc = 0.f;
#pragma unroll
                for (int t = 0; t < VPL; ++t) { m[t] += kc[t] * delta; o_acc += m[t] * s_q[buf][tt][lane + 32 * t]; }
                op[tt] = o_acc;
            }
        }
        {   // eight sums across the warp with the pairing of the plain butterfly (16, 8, 4, 2, 1), but each exchange halves the
            // values a lane carries: 4 + 2 + 1 + 1 + 1 shuffles instead of 8 x 5. Value i ends up in the lanes whose bits 4, 3, 2 spell i.
            const bool hi4 = lane & 16u, hi3 = lane & 8u, hi2 = lane & 4u;
            float a4[4], a2[2], a1;
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float keep = hi4 ? op[4 + i] : op[i], send = hi4 ? op[i] : op[4 + i]; a4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16); }
#pragma unroll
            for (int i = 0; i < 2; ++i) { const float keep = hi3 ? a4[2 + i] : a4[i], send = hi3 ? a4[i] : a4[2 + i]; a2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8); }
            { const float keep = hi2 ? a2[1] : a2[0], send = hi2 ? a2[0] : a2[1]; a1 = keep + __shfl_xor_sync(0xffffffffu, send, 4); }
            a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
            a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
            const uint32_t ti = ((lane >> 4) & 1u) * 4u + ((lane >> 3) & 1u) * 2u + ((lane >> 2) & 1u);
            if ((lane & 3u) == 0u && ti < n) core[(size_t)(tb * DN_TB + ti) * D.d_inner + (size_t)h * S + j] = a1 * scale;
        }
        __syncthreads();                                         // buffer buf may be refilled by the next stage() call
    }
#pragma unroll
    for (int t = 0; t < VPL; ++t) row[lane + 32 * t] = m[t];
}

// ---- the same token-by-token recurrence with a lane group per row (the default scan) -----------------------------------
// k_dn_state_seq spreads ONE row over the 32 lanes of a warp: per token a warp issues about 50 instructions for 4 x 128
// multiply-adds, ten of them the two five-step reductions, and every SM carries 32 such warps. Here LPR = S / CPT lanes
// share a row (CPT columns each, as float4 pieces interleaved over the lanes so that a quarter warp reads 128 contiguous
// bytes of k or q), a thread carries RPT rows (k and q, read from shared memory once, serve all of them: the shared-memory
// pipe delivers 128 bytes per cycle whether or not lanes read the same address, and with one row per thread it was busier
// than the fp32 pipe), the row's partial sums meet in ONE exchange step, and the arithmetic is packed fp32 (two columns
// per instruction). Per element it is the reference's (decay the row, dot with k, add k * delta, dot with q:
// native/redlite_native_engine_cpu.c:198-216); only the order of the sums inside a dot product differs. Whole blocks of
// eight tokens run through a branch-free unrolled body; the block's decays, betas and v are fetched before its first
// token, a token's q and the next token's k before the exchange that the chain waits for, and the eight output sums are
// reduced together after the block. RC_DN_SCAN=warp selects k_dn_state_seq for comparison.
// What bounds it is one warp per scheduler with a chain of about 400 cycles a token, 161 instructions of which 64 are packed fp32 (two cycles each). One
// block an SM is said to the compiler (the second launch bound): it then takes 206 registers instead of 128 and has loads and the rows' chains further ahead.
// With the token in two halves over arrays of the rows, up to the exchange and from it: 2048 tokens 501 -> 447 us (471 by the bound alone); 512 tokens
// of states 256, 64, 32 wide 224 -> 214, 129 -> 121, 77 -> 70. The same to the bit. Tried on that: k of eight tokens as separate values 473; one exchange of three
// steps for both rows 492; one barrier a block with a third buffer 484; loads pinned to their token 455; the rows half a token apart: the same code.
template <uint32_t S, uint32_t CPT, uint32_t RPT, uint32_t WARPS>
__global__ void __launch_bounds__(WARPS * 32u, 1) k_dn_scan(DnDims D, uint32_t T, const float *qk, const float *v,
                                                         const float *beta, const float *gate,
                                                         float *__restrict__ state, float *__restrict__ core) {
    pdl_prologue();
    constexpr uint32_t LPR = S / CPT, RPW = 32u / LPR, RB = RPW * RPT * WARPS, NP = CPT / 4u, NT = WARPS * 32u, V4 = S / 4u;
    static_assert(LPR == 2u || LPR == 4u || LPR == 8u || LPR == 16u || LPR == 32u, "lanes per row");
    static_assert(S % RB == 0u && RB % 4u == 0u && DN_TB == 8u && RPT <= 2u, "rows per block");
    __shared__ __align__(16) float s_q[2][DN_TB][S], s_k[2][DN_TB][S];
    __shared__ __align__(16) float s_v[2][RB][DN_TB];            // v by (row, token): a thread reads its row's eight values as two float4
    __shared__ __align__(16) float s_b[2][DN_TB], s_g[2][DN_TB];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, p = lane % LPR, r = lane / LPR;
    const uint32_t h = blockIdx.x / (S / RB), j0 = (blockIdx.x % (S / RB)) * RB;     // head, first of the block's RB rows
    const uint32_t jr = (warp * RPW + r) * RPT;                                      // this thread's first row inside the block
    const uint32_t kh = h / (D.rank / D.groups);
    const size_t tok_qk = (size_t)2u * D.groups * S;
    const float *q = qk + (size_t)kh * S, *k = qk + (size_t)(D.groups + kh) * S;
    float *rows = state + ((size_t)h * S + j0 + jr) * S;
    const float scale = 1.0f / sqrtf((float)S);

    auto stage = [&](uint32_t tb, uint32_t buf) {               // tokens [tb * DN_TB, ...) -> buffer buf
        const uint32_t t0 = tb * DN_TB, n = min(DN_TB, T - t0);
        for (uint32_t i = tid; i < 2u * DN_TB * V4; i += NT) {
            const uint32_t which = i / (DN_TB * V4), tt = (i / V4) % DN_TB, c = (i % V4) * 4u;
            if (tt < n) {
                const float *src = (which ? k : q) + (size_t)(t0 + tt) * tok_qk + c;
                float *dst = (which ? &s_k[buf][tt][0] : &s_q[buf][tt][0]) + c;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
            }
        }
        for (uint32_t i = tid; i < DN_TB * RB; i += NT) {
            const uint32_t tt = i / RB, rr = i % RB;
            if (tt < n)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(&s_v[buf][rr][tt])),
                             "l"(v + (size_t)(t0 + tt) * D.d_inner + (size_t)h * S + j0 + rr) : "memory");
        }
        for (uint32_t i = tid; i < DN_TB * 2u; i += NT) {
            const uint32_t tt = i >> 1;
            if (tt < n) {
                const float *src = (i & 1u ? gate : beta) + (size_t)(t0 + tt) * D.rank + h;
                float *dst = i & 1u ? &s_g[buf][tt] : &s_b[buf][tt];
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float2 m[RPT][CPT / 2u];                                     // the rows as register pairs: the arithmetic is packed fp32 (two lanes per instruction)
#pragma unroll
    for (uint32_t a = 0; a < RPT; ++a)
#pragma unroll
        for (uint32_t i = 0; i < NP; ++i) {
            const float4 x = *reinterpret_cast<const float4 *>(rows + (size_t)a * S + 4u * (i * LPR + p));
            m[a][2u * i] = make_float2(x.x, x.y); m[a][2u * i + 1u] = make_float2(x.z, x.w);
        }

    auto body = [&](auto full_c, uint32_t buf, uint32_t n, uint32_t t0) {
        constexpr bool FULL = decltype(full_c)::value;
        // the block's scalars first, off the token-to-token chain: eight decays (lane l computes token l % 8's), betas and this
        // thread's v (entries of tokens >= n are stale and never used)
        float dec[DN_TB], bt[DN_TB], vv[RPT][DN_TB];
        {
            const float dec_l = expf(s_g[buf][lane & (DN_TB - 1u)]);
#pragma unroll
            for (uint32_t tt = 0; tt < DN_TB; ++tt) dec[tt] = __shfl_sync(0xffffffffu, dec_l, (int)tt);
            const float4 b0 = *reinterpret_cast<const float4 *>(&s_b[buf][0]), b1 = *reinterpret_cast<const float4 *>(&s_b[buf][4]);
            bt[0] = b0.x; bt[1] = b0.y; bt[2] = b0.z; bt[3] = b0.w; bt[4] = b1.x; bt[5] = b1.y; bt[6] = b1.z; bt[7] = b1.w;
#pragma unroll
            for (uint32_t a = 0; a < RPT; ++a) {
                const float4 v0 = *reinterpret_cast<const float4 *>(&s_v[buf][jr + a][0]), v1 = *reinterpret_cast<const float4 *>(&s_v[buf][jr + a][4]);
                vv[a][0] = v0.x; vv[a][1] = v0.y; vv[a][2] = v0.z; vv[a][3] = v0.w; vv[a][4] = v1.x; vv[a][5] = v1.y; vv[a][6] = v1.z; vv[a][7] = v1.w;
            }
        }
        float op[RPT][DN_TB], x[RPT][LPR <= 8u ? LPR : 1u];
        float4 kk[2][NP], qq[NP];                                // k by token parity
        auto load = [&](float4 (&to)[NP], const float *from) {
#pragma unroll
            for (uint32_t i = 0; i < NP; ++i) to[i] = *reinterpret_cast<const float4 *>(from + 4u * (i * LPR + p));
        };
        auto dot = [&](const float2 (&mr)[CPT / 2u], const float4 (&c)[NP]) {
            float2 s2 = __fmul2_rn(mr[0], make_float2(c[0].x, c[0].y));
            if constexpr (NP == 1u) {
                s2 = __ffma2_rn(mr[1], make_float2(c[0].z, c[0].w), s2);
            } else {
                float2 pb = __fmul2_rn(mr[1], make_float2(c[0].z, c[0].w));
#pragma unroll
                for (uint32_t i = 1; i < NP; ++i) {
                    s2 = __ffma2_rn(mr[2u * i], make_float2(c[i].x, c[i].y), s2);
                    pb = __ffma2_rn(mr[2u * i + 1u], make_float2(c[i].z, c[i].w), pb);
                }
                s2 = __fadd2_rn(s2, pb);
            }
            return s2.x + s2.y;
        };
        // row a, token tt, up to the exchange: decay, dot with k, partial sums on their way
        auto begin = [&](uint32_t a, uint32_t tt) {
            const float2 d2 = make_float2(dec[tt], dec[tt]);
#pragma unroll
            for (uint32_t i = 0; i < 2u * NP; ++i) m[a][i] = __fmul2_rn(m[a][i], d2);
            float sum = dot(m[a], kk[tt & 1u]);
            if constexpr (LPR <= 8u) {
                // one exchange step instead of log2(LPR) dependent ones: every lane of the row fetches all LPR partial sums
                // and adds them in the same order (so the row's lanes agree to the bit)
#pragma unroll
                for (uint32_t l = 0; l < LPR; ++l) x[a][l] = __shfl_sync(0xffffffffu, sum, (int)((lane & ~(LPR - 1u)) + l));
            } else {
#pragma unroll
                for (uint32_t o = LPR / 2u; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, (int)o);
                x[a][0] = sum;
            }
        };
        // ... and from there: correction, update, dot with q
        auto finish = [&](uint32_t a, uint32_t tt) {
            if constexpr (LPR <= 8u) {
#pragma unroll
                for (uint32_t w = LPR; w > 1u; w >>= 1)
#pragma unroll
                    for (uint32_t l = 0; l < w / 2u; ++l) x[a][l] = x[a][2u * l] + x[a][2u * l + 1u];
            }
            const float delta = (vv[a][tt] - x[a][0]) * bt[tt];
            const float2 e2 = make_float2(delta, delta);
#pragma unroll
            for (uint32_t i = 0; i < NP; ++i) {
                m[a][2u * i] = __ffma2_rn(make_float2(kk[tt & 1u][i].x, kk[tt & 1u][i].y), e2, m[a][2u * i]);
                m[a][2u * i + 1u] = __ffma2_rn(make_float2(kk[tt & 1u][i].z, kk[tt & 1u][i].w), e2, m[a][2u * i + 1u]);
            }
            op[a][tt] = dot(m[a], qq);
        };
        load(kk[0], &s_k[buf][0][0]);
#pragma unroll
        for (uint32_t tt = 0; tt < DN_TB; ++tt) {
#pragma unroll
            for (uint32_t a = 0; a < RPT; ++a) op[a][tt] = 0.f;
        }
#pragma unroll
        for (uint32_t tt = 0; tt < DN_TB; ++tt) {
            if (FULL || tt < n) {
                // this token's q and the next token's k are requested before the exchange that the chain waits for
                load(qq, &s_q[buf][tt][0]);
                if (tt + 1u < DN_TB) load(kk[(tt + 1u) & 1u], &s_k[buf][tt + 1u][0]);
#pragma unroll
                for (uint32_t a = 0; a < RPT; ++a) begin(a, tt);
#pragma unroll
                for (uint32_t a = 0; a < RPT; ++a) finish(a, tt);
            }
        }
        // the eight output sums over the row's LPR lanes: while a lane carries more than one value each exchange halves them,
        // so a lane ends with max(1, 8 / LPR) finished tokens (first token `tok`) instead of every lane reducing all eight
        constexpr uint32_t LOW = LPR > DN_TB ? LPR / DN_TB - 1u : 0u;     // lane bits below the halving exchanges: those lanes hold copies
#pragma unroll
        for (uint32_t a = 0; a < RPT; ++a) {
            uint32_t tok = 0u, cnt = DN_TB;
#pragma unroll
            for (uint32_t o = LPR / 2u; o; o >>= 1) {
                if (cnt > 1u) {
                    cnt >>= 1;
                    const bool hi = p & o;
#pragma unroll
                    for (uint32_t i = 0; i < DN_TB / 2u; ++i)
                        if (i < cnt) {
                            const float keep = hi ? op[a][cnt + i] : op[a][i], send = hi ? op[a][i] : op[a][cnt + i];
                            op[a][i] = keep + __shfl_xor_sync(0xffffffffu, send, (int)o);
                        }
                    if (hi) tok += cnt;
                } else {
                    op[a][0] += __shfl_xor_sync(0xffffffffu, op[a][0], (int)o);
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < (LPR < DN_TB ? DN_TB / LPR : 1u); ++i)
                if ((p & LOW) == 0u && (FULL || tok + i < n)) core[(size_t)(t0 + tok + i) * D.d_inner + (size_t)h * S + j0 + jr + a] = op[a][i] * scale;
        }
    };

    const uint32_t nblk = (T + DN_TB - 1u) / DN_TB;
    stage(0u, 0u);
    for (uint32_t tb = 0; tb < nblk; ++tb) {
        const uint32_t buf = tb & 1u, n = min(DN_TB, T - tb * DN_TB);
        if (tb + 1u < nblk) stage(tb + 1u, buf ^ 1u); else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                         // block tb has landed for every warp
        if (n == DN_TB) body(std::true_type{}, buf, n, tb * DN_TB); else body(std::false_type{}, buf, n, tb * DN_TB);
        __syncthreads();                                         // buffer buf may be refilled by the next stage() call
    }
#pragma unroll
    for (uint32_t a = 0; a < RPT; ++a)
#pragma unroll
        for (uint32_t i = 0; i < NP; ++i)
            *reinterpret_cast<float4 *>(rows + (size_t)a * S + 4u * (i * LPR + p)) =
                make_float4(m[a][2u * i].x, m[a][2u * i].y, m[a][2u * i + 1u].x, m[a][2u * i + 1u].y);
}

// ---- the same recurrence four tokens at a time -------------------------------------------------------------------
// Inside a group of four tokens the corrections delta_t depend on each other only through the scalars k_s . k_t, which are
// the same for every state row of a head. With d_t the per-token decay, g_t = d_1 ... d_t, r(t,s) = d_{s+1} ... d_t and
// m the row before the group:
//   delta_t = beta_t (v_t - g_t (m . k_t) - sum_{s<t} r(t,s) (k_s . k_t) delta_s)
//   out_t   = scale (g_t (m . q_t) + sum_{s<=t} r(t,s) (k_s . q_t) delta_s)
//   m      <- g_4 m + sum_s r(4,s) delta_s k_s
// (the delta rule of native/redlite_native_engine_cpu.c:198-216 unrolled over four steps; the sums are reassociated,
// nothing else changes). A warp therefore needs ONE round of reductions per four tokens — the eight dot products of the
// row with k_1..k_4 and q_1..q_4, reduced together — instead of two dependent reductions per token, which is what bounded
// the token-by-token kernel (a chain of about 1100 cycles per token and row).
// k_dn_pairdots  the 16 scalars of a group per key head: k_s . k_t (s < t) and k_s . q_t (s <= t); grid (groups of 4, key heads)
constexpr uint32_t DN_MC = 4u;
__global__ void __launch_bounds__(32) k_dn_pairdots(DnDims D, uint32_t T, const float *qk, float *__restrict__ pd) {
    pdl_prologue();
    const uint32_t c = blockIdx.x, kh = blockIdx.y, lane = threadIdx.x, S = D.S;
    const size_t tok_qk = (size_t)2u * D.groups * S;
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    for (uint32_t i = lane; i < S; i += 32u) {
        float q[4], k[4];
#pragma unroll
        for (uint32_t a = 0; a < 4u; ++a) {
            const uint32_t t = c * 4u + a;
            q[a] = t < T ? qk[(size_t)t * tok_qk + (size_t)kh * S + i] : 0.f;
            k[a] = t < T ? qk[(size_t)t * tok_qk + (size_t)(D.groups + kh) * S + i] : 0.f;
        }
        acc[0] += k[0] * k[1]; acc[1] += k[0] * k[2]; acc[2] += k[1] * k[2]; acc[3] += k[0] * k[3]; acc[4] += k[1] * k[3]; acc[5] += k[2] * k[3];
        acc[6] += k[0] * q[0]; acc[7] += k[0] * q[1]; acc[8] += k[1] * q[1]; acc[9] += k[0] * q[2]; acc[10] += k[1] * q[2]; acc[11] += k[2] * q[2];
        acc[12] += k[0] * q[3]; acc[13] += k[1] * q[3]; acc[14] += k[2] * q[3]; acc[15] += k[3] * q[3];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
        for (int o = 16; o; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    if (lane < 16u) {
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) if ((int)lane == i) v = acc[i];
        pd[((size_t)c * D.groups + kh) * 16u + lane] = v;
    }
}

// Block and staging as k_dn_state_seq (8 warps = 8 rows of one head, eight tokens staged at a time); T4 = the tokens that
// form whole groups of four (the caller runs the rest through k_dn_state_seq).
template <int VPL>
__global__ void __launch_bounds__(256) k_dn_state_seq4(DnDims D, uint32_t T4, const float *qk, const float *v,
                                                       const float *beta, const float *gate, const float *pd,
                                                       float *__restrict__ state, float *__restrict__ core) {
    pdl_prologue();
    constexpr uint32_t S = VPL * 32u;
    __shared__ __align__(16) float s_q[2][DN_TB][S], s_k[2][DN_TB][S];
    __shared__ __align__(16) float s_v[2][DN_TB][8];
    __shared__ __align__(16) float s_pd[2][DN_TB / DN_MC][16];
    __shared__ float s_b[2][DN_TB], s_g[2][DN_TB];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t row0 = blockIdx.x * 8u;
    const uint32_t h = row0 / S, j0 = row0 - h * S, j = j0 + warp;
    const uint32_t kh = h / (D.rank / D.groups);
    const size_t tok_qk = (size_t)2u * D.groups * S;
    const float *q = qk + (size_t)kh * S, *k = qk + (size_t)(D.groups + kh) * S;
    float *row = state + ((size_t)h * S + j) * S;
    const float scale = 1.0f / sqrtf((float)S);

    auto stage = [&](uint32_t tb, uint32_t buf) {               // tokens [tb * DN_TB, ...) -> buffer buf (T4 is a multiple of 4, so n is 4 or 8)
        const uint32_t t0 = tb * DN_TB, n = min(DN_TB, T4 - t0);
        constexpr uint32_t V4 = S / 4u;
        for (uint32_t i = tid; i < 2u * n * V4; i += 256u) {
            const uint32_t which = i / (n * V4), r = i - which * n * V4, tt = r / V4, c = (r - tt * V4) * 4u;
            const float *src = (which ? k : q) + (size_t)(t0 + tt) * tok_qk + c;
            float *dst = (which ? &s_k[buf][tt][0] : &s_q[buf][tt][0]) + c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
        }
        for (uint32_t i = tid; i < n * 2u; i += 256u) {
            const uint32_t tt = i >> 1, c = (i & 1u) * 4u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(&s_v[buf][tt][c])),
                         "l"(v + (size_t)(t0 + tt) * D.d_inner + (size_t)h * S + j0 + c) : "memory");
        }
        for (uint32_t i = tid; i < n * 2u; i += 256u) {
            const uint32_t tt = i >> 1;
            const float *src = (i & 1u ? gate : beta) + (size_t)(t0 + tt) * D.rank + h;
            float *dst = i & 1u ? &s_g[buf][tt] : &s_b[buf][tt];
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
        }
        for (uint32_t i = tid; i < (n / DN_MC) * 4u; i += 256u) {     // the groups' 16 scalars, 16 bytes per copy
            const uint32_t g = i >> 2, c = (i & 3u) * 4u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(&s_pd[buf][g][c])),
                         "l"(pd + ((size_t)(t0 / DN_MC + g) * D.groups + kh) * 16u + c) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float m[VPL];
#pragma unroll
    for (int t = 0; t < VPL; ++t) m[t] = row[lane + 32 * t];
    const uint32_t nblk = (T4 + DN_TB - 1u) / DN_TB;
    if (nblk) stage(0u, 0u);
    for (uint32_t tb = 0; tb < nblk; ++tb) {
        const uint32_t buf = tb & 1u, n = min(DN_TB, T4 - tb * DN_TB);
        if (tb + 1u < nblk) stage(tb + 1u, buf ^ 1u); else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        for (uint32_t g4 = 0; g4 < n / DN_MC; ++g4) {
            const uint32_t t0 = g4 * DN_MC;
            // ---- the row's eight dot products with k_1..k_4 (p[0..3]) and q_1..q_4 (p[4..7]), this lane's share
            float kc[4][VPL], p[8];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                float sk = 0.f, sq = 0.f;
#pragma unroll
                for (int t = 0; t < VPL; ++t) { kc[a][t] = s_k[buf][t0 + a][lane + 32 * t]; sk += m[t] * kc[a][t]; sq += m[t] * s_q[buf][t0 + a][lane + 32 * t]; }
                p[a] = sk; p[4 + a] = sq;
            }
            // ---- reduce the eight values together: each exchange halves the values a lane carries (4 + 2 + 1 shuffles), two
            // more finish the one that is left; value i ends up complete in the lanes whose bits 4, 3, 2 spell i
            {
                const bool hi4 = lane & 16u, hi3 = lane & 8u, hi2 = lane & 4u;
                float a4[4], a2[2], a1;
#pragma unroll
                for (int i = 0; i < 4; ++i) { const float keep = hi4 ? p[4 + i] : p[i], send = hi4 ? p[i] : p[4 + i]; a4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16); }
#pragma unroll
                for (int i = 0; i < 2; ++i) { const float keep = hi3 ? a4[2 + i] : a4[i], send = hi3 ? a4[i] : a4[2 + i]; a2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8); }
                { const float keep = hi2 ? a2[1] : a2[0], send = hi2 ? a2[0] : a2[1]; a1 = keep + __shfl_xor_sync(0xffffffffu, send, 4); }
                a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
                a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
#pragma unroll
                for (int i = 0; i < 8; ++i) p[i] = __shfl_sync(0xffffffffu, a1, ((i >> 2) & 1) * 16 + ((i >> 1) & 1) * 8 + (i & 1) * 4);
            }
            // ---- the four corrections and outputs (every lane computes them; they are scalars of the row)
            const float d0 = expf(s_g[buf][t0]), d1 = expf(s_g[buf][t0 + 1u]), d2 = expf(s_g[buf][t0 + 2u]), d3 = expf(s_g[buf][t0 + 3u]);
            const float g0 = d0, g1 = g0 * d1, g2 = g1 * d2, g3 = g2 * d3;
            const float r10 = d1, r21 = d2, r32 = d3, r20 = d1 * d2, r31 = d2 * d3, r30 = r20 * d3;
            const float4 pa = *reinterpret_cast<const float4 *>(&s_pd[buf][g4][0]), pb = *reinterpret_cast<const float4 *>(&s_pd[buf][g4][4]),
                         pc = *reinterpret_cast<const float4 *>(&s_pd[buf][g4][8]), pe = *reinterpret_cast<const float4 *>(&s_pd[buf][g4][12]);
            // pa = (k0.k1, k0.k2, k1.k2, k0.k3), pb = (k1.k3, k2.k3, k0.q0, k0.q1), pc = (k1.q1, k0.q2, k1.q2, k2.q2), pe = (k0.q3, k1.q3, k2.q3, k3.q3)
            const float e0 = (s_v[buf][t0][warp] - g0 * p[0]) * s_b[buf][t0];
            const float e1 = (s_v[buf][t0 + 1u][warp] - g1 * p[1] - r10 * pa.x * e0) * s_b[buf][t0 + 1u];
            const float e2 = (s_v[buf][t0 + 2u][warp] - g2 * p[2] - r20 * pa.y * e0 - r21 * pa.z * e1) * s_b[buf][t0 + 2u];
            const float e3 = (s_v[buf][t0 + 3u][warp] - g3 * p[3] - r30 * pa.w * e0 - r31 * pb.x * e1 - r32 * pb.y * e2) * s_b[buf][t0 + 3u];
            if (lane == 0) {
                const size_t o = (size_t)(tb * DN_TB + t0) * D.d_inner + (size_t)h * S + j;
                core[o] = (g0 * p[4] + pb.z * e0) * scale;
                core[o + D.d_inner] = (g1 * p[5] + r10 * pb.w * e0 + pc.x * e1) * scale;
                core[o + 2u * (size_t)D.d_inner] = (g2 * p[6] + r20 * pc.y * e0 + r21 * pc.z * e1 + pc.w * e2) * scale;
                core[o + 3u * (size_t)D.d_inner] = (g3 * p[7] + r30 * pe.x * e0 + r31 * pe.y * e1 + r32 * pe.z * e2 + pe.w * e3) * scale;
            }
            // ---- the row after the group
            const float c0 = r30 * e0, c1 = r31 * e1, c2 = r32 * e2;
#pragma unroll
            for (int t = 0; t < VPL; ++t) m[t] = g3 * m[t] + c0 * kc[0][t] + c1 * kc[1][t] + c2 * kc[2][t] + e3 * kc[3][t];
        }
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < VPL; ++t) row[lane + 32 * t] = m[t];
}

int launch_deltanet_seq(const DnDims &D, uint32_t T, const float *conv_kernel, const float *dt_bias, const float *ssm_a, const float *norm_w,
                        const float *qkv, const float *z, const float *ba, float *conv_state, float *rec_state,
                        float *qk, float *v, float *beta, float *gate, float *core, float *out, float *pairdots, cudaStream_t s) {
    RC_REQUIRE(D.S == 32u || D.S == 64u || D.S == 128u || D.S == 256u, "deltanet: state size %u not in {32,64,128,256}", D.S);
    RC_REQUIRE(D.rank && D.groups && D.rank % D.groups == 0 && D.d_inner == D.rank * D.S && D.channels == 2u * D.S * D.groups + D.d_inner && D.d_conv >= 2u,
               "deltanet: inconsistent dimensions");
    if (!T) return 1;
    prof_begin("dn_prep_seq", s);
    RC_LAUNCH((k_dn_prep_seq), dim3(2u * D.groups + D.d_inner / D.S + 1u, (T + DN_PREP_TOK - 1u) / DN_PREP_TOK), D.S, 0, s, D, T, conv_kernel, dt_bias, ssm_a, qkv, ba, (const float *)conv_state, qk, v, beta, gate);
    prof_end(s);
    RC_LAUNCHED();
    prof_begin("dn_conv_roll", s);
    RC_LAUNCH((k_dn_conv_roll), (D.channels + 255u) / 256u, 256, 0, s, D, T, qkv, conv_state);
    prof_end(s);
    RC_LAUNCHED();
    const uint32_t blocks = (D.rank * D.S + 7u) / 8u;
    // RC_DN_SCAN=grouped sends whole groups of four tokens through the grouped recurrence (the token-by-token kernel takes
    // the up to three tokens left over). Off by default: measured on 2048-token chunks it is 1.19x faster (0.98 against
    // 1.16 ms per layer — both forms execute about the same number of instructions) and its reassociated sums leave three
    // times the rounding noise at the 48th layer (1.8e-4 against 5.4e-5 of the layer output), which the full-depth router
    // comparison notices.
    const char *scan = getenv("RC_DN_SCAN");
    const bool grouped = scan && scan[0] == 'g';
    const uint32_t T4 = grouped && pairdots && D.S <= 128u ? T / DN_MC * DN_MC : 0u;
    if (T4) {
        prof_begin("dn_pairdots", s);
        RC_LAUNCH((k_dn_pairdots), dim3(T4 / DN_MC, D.groups), 32, 0, s, D, T4, (const float *)qk, pairdots);
        prof_end(s);
        RC_LAUNCHED();
        prof_begin("dn_state_seq4", s);
        switch (D.S) {
            case 32: RC_LAUNCH((k_dn_state_seq4<1>), blocks, 256, 0, s, D, T4, qk, v, beta, gate, (const float *)pairdots, rec_state, core); break;
            case 64: RC_LAUNCH((k_dn_state_seq4<2>), blocks, 256, 0, s, D, T4, qk, v, beta, gate, (const float *)pairdots, rec_state, core); break;
            default: RC_LAUNCH((k_dn_state_seq4<4>), blocks, 256, 0, s, D, T4, qk, v, beta, gate, (const float *)pairdots, rec_state, core); break;
        }
        prof_end(s);
        RC_LAUNCHED();
    }
    const bool per_warp = scan && scan[0] == 'w';                 // RC_DN_SCAN=warp: the one-row-per-warp kernel, for comparison
    if (T4 < T && !per_warp) {
        const uint32_t Tr = T - T4;
        const size_t tok_qk = (size_t)2u * D.groups * D.S;
        const float *qk_r = qk + (size_t)T4 * tok_qk, *v_r = v + (size_t)T4 * D.d_inner, *b_r = beta + (size_t)T4 * D.rank, *g_r = gate + (size_t)T4 * D.rank;
        float *core_r = core + (size_t)T4 * D.d_inner;
        prof_begin("dn_state_seq", s);
        switch (D.S) {
            case 32: RC_LAUNCH((k_dn_scan<32, 16, 1, 2>), D.rank, 64, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
            case 64: RC_LAUNCH((k_dn_scan<64, 16, 1, 8>), D.rank, 256, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
            // 128-wide states: two rows per thread halve the shared-memory reads of k and q per multiply-add; measured on 2048-token
            // chunks this tile takes 0.45 ms, one row of 16 or 32 columns per thread 0.52 and 0.48 ms, two rows of 8 columns 0.47 ms
            case 128: RC_LAUNCH((k_dn_scan<128, 16, 2, 4>), D.rank * 4u, 128, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
            default: RC_LAUNCH((k_dn_scan<256, 32, 1, 8>), D.rank * 8u, 256, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
        }
        prof_end(s);
        RC_LAUNCHED();
    } else if (T4 < T) {
        const uint32_t Tr = T - T4;
        const size_t tok_qk = (size_t)2u * D.groups * D.S;
        const float *qk_r = qk + (size_t)T4 * tok_qk, *v_r = v + (size_t)T4 * D.d_inner, *b_r = beta + (size_t)T4 * D.rank, *g_r = gate + (size_t)T4 * D.rank;
        float *core_r = core + (size_t)T4 * D.d_inner;
        prof_begin("dn_state_seq", s);
        switch (D.S) {
            case 32: RC_LAUNCH((k_dn_state_seq<1>), blocks, 256, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
            case 64: RC_LAUNCH((k_dn_state_seq<2>), blocks, 256, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
            case 128: RC_LAUNCH((k_dn_state_seq<4>), blocks, 256, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
            default: RC_LAUNCH((k_dn_state_seq<8>), blocks, 256, 0, s, D, Tr, qk_r, v_r, b_r, g_r, rec_state, core_r); break;
        }
        prof_end(s);
        RC_LAUNCHED();
    }
    prof_begin("dn_tail", s);
    const uint32_t rows = D.rank * T, tail_grid = (rows + 7u) / 8u;
    switch (D.S) {
        case 32: RC_LAUNCH((k_dn_tail_seq<1>), tail_grid, 256, 0, s, D, rows, (const float *)core, z, norm_w, out); break;
        case 64: RC_LAUNCH((k_dn_tail_seq<2>), tail_grid, 256, 0, s, D, rows, (const float *)core, z, norm_w, out); break;
        case 128: RC_LAUNCH((k_dn_tail_seq<4>), tail_grid, 256, 0, s, D, rows, (const float *)core, z, norm_w, out); break;
        default: RC_LAUNCH((k_dn_tail_seq<8>), tail_grid, 256, 0, s, D, rows, (const float *)core, z, norm_w, out); break;
    }
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

int launch_deltanet(const DnDims &D, uint32_t batch, const float *conv_kernel, const float *dt_bias, const float *ssm_a, const float *norm_w,
                    const float *qkv, const float *z, const float *ba, float *conv_state, float *rec_state,
                    float *qk, float *v, float *beta, float *gate, float *core, float *out, cudaStream_t s) {
    RC_REQUIRE(D.S >= 32u && D.S <= 256u && D.S % 32u == 0 && (D.S == 32u || D.S == 64u || D.S == 128u || D.S == 256u), "deltanet: state size %u not in {32,64,128,256}", D.S);
    RC_REQUIRE(D.rank && D.groups && D.rank % D.groups == 0 && D.d_inner == D.rank * D.S && D.channels == 2u * D.S * D.groups + D.d_inner && D.d_conv >= 2u,
               "deltanet: inconsistent dimensions");
    if (!batch) return 1;
    // one launch where a head's state fits the registers of a block and the value heads of a key head fit a cluster; else three.
    // Three also where out lies in qkv or ba: only the separate kernels have read all of those before the first output is written.
    const uint32_t width = D.rank / D.groups;
    auto overlap = [](const float *a, uint64_t na, const float *b, uint64_t nb) { return a < b + nb && b < a + na; };
    const uint64_t n_out = (uint64_t)batch * D.d_inner;
    const bool in_place = overlap(out, n_out, qkv, (uint64_t)batch * D.channels) || overlap(out, n_out, ba, (uint64_t)batch * 2u * D.rank);
    if (D.S <= 128u && width <= 8u && !in_place) {
        prof_begin("dn_step", s);
#define RC_DN_STEP(VPL, SPLIT, MINB, RING) do { const dim3 gs(D.rank * SPLIT, batch); \
        if (D.d_conv == 4u) RC_LAUNCH_CLUSTER(width * SPLIT, (k_dn_step<VPL, 4u, SPLIT, MINB, RING>), gs, 256, 0, s, D, conv_kernel, dt_bias, ssm_a, qkv, ba, conv_state, rec_state, z, norm_w, out); \
        else RC_LAUNCH_CLUSTER(width * SPLIT, (k_dn_step<VPL, 0u, SPLIT, MINB, RING>), gs, 256, 0, s, D, conv_kernel, dt_bias, ssm_a, qkv, ba, conv_state, rec_state, z, norm_w, out); } while (0)
        // Heads of 128: as many blocks per head as still fit the chip at once (3 blocks per SM with 4 or 8 rows a warp, 2 with 16) and
        // a cluster (8 blocks), since a second wave costs more than idle SMs and every block repeats the preparation. us a step
        // of 32 heads, graph-replayed, 1 / 3 / 4 / 6 / 8 / 10 sequences: 4 blocks 5.7 / 7.4 / 12.7 / 14.2 / 19.3 / 24.6, 2 blocks at
        // 2 per SM 6.6 / 8.1 / 8.4 / 15.0 / 15.9 / 22.0, 2 blocks at 3 per SM 6.7 / 9.1 / 9.6 / 10.1 / 16.3 / 18.0, one block 7.7 / 10.2 / 10.8 /
        // 11.4 / 11.9 / 18.5, one block at 3 per SM with half of its rows in flight 10.1 / 12.8 / 13.6 / 14.5 / 15.1 / 15.8 (the separate
        // kernels: 7.7 / 8.8 / 10.9 / 11.1 / 12.8 / 15.4).
        static int sms = 0;
        if (!sms) { int dev = 0; RC_CUDA(cudaGetDevice(&dev)); RC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)); }
        const uint64_t blocks = (uint64_t)D.rank * batch, two = 2u * (uint32_t)sms, three = 3u * (uint32_t)sms;
        if (D.S == 32u) RC_DN_STEP(1, 1u, 2, 4u);
        else if (D.S == 64u) RC_DN_STEP(2, 1u, 2, 8u);
        else if (width <= 2u && 4u * blocks <= three) RC_DN_STEP(4, 4u, 2, 4u);
        else if (width <= 4u && 2u * blocks <= two) RC_DN_STEP(4, 2u, 2, 8u);
        else if (width <= 4u && 2u * blocks <= three) RC_DN_STEP(4, 2u, 3, 8u);
        else if (blocks <= two) RC_DN_STEP(4, 1u, 2, 16u);
        else RC_DN_STEP(4, 1u, 3, 8u);
#undef RC_DN_STEP
        prof_end(s);
        RC_LAUNCHED();
        return 1;
    }
    const dim3 gp(2u * D.groups + D.d_inner / D.S + 1u, batch);
    prof_begin("dn_prep", s);
    RC_LAUNCH((k_dn_prep), gp, D.S, 0, s, D, conv_kernel, dt_bias, ssm_a, qkv, ba, conv_state, qk, v, beta, gate);
    prof_end(s);
    RC_LAUNCHED();
    prof_begin("dn_state", s);
    const uint64_t warps = (uint64_t)batch * D.rank * D.S;
    const uint32_t blocks = (uint32_t)((warps + 7u) / 8u);
    switch (D.S) {
        case 32: RC_LAUNCH((k_dn_state<1>), blocks, 256, 0, s, D, batch, qk, v, beta, gate, rec_state, core); break;
        case 64: RC_LAUNCH((k_dn_state<2>), blocks, 256, 0, s, D, batch, qk, v, beta, gate, rec_state, core); break;
        case 128: RC_LAUNCH((k_dn_state<4>), blocks, 256, 0, s, D, batch, qk, v, beta, gate, rec_state, core); break;
        default: RC_LAUNCH((k_dn_state<8>), blocks, 256, 0, s, D, batch, qk, v, beta, gate, rec_state, core); break;
    }
    prof_end(s);
    RC_LAUNCHED();
    prof_begin("dn_tail", s);
    RC_LAUNCH((k_dn_tail), dim3(D.rank, batch), D.S, 0, s, D, core, z, norm_w, out);
    prof_end(s);
    RC_LAUNCHED();
    return 1;
}

}  // namespace rc

using namespace rc;

extern "C" int redcuda_deltanet_step(const redcuda_deltanet_params *p, uint32_t batch, const float *qkv, const float *z, const float *ba,
                                     float *conv_state, float *rec_state, float *out) {
    if (!require_device()) return 0;
    RC_REQUIRE(p && qkv && z && ba && conv_state && rec_state && out && batch, "deltanet step: null or empty argument");
    RC_REQUIRE(p->conv_kernel && p->dt_bias && p->ssm_a && p->ssm_norm, "deltanet step: null parameter array");
    const DnDims D{p->d_conv, p->d_state, p->n_group, p->dt_rank, p->d_inner, p->channels, p->rms_eps};
    RC_REQUIRE(D.rank && D.S && D.groups && D.d_conv >= 2u, "deltanet step: zero dimension");
    const size_t ns = D.d_conv - 1u, nqk = 2u * (size_t)D.groups * D.S;
    const size_t b_ck = (size_t)D.channels * D.d_conv * 4u, b_r = (size_t)D.rank * 4u, b_nw = (size_t)D.S * 4u;
    const size_t b_qkv = (size_t)batch * D.channels * 4u, b_z = (size_t)batch * D.d_inner * 4u, b_ba = (size_t)batch * 2u * D.rank * 4u;
    const size_t b_cs = (size_t)batch * D.channels * ns * 4u, b_rs = (size_t)batch * D.rank * D.S * D.S * 4u;
    const size_t b_qk = batch * nqk * 4u;
    Stage st;
    if (!st.open(Stage::pad(b_ck) + 2u * Stage::pad(b_r) + Stage::pad(b_nw) + Stage::pad(b_qkv) + 4u * Stage::pad(b_z) + Stage::pad(b_ba) + Stage::pad(b_cs) + Stage::pad(b_rs) +
                 Stage::pad(b_qk) + 2u * Stage::pad(batch * b_r))) return 0;
    auto f32 = [&](size_t n) { return st.take<float>(n); };
    float *ck = f32(b_ck), *dt = f32(b_r), *sa = f32(b_r), *nw = f32(b_nw), *dq = f32(b_qkv), *dz = f32(b_z), *dba = f32(b_ba), *cs = f32(b_cs), *rs = f32(b_rs),
          *qk = f32(b_qk), *v = f32(b_z), *beta = f32(batch * b_r), *gate = f32(batch * b_r), *core = f32(b_z), *o = f32(b_z);
    if (!st.upload(ck, p->conv_kernel, b_ck) || !st.upload(dt, p->dt_bias, b_r) || !st.upload(sa, p->ssm_a, b_r) || !st.upload(nw, p->ssm_norm, b_nw) || !st.upload(dq, qkv, b_qkv) ||
        !st.upload(dz, z, b_z) || !st.upload(dba, ba, b_ba) || !st.upload(cs, conv_state, b_cs) || !st.upload(rs, rec_state, b_rs)) return 0;
    if (!launch_deltanet(D, batch, ck, dt, sa, nw, dq, dz, dba, cs, rs, qk, v, beta, gate, core, o, st.stream())) return 0;
    return st.download(conv_state, cs, b_cs) && st.download(rec_state, rs, b_rs) && st.download(out, o, b_z) && st.finish();
}

// ---------------------------------------------------------------------------------------------------------------
// Allocation-free variant of the DeltaNet step.
//
// Where the step runs as three kernels (state size 256, more than eight value heads per key head, an output inside the inputs) it needs
// scratch between them (normalised q/k, conv output v, beta, gate, un-normalised head outputs). redcuda_deltanet_step allocates that scratch per call, which a caller cannot afford when it runs inside a
// serving loop that must never block on the allocator (cudaMalloc / cudaFree synchronise the whole device), or when
// another runtime owns the device memory budget. For those callers the scratch lives in the array below, part of the
// library image: every GPU that loads the library holds these 512 KiB until the process exits.
#define RC_DN_SCRATCH_FLOATS (128u * 1024u)
static __device__ __align__(256) float g_dn_scratch[RC_DN_SCRATCH_FLOATS];

// In host code g_dn_scratch is only a handle for the runtime, not an address a kernel may use; the device address is
// asked for once per device (with that device current) and cached here.
static std::mutex g_dn_scratch_mu;
static float *g_dn_scratch_dev[64] = {nullptr};

extern "C" int redcuda_deltanet_step_noalloc(const redcuda_deltanet_params *p, uint32_t batch, const float *qkv_dev, const float *z_dev,
                                             const float *ba_dev, float *conv_state_dev, float *rec_state_dev, float *out_dev, void *stream) {
    if (!require_device()) return 0;
    RC_REQUIRE(p && qkv_dev && z_dev && ba_dev && conv_state_dev && rec_state_dev && out_dev && batch, "deltanet step (no-alloc): null or empty argument");
    RC_REQUIRE(p->conv_kernel && p->dt_bias && p->ssm_a && p->ssm_norm, "deltanet step (no-alloc): null parameter array");
    const DnDims D{p->d_conv, p->d_state, p->n_group, p->dt_rank, p->d_inner, p->channels, p->rms_eps};
    const uint64_t n_qk = (uint64_t)batch * 2u * D.groups * D.S, n_v = (uint64_t)batch * D.d_inner, n_r = (uint64_t)batch * D.rank;
    const uint64_t need = n_qk + 2u * n_v + 2u * n_r;            // the limit is the call's, whichever form runs
    RC_REQUIRE(need <= RC_DN_SCRATCH_FLOATS,
               "deltanet step (no-alloc): batch %u with these dimensions needs %llu scratch floats, the built-in scratch holds %u; "
               "use a smaller batch or redcuda_deltanet_step", batch, (unsigned long long)need, RC_DN_SCRATCH_FLOATS);
    int dev = 0;
    RC_CUDA(cudaGetDevice(&dev));
    RC_REQUIRE(dev >= 0 && dev < 64, "device index %d out of range", dev);
    float *scr = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_dn_scratch_mu);
        if (!g_dn_scratch_dev[dev]) {      // first call on this device: resolve the symbol (not during stream capture)
            void *sym = nullptr;
            RC_CUDA(cudaGetSymbolAddress(&sym, g_dn_scratch));
            g_dn_scratch_dev[dev] = (float *)sym;
        }
        scr = g_dn_scratch_dev[dev];
    }
    // every scratch region is fully written by k_dn_prep / k_dn_state before it is read, so nothing has to be cleared
    float *qk = scr, *v = qk + n_qk, *core = v + n_v, *beta = core + n_v, *gate = beta + n_r;
    return launch_deltanet(D, batch, p->conv_kernel, p->dt_bias, p->ssm_a, p->ssm_norm, qkv_dev, z_dev, ba_dev, conv_state_dev, rec_state_dev,
                           qk, v, beta, gate, core, out_dev, (cudaStream_t)stream);
}
