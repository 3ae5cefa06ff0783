// Softmax + top-k of one token by one warp, shared by the stand-alone router kernel and the single-token GEMV's tail.
#pragma once
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"

namespace rc {

// NPL = probabilities per lane (expert i sits in lane i % 32, slot i / 32). CG: the logits were written by other blocks of
// the same launch (read past L1).
// A single warp runs this alone while the rest of the layer waits, so what counts is the length of the dependent chain.
// Probabilities are non-negative, so their bit patterns order as they do: a selection round is an integer maximum over the
// lane's slots and one redux over the warp, then the lowest expert id that holds that value (a second redux), with neither
// index nor value carried through shuffle steps. A non-finite softmax leaves every probability NaN: every key is 0, id 0 is
// taken and the status word raised.
template <bool CG, int NPL>
__device__ __forceinline__ void route_one_token_n(const float *__restrict__ l, uint32_t n_expert, uint32_t top_k, uint32_t *__restrict__ ids_row,
                                                  float *__restrict__ weights_row, float *__restrict__ probs_row, const RouteGroup1 &G,
                                                  uint32_t *__restrict__ status, uint32_t lane) {
    float p[NPL];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < NPL; ++j) { const uint32_t i = lane + 32u * j; p[j] = i < n_expert ? (CG ? __ldcg(l + i) : l[i]) : -INFINITY; mx = fmaxf(mx, p[j]); }
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    double den = 0.0;
#pragma unroll
    for (int j = 0; j < NPL; ++j) { const uint32_t i = lane + 32u * j; const float e = i < n_expert ? expf(p[j] - mx) : 0.f; p[j] = e; den += (double)e; }
    for (int o = 16; o; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    const float inv = (float)(1.0 / den);
    uint32_t key[NPL];                 // bits of the probability + 1; 0 = not a candidate (absent, taken or NaN)
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
        const uint32_t i = lane + 32u * j;
        const float v = p[j] * inv;
        key[j] = i < n_expert && v >= 0.f ? __float_as_uint(v) + 1u : 0u;
        if (probs_row && i < n_expert) probs_row[i] = v;
    }
    double sel = 0.0;
    float myw = 0.f;                   // lane k keeps the weight of selection k (top_k <= 64: two per lane)
    float myw2 = 0.f;
    for (uint32_t k = 0; k < top_k; ++k) {
        uint32_t m = key[0];
#pragma unroll
        for (int j = 1; j < NPL; ++j) m = max(m, key[j]);
        m = __reduce_max_sync(0xffffffffu, m);
        uint32_t slot = 0xffffffffu;
#pragma unroll
        for (int j = NPL - 1; j >= 0; --j) if (key[j] == m) slot = (uint32_t)j;
        const uint32_t bi = __reduce_min_sync(0xffffffffu, slot == 0xffffffffu ? slot : lane + 32u * slot);
        const float bv = m ? __uint_as_float(m - 1u) : __int_as_float(0x7fffffff);
        if (!m && status && lane == 0) status[ST_ROUTER_NONFINITE] = 1u;
#pragma unroll
        for (int j = 0; j < NPL; ++j) if (lane + 32u * j == bi) key[j] = 0u;
        if (lane == 0) {
            ids_row[k] = bi;
            if (G.sorted) { G.sorted[k] = k; G.uexp[k] = bi; G.ustart[k] = k; G.item_u[k] = k; G.item_p0[k] = k; }      // single token: pair k = group k = item k
            if (G.ids_mirror) G.ids_mirror[k] = bi;
        }
        if (lane == (k & 31u)) { if (k < 32u) myw = bv; else myw2 = bv; }
        sel += (double)bv;
    }
    if (!(sel > 0.0 && sel < (double)INFINITY) && status && lane == 0) status[ST_ROUTER_NONFINITE] = 1u;
    const float invs = (float)(1.0 / sel);
    if (lane < top_k) weights_row[lane] = myw * invs;
    if (lane + 32u < top_k) weights_row[lane + 32u] = myw2 * invs;
    if (G.sorted && lane == 0) { G.ustart[top_k] = top_k; *G.n_unique = top_k; *G.n_items = top_k; if (G.work) { G.work[0] = 0u; G.work[1] = 0u; } }
}
template <bool CG>
__device__ __forceinline__ void route_one_token(const float *__restrict__ l, uint32_t n_expert, uint32_t top_k, uint32_t *__restrict__ ids_row,
                                                float *__restrict__ weights_row, float *__restrict__ probs_row, const RouteGroup1 &G,
                                                uint32_t *__restrict__ status, uint32_t lane) {
    if (n_expert <= 128u) route_one_token_n<CG, 4>(l, n_expert, top_k, ids_row, weights_row, probs_row, G, status, lane);
    else if (n_expert <= 512u) route_one_token_n<CG, 16>(l, n_expert, top_k, ids_row, weights_row, probs_row, G, status, lane);
    else route_one_token_n<CG, 32>(l, n_expert, top_k, ids_row, weights_row, probs_row, G, status, lane);
}

// The block of a launch that draws the last ticket sees every block's logits (fence before the ticket, fence after it)
// and runs the selection for the launch's single token. Called by all threads of every block.
__device__ __forceinline__ void route_tail(const RouteTail &T) {
    __shared__ uint32_t s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(T.ticket, 1u) == gridDim.x - 1u ? 1u : 0u;
    __syncthreads();
    if (s_last) {
        __threadfence();
        if (threadIdx.x == 0) *T.ticket = 0u;
        if (threadIdx.x < 32u) route_one_token<true>(T.logits, T.n_expert, T.top_k, T.ids, T.weights, nullptr, T.G, T.status, threadIdx.x);
    }
}

}  // namespace rc
