// Further GGUF block types behind the stage entry points: Q8_0, Q2_K, Q4_K, Q5_K (the reference's
// rl_quant_dequant_row / rl_quant_row_dot cases 8, 10, 12, 13: native/redlite_native_quant_cpu.c:40-128, 198-265) and the
// codebook types IQ3_XXS, IQ2_S, IQ4_XS (cases 18, 22, 23 through rl_iq3_group8: native/redlite_native_iq3.c:53-148) and
// IQ2_XS, IQ1_M (17, 29: the weights of rl_native_quant_row_dot, native/redlite_native_reference.c:116-176).
// Rows stay in their GGUF layout; values are decoded with the reference's float operations in the reference's order
// (explicit round-to-nearest multiplies and subtractions, so that no fused multiply-add changes a bit). These types are
// not on the decode path of the Qwen3-Next model files this library was built for (those use Q6_K / IQ2_XXS / IQ3_S);
// they are served for dequantisation and matrix-vector products, not yet by the engine or the expert kernels.
#include "redcuda_common.cuh"
#include "redcuda_kernels.cuh"
#include "redcuda_kquants.cuh"
#include "redcuda_kquants_iq.cuh"
#include "redcuda_stage.cuh"

#include <cuda_fp16.h>
#include <algorithm>
#include <mutex>

namespace rc {

bool kq_supported(uint32_t t) { return kq_type(t) || kq_iq_type(t); }
static uint32_t kq_any_block_values(uint32_t t) { return kq_iq_type(t) ? 256u : kq_block_values(t); }
static uint32_t kq_any_block_bytes(uint32_t t) { return kq_iq_type(t) ? kq_iq_block_bytes(t) : kq_block_bytes(t); }
uint64_t kq_row_bytes(uint32_t t, uint32_t ncols) { return ncols % kq_any_block_values(t) ? 0u : (uint64_t)(ncols / kq_any_block_values(t)) * kq_any_block_bytes(t); }

// tables of the IQ3-family types, one copy per device (module globals), set by redcuda_set_codebooks_ext
__device__ uint32_t d_iq3xxs_grid[256];
__device__ uint64_t d_iq2s_grid[1024];
__device__ int8_t d_iq4nl[16];
__device__ int8_t d_iq2xs_grid[4096];
__device__ int8_t d_iq1m_grid[16384];
static bool g_iq_tabs_set[64], g_xs_tabs_set[64];
static KqIqTabs g_iq_tabs[64];
static std::mutex g_iq_mu;

int kq_set_iq_tables(const uint32_t *iq3xxs, const uint64_t *iq2s, const int8_t *iq4nl) {
    int dev = 0;
    RC_CUDA(cudaGetDevice(&dev));
    RC_REQUIRE(dev >= 0 && dev < 64, "device index %d out of range", dev);
    RC_CUDA(cudaMemcpyToSymbol(d_iq3xxs_grid, iq3xxs, sizeof(d_iq3xxs_grid)));
    RC_CUDA(cudaMemcpyToSymbol(d_iq2s_grid, iq2s, sizeof(d_iq2s_grid)));
    RC_CUDA(cudaMemcpyToSymbol(d_iq4nl, iq4nl, sizeof(d_iq4nl)));
    void *a = nullptr, *b = nullptr, *c = nullptr;
    RC_CUDA(cudaGetSymbolAddress(&a, d_iq3xxs_grid));
    RC_CUDA(cudaGetSymbolAddress(&b, d_iq2s_grid));
    RC_CUDA(cudaGetSymbolAddress(&c, d_iq4nl));
    // a copy from pageable memory may still be on its way when it returns, and the calls that read the tables run on streams of their own
    RC_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    std::lock_guard<std::mutex> lk(g_iq_mu);
    g_iq_tabs[dev].iq3xxs = (const uint32_t *)a; g_iq_tabs[dev].iq2s = (const uint64_t *)b; g_iq_tabs[dev].iq4nl = (const int8_t *)c;
    g_iq_tabs_set[dev] = true;
    return 1;
}
int kq_set_xs_tables(const int8_t *iq2xs, const int8_t *iq1m) {
    int dev = 0;
    RC_CUDA(cudaGetDevice(&dev));
    RC_REQUIRE(dev >= 0 && dev < 64, "device index %d out of range", dev);
    RC_CUDA(cudaMemcpyToSymbol(d_iq2xs_grid, iq2xs, sizeof(d_iq2xs_grid)));
    RC_CUDA(cudaMemcpyToSymbol(d_iq1m_grid, iq1m, sizeof(d_iq1m_grid)));
    void *a = nullptr, *b = nullptr;
    RC_CUDA(cudaGetSymbolAddress(&a, d_iq2xs_grid));
    RC_CUDA(cudaGetSymbolAddress(&b, d_iq1m_grid));
    RC_CUDA(cudaStreamSynchronize(cudaStreamLegacy));      // as in kq_set_iq_tables
    std::lock_guard<std::mutex> lk(g_iq_mu);
    g_iq_tabs[dev].iq2xs = (const int8_t *)a; g_iq_tabs[dev].iq1m = (const int8_t *)b;
    g_xs_tabs_set[dev] = true;
    return 1;
}
// the current device's tables; fails (with a message) for an IQ3-family type before they were set
static int kq_tabs_for(uint32_t type, KqIqTabs &T) {
    T = KqIqTabs{nullptr, nullptr, nullptr, nullptr, nullptr};
    if (!kq_iq_type(type)) return 1;
    int dev = 0;
    RC_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_iq_mu);
    RC_REQUIRE(dev >= 0 && dev < 64, "device index %d out of range", dev);
    if (kq_iq_family3(type)) RC_REQUIRE(g_iq_tabs_set[dev], "type %u needs the IQ3-family tables on device %d: call redcuda_set_codebooks_ext first", type, dev);
    else RC_REQUIRE(g_xs_tabs_set[dev], "type %u needs the IQ2_XS / IQ1_M grids on device %d: call redcuda_set_codebooks_xs first", type, dev);
    T = g_iq_tabs[dev];
    return 1;
}
// values 8 g .. 8 g + 7 of a row in file layout. TYPE is a compile-time constant so that the eight values share their block's
// scale words: a value at a time the decode was some forty instructions per value and bound both kernels below.
template <uint32_t TYPE>
__device__ __forceinline__ void kq_decode8(const uint8_t *__restrict__ row, uint32_t g, const KqIqTabs &T, float (&v)[8]) {
    if (kq_iq_type(TYPE)) {
        const uint8_t *bp = row + (uint64_t)(g >> 5) * kq_iq_block_bytes(TYPE);
        const uint32_t j0 = (g & 31u) << 3;
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) v[j] = kq_iq_value(TYPE, bp, j0 | j, T);
    } else {
        constexpr uint32_t gpb = TYPE == RC_Q8_0 ? 4u : 32u;           // groups of eight per block
        const uint8_t *bp = row + (uint64_t)(g / gpb) * kq_block_bytes(TYPE);
        const uint32_t j0 = (g % gpb) << 3;
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) v[j] = kq_value(TYPE, bp, j0 | j);
    }
}

// out[r][c] for GGUF rows; one thread per eight consecutive values
template <uint32_t TYPE>
__global__ void __launch_bounds__(256) k_kq_dequant(const uint8_t *__restrict__ rows, uint64_t row_bytes, uint32_t gpr, uint64_t groups, KqIqTabs T, float *__restrict__ out) {
    pdl_prologue();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < groups; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = i / gpr; const uint32_t g = (uint32_t)(i - r * gpr);
        float v[8];
        kq_decode8<TYPE>(rows + r * row_bytes, g, T, v);
        float4 *o = reinterpret_cast<float4 *>(out + i * 8u);
        o[0] = make_float4(v[0], v[1], v[2], v[3]);
        o[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// out[t][row] = sum_c W[row][c] * x[t][c]; one warp per row and NT tokens (a row is decoded once per NT tokens), a lane every
// 32nd group of eight columns, fp32 products and sums. The call around it is bound by the link (the rows come from the
// host): an 8192 x 2048 Q4_K matrix for 4 tokens took 224 us here when every value of every token was decoded on its own.
template <uint32_t TYPE, int NT>
__global__ void __launch_bounds__(256) k_kq_gemv(const uint8_t *__restrict__ w, uint64_t row_bytes, uint32_t nrows, uint32_t ncols,
                                                 const float *__restrict__ x, uint32_t ntok, KqIqTabs T, float *__restrict__ out) {
    pdl_prologue();
    const uint32_t row = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u, t0 = blockIdx.y * NT;
    if (row >= nrows) return;
    const uint8_t *rp = w + (uint64_t)row * row_bytes;
    float acc[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t] = 0.f;
    for (uint32_t g = lane; g < (ncols >> 3); g += 32u) {
        float v[8];
        kq_decode8<TYPE>(rp, g, T, v);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            // tokens beyond the batch re-read its last row and are not stored
            const float4 *xp = reinterpret_cast<const float4 *>(x + (size_t)min(t0 + t, ntok - 1u) * ncols + g * 8u);
            const float4 a = __ldg(xp), b = __ldg(xp + 1);
            acc[t] += v[0] * a.x + v[1] * a.y + v[2] * a.z + v[3] * a.w + v[4] * b.x + v[5] * b.y + v[6] * b.z + v[7] * b.w;
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        for (int o = 16; o; o >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
        if (lane == 0 && t0 + t < ntok) out[(size_t)(t0 + t) * nrows + row] = acc[t];
    }
}

#define KQ_FOR_TYPE(type, CALL) switch (type) { \
        case 8u: CALL(8u); break; case 10u: CALL(10u); break; case 12u: CALL(12u); break; case 13u: CALL(13u); break; case 17u: CALL(17u); break; \
        case 18u: CALL(18u); break; case 22u: CALL(22u); break; case 23u: CALL(23u); break; default: CALL(29u); break; }

int kq_dequant_rows(uint32_t type, const uint8_t *rows, uint32_t nrows, uint32_t ncols, float *out) {
    const uint64_t rb = kq_row_bytes(type, ncols), bytes = rb * nrows;
    RC_REQUIRE(rb, "dequant: %u columns is not a valid row length for type %u", ncols, type);
    const uint64_t n = (uint64_t)nrows * ncols, groups = n / 8u;
    KqIqTabs T;
    if (!kq_tabs_for(type, T)) return 0;
    Stage st;
    if (!st.open(Stage::pad(bytes) + Stage::pad(n * 4u))) return 0;
    uint8_t *raw = st.take(bytes);
    float *o = st.take<float>(n * 4u);
    if (!st.upload(raw, rows, bytes)) return 0;
    const unsigned grid = (unsigned)((groups + 255u) / 256u < 4096u ? (groups + 255u) / 256u : 4096u);
#define KQ_DEQ(T_) RC_LAUNCH((k_kq_dequant<T_>), grid, 256, 0, st.stream(), raw, rb, ncols / 8u, groups, T, o)
    KQ_FOR_TYPE(type, KQ_DEQ)
#undef KQ_DEQ
    RC_LAUNCHED();
    return st.download(out, o, n * 4u) && st.finish();
}

int kq_matvec(uint32_t type, const uint8_t *w, uint32_t nrows, uint32_t ncols, const float *x, uint32_t ntok, float *out) {
    const uint64_t rb = kq_row_bytes(type, ncols), bytes = rb * nrows;
    RC_REQUIRE(rb, "matvec: %u columns is not a valid row length for type %u", ncols, type);
    RC_REQUIRE((uint64_t)nrows * ntok < (1ull << 26), "matvec: %u rows x %u tokens exceed the grid", nrows, ntok);
    KqIqTabs T;
    if (!kq_tabs_for(type, T)) return 0;
    const size_t xb = (size_t)ntok * ncols * 4u, ob = (size_t)ntok * nrows * 4u;
    Stage st;
    if (!st.open(Stage::pad(bytes) + Stage::pad(xb) + Stage::pad(ob))) return 0;
    uint8_t *raw = st.take(bytes);
    float *xd = st.take<float>(xb), *od = st.take<float>(ob);
    // one upload, then one launch: multiplying runs of 2 MB while the next run is on the link measured 445 us instead of 370
    if (!st.upload(xd, x, xb) || !st.upload(raw, w, bytes)) return 0;
    for (uint32_t t0 = 0; t0 < ntok; t0 += 4u * 65535u) {       // a batch larger than 65535 x 4 tokens takes several launches
        const uint32_t n = std::min(ntok - t0, 4u * 65535u);
        const float *xt = xd + (size_t)t0 * ncols;
        float *ot = od + (size_t)t0 * nrows;
#define KQ_MV(T_) do { if (n == 1u) RC_LAUNCH((k_kq_gemv<T_, 1>), dim3((nrows + 7u) / 8u), 256, 0, st.stream(), raw, rb, nrows, ncols, xt, n, T, ot); \
                       else RC_LAUNCH((k_kq_gemv<T_, 4>), dim3((nrows + 7u) / 8u, (n + 3u) / 4u), 256, 0, st.stream(), raw, rb, nrows, ncols, xt, n, T, ot); } while (0)
        KQ_FOR_TYPE(type, KQ_MV)
#undef KQ_MV
        RC_LAUNCHED();
    }
    return st.download(out, od, ob) && st.finish();
}

}  // namespace rc
