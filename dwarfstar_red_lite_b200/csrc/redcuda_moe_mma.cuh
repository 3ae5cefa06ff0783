// Launch interface of the integer tensor-core path for IQ2_XXS expert matrices (redcuda_moe_mma.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rc {

struct MmaArgs {
    const uint8_t *w0, *w1;        // planar IQ2_XXS expert matrices of the shard, back to back (gate/up, or down/nullptr)
    uint64_t mat_bytes, nb;        // bytes and 256-blocks of one expert matrix
    uint32_t nrows, ncols;         // per expert matrix
    uint32_t expert_begin, n_local;  // first expert id of the shard and the number of experts it holds (slot = id - expert_begin)
    uint32_t *status;              // sticky status words (redcuda_common.cuh), may be null
    const uint32_t *sorted, *uexp, *ustart;              // pairs grouped by expert (k_group_pairs)
    const uint32_t *item_u, *item_p0, *n_items;          // work items: expert slot and first pair of up to `TOK` pairs
    const int8_t *xq;              // activation digits [row][3][ncols] (wide form [row][4][ncols]); row of pair p = p / x_div
    const float *sx;               // activation scale per row (wide form: per row and 256-column block)
    uint32_t x_div;
    float *out; uint32_t out_stride;                     // result row of pair p = out + p * out_stride
    const uint2 *lut_grid; const uint4 *lut_sign;        // filled by launch_moe_mma
    uint32_t S, tiles_per_warp, item_tok, item_class;    // filled by launch_moe_mma
    float dw1, dw2;                // weights of digits 1 and 2 (2^bits, 4^bits), filled by launch_moe_mma
    uint32_t *work;                // nibble-layout batch kernel: the launch's run counter, zeroed by the grouping kernel
    uint32_t fmt;                  // nibble-layout kernels: NIB_IQ2, NIB_IQ3 or NIB_IQ2W
    const float *x_raw;            // nibble-layout gate/up of a single token: its fp32 activation row, quantised inside the kernel (xq / sx unused)
    uint32_t act_bits;             // digit width, filled by the launcher
};

// Builds the magnitude and sign tables of the tensor-core path from the IQ2_XXS codebook (current device).
int mma_set_luts(const uint8_t *iq2_grid_host);
// Width of one balanced activation digit: 8 bits (24-bit fixed point per row, the default) or 7 (RC_ACT_BITS=7, the
// earlier 21-bit form, kept for A/B runs).
uint32_t act_digit_bits();
// x[rows][x_stride] (first ncols of each row) -> digits xq[rows][3][ncols] and scales sx[rows]
int launch_quant_act(const float *x, uint32_t x_stride, uint32_t rows, uint32_t ncols, int8_t *xq, float *sx, cudaStream_t s);
// the wide form: digits xq[rows][4][ncols] and scales sx[rows][ncols / 256]
int launch_quant_act_wide(const float *x, uint32_t x_stride, uint32_t rows, uint32_t ncols, int8_t *xq, float *sx, cudaStream_t s);
// Pairs one work item of the tensor-core expert kernel covers: 2 in the few-token configuration, 8 for a decode batch,
// 16 when the experts see many pairs each (prefill chunks, expert-parallel shards): an expert's weights are decoded
// once per item, so larger items halve that work where most experts would otherwise need two.
uint32_t mma_item_tokens(bool few_tokens, uint32_t npairs = 0u, uint32_t n_experts = 1u);
// max_items = upper bound of work items (grid.y); item_tok: the size the items were cut with (2, 8 or 16)
int launch_moe_mma(MmaArgs &A, uint32_t max_items, uint32_t item_tok, cudaStream_t s);
// ---- nibble layout of IQ2_XXS / IQ3_S expert matrices (redcuda_moe_nib.cu): 138 bytes per 256 weights, table-free decode ----
constexpr uint32_t NIB_BLOCK_BYTES = 138u;
// What the 4-bit codes of a matrix mean and which digits its activations have (a template parameter of the kernels). NIB_IQ2:
// three digits of 8 bits per value and one scale per row, as k_quant_act makes them. The other two are the wide form: four digits
// and a power-of-two scale per 256-column block (k_quant_act_wide). NIB_IQ2W: IQ2_XXS codes of a layer whose other matrices are IQ3_S.
constexpr uint32_t NIB_IQ2 = 0u, NIB_IQ3 = 1u, NIB_IQ2W = 2u;
constexpr uint32_t NIB_WIDE_PAIRS = 6u;      // pairs of a work item in the wide form: four digits each fill the 24 columns of three tiles
// One record = one 16-row tile x one 256-column block, laid out by the MMA fragments that a warp's lanes (g = lane / 4, t = lane % 4) take
// from it: rows g and g + 8, code words (t, kg) of all eight 32-column groups kg.
constexpr uint32_t NIB_SC_OFF = 2048u, NIB_D_OFF = 2176u, NIB_REC = 2208u;
// where the 16-byte pieces of a lane sit inside each of the record's four runs of 512 bytes (run 2 (row / 8) + kg / 4): a warp's load of
// a run is contiguous, and from shared memory eight lanes (two rows, or the same t of eight rows) hit eight different bank groups
__host__ __device__ __forceinline__ uint32_t nib_lane_off(uint32_t g, uint32_t t) { return (8u * t + (g ^ (2u * t))) * 16u; }
// byte offset of code word (t, kg) of row rr inside a record
__host__ __device__ __forceinline__ uint32_t nib_code_off(uint32_t rr, uint32_t t, uint32_t kg) {
    return (2u * (rr >> 3) + (kg >> 2)) * 512u + nib_lane_off(rr & 7u, t) + (kg & 3u) * 4u;
}
// byte offset of the scale of group kg and of d of row rr: those of four groups together, rows g and g + 8 side by side
__host__ __device__ __forceinline__ uint32_t nib_sc_off(uint32_t rr, uint32_t kg) { return NIB_SC_OFF + (kg >> 2) * 64u + (rr & 7u) * 8u + (rr >> 3) * 4u + (kg & 3u); }
__host__ __device__ __forceinline__ uint32_t nib_d_off(uint32_t rr) { return NIB_D_OFF + (rr & 7u) * 4u + (rr >> 3) * 2u; }
uint64_t nib_matrix_bytes(uint32_t nrows, uint32_t ncols);
bool nib_shape_ok(uint32_t nrows, uint32_t ncols);
// GGUF rows of IQ2_XXS (NIB_IQ2, NIB_IQ2W) or IQ3_S (NIB_IQ3), one matrix or several in a row (nrows = all their rows) -> nibble layout
// (dst: nib_matrix_bytes, 16-byte aligned)
int launch_nib_repack(uint32_t fmt, const uint8_t *raw, uint64_t nrows, uint32_t ncols, uint8_t *dst, cudaStream_t s);
// gate/up (A.w1 set) or down projection of the grouped pairs, work items of at most 8 pairs (wide form: NIB_WIDE_PAIRS), of which there are
// at most max_items; persistent kernel (redcuda_moe_nib_batch.cu). A.work: its counter, zeroed by the grouping kernel
int launch_nib_batch(MmaArgs &A, uint32_t max_items, cudaStream_t s);
// gate/up of the top_k experts of a single token (A.x_raw), quantised inside the kernel
int launch_nib_one(MmaArgs &A, uint32_t top_k, cudaStream_t s);
// Single token, nibble layout: down projection of the token's top_k experts for one 16-row tile per block, the shared
// expert's down rows, and the tail out = resid + sum_k w_k * expert_k + shared * scalar, in router order — the fusion of
// redmetal_topk_down_tail (native/redmetal_topk.m:254-280). The act rows are quantised inside the kernel.
struct NibTailArgs {
    const uint8_t *w_down; uint64_t mat_bytes;       // nibble-layout down matrices of the shard, bytes of one
    uint32_t nrows, ncols, expert_begin, n_local, top_k;
    const uint32_t *ids; const float *wk;            // the token's experts and router weights [top_k]
    const float *act; uint32_t act_stride;            // act[k][ncols]: SiLU(gate) * up of expert k
    const uint8_t *sh_down; uint64_t sh_nb;           // shared expert's down matrix (planar Q6_K), or null
    const float *sh_act, *scalar, *resid;             // shared activation [ncols], its scalar gate [1], residual [nrows] or null
    float *out;
    float dw1, dw2; uint32_t bits;                    // filled by the launcher
    uint32_t fmt;                                     // NIB_IQ2, NIB_IQ3 or NIB_IQ2W
    uint32_t *status;
};
bool nib_tail_ok(uint32_t top_k, uint32_t nrows, uint32_t ncols);
int launch_nib_down_tail(NibTailArgs &A, cudaStream_t s);

#ifdef __CUDACC__
// the three balanced digits of one activation and the row scale: the arithmetic of k_quant_act, shared with the kernels
// that quantise a row themselves
__device__ __forceinline__ float act_qmax(uint32_t bits) { return bits == 8u ? 8355711.0f : 1040000.0f; }    // largest value three digits hold: 127 * (65536 + 256 + 1), or just below 63.5 * 16384
// |v| as bits: they order as the magnitudes do, with infinity and then NaN above every number
__device__ __forceinline__ uint32_t act_mag(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t act_mag4(const float4 &v) { return max(max(act_mag(v.x), act_mag(v.y)), max(act_mag(v.z), act_mag(v.w))); }
// mx: largest act_mag of the row. Digits cannot hold a non-finite value, so a row with one gets a NaN scale: its products are NaN.
__device__ __forceinline__ float act_scale(uint32_t mx, float qmax) { return mx == 0u ? 1.0f : mx < 0x7f800000u ? __uint_as_float(mx) / qmax : __uint_as_float(0x7fffffffu); }
__device__ __forceinline__ void act_digits(float f, float inv, float qmax, uint32_t bits, int &d0, int &d1, int &d2) {
    const int half = 1 << (bits - 1u), mask = (1 << bits) - 1;
    int iv = __float2int_rn(fminf(fmaxf(f * inv, -qmax), qmax));
    d0 = ((iv + half) & mask) - half; iv = (iv - d0) >> bits;
    d1 = ((iv + half) & mask) - half; iv = (iv - d1) >> bits;
    d2 = iv;
}

// The wide form, for layers whose activations were multiplied in fp32 before they came to the digit kernels (IQ3_S). A 24-bit fixed
// point per ROW loses the small elements of a row with a large one. Here a block of 256 columns, which a weight row scales by one d
// as well, has a power-of-two scale that puts its largest magnitude into [2^29, 2^30): elements down to 2^-6 of that are exact and
// the others are within 2^-31 of it, below the rounding of a single fp32 product with any weight of the block (their magnitudes
// lie within a factor of 465). up: the multiplier; the returned scale undoes it. Blocks below 2^-97 keep fewer bits: their quantum
// is 2^-127.
__device__ __forceinline__ float actw_scale(uint32_t mx, float &up) {
    const int e = min(29 - ((int)(mx >> 23) - 127), 126);
    up = __uint_as_float((uint32_t)(e + 127) << 23);
    return mx < 0x7f800000u ? __uint_as_float((uint32_t)(127 - e) << 23) : __uint_as_float(0x7fffffffu);
}
// byte i of a word: digit i of the value. Adding 128 to every digit makes all bytes non-negative, so that the carries resolve themselves.
__device__ __forceinline__ uint32_t actw_digits(float f, float up) { return ((uint32_t)__float2int_rn(f * up) + 0x80808080u) ^ 0x80808080u; }
// the digit words of four values -> plane[i] = digit i of the four
__device__ __forceinline__ void actw_planes(const uint32_t (&w)[4], uint32_t (&plane)[4]) {
    const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140), c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
    plane[0] = __byte_perm(a, b, 0x5410); plane[1] = __byte_perm(a, b, 0x7632); plane[2] = __byte_perm(c, d, 0x5410); plane[3] = __byte_perm(c, d, 0x7632);
}
#endif

// Q6_K matrix (or gate/up pair with SiLU*mul when w1 != nullptr) x ntok activation rows given as digits (redcuda_q6k_mma.cu)
int launch_q6k_mma(const uint8_t *w0, const uint8_t *w1, uint64_t nb, uint32_t nrows, uint32_t ncols, uint32_t ntok,
                   const int8_t *xq, const float *sx, float *out, uint32_t out_stride, const char *tag, cudaStream_t s);
int q6k_mma_init();      // before the first launch on a device

}  // namespace rc
