// Device pieces shared by the expert kernels of the nibble layout (redcuda_moe_nib.cu: one token; redcuda_moe_nib_batch.cu: batches).
#pragma once
#include "redcuda_common.cuh"
#include "redcuda_moe_mma.cuh"

namespace rc {

// ---- small PTX wrappers ----
__device__ __forceinline__ uint32_t nb_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// z: four registers that hold zero for the whole kernel, the accumulator input of every MMA (each 32-weight group gets
// its own exact s32 product sum, scaled by the group's integer scale afterwards)
__device__ __forceinline__ void nb_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const int (&z)[4]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(z[0]), "r"(z[1]), "r"(z[2]), "r"(z[3]));
}
// byte permute with the selector taken as it is (the intrinsic masks bit 3 of every selector nibble first, one more
// instruction per use; the 4-bit codes never set it)
__device__ __forceinline__ uint32_t nb_prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// the 8 codes of a word -> the int8 operands of weights 0..3 (lo) and 4..7 (hi)
template <uint32_t FMT>
__device__ __forceinline__ void nb_expand(uint32_t w, uint32_t &lo, uint32_t &hi);
// one record into a ring slot: the copy engine signals the slot's mbarrier with the bytes it delivered
__device__ __forceinline__ void nb_fetch(uint32_t dst, const void *src, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(NIB_REC) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(NIB_REC), "r"(bar) : "memory");
}
constexpr uint32_t NIB_SPIN_LIMIT = 1u << 22;      // polls of the (itself time-limited) try_wait: far beyond any real wait
__device__ __forceinline__ bool nb_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < NIB_SPIN_LIMIT; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

constexpr uint32_t NIB_TAB_POS = 0x002b1908u, NIB_TAB_NEG = 0x00d5e7f8u;      // bytes 8, 25, 43, 0 and -8, -25, -43, 0

template <>
__device__ __forceinline__ void nb_expand<NIB_IQ2>(uint32_t w, uint32_t &lo, uint32_t &hi) {
    lo = nb_prmt(NIB_TAB_POS, NIB_TAB_NEG, w); hi = nb_prmt(NIB_TAB_POS, NIB_TAB_NEG, w >> 16);
}
template <>
__device__ __forceinline__ void nb_expand<NIB_IQ2W>(uint32_t w, uint32_t &lo, uint32_t &hi) { nb_expand<NIB_IQ2>(w, lo, hi); }
template <>
__device__ __forceinline__ void nb_expand<NIB_IQ3>(uint32_t w, uint32_t &lo, uint32_t &hi) {
    lo = ((w << 4) & 0xf0f0f0f0u) | 0x08080808u; hi = (w & 0xf0f0f0f0u) | 0x08080808u;
}

// One warp: 16 rows x one 256-column block (a record in shared memory) against NT 8-column tiles of activation digits.
// Bl: digits of column g of tile 0 at this block's first column + 8 t (tile n is n * 8 * BPITCH further).
// blk[n]: sums of rows g (0, 1) and g + 8 (2, 3), columns 2 t and 2 t + 1 of tile n; da, db: d / 8 of the two rows.
template <uint32_t FMT, int NT, uint32_t BPITCH>
__device__ __forceinline__ void nib_sums(const uint8_t *st, const int8_t *Bl, uint32_t g, uint32_t t, const int (&z)[4], int (&blk)[NT][4], float &da, float &db) {
    const uint32_t o = nib_lane_off(g, t);
    const uint4 qa0 = *reinterpret_cast<const uint4 *>(st + o), qa1 = *reinterpret_cast<const uint4 *>(st + 512u + o);
    const uint4 qb0 = *reinterpret_cast<const uint4 *>(st + 1024u + o), qb1 = *reinterpret_cast<const uint4 *>(st + 1536u + o);
    const uint2 s0 = *reinterpret_cast<const uint2 *>(st + NIB_SC_OFF + g * 8u), s1 = *reinterpret_cast<const uint2 *>(st + NIB_SC_OFF + 64u + g * 8u);
    const uint2 sa = make_uint2(s0.x, s1.x), sb = make_uint2(s0.y, s1.y);
    const __half2 dab = *reinterpret_cast<const __half2 *>(st + NIB_D_OFF + g * 4u);
    da = 0.125f * __low2float(dab); db = 0.125f * __high2float(dab);
    const uint32_t wa[8] = {qa0.x, qa0.y, qa0.z, qa0.w, qa1.x, qa1.y, qa1.z, qa1.w};
    const uint32_t wb[8] = {qb0.x, qb0.y, qb0.z, qb0.w, qb1.x, qb1.y, qb1.z, qb1.w};
#pragma unroll
    for (int n = 0; n < NT; ++n) { blk[n][0] = blk[n][1] = blk[n][2] = blk[n][3] = 0; }
#pragma unroll
    for (int kg = 0; kg < 8; ++kg) {
        uint32_t a0, a1, a2, a3;
        nb_expand<FMT>(wa[kg], a0, a2);
        nb_expand<FMT>(wb[kg], a1, a3);
        const int sca = (int)nb_prmt(kg < 4 ? sa.x : sa.y, 0u, 0x4440u + (uint32_t)(kg & 3));
        const int scb = (int)nb_prmt(kg < 4 ? sb.x : sb.y, 0u, 0x4440u + (uint32_t)(kg & 3));
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const uint2 bf = *reinterpret_cast<const uint2 *>(Bl + (uint32_t)n * 8u * BPITCH + (uint32_t)kg * 32u);
            int d[4];
            nb_mma(d, a0, a1, a2, a3, bf.x, bf.y, z);
            blk[n][0] += sca * d[0]; blk[n][1] += sca * d[1];
            blk[n][2] += scb * d[2]; blk[n][3] += scb * d[3];
        }
    }
}
template <uint32_t FMT, int NT, uint32_t BPITCH>
__device__ __forceinline__ void nib_chunk(const uint8_t *st, const int8_t *Bl, uint32_t g, uint32_t t, const int (&z)[4], float (&out)[3][4]) {
    int blk[NT][4];
    float da, db;
    nib_sums<FMT, NT, BPITCH>(st, Bl, g, t, z, blk, da, db);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        out[n][0] += da * (float)blk[n][0]; out[n][1] += da * (float)blk[n][1];
        out[n][2] += db * (float)blk[n][2]; out[n][3] += db * (float)blk[n][3];
    }
}
// The wide form: column 4 p + i is digit i of pair p, so lane t holds two digits of pair 2 n + t / 2 of tile n, the upper two where
// t is odd. sx[n * 2 * SXP]: that pair's scale of this block. out[n]: rows g and g + 8.
template <uint32_t FMT, int NT, uint32_t BPITCH, uint32_t SXP>
__device__ __forceinline__ void nib_chunk_wide(const uint8_t *st, const int8_t *Bl, const float *sx, uint32_t g, uint32_t t, const int (&z)[4], float (&out)[NT][2]) {
    int blk[NT][4];
    float da, db;
    nib_sums<FMT, NT, BPITCH>(st, Bl, g, t, z, blk, da, db);
    const float up = t & 1u ? 65536.0f : 1.0f;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const float w = sx[n * 2u * SXP] * up;              // a power of two: da * w and db * w are exact
        out[n][0] += (da * w) * fmaf(256.0f, (float)blk[n][1], (float)blk[n][0]);
        out[n][1] += (db * w) * fmaf(256.0f, (float)blk[n][3], (float)blk[n][2]);
    }
}
// a lane's row g and g + 8 sums of its two digits -> the full sum of row g (even t) or g + 8 (odd t)
__device__ __forceinline__ float nib_pair_sum(float r0, float r1, uint32_t t) {
    const float got = __shfl_xor_sync(0xffffffffu, t & 1u ? r0 : r1, 1);
    return (t & 1u ? r1 : r0) + got;
}

}  // namespace rc
