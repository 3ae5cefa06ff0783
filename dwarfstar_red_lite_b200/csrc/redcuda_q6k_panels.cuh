// Host and device pieces of k_q6k_mma (redcuda_q6k_mma.cu): how a launch is cut up, and the order of steps in which a block stages one
// panel of columns after the other. A plain C++ build runs both on the CPU.
#pragma once
#include <stdint.h>
#include <stddef.h>
#ifdef __CUDACC__
#define Q6M_HD __host__ __device__ __forceinline__
#else
#define Q6M_HD inline
#endif

namespace rc {

constexpr uint32_t Q6M_PANEL = 4096u;       // most columns staged at a time
constexpr uint32_t Q6M_SMEM = 216u * 1024u; // most shared memory of a block
// bytes of a staged panel of pc columns: 16 rows of a matrix, 8 tokens
Q6M_HD constexpr uint32_t q6m_a_bytes(uint32_t pc) { return 16u * (pc / 2u + 16u + pc / 4u + 16u + pc / 16u + 16u); }
Q6M_HD constexpr uint32_t q6m_b_bytes(uint32_t pc) { return 24u * (pc + 16u); }

// MS matrices, KS column splits, groups of 8 tokens that a block really has, columns staged at a time
struct Q6Plan { uint32_t MS, KS, groups, panel; size_t smem; };
inline Q6Plan q6m_plan(bool pair, uint32_t nrows, uint32_t ncols, uint32_t ntok) {
    Q6Plan P{};
    P.MS = pair ? 2u : 1u;
    const uint32_t nsteps = ncols / 16u, tgroups = (ntok + 7u) / 8u, tiles = nrows / 16u;
    // Column splits while the launch would leave SMs or warps idle and every split keeps 256 columns or more (whole runs of 128). Warps idle
    // where there are fewer groups of tokens than warps, as in a prompt of 3 to 7 tokens, even if the blocks fill the chip: a projection of 8192 rows
    // is split by eight there. The order of a row's fp32 sums follows from the split.
    uint32_t KS = 1u;
    while (P.MS * KS * 2u <= 8u && nsteps / (KS * 2u) >= 16u && nsteps % (KS * 16u) == 0 &&
           ((uint64_t)tiles * ((tgroups + 8u / (P.MS * KS) - 1u) / (8u / (P.MS * KS))) < 148u * 2u || tgroups < 8u / (P.MS * KS))) KS <<= 1;
    P.KS = KS;
    const uint32_t TGB = 8u / (P.MS * KS);
    P.groups = TGB < tgroups ? TGB : tgroups;
    auto bytes = [&](uint32_t pc) { return (size_t)P.MS * q6m_a_bytes(pc) + (size_t)P.groups * q6m_b_bytes(pc); };
    for (P.panel = ncols < Q6M_PANEL ? ncols : Q6M_PANEL; bytes(P.panel) > Q6M_SMEM;) P.panel = (P.panel / 2u + 255u) / 256u * 256u;
    P.smem = bytes(P.panel);
    return P;
}

// The panels of a row of nblk_row blocks of 256 columns, at most nblk_panel at a time. B.send arms the barrier's phase and sends for a
// panel, B.arrived waits for the phase of the given parity and answers the same in every thread of the block, B.multiply uses the panel.
// A phase that did not end in time ends the work: its barrier must not be armed again and its copies may still be on their way into the
// buffers, so nothing further is sent for and that phase is given as long again. False: the results are void.
template <class B>
Q6M_HD bool q6m_panels(B &b, uint32_t nblk_row, uint32_t nblk_panel) {
    uint32_t parity = 0u;
    for (uint32_t blk0 = 0u; blk0 < nblk_row; blk0 += nblk_panel, parity ^= 1u) {
        const uint32_t nblk = nblk_row - blk0 < nblk_panel ? nblk_row - blk0 : nblk_panel;
        b.send(blk0, nblk);
        if (!b.arrived(parity)) { b.arrived(parity); return false; }
        b.multiply(blk0, nblk);
    }
    return true;
}

}  // namespace rc
