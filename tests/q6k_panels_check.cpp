// Test helper (compiled for the host by tests/test_q6k_panels_host.py): the panel steps and the launch rule of k_q6k_mma
// (csrc/redcuda_q6k_panels.cuh), the steps against a model of the staging barrier.
#include "../dwarfstar_red_lite_b200/csrc/redcuda_q6k_panels.cuh"
#include <vector>

enum : int { DOUBLE_ARM = 1, SENT_OVER_LIVE = 2, ENDED_LIVE = 4, WRONG_PHASE = 8, BAD_PANEL = 16, WRONG_RESULT = 32 };

// one mbarrier of one arrival and the copies that it counts; the copies of panel `late` come `waits_late` waits late (2: never)
struct Block {
    int faults = 0, late, waits_late, panels = 0;
    bool armed = false, live = false;
    uint32_t phase = 0, next = 0;
    int waits = 0;
    void send(uint32_t blk0, uint32_t nblk) {
        if (armed) faults |= DOUBLE_ARM;
        if (live) faults |= SENT_OVER_LIVE;
        if (blk0 != next || nblk == 0) faults |= BAD_PANEL;
        next = blk0 + nblk;
        armed = live = true; waits = 0; ++panels;
    }
    bool arrived(uint32_t parity) {
        if (parity != (phase & 1u)) faults |= WRONG_PHASE;
        if (panels - 1 == late && waits++ < waits_late) return false;
        if (armed) { armed = live = false; ++phase; }
        return true;
    }
    void multiply(uint32_t, uint32_t) { if (live) faults |= SENT_OVER_LIVE; }
};

// the loop that went on after a wait that had run out
static bool goes_on(Block &b, uint32_t row, uint32_t panel) {
    uint32_t parity = 0u;
    bool ok = true;
    for (uint32_t blk0 = 0u; blk0 < row; blk0 += panel, parity ^= 1u) {
        const uint32_t nblk = row - blk0 < panel ? row - blk0 : panel;
        b.send(blk0, nblk);
        if (ok) ok = b.arrived(parity);
        if (ok) b.multiply(blk0, nblk);
    }
    if (!ok) b.arrived(parity ^ 1u);
    return ok;
}

extern "C" int check_panels(uint32_t row, uint32_t panel, int late, int waits_late, int planted) {
    Block b; b.late = late; b.waits_late = waits_late;
    const bool ok = planted ? goes_on(b, row, panel) : rc::q6m_panels(b, row, panel);
    if (ok != (late < 0 || waits_late == 0)) b.faults |= WRONG_RESULT;
    if (ok && b.next != row) b.faults |= BAD_PANEL;
    if (b.live && waits_late < 2) b.faults |= ENDED_LIVE;      // copies that were late, not lost, must have been waited for
    return b.faults;
}

extern "C" void plan(int pair, uint32_t nrows, uint32_t ncols, uint32_t ntok, uint32_t *out) {
    const rc::Q6Plan P = rc::q6m_plan(pair != 0, nrows, ncols, ntok);
    out[0] = P.MS; out[1] = P.KS; out[2] = P.groups; out[3] = P.panel; out[4] = (uint32_t)P.smem;
}
