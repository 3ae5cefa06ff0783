// Test helper (tests/test_gemv_norm_host.py): asks the library which single-token GEMVs it normalises on the way, and that others with a norm are
// refused before anything is launched. No device is needed.
#include "../dwarfstar_red_lite_b200/csrc/redcuda_kernels.cuh"
#include "../dwarfstar_red_lite_b200/csrc/redcuda_formats.cuh"
#include <stdlib.h>

extern "C" {
const char *redcuda_last_error(void);
// offsets in floats into one buffer; negative: null
int norm_ok(uint32_t type, uint32_t ncols, long x, long branch, long w, long resid, long normed) {
    static float *buf = (float *)aligned_alloc(4096, 1 << 20);
    auto at = [&](long o) { return o < 0 ? nullptr : buf + o; };
    rc::GemvArgs A{};
    A.ntok = 1u; A.njobs = 1u; A.x = at(x);
    A.job[0].type = type; A.job[0].ncols = ncols; A.job[0].nrows = 16u;
    A.norm = rc::GemvNorm{at(w), at(branch), 1e-6f, at(resid), at(normed)};
    return rc::gemv1_norm_ok(A) ? 1 : 0;
}
// a launch that the single-token kernel does not take, with a norm: 0 and the message
const char *refused(uint32_t type, uint32_t ntok) {
    static float *buf = (float *)aligned_alloc(4096, 1 << 20);
    rc::GemvArgs A{};
    A.ntok = ntok; A.njobs = 1u; A.x = buf; A.x_stride = 256u;
    A.job[0].type = type; A.job[0].ncols = 256u; A.job[0].nrows = 16u; A.job[0].w0 = (const uint8_t *)buf; A.job[0].out = buf;
    A.norm = rc::GemvNorm{buf + 1024, nullptr, 1e-6f, nullptr, buf + 2048};
    return rc::launch_gemv(A, nullptr) ? "accepted" : redcuda_last_error();
}
}
