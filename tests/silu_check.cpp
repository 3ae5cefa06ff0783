// Test helper (tests/test_chunk_silu.py): the SiLU of a chunk's rows compiled for the host, and the library's chunk kernels on a caller's device pointers.
#include <cuda_runtime.h>
#include "../dwarfstar_red_lite_b200/csrc/redcuda_silu.cuh"
#include "../dwarfstar_red_lite_b200/csrc/redcuda_kernels.cuh"

extern "C" {
void silu_of(const double *a, double *out, long n) { for (long i = 0; i < n; ++i) out[i] = rc::silu_d(a[i]); }
int chunk(const unsigned *d, float eps, unsigned T, const float *conv_kernel, const float *dt_bias, const float *ssm_a, const float *norm_w, const float *qkv, const float *z, const float *ba,
          float *conv_state, float *rec_state, float *qk, float *v, float *beta, float *gate, float *core, float *out) {
    const rc::DnDims D{d[0], d[1], d[2], d[3], d[4], d[5], eps};
    return rc::launch_deltanet_seq(D, T, conv_kernel, dt_bias, ssm_a, norm_w, qkv, z, ba, conv_state, rec_state, qk, v, beta, gate, core, out, nullptr, nullptr);
}
}
