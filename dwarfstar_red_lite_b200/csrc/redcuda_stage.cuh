// Staging of the host-buffer entry points (quant_matvec, quant_dequant_rows, router_select, deltanet_step, ...): a call
// leases a stream, a device work area and a pinned buffer, moves its arrays through the pinned buffer and gives the lease
// back. What bounded those calls was not the GPU: one cudaMalloc / cudaFree pair per array (each stalls the device) and
// the driver's single-threaded copy of pageable memory.
#pragma once
#include "redcuda_common.cuh"

namespace rc {

struct StageLease;      // redcuda_stage.cu

// One host-buffer call. Arrays are carved out of the lease's device area with take() after open() has sized it; upload() and
// download() queue copies of host arrays, finish() waits for them. Every method returns 0 (with a message) on failure.
class Stage {
  public:
    Stage() = default;
    ~Stage();
    Stage(const Stage &) = delete;
    Stage &operator=(const Stage &) = delete;
    // the device bytes of all arrays of the call (each rounded up to 256 by pad())
    int open(size_t device_bytes);
    static size_t pad(size_t n) { return (n + 255u) / 256u * 256u; }
    template <class T = uint8_t> T *take(size_t bytes) { uint8_t *p = dev_ + used_; used_ += pad(bytes); return reinterpret_cast<T *>(p); }
    // the host array may be changed by its owner only after finish(); dst is ready for work queued on stream() afterwards
    int upload(void *dst_dev, const void *src_host, size_t bytes);
    int download(void *dst_host, const void *src_dev, size_t bytes);
    int finish();
    cudaStream_t stream() const;

  private:
    int open_or_throw(size_t device_bytes);
    int upload_or_throw(void *dst_dev, const void *src_host, size_t bytes);
    int download_or_throw(void *dst_host, const void *src_dev, size_t bytes);
    int follow_default_stream();
    int drain_pinned();      // waits until no copy reads or writes the pinned buffer any more
    StageLease *lease_ = nullptr;
    DevMem own_;             // the device area of a call too large for a lease to keep
    uint8_t *dev_ = nullptr;
    size_t used_ = 0, pinned_used_ = 0;
    bool followed_ = false;
};

// Gives back every device and pinned buffer that idle leases keep (called when an allocation of the library fails, and by redcuda_trim)
void stage_trim();

}  // namespace rc
