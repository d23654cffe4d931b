// Copies between pageable host memory and the device, for the state's import
// and export.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace pe {

// One world's copier. Large copies go through pinned slots of its own
// (kSlots * kSlotBytes, allocated by the first large copy and kept until the
// object goes), which several host threads of the call fill or empty; all are
// joined before the call returns. Small copies, memory that is not pageable
// and worlds without the slots (no memory for them) take one cudaMemcpyAsync.
class HostTransfer {
   public:
    HostTransfer() = default;
    HostTransfer(const HostTransfer&) = delete;
    HostTransfer& operator=(const HostTransfer&) = delete;
    ~HostTransfer();
    // The device copy is ordered on st. A pageable source may be written to again
    // when the call returns, a pinned one when the copy has been done.
    cudaError_t to_device(void* dst, const void* src, size_t bytes, int device, cudaStream_t st);
    // The bytes are in dst when the call returns without an error.
    cudaError_t to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t st);

    static constexpr int kThreads = 8;  // at most
    static constexpr int kSlots = 2 * kThreads;
    static constexpr size_t kSlotBytes = 256u << 10;

   private:
    bool prepare(const void* host, size_t bytes, int device, int* threads);
    template <class F>
    cudaError_t share_out(size_t bytes, int threads, int device, F&& part);
    char* pinned_ = nullptr;
    cudaEvent_t done_[kSlots] = {};  // the slot's last device copy
    bool failed_ = false;
};

}  // namespace pe
