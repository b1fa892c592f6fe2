// host_io.cuh -- pinned staging of pageable host arrays (host_io.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <mutex>

namespace gvc {

class Stage {
public:
    static constexpr int kThreads = 8;
    static constexpr int kSlots = 2 * kThreads;
    // Queues host -> device copies of n arrays on `st`; on return the host arrays have been read.
    cudaError_t upload(int device, int n, void* const* dst, const void* const* src, const int64_t* bytes,
                       cudaStream_t st);
    // Device -> host; on return the data has arrived (and `st` has finished what was before).
    cudaError_t download(int device, void* dst, const void* src, int64_t bytes, cudaStream_t st);
    void release();

private:
    cudaError_t prepare();
    std::mutex mutex_;
    char* pinned_ = nullptr;
    cudaEvent_t event_[kSlots] = {};
};

}  // namespace gvc
