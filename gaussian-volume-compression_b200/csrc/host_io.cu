// host_io.cu -- copies between pageable host arrays and the device through pinned chunks.
//
// The mesh samplers take and return the caller's own (pageable) arrays.  One thread's copy
// into the driver's staging buffer bounds such a transfer, and a fresh result array costs a
// page fault per 4 KB on top: 131 MB in and out took 13.6 ms.  Here a few threads copy chunks
// into pinned slots, two per thread, while the chunks before them are on their way, so that
// copying and the link overlap: 3.9 to 4.7 ms, with 6 or 8 threads and chunks of 1 or 2 MB alike
// (12 threads or 0.5 MB 5.5).
//
// A Stage belongs to a context: 16 MB pinned, made at its first use and freed with it, for one
// transfer at a time.  The threads live as long as a call; where none can be started the
// caller's does the work.
#include <sched.h>
#include <cstring>
#include <thread>

#include "host_io.cuh"

namespace gvc {

namespace {

constexpr int64_t kChunk = 1 << 20;  // 1 MB: about 20 us on the link

int worker_count(int64_t chunks) {
    cpu_set_t set;
    CPU_ZERO(&set);
    int cpus = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : 1;
    int64_t n = cpus / 2 < Stage::kThreads ? cpus / 2 : Stage::kThreads;  // the caller's other threads go on
    if (n > chunks / 2) n = chunks / 2;  // below two chunks each a thread is not worth its start
    return n < 1 ? 1 : (int)n;
}

// Runs work(0) .. work(n - 1), work(0) on this thread; work must not throw.
template <class Work>
void run_workers(int n, Work& work) {
    std::thread th[Stage::kThreads];
    for (int t = 1; t < n; t++) {
        try {
            th[t] = std::thread([&work, t] { work(t); });
        } catch (...) {
            break;  // the others take its chunks
        }
    }
    work(0);
    for (int t = 1; t < n; t++)
        if (th[t].joinable()) th[t].join();
}

}  // namespace

cudaError_t Stage::prepare() {
    if (pinned_) return cudaSuccess;
    for (cudaEvent_t& e : event_) {
        if (e) continue;
        const cudaError_t r = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
        if (r != cudaSuccess) return r;
    }
    return cudaHostAlloc((void**)&pinned_, (size_t)kChunk * kSlots, cudaHostAllocDefault);
}

void Stage::release() {
    for (cudaEvent_t& e : event_) {
        if (!e) continue;
        cudaEventSynchronize(e);
        cudaEventDestroy(e);
        e = nullptr;
    }
    if (pinned_) cudaFreeHost(pinned_);
    pinned_ = nullptr;
}

cudaError_t Stage::upload(int device, int n, void* const* dst, const void* const* src, const int64_t* bytes,
                          cudaStream_t st) {
    std::lock_guard<std::mutex> lock(mutex_);
    if (prepare() != cudaSuccess) {
        // no pinned memory to be had: the driver's own staging, which reads the arrays before it returns
        (void)cudaGetLastError();
        for (int i = 0; i < n; i++) {
            if (bytes[i] == 0) continue;
            const cudaError_t e = cudaMemcpyAsync(dst[i], src[i], (size_t)bytes[i], cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess) return e;
        }
        return cudaStreamSynchronize(st);
    }
    int64_t total = 0;
    for (int i = 0; i < n; i++) total += (bytes[i] + kChunk - 1) / kChunk;
    std::atomic<int64_t> next{0};
    std::atomic<int> failed{0};
    auto work = [&](int t) {
        cudaError_t r = t ? cudaSetDevice(device) : cudaSuccess;
        for (int k = 0; r == cudaSuccess && failed.load(std::memory_order_relaxed) == 0; k++) {
            int64_t c = next.fetch_add(1, std::memory_order_relaxed);
            if (c >= total) break;
            int i = 0;
            for (; c >= (bytes[i] + kChunk - 1) / kChunk; i++) c -= (bytes[i] + kChunk - 1) / kChunk;
            const int64_t off = c * kChunk, len = bytes[i] - off < kChunk ? bytes[i] - off : kChunk;
            const int slot = 2 * t + (k & 1);
            char* pin = pinned_ + slot * kChunk;
            // the slot's last transfer, this call's or an earlier one's
            if ((r = cudaEventSynchronize(event_[slot])) != cudaSuccess) break;
            std::memcpy(pin, (const char*)src[i] + off, (size_t)len);
            if ((r = cudaMemcpyAsync((char*)dst[i] + off, pin, (size_t)len, cudaMemcpyHostToDevice, st)) != cudaSuccess)
                break;
            r = cudaEventRecord(event_[slot], st);
        }
        if (r != cudaSuccess) failed.store((int)r, std::memory_order_relaxed);
    };
    run_workers(worker_count(total), work);
    return (cudaError_t)failed.load();
}

cudaError_t Stage::download(int device, void* dst, const void* src, int64_t bytes, cudaStream_t st) {
    std::lock_guard<std::mutex> lock(mutex_);
    cudaError_t e;
    if (prepare() != cudaSuccess) {
        (void)cudaGetLastError();
        e = bytes ? cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyDeviceToHost, st) : cudaSuccess;
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    // one thread waits for the work before the copies
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    const int64_t total = (bytes + kChunk - 1) / kChunk;
    std::atomic<int64_t> next{0};
    std::atomic<int> failed{0};
    auto work = [&](int t) {
        cudaError_t r = t ? cudaSetDevice(device) : cudaSuccess;
        int64_t held[2] = {-1, -1};
        auto drain = [&](int h) {  // the chunk in this thread's slot h, once it has arrived
            if (held[h] < 0 || r != cudaSuccess) return;
            const int64_t off = held[h] * kChunk, len = bytes - off < kChunk ? bytes - off : kChunk;
            held[h] = -1;
            if ((r = cudaEventSynchronize(event_[2 * t + h])) == cudaSuccess)
                std::memcpy((char*)dst + off, pinned_ + (2 * t + h) * kChunk, (size_t)len);
        };
        int k = 0;
        for (; r == cudaSuccess && failed.load(std::memory_order_relaxed) == 0; k++) {
            const int h = k & 1;
            drain(h);
            const int64_t c = next.fetch_add(1, std::memory_order_relaxed);
            if (c >= total || r != cudaSuccess) break;
            const int64_t off = c * kChunk, len = bytes - off < kChunk ? bytes - off : kChunk;
            const int slot = 2 * t + h;
            // an earlier upload may still read the slot
            if ((r = cudaEventSynchronize(event_[slot])) != cudaSuccess) break;
            if ((r = cudaMemcpyAsync(pinned_ + slot * kChunk, (const char*)src + off, (size_t)len,
                                     cudaMemcpyDeviceToHost, st)) != cudaSuccess) break;
            if ((r = cudaEventRecord(event_[slot], st)) != cudaSuccess) break;
            held[h] = c;
        }
        drain(0);
        drain(1);
        if (r != cudaSuccess) failed.store((int)r, std::memory_order_relaxed);
    };
    run_workers(worker_count(total), work);
    return (cudaError_t)failed.load();
}

}  // namespace gvc
