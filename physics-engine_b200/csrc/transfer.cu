// State import and export through pageable memory. What bounds it is the
// caller's memory, not the link: one thread copies 12 to 17 GB/s, and takes 0.2
// to 0.45 ms a megabyte where the destination's pages are touched for the first
// time (every array a caller has just allocated), while the link moves 54 GB/s.
// 32 MB with 1 / 2 / 4 / 8 / 16 threads, ms: pinned to fresh pages 14.2 / 7.2 /
// 3.8 / 2.1 / 1.7, to warm pages 2.0 / 1.9 / 0.9 / 0.9 / 0.7, warm pages to pinned
// 2.5 / 1.9 / 1.2 / 1.0 / 0.5. So up to eight threads, at most half the
// machine's, each move a contiguous part through two slots of their own (of 256
// kB: 33 MB out takes 1.7 ms to warm pages; 1.4 with 512 kB, 2.1 with 128). At
// 1.4M particles positions and velocities in and positions, velocities and
// densities out, into new arrays, take 9 ms where they took 26.
#include "transfer.cuh"

#include <algorithm>
#include <cstring>
#include <thread>

#include "parts.cuh"

namespace pe {

namespace {

// A thread's least share, and the least copy that is shared out: below, starting
// the threads takes what they save (5.7 MB to warm pages: 0.34 ms by one copy,
// 0.5 by two threads). The slots cost 2 to 4 ms to allocate, so the first copy
// that makes them is a large one.
constexpr size_t kThreadBytes = 1u << 20, kLeastBytes = 8u << 20, kFirstBytes = 16u << 20;

struct DeviceScope {  // the calling thread's current device
    int old = -1;
    explicit DeviceScope(int device) {
        if (cudaGetDevice(&old) != cudaSuccess || old == device || cudaSetDevice(device) != cudaSuccess) old = -1;
    }
    ~DeviceScope() {
        if (old >= 0) cudaSetDevice(old);
    }
};

}  // namespace

HostTransfer::~HostTransfer() {
    for (cudaEvent_t e : done_)
        if (e) cudaEventDestroy(e);
    if (pinned_) cudaFreeHost(pinned_);
}

// Whether the copy goes through the slots, and by how many threads.
bool HostTransfer::prepare(const void* host, size_t bytes, int device, int* threads) {
    const size_t half = std::thread::hardware_concurrency() / 2u;
    *threads = (int)std::min({(size_t)kThreads, half, bytes / kThreadBytes});
    if (*threads < 2 || failed_ || bytes < (pinned_ ? kLeastBytes : kFirstBytes)) return false;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type != cudaMemoryTypeUnregistered) return false;
    if (pinned_) return true;
    DeviceScope scope(device);
    void* p = nullptr;
    if (cudaMallocHost(&p, kSlots * kSlotBytes) != cudaSuccess) {
        cudaGetLastError();
        failed_ = true;
        return false;
    }
    pinned_ = static_cast<char*>(p);
    for (cudaEvent_t& e : done_)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            e = nullptr;
            failed_ = true;
            return false;
        }
    return true;
}

// Calls part(t, begin, end) for `threads` parts of the bytes, each by its own thread.
template <class F>
cudaError_t HostTransfer::share_out(size_t bytes, int threads, int device, F&& part) {
    cudaError_t err[kThreads] = {};
    const size_t step = (bytes / (size_t)threads + 4095u) & ~(size_t)4095u;
    auto run = [&](int t) noexcept {
        DeviceScope scope(device);
        const size_t b = std::min(bytes, step * (size_t)t), e = t == threads - 1 ? bytes : std::min(bytes, b + step);
        err[t] = b < e ? part(t, b, e) : cudaSuccess;
    };
    run_parts<kThreads>(threads, run);
    for (int t = 0; t < threads; ++t)
        if (err[t] != cudaSuccess) return err[t];
    return cudaSuccess;
}

cudaError_t HostTransfer::to_device(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
    int threads = 0;
    if (!prepare(src, bytes, device, &threads)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    return share_out(bytes, threads, device, [&](int t, size_t b, size_t e) noexcept {
        cudaError_t r = cudaSuccess;
        for (int k = 2 * t; b < e && r == cudaSuccess; k ^= 1) {
            const size_t n = std::min(kSlotBytes, e - b);
            char* const slot = pinned_ + (size_t)k * kSlotBytes;
            r = cudaEventSynchronize(done_[k]);  // the slot's last copy, also one of an earlier call
            if (r != cudaSuccess) break;
            std::memcpy(slot, static_cast<const char*>(src) + b, n);
            r = cudaMemcpyAsync(static_cast<char*>(dst) + b, slot, n, cudaMemcpyHostToDevice, st);
            if (r == cudaSuccess) r = cudaEventRecord(done_[k], st);
            b += n;
        }
        return r;
    });
}

cudaError_t HostTransfer::to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
    int threads = 0;
    if (!prepare(dst, bytes, device, &threads)) {
        const cudaError_t r = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        return r != cudaSuccess ? r : cudaStreamSynchronize(st);
    }
    return share_out(bytes, threads, device, [&](int t, size_t b, size_t e) noexcept {
        // A slot is handed to the next copy only once it has been emptied; an
        // earlier call's copy out of it is ahead on the stream.
        auto fetch = [&](int k, size_t at) noexcept {
            const cudaError_t r = cudaMemcpyAsync(pinned_ + (size_t)k * kSlotBytes, static_cast<const char*>(src) + at,
                                                  std::min(kSlotBytes, e - at), cudaMemcpyDeviceToHost, st);
            return r != cudaSuccess ? r : cudaEventRecord(done_[k], st);
        };
        int k = 2 * t;
        cudaError_t r = fetch(k, b);
        if (r == cudaSuccess && b + kSlotBytes < e) r = fetch(k ^ 1, b + kSlotBytes);
        for (; b < e && r == cudaSuccess; b += kSlotBytes, k ^= 1) {
            r = cudaEventSynchronize(done_[k]);
            if (r != cudaSuccess) break;
            std::memcpy(static_cast<char*>(dst) + b, pinned_ + (size_t)k * kSlotBytes, std::min(kSlotBytes, e - b));
            if (b + 2 * kSlotBytes < e) r = fetch(k, b + 2 * kSlotBytes);
        }
        return r;
    });
}

}  // namespace pe
