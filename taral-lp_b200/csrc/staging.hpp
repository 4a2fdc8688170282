// Copies between the device and pageable host memory. The runtime's own path moves such a copy through one staging buffer
// with one host thread: page faults and a core's copy rate hold it to 4.7 GB/s into fresh memory and 11 GB/s out of it, on
// a link of 55 GB/s. Here up to 16 threads take chunks in turn, each through its own pinned slot, so that the link, the page
// faults and the host copies of different chunks overlap. 16 cores, a prediction of 128 x 132,001 (68 MB): 14.6 -> 3.3 ms;
// reading the weights of that network (272 MB) 58 -> 13 ms, setting them 25 -> 11 ms. Chunks of 1 MB gain another 15 %
// but take 10 ms to pin, 512 KB 4 ms; 256 KB lose 20 %.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>

namespace taral {

class Staging {
    static constexpr size_t kChunk = size_t(1) << 19;
    static constexpr int kThreadsMax = 16;
    static constexpr size_t kLeast = size_t(4) << 20;  // bytes; below, the threads' start costs more than they save
    unsigned char* pinned = nullptr;
    std::array<cudaEvent_t, kThreadsMax> done{};
    int slots = 0, dev = 0;
    std::mutex one;  // transfer at a time

public:
    Staging() = default;
    Staging(const Staging&) = delete;
    Staging& operator=(const Staging&) = delete;
    ~Staging() { release(); }

    // Slots for transfers of up to `largest` bytes; none where they cannot be had, and copy() then leaves it to the runtime.
    void prepare(size_t largest) {
        if (largest < kLeast || cudaGetDevice(&dev) != cudaSuccess) return;
        // a slot for every 2 MB, so that pinning them (0.5 ms a MB) stays well below what one transfer of that size takes
        int want = int(std::min<size_t>(largest >> 21, std::min<unsigned>(kThreadsMax, std::thread::hardware_concurrency())));
        if (const char* e = std::getenv("TARAL_STAGING")) want = std::min(kThreadsMax, std::atoi(e));  // 0: none (tests)
        if (want < 2 || cudaHostAlloc(reinterpret_cast<void**>(&pinned), size_t(want) * kChunk, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            pinned = nullptr;
            return;
        }
        for (; slots < want; ++slots)
            if (cudaEventCreateWithFlags(&done[size_t(slots)], cudaEventDisableTiming) != cudaSuccess) break;
        if (slots < want) cudaGetLastError(), release();
    }
    void release() {
        while (slots > 0) cudaEventDestroy(done[size_t(--slots)]);
        if (pinned) cudaFreeHost(pinned);
        pinned = nullptr;
    }

    // As cudaMemcpyAsync on `s`. A staged transfer has ended on return, with whatever was queued on `s` before it.
    cudaError_t copy(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s) {
        const bool down = kind == cudaMemcpyDeviceToHost;
        if (slots == 0 || bytes < kLeast || !pageable(down ? dst : src)) return cudaMemcpyAsync(dst, src, bytes, kind, s);
        std::lock_guard<std::mutex> lock(one);
        const size_t chunks = (bytes + kChunk - 1) / kChunk;
        std::atomic<size_t> next{0};
        std::atomic<int> failed{int(cudaSuccess)};
        auto work = [&](int slot) {
            unsigned char* buf = pinned + size_t(slot) * kChunk;
            const cudaEvent_t ev = done[size_t(slot)];
            cudaError_t e = slot ? cudaSetDevice(dev) : cudaSuccess;
            for (size_t c; e == cudaSuccess && failed.load() == int(cudaSuccess) && (c = next.fetch_add(1)) < chunks;) {
                const size_t at = c * kChunk, n = std::min(kChunk, bytes - at);
                unsigned char* to = static_cast<unsigned char*>(dst) + at;
                const unsigned char* from = static_cast<const unsigned char*>(src) + at;
                if (!down) std::memcpy(buf, from, n);
                e = cudaMemcpyAsync(down ? buf : to, down ? from : buf, n, kind, s);
                if (e == cudaSuccess) e = cudaEventRecord(ev, s);
                if (e == cudaSuccess) e = cudaEventSynchronize(ev);  // also before the slot is filled again
                if (e == cudaSuccess && down) std::memcpy(to, buf, n);
            }
            if (e != cudaSuccess) failed = int(e);
        };
        std::array<std::thread, kThreadsMax> threads;
        for (int t = 1; t < slots && size_t(t) < chunks; ++t) {
            try {
                threads[size_t(t)] = std::thread(work, t);
            } catch (...) {  // no more threads to be had
                break;
            }
        }
        work(0);
        for (std::thread& t : threads)
            if (t.joinable()) t.join();
        return cudaError_t(failed.load());
    }

private:
    static bool pageable(const void* p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }
};

}  // namespace taral
