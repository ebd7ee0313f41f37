#include "vs_host_copy.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace vs {

namespace {
constexpr size_t kSlots = 8;
constexpr size_t kChunk = 512u << 10;
// Below this the threads' wake-up costs what they save.  Into arrays whose pages
// are new, as a program's that keeps its films, on 16 cores, one thread / several:
// a box room and its 1.05 MB film 1.92 / 1.84 ms, a principled room and its films
// of 1.4 and 2.8 MB 2.14 / 1.89.  Into memory that the last film's array has just
// given back: 1.05 MB 0.22 to 0.30 / 0.27 ms, 2.1 MB 0.35 to 0.48 / 0.41 to 0.45,
// 2.8 MB 0.43 to 0.50 / 0.46, 3.6 MB 0.54 to 0.57 / 0.41, 4.2 MB 0.65 / 0.35, 17 MB
// 2.2 / 1.1, 33 MB 4.2 / 2.6.
constexpr size_t kMinBytes = 1u << 20;
constexpr unsigned kMaxHelpers = 3;
}  // namespace

struct HostCopy::Impl {
    uint8_t *ring = nullptr;
    cudaEvent_t ev[kSlots] = {};
    cudaEvent_t ready = nullptr;  // the work before the copy has ended
    // The chunks' own stream: the later ones are queued as slots empty, and on
    // the caller's stream another thread's render could have come before them.
    cudaStream_t st = nullptr;
    std::vector<std::thread> helpers;
    std::mutex one;  // one copy at a time

    // The current copy.  Chunk k uses slot k % kSlots; the thread that has
    // emptied a slot queues the slot's next chunk.
    uint8_t *dst = nullptr;
    const uint8_t *src = nullptr;
    size_t bytes = 0, chunks = 0;
    int device = 0;
    std::atomic<size_t> next{0};
    std::atomic<size_t> queued[kSlots];  // chunks queued into the slot so far
    std::atomic<int> error{0};

    std::mutex mu;
    std::condition_variable cv_start, cv_end;
    uint64_t generation = 0;
    unsigned running = 0;
    bool stop = false;

    cudaError_t init() {
        cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&ring), kSlots * kChunk, cudaHostAllocPortable);
        if (e != cudaSuccess) {
            ring = nullptr;
            return e;
        }
        for (size_t i = 0; i < kSlots && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            release();
            return e;
        }
        const unsigned n = std::min(kMaxHelpers, std::max(1u, std::thread::hardware_concurrency()) - 1u);
        try {
            for (unsigned i = 0; i < n; ++i) helpers.emplace_back([this] { helper(); });
        } catch (...) {
            // Fewer helpers than asked for: the caller's thread copies anyway.
        }
        return cudaSuccess;
    }

    void release() {
        for (cudaEvent_t &e : ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        if (st) cudaStreamDestroy(st);
        st = nullptr;
        if (ready) cudaEventDestroy(ready);
        ready = nullptr;
        if (ring) cudaFreeHost(ring);
        ring = nullptr;
    }

    size_t size_of(size_t k) const { return std::min(kChunk, bytes - k * kChunk); }

    bool queue(size_t k) {
        const size_t s = k % kSlots;
        cudaError_t e = cudaMemcpyAsync(ring + s * kChunk, src + k * kChunk, size_of(k), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev[s], st);
        if (e != cudaSuccess) {
            error = e;
            return false;
        }
        queued[s].fetch_add(1, std::memory_order_release);
        return true;
    }

    void work() {
        for (;;) {
            const size_t k = next.fetch_add(1);
            if (k >= chunks) return;
            const size_t s = k % kSlots;
            while (queued[s].load(std::memory_order_acquire) <= k / kSlots) {
                if (error.load()) return;
                std::this_thread::yield();
            }
            const cudaError_t e = cudaEventSynchronize(ev[s]);
            if (e != cudaSuccess) {
                error = e;
                return;
            }
            std::memcpy(dst + k * kChunk, ring + s * kChunk, size_of(k));
            if (k + kSlots < chunks && !queue(k + kSlots)) return;
        }
    }

    void helper() {
        uint64_t seen = 0;
        std::unique_lock<std::mutex> lk(mu);
        for (;;) {
            cv_start.wait(lk, [&] { return stop || generation != seen; });
            if (stop) return;
            seen = generation;
            lk.unlock();
            if (cudaSetDevice(device) == cudaSuccess) work();
            lk.lock();
            if (--running == 0) cv_end.notify_one();
        }
    }

    cudaError_t copy(void *d, const void *s, size_t n, int dev, cudaStream_t stream) {
        std::lock_guard<std::mutex> guard(one);
        dst = static_cast<uint8_t *>(d);
        src = static_cast<const uint8_t *>(s);
        bytes = n;
        chunks = (n + kChunk - 1) / kChunk;
        device = dev;
        next = 0;
        error = 0;
        for (auto &q : queued) q = 0;
        cudaError_t e = cudaEventRecord(ready, stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(st, ready, 0);
        if (e != cudaSuccess) return e;
        for (size_t k = 0; k < std::min(chunks, kSlots); ++k)
            if (!queue(k)) break;
        // Only this thread waits for the work before the copy (which may be a
        // long render); the helpers start as the first chunk is on its way.
        if (!error.load() && (e = cudaEventSynchronize(ready)) != cudaSuccess) error = e;
        {
            std::lock_guard<std::mutex> lk(mu);
            ++generation;
            running = static_cast<unsigned>(helpers.size());
        }
        cv_start.notify_all();
        work();
        std::unique_lock<std::mutex> lk(mu);
        cv_end.wait(lk, [&] { return running == 0; });
        if (error.load()) {
            // Nothing may still be writing the ring when the next copy starts.
            (void)cudaStreamSynchronize(st);
        }
        return static_cast<cudaError_t>(error.load());
    }

    ~Impl() {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
        }
        cv_start.notify_all();
        for (std::thread &t : helpers) t.join();
        release();
    }
};

HostCopy::HostCopy() : impl(new Impl()) {}
HostCopy::~HostCopy() { delete impl; }

void HostCopy::prepare() {
    // Where no page-locked memory is to be had, copies go without it.
    if (impl->init() != cudaSuccess) (void)cudaGetLastError();
}

cudaError_t HostCopy::copy(void *dst, const void *src, size_t bytes, int device, cudaStream_t st) {
    // Page-locked (or device) destinations take the copy directly.
    cudaPointerAttributes at{};
    const bool pageable = cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
    (void)cudaGetLastError();
    if (bytes < kMinBytes || !pageable || !impl->ring) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    return impl->copy(dst, src, bytes, device, st);
}

}  // namespace vs
