// Launch facts that differ by device, looked up once for each.  Calls may come
// from several threads, and a process may have contexts on several devices, so
// each device has its own entry, written once whole (two threads that look the
// same one up write the same value).
#pragma once

#include <algorithm>
#include <atomic>

#include <cuda_runtime.h>

namespace vs {

constexpr int kMaxDevices = 64;

// The current device's index, checked against the tables below.
inline cudaError_t current_device(int *dev) {
    const cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return e;
    return *dev >= 0 && *dev < kMaxDevices ? cudaSuccess : cudaErrorInvalidDevice;
}

// SMs of the current device.
inline cudaError_t device_sms(int *sms) {
    static std::atomic<int> cache[kMaxDevices];
    int dev = 0;
    cudaError_t e = current_device(&dev);
    if (e != cudaSuccess) return e;
    *sms = cache[dev].load();
    if (*sms != 0) return cudaSuccess;
    e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) cache[dev].store(*sms);
    return e;
}

// Blocks of `threads` threads that are resident at once on the current device
// (one entry per kernel: call it with one block size for each).
template <auto Kernel>
cudaError_t resident_blocks(unsigned *grid, int threads = 128) {
    static std::atomic<unsigned> cache[kMaxDevices];
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = current_device(&dev);
    if (e != cudaSuccess) return e;
    *grid = cache[dev].load();
    if (*grid != 0u) return cudaSuccess;
    e = device_sms(&sms);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void *>(Kernel),
                                                                              threads, 0);
    if (e != cudaSuccess) return e;
    *grid = static_cast<unsigned>(std::max(1, sms * std::max(per_sm, 1)));
    cache[dev].store(*grid);
    return cudaSuccess;
}

// The same as a value; zero, which no launch takes, when a query fails.
template <auto Kernel>
unsigned wave_grid(int threads = 128) {
    unsigned grid = 0;
    return resident_blocks<Kernel>(&grid, threads) == cudaSuccess ? grid : 0u;
}

// Lets a kernel be launched with `bytes` of dynamic shared memory on the
// current device.
template <auto Kernel>
cudaError_t allow_shared(int bytes) {
    static std::atomic<bool> done[kMaxDevices];
    int dev = 0;
    cudaError_t e = current_device(&dev);
    if (e != cudaSuccess || done[dev].load()) return e;
    e = cudaFuncSetAttribute(reinterpret_cast<const void *>(Kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done[dev].store(true);
    return e;
}

}  // namespace vs
