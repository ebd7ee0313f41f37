// Device-to-host copies into pageable memory, spread over a few threads.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace vs {

// A copy to pageable memory ends in one host thread that writes fresh pages
// (a new film array's pages are faulted and zeroed by that write) at 10 to 15
// GB/s, a quarter of what the bus delivers.  Here the device writes chunks
// into a page-locked ring and several threads take them in order from there.
// The ring (4 MB) and the threads are made by prepare and live as long as the
// object; copies of one object run one at a time.
class HostCopy {
public:
    HostCopy();
    ~HostCopy();
    HostCopy(const HostCopy &) = delete;
    HostCopy &operator=(const HostCopy &) = delete;
    // Makes the ring and the threads, on the current device: about 3 ms, which
    // the first film of a program would wait for otherwise.  Without it, or
    // where no page-locked memory is to be had, copies go straight through.
    void prepare();
    // Copies `bytes` from device memory to dst after the work queued on `st`;
    // returns when dst holds them.  Small copies go straight through.
    cudaError_t copy(void *dst, const void *src, size_t bytes, int device, cudaStream_t st);

private:
    struct Impl;
    Impl *impl;
};

}  // namespace vs
