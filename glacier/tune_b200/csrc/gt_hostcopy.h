// Copies between pageable host memory and the device, at the rate of the link.
//
// cudaMemcpyAsync from or to pageable memory goes through the driver's own staging buffers with one thread copying:
// 16 - 18 GB/s here, a third of what the link carries.  A HostCopier keeps a small ring of page-locked pieces and a few
// worker threads: the workers copy pieces between the caller's buffer and the ring side by side while the copies of other
// pieces are on the link.  Buffers that are page-locked already, and small ones, go to cudaMemcpyAsync directly.
//
// One copier belongs to one engine and is used under its lock.  Workers are started by the first large copy, sleep when
// there is nothing to do, and end with the engine, which also frees the ring (8 MB).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace gt {

class HostCopier {
public:
    HostCopier() = default;
    ~HostCopier();
    HostCopier(const HostCopier &) = delete;
    HostCopier &operator=(const HostCopier &) = delete;
    // dst <- src on `s`.  Returns when src has been read (the copy to the device may still be under way on `s`).
    cudaError_t to_device(void *dst, const void *src, size_t bytes, cudaStream_t s);
    // dst <- src, after everything queued on `s` so far.  Returns with dst filled.
    cudaError_t to_host(void *dst, const void *src, size_t bytes, cudaStream_t s);
    // whether a buffer goes through the ring (pageable and large enough)
    static bool staged(const void *host, size_t bytes);

private:
    struct Impl;
    Impl *impl_ = nullptr;
    cudaError_t start();
};

}  // namespace gt
