// devbuf.h -- owning device buffer used by the host-side objects of the library.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "status.h"

namespace cgppd {

// A clear of device memory (and the end of a copy from pageable memory) runs on the legacy
// stream after the call has returned, behind whatever is queued there; the objects' own
// streams don't wait for that stream, so the host does: after each buffer, or once after
// several that were set up without waiting.
inline int buffers_settled()
{
    return cgppd_check(cudaStreamSynchronize(cudaStreamLegacy), "device buffer set-up");
}

template <typename T>
struct DevBuf {
    T *ptr = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release()
    {
        if (ptr)
            cudaFree(ptr);
        ptr = nullptr;
        n = 0;
    }
    int alloc(size_t count)
    {
        release();
        const size_t want = std::max<size_t>(count, 1);
        if (cgppd_check(cudaMalloc(&ptr, want * sizeof(T)), "device allocation") != 0) {
            ptr = nullptr;
            return -1;
        }
        n = want;
        return 0;
    }
    // Room for at least `count` elements (the contents are lost if it grows).
    int reserve(size_t count) { return n >= count ? 0 : alloc(count); }
    int upload(const std::vector<T> &v, bool wait = true)
    {
        if (v.empty())
            return zero(1, wait);
        if (alloc(v.size()) != 0 ||
            cgppd_check(cudaMemcpy(ptr, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice), "device upload") != 0)
            return -1;
        return wait ? buffers_settled() : 0;
    }
    int zero(size_t count, bool wait = true)
    {
        if (alloc(count) != 0 || cgppd_check(cudaMemset(ptr, 0, n * sizeof(T)), "device memset") != 0)
            return -1;
        return wait ? buffers_settled() : 0;
    }
};

}  // namespace cgppd
