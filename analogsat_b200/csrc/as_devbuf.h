// A device buffer that grows on demand and knows the GPU it lies on: asked for while
// another GPU is current, it moves there (a pointer of the first one would fault on the
// second), and it is freed with its own GPU current.  No kernel code, so a host build
// can check it against a fake runtime.
#pragma once

#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstddef>
#include <utility>

namespace asb {

struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    int dev = -1;  // GPU that holds p

    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }

    void release() {
        if (p) {
            int cur = dev;
            const bool other = cudaGetDevice(&cur) == cudaSuccess && cur != dev;
            if (other) cudaSetDevice(dev);
            cudaFree(p);
            if (other) cudaSetDevice(cur);
        }
        p = nullptr;
        bytes = 0;
        dev = -1;
    }
    // True if alloc(b) on the current device would keep the buffer.
    bool holds(size_t b, int current) const { return p && b <= bytes && dev == current; }
    cudaError_t alloc(size_t b) {
        int cur = 0;
        cudaError_t e = cudaGetDevice(&cur);
        if (e != cudaSuccess) return e;
        if (holds(b, cur)) return cudaSuccess;
        release();
        e = cudaMalloc(&p, std::max<size_t>(b, 16));
        if (e == cudaSuccess) {
            bytes = b;
            dev = cur;
        } else {
            p = nullptr;
        }
        return e;
    }
    // The other's buffer, which is left empty.
    void take(DevBuf& o) {
        release();
        std::swap(p, o.p);
        std::swap(bytes, o.bytes);
        std::swap(dev, o.dev);
    }
    template <typename T> T* as() const { return static_cast<T*>(p); }
};

}  // namespace asb
