// cuda_check.h — CUDA error checking that converts failures into cellsim::Error.
#pragma once
#include <cuda_runtime.h>

#include <string>

#include "internal.h"

#define CS_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t err__ = (call);                                                                \
        if (err__ != cudaSuccess)                                                                  \
            throw ::cellsim::Error(CS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(err__)); \
    } while (0)

#define CS_LAUNCH_CHECK()                                                                          \
    do {                                                                                           \
        cudaError_t err__ = cudaGetLastError();                                                    \
        if (err__ != cudaSuccess)                                                                  \
            throw ::cellsim::Error(CS_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(err__)); \
    } while (0)

namespace cellsim {

// The device has no room for an allocation; nothing else is wrong.
struct OutOfMemory : Error {
    using Error::Error;
};

// RAII device buffer (empty after a failed alloc).
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { reset(); }
    void alloc(size_t count) {
        reset();
        if (count == 0) return;
        const cudaError_t e = cudaMalloc((void**)&p, sizeof(T) * count);
        if (e != cudaSuccess) {
            p = nullptr;
            cudaGetLastError();  // or the next launch check would report it again
            const std::string what = std::string("device allocation: ") + cudaGetErrorString(e);
            if (e == cudaErrorMemoryAllocation) throw OutOfMemory(CS_ERR_CUDA, what);
            throw Error(CS_ERR_CUDA, what);
        }
        n = count;
    }
    void reset() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    size_t bytes() const { return sizeof(T) * n; }
};

// Makes `device` current for the lifetime of the guard and restores the
// previous device afterwards.
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        CS_CUDA(cudaSetDevice(dev));
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

}  // namespace cellsim
