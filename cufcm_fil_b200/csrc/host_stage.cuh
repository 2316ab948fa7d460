// host_stage.cuh -- staging of the host entry points' arrays.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdlib>
#include <cstring>

namespace cufil {

// Page-locked host memory for a handle's calls, taken at the second of them: it costs 1 to 3 ms whatever its size (a
// handle's creation takes 3), which a handle that makes one call, or serves device arrays alone, would not get back.
// Where it is refused the calls go on without.
struct PinnedBuffer {
    void *ptr = nullptr;
    int calls = 0;
    // At the start of each call: the buffer, or null.
    void *open(size_t bytes) {
        if (calls < 2 && ++calls == 2) {
            // the allocation must not break another thread's stream capture
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (cudaMallocHost(&ptr, bytes) != cudaSuccess) {
                ptr = nullptr;
                cudaGetLastError();
            }
            cudaThreadExchangeStreamCaptureMode(&mode);
        }
        return ptr;
    }
    void release() {
        if (ptr) cudaFreeHost(ptr);
        ptr = nullptr;
    }
};

// Device buffer behind a host entry point and, up to kGatherMax, a host buffer of the same layout, page-locked from the
// second call on: the call's arrays are gathered into one copy each way.  (A copy from the caller's pageable memory is
// staged by CUDA, array by array: a swimmer's product of 3,180 segments and its blobs takes 265 us so the first time, 193
// gathered, 138 gathered into page-locked memory; a flow field of 16,000 points 352, 334 and 256.)  Above the limit the
// copy itself is what costs, so the arrays are copied as they are.  Offsets and sizes in bytes.
struct HostStage {
    static constexpr size_t kGatherMax = size_t{4} << 20;
    char *host = nullptr, *dev = nullptr;
    void *plain = nullptr;  // until there is page-locked memory
    size_t size = 0;
    PinnedBuffer pinned;
    cudaError_t alloc(size_t bytes) {
        size = bytes > 0 ? bytes : 1;
        return cudaMalloc(reinterpret_cast<void **>(&dev), size);
    }
    void release() {
        pinned.release();
        std::free(plain);
        if (dev) cudaFree(dev);
        host = dev = nullptr;
        plain = nullptr;
    }
    template <typename T>
    T *at(size_t off) const { return reinterpret_cast<T *>(dev + off); }
    // A call: open(), put() the inputs, then up() their whole range; after the work, down() the results' range,
    // synchronize, take().
    void open() {
        if (size > kGatherMax) return;
        void *p = pinned.open(size);
        if (!p) {
            if (!plain) plain = std::malloc(size);
            p = plain;
        } else if (plain) {
            std::free(plain);
            plain = nullptr;
        }
        host = static_cast<char *>(p);
    }
    cudaError_t put(size_t off, const void *src, size_t bytes, cudaStream_t st) const {
        if (!bytes) return cudaSuccess;
        if (!host) return cudaMemcpyAsync(dev + off, src, bytes, cudaMemcpyHostToDevice, st);
        std::memcpy(host + off, src, bytes);
        return cudaSuccess;
    }
    cudaError_t up(size_t bytes, cudaStream_t st) const {
        return host && bytes ? cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st) : cudaSuccess;
    }
    cudaError_t down(size_t off, size_t bytes, cudaStream_t st) const {
        return host && bytes ? cudaMemcpyAsync(host + off, dev + off, bytes, cudaMemcpyDeviceToHost, st) : cudaSuccess;
    }
    cudaError_t take(void *dst, size_t off, size_t bytes, cudaStream_t st) const {
        if (!bytes) return cudaSuccess;
        if (host) {
            std::memcpy(dst, host + off, bytes);
            return cudaSuccess;
        }
        cudaError_t e = cudaMemcpyAsync(dst, dev + off, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
};

}  // namespace cufil
