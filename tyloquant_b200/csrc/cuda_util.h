// CUDA-side helpers shared by the .cu files of the library.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "common.h"

namespace mfqb {

#define MFQB_CUDA(expr)                                                                         \
    do {                                                                                        \
        const cudaError_t e_ = (expr);                                                          \
        if (e_ != cudaSuccess) ::mfqb::fail(MFQB_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

// Makes `device` current for the scope and restores the previous device afterwards.
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int device) {
        MFQB_CUDA(cudaGetDevice(&prev));
        if (prev != device) MFQB_CUDA(cudaSetDevice(device));
        else prev = -1;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

int device_sm_count(int device);

// cudaMalloc on the current device; where there is no room, after parked blocks of freed tensors have been given back.
void device_malloc(void** p, size_t bytes);

// Owning device buffer.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), bytes(o.bytes) {
        o.p = nullptr;
        o.bytes = 0;
    }
    void alloc(size_t n) {
        release();
        if (n) device_malloc(&p, n);
        bytes = n;
    }
    void upload(const void* src, size_t n) {
        alloc(n);
        if (n) MFQB_CUDA(cudaMemcpy(p, src, n, cudaMemcpyHostToDevice));
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    ~DevBuf() { release(); }
};

#if defined(__CUDACC__)
// Four neighbouring decoded weights, `live` of them inside the row: one vector store where the four are aligned.
__device__ __forceinline__ void store_quad(void* out, int out_dtype, size_t off, const float (&v)[4], int live) {
    if (out_dtype == MFQB_F32) {
        float* p = static_cast<float*>(out) + off;
        if (live == 4 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        else
            for (int e = 0; e < live; ++e) p[e] = v[e];
    } else {
        __nv_bfloat16* p = static_cast<__nv_bfloat16*>(out) + off;
        if (live == 4 && (reinterpret_cast<uintptr_t>(p) & 7) == 0) {
            const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
            *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        } else {
            for (int e = 0; e < live; ++e) p[e] = __float2bfloat16_rn(v[e]);
        }
    }
}
#endif

// Library scratch that only ever grows: one block per device, handed to kernels that may still be
// in flight (or baked into a captured graph) when a later call needs more.  A larger request
// allocates a new block and keeps the old one alive until the process exits, so a pointer handed
// out once stays valid.  Growing allocates, which a stream capture does not allow: the call then
// fails with a message instead of breaking the capture.  Calls that share a block on one device
// must be ordered by their streams (the block holds one call's intermediates at a time).
struct GrowOnlyScratch {
    void* get(int device, size_t bytes, cudaStream_t stream, const char* what, bool exact = false);   // exact: no room for growth
    // Grows the block for a call that may follow, which could be captured; does nothing while the stream is.
    void reserve(int device, size_t bytes, cudaStream_t stream, const char* what);

private:
    struct PerDevice {
        void* p = nullptr;
        size_t bytes = 0;
    };
    PerDevice dev_[64];
};

}  // namespace mfqb
