// frame_copy.cu -- page-locked host frames to the device over few SMs.
//
// The serving loop's frames arrive over the host link.  Read by the row
// kernel itself, a frame holds the registers of every SM for as long as the
// link takes, and the column kernels of other requests (a whole SM's
// registers each) wait; this kernel keeps the link full from a few blocks --
// 16 x 256 threads x 8 loads of 16 bytes, 0.5 MB in flight; 8 blocks already
// measured the link's rate, 16 MB in 86 us with 8 to 304 blocks -- and leaves
// the other SMs to them.
// The next frame's copy, launched as this one's programmatic dependent, may
// start when every block has issued its last loads.
#include <cstdint>

#include "glsfft_internal.h"
#include "pdl.cuh"

namespace glsfft {

namespace {

constexpr int kThreads = 256, kBlocks = 16, kBatch = 8;

template <class V>
__device__ __forceinline__ void copy_part(const V *__restrict__ src, V *__restrict__ dst, size_t n) {
    const size_t stride = (size_t)gridDim.x * kThreads;
    bool told = false;
    for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < n; i += kBatch * stride) {
        V v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; k++)
            if (i + k * stride < n) v[k] = src[i + k * stride];
        if (i + kBatch * stride >= n) {
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            told = true;
        }
#pragma unroll
        for (int k = 0; k < kBatch; k++)
            if (i + k * stride < n) dst[i + k * stride] = v[k];
    }
    if (!told) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__global__ void __launch_bounds__(kThreads) frame_copy_kernel(const float *src, float *dst, size_t n) {
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 && n % 4 == 0)
        copy_part(reinterpret_cast<const float4 *>(src), reinterpret_cast<float4 *>(dst), n / 4);
    else
        copy_part(src, dst, n);
}

}  // namespace

cudaError_t launch_frame_copy(const float *host, float *dst, size_t n, cudaStream_t s) {
    const size_t want = (n / 4 + kThreads - 1) / kThreads;
    const unsigned grid = (unsigned)(want < kBlocks ? (want ? want : 1) : kBlocks);
    return launch_maybe_pdl(true, frame_copy_kernel, dim3(grid), dim3(kThreads), 0, s, host, dst, n);
}

}  // namespace glsfft
