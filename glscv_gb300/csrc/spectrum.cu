// spectrum.cu -- the spectrum operations next to the FFT (mulSpectrums,
// mulSpectrumsPhaseOnly, magSpectrums, logMagSpectrums), gls::minMaxLoc,
// gls::normalize(NORM_MINMAX) and glsCam's FFT display pipeline, on device
// buffers.  The element kernels are HBM-bound streams (grid-stride, one
// complex or float per thread per step); minMaxLoc is a key reduction with one
// atomic per block; normalize reads the min / max keys on the device, so the
// display pipeline needs no host round trip.
//
// Reference (paths inside glsCV):
//   mulSpectrums / PhaseOnly / magSpectrums / logMagSpectrums
//                          glsCV/glsBasicOperation.cpp:320-351, shaders :92-212
//   minMaxLoc              glsCV/glsMinMaxLoc.cpp:65-119, :149-200
//   normalize NORM_MINMAX  glsCV/glsNormalize.cpp:52-68
//   glsCam FFT view        glsCam/glsCam.cpp:196-203
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "capi_internal.h"
#include "fft_device.cuh"
#include "glsfft.h"
#include "glsfft_internal.h"
#include "pdl.cuh"
#include "spectrum_device.cuh"

using namespace glsfft;

namespace {

constexpr int kThreads = 256;

// Blocks for n elements: one wave of the kernel's resident blocks at most
// (grid-stride beyond).  A grid of more blocks than fit at once would run a
// partial second wave at a fraction of the occupancy.  KERN's resident blocks
// are looked up once per device.
template <auto KERN>
int grid_for(size_t n) {
    static std::atomic<int> known[64];  // resident blocks per device, 0 = not looked up
    int dev = 0, cap = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) cap = known[dev].load(std::memory_order_relaxed);
    if (!cap) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, kThreads, 0) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 1;
        }
        cap = std::max(sm_count(), 1) * std::max(per_sm, 1);
        if (dev >= 0 && dev < 64) known[dev].store(cap, std::memory_order_relaxed);
    }
    const size_t want = (n + kThreads - 1) / kThreads;
    return (int)(want < (size_t)cap ? (want ? want : 1) : (size_t)cap);
}

// The element kernels move 16 bytes per load and store (two complex or four
// float values per step; a scalar loop covers a misaligned or odd tail) and
// issue the loads of two steps (four for the float-input kernels) before
// using them, so each thread keeps several loads in flight and a grid of
// eight resident blocks per SM streams at HBM rate.
__device__ __forceinline__ bool al16(const void *p) {
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// d may equal a or b (in place): each element is read, then written, by one thread
template <int OP>  // 0: a*b, 1: a*conj(b), 2: phase only
__device__ __forceinline__ float2 spec_binary_op(float2 x, float2 y) {
    return OP == 0 ? spec_mul<false>(x, y) : OP == 1 ? spec_mul<true>(x, y) : spec_poc(x, y);
}
template <int OP>
__global__ void __launch_bounds__(kThreads) spec_binary_kernel(const float2 *a, const float2 *b,
                                                              float2 *d, size_t n) {
    pdl_wait();
    const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t done = 0;
    if (al16(a) && al16(b) && al16(d)) {
        const size_t nv = n / 2;
        const float4 *a4 = reinterpret_cast<const float4 *>(a);
        const float4 *b4 = reinterpret_cast<const float4 *>(b);
        float4 *d4 = reinterpret_cast<float4 *>(d);
        auto step = [&](const float4 x, const float4 y) {
            const float2 r0 = spec_binary_op<OP>(make_float2(x.x, x.y), make_float2(y.x, y.y));
            const float2 r1 = spec_binary_op<OP>(make_float2(x.z, x.w), make_float2(y.z, y.w));
            return make_float4(r0.x, r0.y, r1.x, r1.y);
        };
        size_t i = tid;
        for (; i + stride < nv; i += 2 * stride) {  // both steps' loads in flight
            const float4 x0 = a4[i], y0 = b4[i], x1 = a4[i + stride], y1 = b4[i + stride];
            d4[i] = step(x0, y0);
            d4[i + stride] = step(x1, y1);
        }
        if (i < nv) d4[i] = step(a4[i], b4[i]);
        done = nv * 2;
    }
    pdl_trigger();
    for (size_t i = done + tid; i < n; i += stride) d[i] = spec_binary_op<OP>(a[i], b[i]);
}

// magnitude or log-magnitude; with KEYS, also the minMaxLoc keys of the
// output (row-major index = element index)
template <bool LOG>
__device__ __forceinline__ float mag_op(float2 x, float offset) {
    return LOG ? spec_log_mag(x, offset) : spec_mag(x);
}
__device__ __forceinline__ void keys_add(float v, size_t i, unsigned long long &kmin,
                                         unsigned long long &kmax) {
    const unsigned long long k0 = min_key(v, (unsigned)i), k1 = max_key(v, (unsigned)i);
    kmin = k0 > kmin ? k0 : kmin;
    kmax = k1 > kmax ? k1 : kmax;
}
template <bool LOG, bool KEYS>
__global__ void __launch_bounds__(kThreads) spec_mag_kernel(const float2 *a, float *d, size_t n,
                                                           float offset,
                                                           unsigned long long *keys) {
    __shared__ unsigned long long red[2 * (kThreads / 32)];
    unsigned long long kmin = 0, kmax = 0;
    pdl_wait();
    const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t done = 0;
    if (al16(a) && al16(d)) {  // four complex in, four float out per step
        const size_t nv = n / 4;
        const float4 *a4 = reinterpret_cast<const float4 *>(a);
        float4 *d4 = reinterpret_cast<float4 *>(d);
        auto step = [&](size_t i, const float4 p, const float4 q) {
            const float4 r = make_float4(mag_op<LOG>(make_float2(p.x, p.y), offset),
                                         mag_op<LOG>(make_float2(p.z, p.w), offset),
                                         mag_op<LOG>(make_float2(q.x, q.y), offset),
                                         mag_op<LOG>(make_float2(q.z, q.w), offset));
            d4[i] = r;
            if constexpr (KEYS) {
                keys_add(r.x, 4 * i, kmin, kmax);
                keys_add(r.y, 4 * i + 1, kmin, kmax);
                keys_add(r.z, 4 * i + 2, kmin, kmax);
                keys_add(r.w, 4 * i + 3, kmin, kmax);
            }
        };
        size_t i = tid;
        for (; i + stride < nv; i += 2 * stride) {  // both steps' loads in flight
            const float4 p0 = a4[2 * i], q0 = a4[2 * i + 1];
            const float4 p1 = a4[2 * (i + stride)], q1 = a4[2 * (i + stride) + 1];
            step(i, p0, q0);
            step(i + stride, p1, q1);
        }
        if (i < nv) step(i, a4[2 * i], a4[2 * i + 1]);
        done = nv * 4;
    }
    pdl_trigger();
    for (size_t i = done + tid; i < n; i += stride) {
        const float v = mag_op<LOG>(a[i], offset);
        d[i] = v;
        if constexpr (KEYS) keys_add(v, i, kmin, kmax);
    }
    if constexpr (KEYS) block_minmax_commit(kmin, kmax, red, keys);
}

// Each thread visits its indices in increasing order, so a running strict
// compare keeps its first occurrence; keys are formed once per thread for the
// block reduction.  Starting from the literal excludes what the reference
// excludes (NaN and values at or beyond it never compare).
struct MinMaxRun {
    float vmin = kMinMaxLiteral, vmax = -kMinMaxLiteral;
    unsigned imin = 0, imax = 0;
    __device__ __forceinline__ void add(float v, unsigned i) {
        if (v < vmin) {
            vmin = v;
            imin = i;
        }
        if (v > vmax) {
            vmax = v;
            imax = i;
        }
    }
    __device__ __forceinline__ void commit(unsigned long long *red, unsigned long long *keys) const {
        block_minmax_commit(min_key(vmin, imin), max_key(vmax, imax), red, keys);
    }
};

// The key reset in front of minmax_kernel: launched in stream order (so no
// earlier reader of the keys can still be running), it lets the min / max
// pass, launched as its programmatic dependent, start streaming at once.
__global__ void minmax_reset_kernel(unsigned long long *keys) {
    keys[0] = 0ull;
    keys[1] = 0ull;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// 16-byte loads in flight per thread of the min / max pass
constexpr int kMinMaxBatch = 8;
// Its blocks: enough for every thread to fill one batch, or two per SM while
// that is fewer (a thread runs its whole batch, so a grid of one load per
// thread spends seven of eight slots on nothing: 1081 x 1919 with
// normalisation 10.1 us, 6.7 with this).
template <bool PARTIAL>
int minmax_grid(size_t n);

// PARTIAL = false: after minmax_reset_kernel, the keys are reduced over the
// grid by atomics.  The input was complete before the reset kernel started
// (stream order); only the keys come from it, so the pass waits for its
// predecessor grid (griddepcontrol.wait, a no-op without programmatic launch)
// just before it commits them.
// PARTIAL = true: block b leaves its two keys in keys[2b], keys[2b + 1], for
// a reader that reduces them itself (normalize_kernel): no reset and no
// atomics.  The input may come from the grid before, so the wait comes first.
template <bool PARTIAL>
__global__ void __launch_bounds__(kThreads) minmax_kernel(const float *x, size_t n,
                                                          unsigned long long *keys) {
    __shared__ unsigned long long red[2 * (kThreads / 32)];
    MinMaxRun run;
    if constexpr (PARTIAL) pdl_wait();
    const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t done = 0;
    if (al16(x)) {
        const size_t nv = n / 4;
        const float4 *x4 = reinterpret_cast<const float4 *>(x);
        // eight independent 16-byte loads in flight before the compares (a
        // read-only stream needs more bytes in flight per thread than a copy;
        // the visiting order per thread stays increasing).  The last batch is
        // predicated, its missing slots NaN, which never compares, so the
        // ragged end costs one round trip rather than one per load.
        constexpr int kBatch = kMinMaxBatch;
        const float4 none = make_float4(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff),
                                        __int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
        for (size_t i = tid; i < nv; i += kBatch * stride) {
            float4 v[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; k++) v[k] = i + k * stride < nv ? x4[i + k * stride] : none;
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const unsigned b = (unsigned)(4 * (i + k * stride));
                run.add(v[k].x, b);
                run.add(v[k].y, b + 1);
                run.add(v[k].z, b + 2);
                run.add(v[k].w, b + 3);
            }
        }
        done = nv * 4;
    }
    if constexpr (PARTIAL) pdl_trigger();
    for (size_t i = done + tid; i < n; i += stride) run.add(x[i], (unsigned)i);
    if constexpr (PARTIAL) {
        const ulonglong2 k = block_minmax(min_key(run.vmin, run.imin), max_key(run.vmax, run.imax), red);
        if (threadIdx.x == 0) reinterpret_cast<ulonglong2 *>(keys)[blockIdx.x] = k;
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the keys are reset
        run.commit(red, keys);
    }
}

// dst = (float)(alpha - scl*min) + scl*src, scl = (float)(beta-alpha) / (float)(max-min)
// The keys are `parts` pairs, the result their extremes.  Before the grid in
// front (which made them) is over, a block already has its first values: the
// source is complete when that grid runs (it reads it), and an in-place
// destination is written only after the wait.
// RAW: the source is written by the grid in front (the FFT display's column
// pass), so the values wait too.
template <bool RAW>
__global__ void __launch_bounds__(kThreads) normalize_kernel(const float *x, float *d, size_t n,
                                                             const unsigned long long *keys,
                                                             int parts, double alpha, double beta) {
    __shared__ unsigned long long red[2 * (kThreads / 32)];
    __shared__ float2 s_lin;
    const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const bool vec = al16(x) && al16(d);
    const size_t nv = vec ? n / 4 : 0;
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    float4 *d4 = reinterpret_cast<float4 *>(d);
    constexpr int kBatch = 4;  // loads in flight; the last batch predicated (one round trip)
    float4 v[kBatch];
    auto fetch = [&](size_t i) {
#pragma unroll
        for (int k = 0; k < kBatch; k++)
            v[k] = i + k * stride < nv ? x4[i + k * stride] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    if constexpr (RAW) pdl_wait();
    fetch(tid);
    if constexpr (!RAW) pdl_wait();
    unsigned long long kmin = 0, kmax = 0;
    for (int i = threadIdx.x; i < parts; i += kThreads) {
        const ulonglong2 k = __ldcg(reinterpret_cast<const ulonglong2 *>(keys) + i);
        kmin = k.x > kmin ? k.x : kmin;
        kmax = k.y > kmax ? k.y : kmax;
    }
    if (parts > 1) {
        const ulonglong2 k = block_minmax(kmin, kmax, red);
        kmin = k.x;
        kmax = k.y;
    }
    // one thread runs the FP64 steps: GB300's FP64 pipe takes 16 cycles a
    // warp instruction (1081 x 1919, min / max and normalisation: 8.0 us with
    // every thread computing them, 6.7 with one)
    if (threadIdx.x == 0) {
        const double mn = min_key_value(kmin), mx = max_key_value(kmax);
        const float f = __fdiv_rn((float)(beta - alpha), (float)(mx - mn));
        s_lin = make_float2(f, (float)__dsub_rn(alpha, __dmul_rn((double)f, mn)));
    }
    __syncthreads();
    pdl_trigger();
    const float scl = s_lin.x, c = s_lin.y;
    auto step = [&](const float4 q) {
        return make_float4(__fadd_rn(c, __fmul_rn(scl, q.x)), __fadd_rn(c, __fmul_rn(scl, q.y)),
                           __fadd_rn(c, __fmul_rn(scl, q.z)), __fadd_rn(c, __fmul_rn(scl, q.w)));
    };
    for (size_t i = tid; i < nv;) {
#pragma unroll
        for (int k = 0; k < kBatch; k++)
            if (i + k * stride < nv) d4[i + k * stride] = step(v[k]);
        i += kBatch * stride;
        if (i < nv) fetch(i);
    }
    for (size_t i = nv * 4 + tid; i < n; i += stride) d[i] = __fadd_rn(c, __fmul_rn(scl, x[i]));
}

template <bool PARTIAL>
int minmax_grid(size_t n) {
    const size_t nv = (n + 3) / 4;
    const size_t least = std::min(nv, (size_t)2 * kThreads * (size_t)std::max(sm_count(), 1));
    return grid_for<minmax_kernel<PARTIAL>>(std::max((nv + kMinMaxBatch - 1) / kMinMaxBatch, least));
}

bool misaligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) != 0; }

// whether [p, p + pb) and [q, q + qb) overlap
bool overlap(const void *p, size_t pb, const void *q, size_t qb) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
    return a < b + qb && b < a + pb;
}

int check_elem(glsfft_context ctx, const void *p0, const void *p1, const void *p2, size_t al,
               int rows, int cols) {
    if (!ctx || !p0 || !p1 || !p2) return GLSFFT_ERROR_INVALID_VALUE;
    if (rows < 1 || cols < 1 || (long long)rows * cols > (1ll << 31)) return GLSFFT_ERROR_SIZE;
    if (misaligned(p0, al) || misaligned(p1, al)) return GLSFFT_ERROR_MISALIGNED;
    return GLSFFT_SUCCESS;
}

// the context's workspace holds the two keys at offset `off`
int keys_at(glsfft_context ctx, size_t off, unsigned long long **keys) {
    const int st = ensure_workspace(ctx, off + 256);
    if (st) return st;
    *keys = reinterpret_cast<unsigned long long *>(static_cast<char *>(ctx->ws) + off);
    return GLSFFT_SUCCESS;
}

}  // namespace

extern "C" {

int glsfft_mul_spectrums(glsfft_context ctx, const void *src0, const void *src1, void *dst,
                         int rows, int cols, int conj, void *stream) {
    int st = check_elem(ctx, src0, src1, dst, sizeof(float2), rows, cols);
    if (!st && misaligned(dst, sizeof(float2))) st = GLSFFT_ERROR_MISALIGNED;
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    const auto *a = static_cast<const float2 *>(src0);
    const auto *b = static_cast<const float2 *>(src1);
    auto *d = static_cast<float2 *>(dst);
    cudaStream_t s = (cudaStream_t)stream;
    // every element kernel is launched as its predecessor's programmatic
    // dependent: resident while that drains
    return cuda_status(conj ? launch_maybe_pdl(true, spec_binary_kernel<1>, grid_for<spec_binary_kernel<1>>(n),
                                               kThreads, 0, s, a, b, d, n)
                            : launch_maybe_pdl(true, spec_binary_kernel<0>, grid_for<spec_binary_kernel<0>>(n),
                                               kThreads, 0, s, a, b, d, n));
}

int glsfft_mul_spectrums_phase_only(glsfft_context ctx, const void *src0, const void *src1,
                                    void *dst, int rows, int cols, void *stream) {
    int st = check_elem(ctx, src0, src1, dst, sizeof(float2), rows, cols);
    if (!st && misaligned(dst, sizeof(float2))) st = GLSFFT_ERROR_MISALIGNED;
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    return cuda_status(launch_maybe_pdl(true, spec_binary_kernel<2>, grid_for<spec_binary_kernel<2>>(n),
                                        kThreads, 0, (cudaStream_t)stream,
                                        static_cast<const float2 *>(src0),
                                        static_cast<const float2 *>(src1), static_cast<float2 *>(dst), n));
}

int glsfft_mag_spectrums(glsfft_context ctx, const void *src, float *dst, int rows, int cols,
                         void *stream) {
    int st = check_elem(ctx, src, src, dst, sizeof(float2), rows, cols);
    if (!st && misaligned(dst, sizeof(float))) st = GLSFFT_ERROR_MISALIGNED;
    // the CV_32FC1 output must not overlap the CV_32FC2 input (a new GlsMat, as getDstMat gives)
    if (!st && overlap(src, 8 * (size_t)rows * cols, dst, 4 * (size_t)rows * cols))
        st = GLSFFT_ERROR_INVALID_VALUE;
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    auto kern = spec_mag_kernel<false, false>;
    return cuda_status(launch_maybe_pdl(true, kern, grid_for<spec_mag_kernel<false, false>>(n), kThreads, 0,
                                        (cudaStream_t)stream, static_cast<const float2 *>(src), dst, n,
                                        0.0f, nullptr));
}

int glsfft_log_mag_spectrums(glsfft_context ctx, const void *src, float *dst, int rows, int cols,
                             float offset, void *stream) {
    int st = check_elem(ctx, src, src, dst, sizeof(float2), rows, cols);
    if (!st && misaligned(dst, sizeof(float))) st = GLSFFT_ERROR_MISALIGNED;
    if (!st && overlap(src, 8 * (size_t)rows * cols, dst, 4 * (size_t)rows * cols))
        st = GLSFFT_ERROR_INVALID_VALUE;
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    auto kern = spec_mag_kernel<true, false>;
    return cuda_status(launch_maybe_pdl(true, kern, grid_for<spec_mag_kernel<true, false>>(n), kThreads, 0,
                                        (cudaStream_t)stream, static_cast<const float2 *>(src), dst, n,
                                        offset, nullptr));
}

int glsfft_min_max_loc_async(glsfft_context ctx, const float *src, int rows, int cols,
                             unsigned long long *d_keys, void *stream) {
    int st = check_elem(ctx, src, src, d_keys, sizeof(float), rows, cols);
    if (!st && misaligned(d_keys, 8)) st = GLSFFT_ERROR_MISALIGNED;
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    minmax_reset_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(d_keys);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_status(e);
    return cuda_status(launch_maybe_pdl(true, minmax_kernel<false>, minmax_grid<false>(n),
                                        kThreads, 0, (cudaStream_t)stream, src, n, d_keys));
}

int glsfft_min_max_loc(glsfft_context ctx, const float *src, int rows, int cols,
                       double *min_val, double *max_val, int *min_loc, int *max_loc,
                       void *stream) {
    int st = check_elem(ctx, src, src, src, sizeof(float), rows, cols);
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    unsigned long long *keys = nullptr;
    st = keys_at(ctx, 0, &keys);
    if (st) return st;
    st = glsfft_min_max_loc_async(ctx, src, rows, cols, keys, stream);
    if (st) return st;
    unsigned long long *h = reinterpret_cast<unsigned long long *>(ctx->h_result);
    cudaError_t e = cudaMemcpyAsync(h, keys, 2 * sizeof(unsigned long long),
                                    cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_status(e);
    const unsigned imin = key_idx(h[0]), imax = key_idx(h[1]);
    if (min_val) *min_val = min_key_value(h[0]);
    if (max_val) *max_val = max_key_value(h[1]);
    if (min_loc) {
        min_loc[0] = (int)(imin % (unsigned)cols);
        min_loc[1] = (int)(imin / (unsigned)cols);
    }
    if (max_loc) {
        max_loc[0] = (int)(imax % (unsigned)cols);
        max_loc[1] = (int)(imax / (unsigned)cols);
    }
    return GLSFFT_SUCCESS;
}

int glsfft_normalize_minmax(glsfft_context ctx, const float *src, float *dst, int rows, int cols,
                            double alpha, double beta, void *stream) {
    int st = check_elem(ctx, src, dst, dst, sizeof(float), rows, cols);
    if (st) return st;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    // two launches: every block's keys, then the normalisation, whose blocks
    // reduce them (a reset and atomics would be a third)
    const int parts = std::min(minmax_grid<true>(n), ctx->key_pairs);
    unsigned long long *keys = nullptr;
    // the blocks' keys have memory of their own (d_keys), but the call keeps
    // its contract: it claims the workspace like the other reductions, so it
    // ends the last phaseCorrelate's surface and fails where the budget has no
    // room for them
    st = keys_at(ctx, 0, &keys);
    if (st) return st;
    keys = ctx->d_keys;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = launch_maybe_pdl(true, minmax_kernel<true>, parts, kThreads, 0, s, src, n, keys);
    if (e != cudaSuccess) return cuda_status(e);
    return cuda_status(launch_maybe_pdl(true, normalize_kernel<false>, grid_for<normalize_kernel<false>>(n / 4),
                                        kThreads, 0, s, src, dst, n, (const unsigned long long *)keys, parts,
                                        alpha, beta));
}

int glsfft_fft_display(glsfft_context ctx, const float *frame, const float *window, float *dst,
                       int rows, int cols, float offset, void *stream) {
    if (!ctx || !frame || !dst) return GLSFFT_ERROR_INVALID_VALUE;
    int st = check_dims(rows, cols);
    if (st) return st;
    if (misaligned(frame, 4) || misaligned(dst, 4) || (window && misaligned(window, 4)))
        return GLSFFT_ERROR_MISALIGNED;
    DeviceGuard g(ctx->device);
    if (!g.ok()) return GLSFFT_ERROR_CUDA;
    const size_t n = (size_t)rows * cols;
    const size_t spec_bytes = (n * sizeof(float2) + 255) / 256 * 256;
    unsigned long long *keys = nullptr;
    st = keys_at(ctx, spec_bytes, &keys);
    if (st) return st;
    cudaStream_t s = (cudaStream_t)stream;
    float2 *spec = static_cast<float2 *>(ctx->ws);
    // rows: window * frame promoted to complex, FFT of every row, half swap;
    // the row kernel also zeroes the min / max keys
    PassArgs r{};
    r.in0 = frame;
    r.out0 = spec;
    r.window = window;
    r.rows = rows;
    r.cols = cols;
    r.scale = 1.0f;
    r.flags = PF_SHIFT_COLS;
    r.tw = ctx->d_tw;
    r.key = keys;
    r.pdl = r.spread = 1;  // the three launches are chained by programmatic dependent launch
    cudaError_t e = launch_rows(cols, window ? LD_R1W : LD_R1, ST_C2, r, 1, s);
    if (e != cudaSuccess) return cuda_status(e);
    if (rows > 1) {
        // columns: FFT of every column, half swap, log(|X| + offset) and its min / max
        PassArgs c{};
        c.in0 = spec;
        c.out0 = dst;
        c.rows = rows;
        c.cols = cols;
        c.scale = 1.0f;
        c.flags = PF_SHIFT_ROWS;
        c.key = keys;
        c.tw = ctx->d_tw;
        c.param = offset;
        c.err = ctx->d_status;
        c.stall_ns = ctx->stall_ns;
        c.pdl = c.spread = 1;  // the plain column kernel; the streamed pass launches as usual
        // 4096-point columns: the streamed pass (TMA-fed, one block per SM)
        e = rows == 4096 && stream_pass_applies(rows, true, c, 1, ST_LOGMAG_MINMAX)
                ? launch_stream_pass(rows, true, c, 1, s, ST_LOGMAG_MINMAX)
                : launch_cols(rows, LD_C2, ST_LOGMAG_MINMAX, c, 1, s);
    } else {
        auto kern = spec_mag_kernel<true, true>;
        kern<<<grid_for<spec_mag_kernel<true, true>>(n), kThreads, 0, s>>>(spec, dst, n, offset, keys);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return cuda_status(e);
    // normalize(0, 1, NORM_MINMAX) in place
    return cuda_status(launch_maybe_pdl(true, normalize_kernel<true>, grid_for<normalize_kernel<true>>(n / 4),
                                        kThreads, 0, s, (const float *)dst, dst, n,
                                        (const unsigned long long *)keys, 1, 0.0, 1.0));
}

}  // extern "C"
