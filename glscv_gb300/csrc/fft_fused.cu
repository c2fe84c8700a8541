// fft_fused.cu -- a whole 2-D FFT of a small image in one launch.
//
// An image of 16..256 points a side and at most 4,096 pixels (64 x 64) fits
// one block's registers: every thread holds 16 values (8 where both sides are
// 32 or 64 points, whose radices are 8 or less: twice the warps for the same
// work).  The block loads the rows, transforms them, turns the image in
// shared memory, transforms the columns and stores them: one launch and one
// read and write of the image, where the two pass kernels need two launches
// and an intermediate in L2.  One block per image.  The lines are the pass
// kernels' own (same radix order, tables and rounding), so the results are
// bit-identical to theirs.
//
// What bounds it: for one image the host's launch rate and the latency of
// the chain load - line - turn - line - store.  Measured on GB300, 64 x 64
// forward + inverse, calls back to back: 9.9 us in four pass launches, 7.6
// us in two of these with 16 values a thread, 6.9 with 8.  Images of up to
// 65,536 pixels as a cluster of such blocks that exchange the columns through
// distributed shared memory were built too: no faster than two pass launches
// (128 x 128 5.5 against 5.0 us, 40 images of 256 x 256 13.2 against 13.3), so
// larger images take the pass kernels.
#include <type_traits>

#include "fft_config.h"
#include "fft_kernels.cuh"
#include "glsfft_internal.h"

namespace glsfft {

namespace {

constexpr int kFusedPx = 4096;  // pixels per image at most

// With 8 values per thread two buffers: the exchanges of the rows (inside one
// warp each) and of the columns go through the first, the turned image through
// the second, so the block meets at two barriers only (64 x 64: 3.51 -> 3.26
// us a call).  With 16 values one buffer serves all three in turn, each use
// behind a barrier (256 x 16: 4.9 us, with two buffers 5.7).
__host__ __device__ constexpr bool fused_two(int e) { return e == 8; }
template <int N, int E, int LD>
__device__ __forceinline__ void fused_rows(const PassArgs &a, const void *in, float2 *xch, float2 *turned,
                                           float2 (&x)[E]) {
    constexpr int T = N / E;
    const int l = threadIdx.x / T, t = threadIdx.x % T;
    const bool active = l < a.rows;
#pragma unroll
    for (int m = 0; m < E; m++)
        x[m] = active ? load_elem<LD>(in, nullptr, (size_t)l * N + t + m * T) : make_float2(0.f, 0.f);
    conj_line(x, a.flags & PF_CONJ_IN);
    using Sync = std::conditional_t<fused_two(E), SyncLines<T, 1>, SyncBlock>;
    LineFft<N, E, Sync>::run(x, t, RowSm{xch + l * padded_count(N)}, a.tw);
    finish_line(x, a.scale, false);
    if constexpr (!fused_two(E)) __syncthreads();
    if (active) {
        // row l of the image, in the column lines' [position][column] order:
        // kFusedPx / rows columns (those past the image are never read)
        const int lw = __ffs(kFusedPx / a.rows) - 1;
        const int sh = (a.flags & PF_SHIFT_COLS) ? N >> 1 : 0;
#pragma unroll
        for (int m = 0; m < E; m++) {
            const int i = (l << lw) + ((t + m * T + sh) & (N - 1));
            turned[i + (i >> 4)] = x[m];
        }
    }
    __syncthreads();
}

template <int N, int E>
__device__ __forceinline__ void fused_cols(const PassArgs &a, float scale, float2 *out, float2 *xch,
                                           const float2 *turned, float2 (&x)[E]) {
    constexpr int T = N / E, W = kFusedPx / N;
    const int c = threadIdx.x % W, t = threadIdx.x / W;
    const bool active = c < a.cols;
    const float2 *p = ColSm<W>{const_cast<float2 *>(turned), c}.at(t);
#pragma unroll
    for (int m = 0; m < E; m++) x[m] = active ? p[slot_step<ColSm<W>, T>(m)] : make_float2(0.f, 0.f);
    if constexpr (!fused_two(E)) __syncthreads();
    LineFft<N, E>::run(x, t, ColSm<W>{xch, c}, a.tw);
    finish_line(x, scale, a.flags & PF_CONJ_OUT);
    if (active) store_line<N, E, T>(out + c, (size_t)a.cols, x, t, a.flags & PF_SHIFT_ROWS);
}

template <int E, int LD>
__global__ void __launch_bounds__(kFusedPx / E) fft2d_fused_kernel(const PassArgs a, float scale_cols) {
    extern __shared__ float4 smem_raw[];
    float2 *xch = reinterpret_cast<float2 *>(smem_raw), *turned = fused_two(E) ? xch + padded_count(kFusedPx) : xch;
    pdl_enter();
    const void *in = image_in(a, blockIdx.x);
    float2 *out = static_cast<float2 *>(image_out(a, blockIdx.x));
    float2 x[E];
    if constexpr (E == 8) {
        if (a.cols == 32) fused_rows<32, E, LD>(a, in, xch, turned, x);
        else fused_rows<64, E, LD>(a, in, xch, turned, x);
        if (a.rows == 32) fused_cols<32, E>(a, scale_cols, out, xch, turned, x);
        else fused_cols<64, E>(a, scale_cols, out, xch, turned, x);
    } else {
        switch (a.cols) {
        case 16: fused_rows<16, E, LD>(a, in, xch, turned, x); break;
        case 32: fused_rows<32, E, LD>(a, in, xch, turned, x); break;
        case 64: fused_rows<64, E, LD>(a, in, xch, turned, x); break;
        case 128: fused_rows<128, E, LD>(a, in, xch, turned, x); break;
        default: fused_rows<256, E, LD>(a, in, xch, turned, x); break;
        }
        switch (a.rows) {
        case 16: fused_cols<16, E>(a, scale_cols, out, xch, turned, x); break;
        case 32: fused_cols<32, E>(a, scale_cols, out, xch, turned, x); break;
        case 64: fused_cols<64, E>(a, scale_cols, out, xch, turned, x); break;
        case 128: fused_cols<128, E>(a, scale_cols, out, xch, turned, x); break;
        default: fused_cols<256, E>(a, scale_cols, out, xch, turned, x); break;
        }
    }
}

template <int E, int LD>
cudaError_t fused_launch(const PassArgs &a, float scale_cols, int images, cudaStream_t s) {
    constexpr size_t smem = (fused_two(E) ? 2 : 1) * sizeof(float2) * (size_t)padded_count(kFusedPx);
    if constexpr (smem > 48 * 1024) {
        const cudaError_t e = smem_opt_in(reinterpret_cast<const void *>(fft2d_fused_kernel<E, LD>), smem);
        if (e != cudaSuccess) return e;
    }
    return launch_maybe_pdl(true, fft2d_fused_kernel<E, LD>, dim3(images), dim3(kFusedPx / E), smem, s,
                            a, scale_cols);
}

}  // namespace

bool fused_applies(int rows, int cols) {
    return rows >= 16 && cols >= 16 && rows * cols <= kFusedPx;
}

cudaError_t launch_fused(const PassArgs &a, bool real_in, float scale_cols, int images,
                         cudaStream_t s) {
    if ((a.rows == 32 || a.rows == 64) && (a.cols == 32 || a.cols == 64))
        return real_in ? fused_launch<8, LD_R1>(a, scale_cols, images, s)
                       : fused_launch<8, LD_C2>(a, scale_cols, images, s);
    return real_in ? fused_launch<16, LD_R1>(a, scale_cols, images, s)
                   : fused_launch<16, LD_C2>(a, scale_cols, images, s);
}

}  // namespace glsfft
