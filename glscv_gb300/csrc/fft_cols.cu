// fft_cols.cu -- instantiations and launcher of the column-pass kernel.
#include "fft_config.h"
#include "fft_kernels.cuh"

namespace glsfft {

template <int N, int W, int LD, int ST>
static cudaError_t cols_w(const PassArgs &a, int images, cudaStream_t s) {
    constexpr int E = cols_E(N), T = cols_T(N);
    constexpr int threads = W * T;
    constexpr size_t smem = num_passes(N) > 1 ? sizeof(float2) * (size_t)padded_count(N * W) : 0;
    auto kern = fft_cols_kernel<N, E, W, LD, ST>;
    dim3 grid((a.cols + W - 1) / W, images);
    return launch_pass(kern, grid, threads, smem, s, a);
}

// Columns per block: the fixed shape's W, or half as many while that leaves
// more than a third of the SMs without a block, down to one warp or 4 columns
// (32-byte row segments, whole DRAM sectors): 512 columns of 512 points are
// 128 blocks of 4 rather than 32 of 16.
template <int N, int W, int LD, int ST>
static cudaError_t cols_t(const PassArgs &a, int images, cudaStream_t s) {
    if constexpr (N >= 64 && W >= 8 && W / 2 * cols_T(N) >= 32) {
        if (a.spread && 3 * (((long long)a.cols * images + W - 1) / W) < 2 * sm_count())
            return cols_t<N, W / 2, LD, ST>(a, images, s);
    }
    return cols_w<N, W, LD, ST>(a, images, s);
}

// 2048-point columns.  Up to two rounds of one 8-column block per SM take
// that (64-byte row segments), many rounds the streamed pass, which overlaps a
// tile's copy with the one before it; between them 4 columns, two blocks per
// SM.  GB300, us with 4 columns / 8 / streamed: 1024 columns 12.5 / 10.6 /
// 12.6, 2048 20.7 / 18.7 / 20.7, 4096 39.6 / 43.7 / 42.6, 9472 82 / 84 / 72.
// All give the same bits.
template <int LD, int ST>
static cudaError_t cols_2048(const PassArgs &a, int images, cudaStream_t s) {
    const long long total = (long long)a.cols * images, round = 8LL * sm_count();
    if (a.spread && total <= 2 * round && total >= round / 2) return cols_w<2048, 8, LD, ST>(a, images, s);
    if (a.spread && total >= 5 * round && stream_pass_applies(2048, true, a, images, ST))
        return launch_stream_pass(2048, true, a, images, s, ST);
    return cols_t<2048, cols_W(2048), LD, ST>(a, images, s);
}

template <int LD, int ST>
static cudaError_t cols_n(int n, const PassArgs &a, int images, cudaStream_t s) {
    switch (n) {
    case 1: return cols_t<1, cols_W(1), LD, ST>(a, images, s);
    case 2: return cols_t<2, cols_W(2), LD, ST>(a, images, s);
    case 4: return cols_t<4, cols_W(4), LD, ST>(a, images, s);
    case 8: return cols_t<8, cols_W(8), LD, ST>(a, images, s);
    case 16: return cols_t<16, cols_W(16), LD, ST>(a, images, s);
    case 32: return cols_t<32, cols_W(32), LD, ST>(a, images, s);
    case 64: return cols_t<64, cols_W(64), LD, ST>(a, images, s);
    case 128: return cols_t<128, cols_W(128), LD, ST>(a, images, s);
    case 256: return cols_t<256, cols_W(256), LD, ST>(a, images, s);
    case 512: return cols_t<512, cols_W(512), LD, ST>(a, images, s);
    case 1024: return cols_t<1024, cols_W(1024), LD, ST>(a, images, s);
    case 2048: return cols_2048<LD, ST>(a, images, s);
    case 4096: return cols_t<4096, cols_W(4096), LD, ST>(a, images, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_cols(int n, int ld, int st, const PassArgs &a, int images, cudaStream_t s) {
    if (ld == LD_C2 && st == ST_C2) return cols_n<LD_C2, ST_C2>(n, a, images, s);
    if (ld == LD_C2 && st == ST_LOGMAG_MINMAX) return cols_n<LD_C2, ST_LOGMAG_MINMAX>(n, a, images, s);
    return cudaErrorInvalidValue;
}

}  // namespace glsfft
