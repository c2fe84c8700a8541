// fft_rows.cu -- instantiations and launcher of the row-pass kernel.
#include "fft_config.h"
#include "fft_kernels.cuh"

namespace glsfft {

// The real-input and argmax row passes (phaseCorrelate, the FFT display,
// promoted CV_32FC1 input) take row schedule 2's shape on 2048- and
// 4096-point rows -- 32 values per thread, as the complex pass does by
// default there -- with the same radix order, so the same results.
template <int N, int LD, int ST>
constexpr PassShape rows_fixed_shape() {
    return (N >= 2048 && !(LD == LD_C2 && ST == ST_C2)) ? row_shape(N, 2) : row_shape(N, 0);
}

// Rows per block.  Grids of many blocks take the fixed shape's; a grid that
// would leave SMs idle or unevenly loaded takes the SMs' even share of its
// rows instead, in one block per SM where that fits 512 threads: 512 rows of
// 512 points are 128 blocks of 4 rather than 64 of 8.
// Whole warps only.
static int row_lines(int fixed, int threads_per_line, int max_lines, long long total) {
    const int sms = sm_count();
    if (sms <= 0 || total >= 4LL * fixed * sms) return fixed;
    const int unit = threads_per_line < 32 ? 32 / threads_per_line : 1;
    for (int k = 1;; k++) {
        int lines = (int)((total + (long long)sms * k - 1) / ((long long)sms * k));
        lines = (lines + unit - 1) / unit * unit;
        if (lines <= max_lines) return lines;
    }
}

template <int N, int LD, int ST>
static cudaError_t rows_t(const PassArgs &a, int images, cudaStream_t s) {
    // Up to eight 1024- or 2048-point rows per SM: blocks of 128 threads with 16
    // values each, two rows or one.  GB300, CV_32FC1 512 x 2048 8.74 -> 8.20
    // us, phaseCorrelate 128 x 2048 23.5 -> 21.2 (from blocks of 4 and 1 rows
    // with 32 values a thread); 512 x 1024 forward + inverse 12.18 -> 11.82.
    // At 4096 points 32 values stay the better (28.5 us against 29.4 on 512
    // rows), at 512 points the even share (1024 rows 11.97 against 12.23).
    if constexpr (N == 1024 || (N == 2048 && !(LD == LD_C2 && ST == ST_C2))) {
        const long long total = (long long)a.rows * images, sms = sm_count();
        if (a.spread && total <= 8 * sms && (N == 2048 || total > sms)) {
            constexpr int LINES = 2048 / N;
            const size_t smem = sizeof(float2) * (size_t)LINES * padded_count(N);
            return launch_pass(fft_rows_kernel<N, 16, LINES, LD, ST>, dim3((a.rows + LINES - 1) / LINES, images),
                               LINES * (N / 16), smem, s, a);
        }
    }
    constexpr PassShape sh = rows_fixed_shape<N, LD, ST>();
    constexpr int E = sh.E, T = N / E, MAXL = cmax(sh.G, 512 / T);
    const int lines = a.spread ? row_lines(sh.G, T, MAXL, (long long)a.rows * images) : sh.G;
    const size_t smem =
        num_passes(N) > 1 ? sizeof(float2) * (size_t)lines * padded_count(N) : 0;
    auto kern = fft_rows_kernel<N, E, MAXL, LD, ST, sh.MB>;
    dim3 grid((a.rows + lines - 1) / lines, images);
    return launch_pass(kern, grid, lines * T, smem, s, a);
}

template <int LD, int ST>
static cudaError_t rows_n(int n, const PassArgs &a, int images, cudaStream_t s) {
    switch (n) {
    case 1: return rows_t<1, LD, ST>(a, images, s);
    case 2: return rows_t<2, LD, ST>(a, images, s);
    case 4: return rows_t<4, LD, ST>(a, images, s);
    case 8: return rows_t<8, LD, ST>(a, images, s);
    case 16: return rows_t<16, LD, ST>(a, images, s);
    case 32: return rows_t<32, LD, ST>(a, images, s);
    case 64: return rows_t<64, LD, ST>(a, images, s);
    case 128: return rows_t<128, LD, ST>(a, images, s);
    case 256: return rows_t<256, LD, ST>(a, images, s);
    case 512: return rows_t<512, LD, ST>(a, images, s);
    case 1024: return rows_t<1024, LD, ST>(a, images, s);
    case 2048: return rows_t<2048, LD, ST>(a, images, s);
    case 4096: return rows_t<4096, LD, ST>(a, images, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_rows(int n, int ld, int st, const PassArgs &a, int images, cudaStream_t s) {
    if (ld == LD_C2 && st == ST_C2) return rows_n<LD_C2, ST_C2>(n, a, images, s);
    if (ld == LD_R1 && st == ST_C2) return rows_n<LD_R1, ST_C2>(n, a, images, s);
    if (ld == LD_R1W && st == ST_C2) return rows_n<LD_R1W, ST_C2>(n, a, images, s);
    if (ld == LD_C2 && st == ST_RE_ARGMAX) return rows_n<LD_C2, ST_RE_ARGMAX>(n, a, images, s);
    return cudaErrorInvalidValue;
}

}  // namespace glsfft
