// poc.cu -- fused phaseCorrelate column kernel (the centroid finish is fused
// into the inverse row pass, fft_kernels.cuh).
#include "fft_config.h"
#include "fft_kernels.cuh"

namespace glsfft {

// W columns per block, or half as many while that leaves more than a third of
// the SMs without a block (as the plain column pass, fft_cols.cu): 1024 x 512
// 32.0 -> 28.3 us a call, 64 x 64 24.3 -> 22.2.  Not below 4 columns: 16-byte
// pieces write half sectors (1024 x 64 complex columns 10.6 us with 4, 13.5
// with 2).
template <int N, int W = poc_W(N)>
static cudaError_t poc_t(const PassArgs &a, cudaStream_t s) {
    constexpr int E = poc_E(N), T = poc_T(N);
    if constexpr (N >= 64 && W >= 8 && W / 2 * T >= 32) {
        if (a.spread && 3 * ((a.cols + W - 1) / W) < 2 * sm_count()) return poc_t<N, W / 2>(a, s);
    }
    constexpr int threads = W * T;
    constexpr size_t one = num_passes(N) > 1 ? sizeof(float2) * (size_t)padded_count(N * W) : 0;
    const size_t smem = a.flags & PF_F1_SPECTRUM ? one : 2 * one;  // an exchange buffer per spectrum
    auto kern = poc_cols_kernel<N, E, W>;
    dim3 grid((a.cols + W - 1) / W, 1);
    return launch_pass(kern, grid, threads, smem, s, a);
}

cudaError_t launch_poc_cols(int n, const PassArgs &a, cudaStream_t s) {
    // more tiles than SMs: the persistent pass, whose blocks copy the next
    // tile while they finish one.  GB300, us a synchronous call, this / the
    // plain kernel: 2048^2 82.6 / 89.4, 2048 x 4096 148 / 170, 4096^2 297 /
    // 387, 2048 x 1024 48.7 / 50.0, 1024 x 2048 49.0 / 49.0; with one tile per
    // SM or fewer there is nothing to overlap: 1024^2 33.3 / 31.9.
    if ((long long)a.cols * n > 8192LL * sm_count() && poc_stream_applies(n, a)) return launch_poc_stream(n, a, s);
    switch (n) {
    case 1: return poc_t<1>(a, s);
    case 2: return poc_t<2>(a, s);
    case 4: return poc_t<4>(a, s);
    case 8: return poc_t<8>(a, s);
    case 16: return poc_t<16>(a, s);
    case 32: return poc_t<32>(a, s);
    case 64: return poc_t<64>(a, s);
    case 128: return poc_t<128>(a, s);
    case 256: return poc_t<256>(a, s);
    case 512: return poc_t<512>(a, s);
    case 1024: return poc_t<1024>(a, s);
    case 2048: return poc_t<2048>(a, s);
    case 4096: return poc_t<4096>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace glsfft
