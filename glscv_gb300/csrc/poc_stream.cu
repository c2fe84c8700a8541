// poc_stream.cu -- the fused phaseCorrelate column pass over many tiles
// (1024-, 2048- and 4096-point columns): one persistent block per SM that
// copies the next tile of both spectra in while it finishes the current one.
//
// A tile is 8192 values of each spectrum (8, 4 or 2 columns).  The plain
// kernel (fft_kernels.cuh) holds both in the registers of a whole SM, so each
// SM loads, transforms and stores a tile in turn: at 2048 points 2.7 us of
// load and 1.4 us of stores around 8 us of arithmetic, the accesses in 32-byte
// segments that each take a wavefront of the load / store unit.  Here three
// shared buffers of one tile take turns:
//   * the TMA copies the two spectra into buffers 1 and 2, each as one box (as
//     boxes of 256 rows, 16 or 32 of them, their issue held thread 0's warp,
//     and at the next barrier the block, for 800 to 4,000 of a tile's 20,000
//     cycles: 4096^2 311 us a call, 297 this way; 4096 x 1024 94.4 and 88.9);
//     the threads take their values to registers and both forward
//     transforms exchange through the same two buffers;
//   * then those are free, and the next tile's copy runs behind the phase, the
//     inverse transform (exchanging through buffer 0) and the store;
//   * the result is laid out in buffer 0 and stored by the TMA.
// Same lines, same order of operations: the bits are the plain kernel's.
// Measured on GB300 (a synchronous call): see launch_poc_cols.
//
// Every wait for a tile is bounded: on expiry the kernel marks the call's key
// words, from which the last pass makes a result that says so, records
// GLSFFT_ERROR_TIMEOUT in the status word if there is one, waits (bounded) for
// its copies in flight and returns.  Host-side fault injection (stall_ns): each
// block's first tile is not copied, and the wait for it runs out after that.
#include <cuda.h>

#include "fft_config.h"
#include "fft_kernels.cuh"
#include "glsfft.h"
#include "glsfft_internal.h"
#include "tma_device.cuh"

namespace glsfft {

namespace {

constexpr int kPocTile = 8192;  // values of one spectrum per tile
constexpr int kPocThreads = kPocTile / 16;
constexpr size_t kPocBuf = sizeof(float2) * (size_t)padded_count(kPocTile);
constexpr unsigned kPocTileBytes = kPocTile * sizeof(float2);
constexpr long long kPocWaitNs = 2000000000ll;
static_assert(kPocBuf % 128 == 0, "tensor boxes need 128-byte aligned buffers");

struct PocMaps {
    CUtensorMap in0, in1, out;
};

template <int N>
__global__ void __launch_bounds__(kPocThreads, 1)
    poc_stream_cols(const __grid_constant__ PocMaps maps, const PassArgs a) {
    constexpr int E = 16, T = N / E, W = kPocTile / N;
    using F = LineFft<N, E>;
    extern __shared__ unsigned char poc_raw[];
    unsigned char *base = poc_raw + ((128u - (smem_u32(poc_raw) & 127u)) & 127u);
    float2 *buf0 = reinterpret_cast<float2 *>(base);
    float2 *buf1 = reinterpret_cast<float2 *>(base + kPocBuf);
    float2 *buf2 = reinterpret_cast<float2 *>(base + 2 * kPocBuf);
    unsigned long long *full = reinterpret_cast<unsigned long long *>(base + 3 * kPocBuf);

    const int tid = threadIdx.x, c = tid % W, t = tid / W;
    const int total = a.cols / W;
    int tile = blockIdx.x;
    // both spectra of one tile: y (in1) into buffer 1, x (in0) into buffer 2
    auto issue = [&](int which) {
        mbar_arrive_tx(full, 2 * kPocTileBytes);
        tensor3d_g2s(buf1, &maps.in1, which * W, 0, 0, full);
        tensor3d_g2s(buf2, &maps.in0, which * W, 0, 0, full);
    };
    if (tid == 0) {
        mbar_init(full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_enter();
    const bool inject = a.stall_ns > 0;
    const long long limit = inject ? a.stall_ns : kPocWaitNs;
    if (tid == 0 && tile < total && !inject) issue(tile);
    unsigned parity = 0;
    for (; tile < total; tile += gridDim.x) {
        const bool ok = mbar_wait(full, parity, limit);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.key + 2, 1ull);
                if (a.err) atomicExch(a.err, (int)GLSFFT_ERROR_TIMEOUT);
                if (!inject) mbar_wait(full, parity, kPocWaitNs);
                bulk_wait<0>();
            }
            __syncthreads();
            return;
        }
        parity ^= 1u;
        float2 x[E], y[E];
#pragma unroll
        for (int m = 0; m < E; m++) {
            y[m] = buf1[(t + m * T) * W + c];
            x[m] = buf2[(t + m * T) * W + c];
        }
        __syncthreads();  // the exchanges overwrite the staged tile
        if (a.flags & PF_F1_SPECTRUM) F::run(y, t, ColSm<W>{buf1, c}, a.tw);
        else F::run2(x, y, t, ColSm<W>{buf2, c}, ColSm<W>{buf1, c}, a.tw);
        // this thread's exchange accesses are ordered before the next copy,
        // and the store of the tile before has read buffer 0
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (tid == 0) bulk_wait_read<0>();
        __syncthreads();
        const int next = tile + gridDim.x;
        if (tid == 0 && next < total) issue(next);
#pragma unroll
        for (int m = 0; m < E; m++) x[m] = poc_conj_phase(x[m], y[m]);
        F::run(x, t, ColSm<W>{buf0, c}, a.tw);
        __syncthreads();  // the last exchange has been read
#pragma unroll
        for (int m = 0; m < E; m++) buf0[(t + m * T) * W + c] = x[m];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            tensor3d_s2g(&maps.out, tile * W, 0, 0, buf0);
            bulk_commit();
        }
    }
    if (tid == 0) bulk_wait<0>();  // the stores are complete
}

template <int N>
cudaError_t poc_stream_t(const PassArgs &a, cudaStream_t s) {
    constexpr int W = kPocTile / N;
    PocMaps maps{};
    if (make_tmap_rows(&maps.in0, a.in0, a.cols, a.rows, W, N) != GLSFFT_SUCCESS ||
        make_tmap_rows(&maps.in1, a.in1, a.cols, a.rows, W, N) != GLSFFT_SUCCESS)
        return cudaErrorNotSupported;
    if (a.out0 == a.in0) maps.out = maps.in0;
    else if (a.out0 == a.in1) maps.out = maps.in1;
    else if (make_tmap_rows(&maps.out, a.out0, a.cols, a.rows, W, N) != GLSFFT_SUCCESS)
        return cudaErrorNotSupported;
    constexpr size_t smem = 128 + 3 * kPocBuf + 16;
    auto kern = poc_stream_cols<N>;
    const cudaError_t e = smem_opt_in(reinterpret_cast<const void *>(kern), smem);
    if (e != cudaSuccess) return e;
    const int tiles = a.cols / W, sms = sm_count();
    if (sms <= 0) return cudaErrorNotSupported;
    return launch_maybe_pdl(a.pdl != 0, kern, dim3(tiles < sms ? tiles : sms), dim3(kPocThreads), smem, s,
                            maps, a);
}

}  // namespace

bool poc_stream_applies(int n, const PassArgs &a) {
    if ((n != 1024 && n != 2048 && n != 4096) || a.rows != n || !a.key) return false;
    const int w = kPocTile / n;
    auto al16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return a.cols >= w && a.cols % w == 0 && al16(a.in0) && al16(a.in1) && al16(a.out0);
}

cudaError_t launch_poc_stream(int n, const PassArgs &a, cudaStream_t s) {
    return n == 1024 ? poc_stream_t<1024>(a, s)
         : n == 2048 ? poc_stream_t<2048>(a, s)
                     : poc_stream_t<4096>(a, s);
}

}  // namespace glsfft
