// fft_stream.cu -- the streamed column pass for 2048- and 4096-point columns
// (pass schedule kSchedStreamed).
//
// A tile of the plain column kernel for 4096-point columns (4 columns, 32
// bytes of each image row: the narrowest segment that keeps whole DRAM
// sectors) is 128 KB, so an SM holds one tile at a time and loads,
// transforms and stores it in turn: HBM idles while the SM computes.  Here
// one persistent 1024-thread block per SM walks the column tiles of the
// batch (image-major, then tile) and keeps the NEXT tile's copy in flight
// while it transforms the current one:
//   * the tile (L columns x N rows, L * N * 8 = 128 KB) lands in a
//     shared-memory stage as one tensor box (Tensor Memory Accelerator, one
//     tensor map over the whole batch), completing on an mbarrier;
//   * every thread copies its 16 values of one column to registers, the
//     block syncs, and thread 0 at once issues the next tile's copy;
//   * the Stockham passes exchange through a separate buffer of half the
//     tile's size, so that stage + exchange fit one SM (128 KB + 68 KB).  For
//     complex results the threads are two groups, each with half the columns,
//     that take turns on it (SyncTurns); for log-magnitudes, whose register
//     stores want a warp to have whole row segments, all columns exchange
//     together, real and imaginary parts one after the other.  GB300, there
//     and back, halves -> turns: 4 x 2048^2 233.5 -> 226.3 us, 4096 x 1024
//     65.1 -> 64.2, 4096^2 231.6 -> 229.1; the 4096^2 display 135.7 -> 164.4,
//     and 152.1 with its stores by the TMA;
//   * complex results go out the same way: a quarter of the tile's rows at a
//     time is laid out in one of two halves of the exchange buffer and stored
//     by the TMA while the next quarter is written and the next tile read.
//     Stored from registers, every 32-byte row segment (4096 points) is a
//     wavefront of its own in the load / store unit, 2.9 of a tile's 9.7 us
//     (GB300, 4096^2 image: 72.0 us a pass with register stores, 67.9 with
//     these).  Log-magnitudes are stored from registers.
// The arithmetic is the plain kernels' (same radix order, twiddle tables and
// rounding), so the results are bit-identical to schedule 0.  The wait for a
// tile is bounded: on expiry the kernel records GLSFFT_ERROR_TIMEOUT in the
// context's device status word, waits (bounded) for its copy in flight and
// returns.  Row variants of the same design measured slower than row
// schedule 2 and are not built.
#include <cuda.h>

#include "fft_config.h"
#include "fft_kernels.cuh"
#include "glsfft.h"
#include "glsfft_internal.h"
#include "sched_internal.h"
#include "tma_device.cuh"

namespace glsfft {

namespace {

constexpr unsigned kStreamTileBytes = 128u * 1024u;
constexpr long long kStreamWaitNs = 2000000000ll;  // 2 s per tile: a safety bound only

template <int N>
__host__ __device__ constexpr int stream_lines() {
    return (int)(kStreamTileBytes / (N * sizeof(float2)));
}
// Complex results: the exchanges by turns; log-magnitudes: in halves (above).
template <int ST>
__host__ __device__ constexpr bool stream_turns() {
    return ST == ST_C2;
}
// half the tile's columns at once, or all, one component at a time
template <int N>
__host__ __device__ constexpr size_t stream_xchg_bytes() {
    static_assert(sizeof(float) * (size_t)col_split_floats(stream_lines<N>() * N) <=
                  sizeof(float2) * (size_t)padded_count(stream_lines<N>() / 2 * N), "exchange buffer");
    constexpr size_t b = sizeof(float2) * (size_t)padded_count(stream_lines<N>() / 2 * N);
    return (b + 15) & ~size_t(15);
}
template <int N>
__host__ __device__ constexpr size_t stream_smem() {
    return 512 + kStreamTileBytes + stream_xchg_bytes<N>() + 16;
}
template <int N, int E>
__host__ __device__ constexpr int stream_threads() {
    return stream_lines<N>() * (N / E);
}

// The maps of one launch; each views the batch as (rows * images) x cols
// 8-byte elements.
struct StreamMaps {
    CUtensorMap in;   // L x N boxes of the input: a tile in one copy
    CUtensorMap out;  // L x 256 boxes of the output
};

// Issue the copy of tile `tile` (image tile / tpi, columns (tile % tpi) * L
// onward) into the stage, completing on `full`.  FIRST: the block's first
// tile, when nothing else is to be done: in 256-row boxes through the output's
// map if the pass is in place, which arrive sooner (4096 x 256 there and back
// 29.9 -> 29.7 us).  Later tiles are one copy each: a thread that issues
// 16 boxes is held until the TMA has taken them, 2 us at 4096 points, and the
// others wait for it at the next barrier (4096^2 there and back 237.2 -> 233.1
// us, its FFT display 147.1 -> 136.4).
template <int N, bool FIRST>
__device__ __forceinline__ void stream_issue(const StreamMaps &maps, const PassArgs &a, int tile,
                                             int tpi, float2 *stage, unsigned long long *full,
                                             bool inject = false) {
    constexpr int L = stream_lines<N>();
    const int x = (tile % tpi) * L, img = tile / tpi;
    mbar_arrive_tx(full, kStreamTileBytes);
    if (inject) return;  // fault injection: the copy is never issued
    if (FIRST && a.in0 == a.out0) {
#pragma unroll
        for (int b = 0; b < N / 256; b++)
            tensor2d_g2s(stage + b * 256 * L, &maps.out, x, img * N + b * 256, full);
    } else {
        tensor3d_g2s(stage, &maps.in, x, 0, img * (N / 256), full);
    }
}

// ST: ST_C2 (complex out), or, over one image, ST_LOGMAG_MINMAX (the FFT
// display epilogue of the plain column kernel: log(|X| + param) as CV_32FC1
// and the minMaxLoc keys of what is stored, reduced over all of the block's
// tiles and committed once)
template <int N, int E, int ST>
__global__ void __launch_bounds__(stream_threads<N, E>(), 1)
    fft_stream_cols(const __grid_constant__ StreamMaps maps, const PassArgs a, int images) {
    constexpr int L = stream_lines<N>(), T = N / E;
    static_assert(N % 256 == 0, "column tiles are read as 256-row boxes");
    static_assert(ST == ST_C2 || ST == ST_LOGMAG_MINMAX, "stream store modes");
    extern __shared__ unsigned char stream_raw[];
    // 512-byte aligned stage (the period of the boxes' swizzle); offsetting the shared array itself (not a cast
    // integer) keeps the compiler's shared-window addressing
    unsigned char *base = stream_raw + ((512u - (smem_u32(stream_raw) & 511u)) & 511u);
    float2 *stage = reinterpret_cast<float2 *>(base);
    float2 *xch = reinterpret_cast<float2 *>(base + kStreamTileBytes);
    unsigned long long *full =
        reinterpret_cast<unsigned long long *>(base + kStreamTileBytes + stream_xchg_bytes<N>());

    pdl_enter();  // before the first tile copy reads the input
    const int tid = threadIdx.x;
    const int tpi = a.cols / L;  // tiles per image
    const int total = tpi * images;
    // c: column among the thread's group's, t: position thread, l: column of
    // the tile, slot: where row t of a box has that column.  With turns, a
    // group has every other 16-byte pair of columns, and the boxes' 16-byte
    // chunks are permuted by the TMA (rows of 32 or 64 bytes: its 32B or 64B
    // mode), so that a group's accesses fall on distinct banks.
    constexpr bool TURNS = stream_turns<ST>();
    constexpr int HALF = L / 2 * T;
    const int c = TURNS ? tid % HALF % (L / 2) : tid % L;
    const int t = TURNS ? tid % HALF / (L / 2) : tid / L;
    const int l = TURNS ? 4 * (c / 2) + 2 * (tid / HALF) + c % 2 : c;
    const int slot = t * L + (!TURNS ? l : l ^ ((L == 4 ? t >> 2 & 1 : t >> 1 & 3) << 1));

    if (tid == 0) {
        mbar_init(full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int tile = blockIdx.x;
    const bool inject = a.stall_ns > 0;
    if (tid == 0 && tile < total) stream_issue<N, true>(maps, a, tile, tpi, stage, full, inject);
    // a half swap of the columns inside one tile (a.cols == L) is no box
    const bool tma_out = ST == ST_C2 && (!(a.flags & PF_SHIFT_COLS) || a.cols > L);
    unsigned parity = 0;
    MinMaxAny run;  // ST_LOGMAG_MINMAX only
    const long long limit = inject ? a.stall_ns : kStreamWaitNs;
    for (; tile < total; tile += gridDim.x) {
        const bool ok = mbar_wait(full, parity, limit);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                if (a.err) atomicExch(a.err, (int)GLSFFT_ERROR_TIMEOUT);
                // the copy in flight, if one was issued, and the stores
                if (!inject) mbar_wait(full, parity, kStreamWaitNs);
                bulk_wait<0>();
            }
            __syncthreads();
            return;
        }
        parity ^= 1u;
        float2 x[E];
#pragma unroll
        for (int m = 0; m < E; m++) x[m] = stage[slot + m * T * L];
        if (tid == 0) bulk_wait_read<0>();  // the exchange buffer is free
        __syncthreads();  // every thread has its values: the stage is free
        const int next = tile + gridDim.x;
        if (tid == 0 && next < total) stream_issue<N, false>(maps, a, next, tpi, stage, full);

        conj_line(x, a.flags & PF_CONJ_IN);
        if constexpr (TURNS)
            LineFft<N, E, SyncTurns<HALF>, 4>::run(x, t, ColSm<L / 2>{xch, c}, a.tw);
        else
            LineFft<N, E, SyncBlock, 4>::run(x, t, ColSmF<L>{reinterpret_cast<float *>(xch), l}, a.tw);
        finish_line(x, a.scale, a.flags & PF_CONJ_OUT);

        const int col = (tile % tpi) * L + l;
        const int ocol = (a.flags & PF_SHIFT_COLS) ? (col + (a.cols >> 1)) & (a.cols - 1) : col;
        char *out = static_cast<char *>(a.out0) + (size_t)(tile / tpi) * a.out_img_bytes;
        if constexpr (ST == ST_LOGMAG_MINMAX) {
            float *fo = reinterpret_cast<float *>(out);
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int pos = t + m * T;
                const int orow = (a.flags & PF_SHIFT_ROWS) ? (pos + (N >> 1)) & (N - 1) : pos;
                const unsigned o = (unsigned)orow * (unsigned)a.cols + (unsigned)ocol;
                const float v = spec_log_mag(x[m], a.param);
                fo[o] = v;
                run.add(v, o);
            }
        } else if (tma_out) {
            const int ox = ocol - l, y0 = (tile / tpi) * a.rows;
            constexpr int QROWS = N / 4, QM = E / 4;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float2 *buf = xch + (q & 1) * (QROWS * L);
                // q = 0: the exchange's last reads are done; from q = 2 on,
                // the store of two quarters ago has read the buffer
                if (q >= 2 && tid == 0) bulk_wait_read<1>();
                if (q != 1) __syncthreads();
#pragma unroll
                for (int m = 0; m < QM; m++) buf[slot + m * T * L] = x[q * QM + m];
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncthreads();
                if (tid == 0) {
                    const int row = (q * QROWS + ((a.flags & PF_SHIFT_ROWS) ? N / 2 : 0)) & (N - 1);
#pragma unroll
                    for (int b = 0; b < QROWS / 256; b++)
                        tensor2d_s2g(&maps.out, ox, y0 + row + b * 256, buf + b * 256 * L);
                    bulk_commit();
                }
            }
        } else {
            store_line<N, E, T>(reinterpret_cast<float2 *>(out) + ocol, (size_t)a.cols, x, t,
                                a.flags & PF_SHIFT_ROWS);
        }
    }
    if (tid == 0) bulk_wait<0>();  // the stores are complete
    if constexpr (ST == ST_LOGMAG_MINMAX) {
        __shared__ unsigned long long red[2 * (stream_threads<N, E>() / 32)];
        block_minmax_commit(run.kmin(), run.kmax(), red, a.key);
    }
}

template <int N, int E, int ST>
cudaError_t stream_launch(const PassArgs &a, int images, cudaStream_t s) {
    constexpr int L = stream_lines<N>();
    StreamMaps maps{};
    const long long height = (long long)a.rows * images;
    if (make_tmap_rows(&maps.in, a.in0, a.cols, height, L, N, stream_turns<ST>()) != GLSFFT_SUCCESS)
        return cudaErrorNotSupported;
    maps.out = maps.in;
    if (ST == ST_C2 && make_tmap_2d(&maps.out, a.out0, a.cols, height, L, 256, true) != GLSFFT_SUCCESS)
        return cudaErrorNotSupported;
    constexpr size_t smem = stream_smem<N>();
    auto kern = fft_stream_cols<N, E, ST>;
    cudaError_t e = smem_opt_in(reinterpret_cast<const void *>(kern), smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (sms <= 0) return cudaErrorNotSupported;
    const long long total = (long long)(a.cols / L) * images;
    const int grid = (int)(total < sms ? total : sms);
    return launch_maybe_pdl(a.pdl != 0, kern, dim3(grid), dim3(stream_threads<N, E>()), smem, s,
                            maps, a, images);
}

}  // namespace

bool stream_pass_applies(int n, bool cols, const PassArgs &a, int images, int st) {
    if (!cols || (n != 2048 && n != 4096)) return false;
    if (a.in1 || a.out1 || !a.in0 || !a.out0 || images < 1) return false;
    if (st != ST_C2 && !(st == ST_LOGMAG_MINMAX && images == 1 && a.key)) return false;
    const int L = (int)(kStreamTileBytes / (n * sizeof(float2)));
    if (a.rows != n || a.cols < L || a.cols % L) return false;
    const size_t img = (size_t)a.rows * a.cols * sizeof(float2);
    if (images > 1 && (a.in_img_bytes != img || a.out_img_bytes != img)) return false;
    const uintptr_t in = reinterpret_cast<uintptr_t>(a.in0), out = reinterpret_cast<uintptr_t>(a.out0);
    return (in % 16) == 0 && (out % (st == ST_C2 ? 16 : 4)) == 0;
}

cudaError_t launch_stream_pass(int n, bool cols, const PassArgs &a, int images, cudaStream_t s,
                               int st) {
    if (!stream_pass_applies(n, cols, a, images, st)) return cudaErrorNotSupported;
    // 16 values per thread (1024 threads); 32 per thread (512 threads)
    // measured the same on GB300
    if (st == ST_LOGMAG_MINMAX)
        return n == 2048 ? stream_launch<2048, 16, ST_LOGMAG_MINMAX>(a, images, s)
                         : stream_launch<4096, 16, ST_LOGMAG_MINMAX>(a, images, s);
    return n == 2048 ? stream_launch<2048, 16, ST_C2>(a, images, s)
                     : stream_launch<4096, 16, ST_C2>(a, images, s);
}

}  // namespace glsfft
