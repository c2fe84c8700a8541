// glsfft_internal.h -- shared declarations between the C ABI and the kernel
// translation units.  Not a public header.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace glsfft {

constexpr int kMaxLen = 4096;  // largest supported FFT length per dimension

// Per-pass twiddle tables: for a pass of radix R whose sub-transforms have
// length L (= span * R), butterfly position k < L/R needs w^r =
// e^{-2 pi i k r / L}, r < R/2 (the line engine derives the rest).  They are
// stored as L/R-entry vectors of two neighbouring r each -- entry (k, r) at
// ((r / 2) * (L / R) + k) * 2 + r % 2 (radix 2: at k) -- so the consecutive
// butterflies of a warp read consecutive 16-byte words: a warp's load is four
// 128-byte lines, where rows of R/2 entries per k made it touch up to 32.
// Measured on GB300 against such rows: 4096^2 forward + inverse 292 -> 254
// us, 1024^2 22.3 -> 20.9 us, 37 x 256 x 512 26.6 -> 24.6 us.  All tables
// live in one buffer of kTwEntries float2, table (R, L) at tw_offset(R, L).
constexpr int kTwRadixSpan = 8192;
constexpr int kTwEntries = 4 * kTwRadixSpan;
__host__ __device__ constexpr int tw_radix_index(int r) {
    return r == 2 ? 0 : r == 4 ? 1 : r == 8 ? 2 : 3;
}
__host__ __device__ constexpr int tw_offset(int r, int l) {
    return tw_radix_index(r) * kTwRadixSpan + l;
}
__host__ __device__ constexpr int tw_entry(int radix, int l, int k, int r) {
    return radix == 2 ? k : ((r / 2) * (l / radix) + k) * 2 + r % 2;
}

// load modes of the first pass
enum { LD_C2 = 0, LD_R1 = 1, LD_R1W = 2 };
// store modes of the last pass
// ST_LOGMAG_MINMAX: log(|sqrt(re^2 + im^2) + param|) stored as CV_32FC1, with
// the minMaxLoc keys of the stored values reduced into key[0] (min), key[1] (max)
enum { ST_C2 = 0, ST_RE = 1, ST_RE_ARGMAX = 2, ST_LOGMAG_MINMAX = 3 };
// per-pass flags
enum : unsigned {
    PF_CONJ_IN = 1u << 0,
    PF_CONJ_OUT = 1u << 1,
    PF_SHIFT_ROWS = 1u << 2,
    PF_SHIFT_COLS = 1u << 3,
    PF_F1_SPECTRUM = 1u << 4,
    PF_EVICT_IN = 1u << 5,  // row passes: the input leaves the L2 first
};

// PF_EVICT_IN (2048- and 4096-point rows) where a row pass's input and result
// overflow the 129 MB L2 and the result alone does not: the input is read
// once, and the lines it leaves behind push out the result's rows that the
// column pass reads next.  Measured on GB300, forward + inverse: 2048 x 4096
// 110.1 -> 105.0 us, 4096 x 2048 128.0 -> 122.1, 40 x 64x4096 98.8 -> 91.2, one
// 4096^2 241.0 -> 236.1.  Not where both fit, as a caller that transforms the
// same image again would lose it (2048^2 forward 26.4 -> 27.4), nor for larger
// results (8 x 1024x2048 197.4 -> 199.0).  1024-point rows gain less than the
// policy operand costs 1024^2 (17.8 -> 18.0).
inline unsigned evict_in(size_t in_bytes, size_t out_bytes, int images) {
    constexpr size_t kL2 = size_t(1) << 27;
    return in_bytes + out_bytes >= kL2 && (out_bytes < kL2 || images == 1) ? PF_EVICT_IN : 0u;
}

struct PassArgs {
    const void *in0;
    const void *in1;
    void *out0;
    void *out1;
    const float *window;
    int rows, cols;
    float scale;
    unsigned flags;
    unsigned long long *key;
    const float2 *tw;  // twiddle table of this pass's length
    size_t in_img_bytes;   // batch: byte stride between images (0 = single / in1 mode)
    size_t out_img_bytes;
    float param;       // ST_LOGMAG_MINMAX: the log-magnitude offset
    // ST_RE_ARGMAX with `result` set: the last block to finish computes the
    // phaseCorrelate centroid (box edge `box`) into result[0..4].  key[0] is
    // the argmax key, key[1] the block counter, key[2] nonzero if a tile wait
    // of the column pass ran out (the result then says so: poc_result); the
    // call's first row pass zeroes all three
    double *result;
    int box;
    // with `result`: set to 1 (after a system-scope fence) once result[0..4]
    // are written, for a host that waits on it instead of the stream; or null
    unsigned long long *done_flag;
    // device status word for bounded waits (the streamed passes record
    // GLSFFT_ERROR_TIMEOUT there), or null
    int *err;
    // fault injection for tests (the TMA-fed passes): when > 0, each block
    // leaves its first tile's copy unissued and waits this many nanoseconds
    // for it, so the wait runs out
    long long stall_ns;
    // a small grid may take other block shapes, to spread evenly over the SMs
    // (row_lines, cols_t), and lets its successor in late (launch_pass): not a
    // launch that always runs beside other streams' (the server's)
    int spread;
    // launch with programmatic dependent launch (every pass kernel begins
    // with griddepcontrol.wait): the grid may become resident before its
    // stream predecessor ends
    int pdl;
};

// Launchers (fft_rows.cu, fft_cols.cu, poc.cu).  They return cudaSuccess or
// the launch error; `images` is the grid's y extent (blockIdx.y = image).
cudaError_t launch_rows(int n, int ld, int st, const PassArgs &a, int images, cudaStream_t s);
cudaError_t launch_cols(int n, int ld, int st, const PassArgs &a, int images, cudaStream_t s);
cudaError_t launch_poc_cols(int n, const PassArgs &a, cudaStream_t s);

// A whole 2-D FFT in one launch (fft_fused.cu): whether the image size is
// one it takes, and the launch over `images` contiguous images -- in0, out0,
// rows, cols, tw, in_img_bytes, both passes' flags, `scale` after the rows
// and `scale_cols` after the columns; real_in: in0 holds CV_32FC1 images.
bool fused_applies(int rows, int cols);
cudaError_t launch_fused(const PassArgs &a, bool real_in, float scale_cols, int images,
                         cudaStream_t s);

// n floats of page-locked host memory to dst by a kernel on a few SMs
// (frame_copy.cu).  It does not wait for its predecessor on the stream beyond
// that one's last loads: the caller makes sure nobody else uses dst.
cudaError_t launch_frame_copy(const float *host, float *dst, size_t n, cudaStream_t s);

// The persistent phaseCorrelate column pass (poc_stream.cu): whether it takes
// these arguments (1024-, 2048- or 4096-point columns, whole tiles, 16-byte
// aligned, the call's key words), and its launch.
bool poc_stream_applies(int n, const PassArgs &a);
cudaError_t launch_poc_stream(int n, const PassArgs &a, cudaStream_t s);

// The streamed column pass for 2048- and 4096-point columns (fft_stream.cu;
// cols must be true): whether it applies to these arguments (contiguous
// complex images, 16-byte aligned, the column count a multiple of the
// tile's; store mode ST_C2, or ST_LOGMAG_MINMAX over one image), and the
// launch, which gives cudaErrorNotSupported when it does not apply.
bool stream_pass_applies(int n, bool cols, const PassArgs &a, int images, int st = ST_C2);
cudaError_t launch_stream_pass(int n, bool cols, const PassArgs &a, int images, cudaStream_t s,
                               int st = ST_C2);

// A 2-D tensor map over a row-major array of 8-byte elements (width x
// height, rows `width` elements apart) with a box_w x box_h box, for TMA
// copies (batch.cpp); `swizzle`: the 16-byte chunks of a box's rows of 32 or
// 64 bytes permuted (the TMA's 32B or 64B mode).  GLSFFT_SUCCESS or an error
// status.
int make_tmap_2d(void *tmap128, const void *base, long long width, long long height, int box_w,
                 int box_h, bool swizzle = false);
// The same with boxes higher than the 256 elements a box dimension may have:
// a 3-D map (width, 256, height / 256) whose box is box_w x box_rows; height
// and box_rows are multiples of 256.
int make_tmap_rows(void *tmap128, const void *base, long long width, long long height, int box_w,
                   int box_rows, bool swizzle = false);

// SMs of the current device (0 on failure), looked up once per device.
int sm_count();

// Opt kernel `kern` into `bytes` of dynamic shared memory on the current
// device.  The attribute belongs to the kernel's instance on one device, so
// this runs once per (kernel, device) (thread-safe; capi.cpp).
cudaError_t smem_opt_in(const void *kern, size_t bytes);

// Twiddle tables: one device buffer of kTwEntries float2 holding the
// per-pass tables of fft_device.cuh (tw_offset).  Generated in FP64 on the
// host and rounded once to FP32.
void make_twiddle_host(float2 *dst /* kTwEntries entries */);

}  // namespace glsfft
