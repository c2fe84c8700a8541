// Host unit test of the serving loop's failure path (glscv_gb300/csrc/serve.cpp)
// against a fake CUDA runtime, built by the host compiler: when a launch fails
// after a request's frame copy and row pass were issued, the request's device
// memory goes to the next request only once those have finished.
#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "capi_internal.h"
#include "glsfft.h"
#include "glsfft_internal.h"

using namespace glsfft;

namespace {

std::mutex mu;
std::condition_variable changed;
bool open_ = false;     // nothing is issued before every request is queued
int at_columns = 0;     // requests that reached their failing launch
int reused = 0, copies = 0;
std::atomic<long> next_handle{16};

struct Use {  // issued work that writes [from, to) and is not known to have finished
    cudaStream_t s;
    const char *from, *to;
};
std::vector<Use> in_use;

void *handle() { return reinterpret_cast<void *>(next_handle.fetch_add(16)); }

void issue(cudaStream_t s, const void *dst, size_t bytes) {
    std::lock_guard<std::mutex> lock(mu);
    const Use u{s, static_cast<const char *>(dst), static_cast<const char *>(dst) + bytes};
    for (const Use &o : in_use) reused += o.s != s && o.from < u.to && u.from < o.to;
    in_use.push_back(u);
}

}  // namespace

// ---------------------------------------------------- the fake CUDA runtime
extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { *a = *b = 0; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = static_cast<cudaStream_t>(handle()); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return cudaStreamCreateWithFlags(s, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    for (size_t i = in_use.size(); i-- > 0;)
        if (in_use[i].s == s) in_use.erase(in_use.begin() + i);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = static_cast<cudaEvent_t>(handle()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) {
    std::unique_lock<std::mutex> lock(mu);
    changed.wait(lock, [] { return open_; });
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *, size_t n, cudaMemcpyKind, cudaStream_t s) {
    issue(s, dst, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *at, const void *p) {
    *at = cudaPointerAttributes{};
    at->type = cudaMemoryTypeHost;
    at->devicePointer = at->hostPointer = const_cast<void *>(p);
    return cudaSuccess;
}
}

// ------------------------------------------- the library behind the server
namespace glsfft {
DeviceGuard::DeviceGuard(int) {}
DeviceGuard::~DeviceGuard() {}
int cuda_status(cudaError_t e) { return e == cudaSuccess ? GLSFFT_SUCCESS : GLSFFT_ERROR_CUDA; }
int check_dims(int, int) { return GLSFFT_SUCCESS; }
cudaError_t launch_frame_copy(const float *, float *dst, size_t n, cudaStream_t s) {
    copies++;
    issue(s, dst, 4 * n);
    return cudaSuccess;
}
cudaError_t launch_rows(int, int, int st, const PassArgs &a, int, cudaStream_t s) {
    if (st == ST_C2) issue(s, a.out0, 8 * (size_t)a.rows * a.cols);
    return cudaSuccess;
}
cudaError_t launch_cols(int, int, int, const PassArgs &, int, cudaStream_t) { return cudaSuccess; }
// fails, the first two requests' launches only once both have come so far
cudaError_t launch_poc_cols(int, const PassArgs &, cudaStream_t) {
    std::unique_lock<std::mutex> lock(mu);
    at_columns++;
    changed.notify_all();
    changed.wait(lock, [] { return at_columns >= 2; });
    return cudaErrorLaunchOutOfResources;
}
}  // namespace glsfft

// Queue the requests on a server of its own, then let it run: every one fails.
static bool all_fail(int slots, bool direct, const std::vector<int> &sides) {
    constexpr int SMALL = 512, BIG = 1024;
    constexpr size_t PX = (size_t)BIG * BIG, REFS = 8 * (PX + (size_t)SMALL * SMALL);
    open_ = false;
    glsfft_context_s ctx;
    glsfft_server srv = nullptr;
    // the references (8 bytes a pixel) and one big request (16) or several small ones
    int bad = glsfft_server_create(&ctx, slots, REFS + 16 * PX + 4096, &srv);
    std::vector<float> frame(PX);
    int big = -1, small = -1;
    bad |= glsfft_server_add_reference(srv, frame.data(), nullptr, BIG, BIG, &big);
    bad |= glsfft_server_add_reference(srv, frame.data(), nullptr, SMALL, SMALL, &small);
    bad |= glsfft_server_set_frame_read(srv, direct);
    std::vector<long long> tickets(sides.size());
    for (size_t k = 0; k < sides.size(); k++)
        bad |= glsfft_server_submit(srv, sides[k] == BIG ? big : small, frame.data(), 5, &tickets[k]);
    {
        std::lock_guard<std::mutex> lock(mu);
        open_ = true;
    }
    changed.notify_all();
    size_t failed = 0;
    for (long long t : tickets) failed += glsfft_server_wait(srv, t, nullptr, nullptr, 30.0) == GLSFFT_ERROR_CUDA;
    glsfft_server_destroy(srv);
    return !bad && failed == sides.size();
}

int main() {
    bool ok = true;
    for (bool direct : {true, false}) {
        // two small requests side by side on two slots; the big one takes the
        // memory of both on the first slot
        at_columns = 0;
        ok = all_fail(4, direct, {512, 512, 1024}) && ok;
    }
    // a big frame by the link stream's copy kernel, then a small request in its memory
    ok = all_fail(1, true, {1024, 512}) && ok && copies == 1;
    std::printf("frame copies %d, memory reused too early %d times\n", copies, reused);
    ok = ok && reused == 0;
    std::printf(ok ? "ALL OK\n" : "FAILED\n");
    return !ok;
}
