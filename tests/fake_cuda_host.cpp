// The library's host-only sources (memory.cu, host_copy.cu, host_spmm.cu) over a fake CUDA runtime of two devices
// whose memory is the host's: what the calls do to devices, streams and copies can be looked at without a GPU, and a
// failing call costs nothing.  Built and run by test_host_fake_cuda.py; argv[1] names the scenario.
#include "../iccad-accel-gcn_b200/csrc/internal.h"
#include "../iccad-accel-gcn_b200/csrc/host_copy.h"

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

static int failures = 0;
#define CHECK(cond) do { if (!(cond)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #cond); failures++; } } while (0)

// ---- the fake runtime --------------------------------------------------------------------------
namespace {
std::mutex g_mutex;
thread_local int t_device = 0;
std::map<void *, int> g_block_device;                    // device of every live block
std::map<cudaStream_t, int> g_stream_device;
int g_syncs[2] = {0, 0};                                 // device-wide waits
int g_wrong_device = 0;                                  // frees, allocations or copies on a stream of another device
int g_fail_free = 0;
bool g_capturing = false;
std::atomic<int> g_copies{0}, g_copies_waited_for{0};    // copies issued; how many of them the last stream wait covered
int g_fail_copy = 0;                                     // number of the copy that fails
thread_local int t_news_left = -1;                       // allocations of this thread until one fails

int stream_device(cudaStream_t s)
{
    std::lock_guard<std::mutex> l(g_mutex);
    const auto it = g_stream_device.find(s);
    return it == g_stream_device.end() ? t_device : it->second;      // the default and per-thread streams
}
cudaError_t event_of(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(std::malloc(8)); return cudaSuccess; }
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { std::lock_guard<std::mutex> l(g_mutex); g_syncs[t_device]++; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *props) { *p = reinterpret_cast<cudaMemPool_t>((intptr_t)props->location.id + 1); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **out, size_t bytes, cudaMemPool_t pool, cudaStream_t s)
{
    const int dev = (int)reinterpret_cast<intptr_t>(pool) - 1;
    if (stream_device(s) != dev) g_wrong_device++;
    *out = std::calloc(1, bytes);
    std::lock_guard<std::mutex> l(g_mutex);
    g_block_device[*out] = dev;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s)
{
    const int dev = stream_device(s);
    std::lock_guard<std::mutex> l(g_mutex);
    const auto it = g_block_device.find(p);
    if (it == g_block_device.end()) return cudaErrorInvalidValue;
    if (it->second != dev) { g_wrong_device++; return cudaErrorInvalidValue; }
    g_block_device.erase(it);
    std::free(p);
    return g_fail_free ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaHostAlloc(void **out, size_t bytes, unsigned) { *out = std::calloc(1, bytes); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = reinterpret_cast<cudaStream_t>(std::malloc(8));
    std::lock_guard<std::mutex> l(g_mutex);
    g_stream_device[*s] = t_device;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st)
{
    *st = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { g_copies_waited_for = g_copies.load(); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return event_of(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return event_of(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(reinterpret_cast<void *>(e)); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { if (stream_device(s) != t_device) g_wrong_device++; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (++g_copies == g_fail_copy) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
}

// ---- allocations that fail ---------------------------------------------------------------------
void *operator new(size_t bytes)
{
    if (t_news_left >= 0 && t_news_left-- == 0) throw std::bad_alloc();
    return std::malloc(bytes > 0 ? bytes : 1);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

// ---- what the sources under test call in the others --------------------------------------------
namespace agcn {
static std::string g_error;
void set_error(const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_error = buf;
}
void clear_error() { g_error.clear(); }
int env_int(const char *, int dflt) { return dflt; }
int spmm_create(agcn_spmm_plan **out, const int *, int64_t n_blocks, const int *, int64_t n_rows, int64_t n_cols, int64_t nnz, cudaStream_t)
{
    agcn_spmm_plan *p = new agcn_spmm_plan;
    p->n_blocks = n_blocks; p->n_rows = n_rows; p->n_cols = n_cols; p->nnz = nnz; p->n_units = ceil_div(n_blocks, 8);
    CHECK(cudaGetDevice(&p->device) == cudaSuccess);
    *out = p;
    return AGCN_OK;
}
void plan_free(agcn_spmm_plan *p) { delete p; }
int spmm_run(agcn_spmm_plan *p, const int *, const float *, const float *, int64_t, float *, int64_t, int, cudaStream_t, int, int)
{
    CHECK(p->device == t_device);
    return AGCN_OK;
}
int spmm_run_prepared(agcn_spmm_plan *p, const int *, const float *, const float *, int64_t, bool, float *, int64_t, int, cudaStream_t, int, int, const SpmmLaunchPart &)
{
    CHECK(p->device == t_device);
    return AGCN_OK;
}
int spmm_pad_rows(const float *, int64_t, int, float *, int64_t, cudaStream_t) { return AGCN_OK; }
int spmm_check_cols(const int *, int64_t, int64_t, int *, cudaStream_t) { return AGCN_OK; }
bool spmm_plan_splits(int64_t, int64_t, int64_t) { return false; }
}  // namespace agcn

// ---- scenarios ---------------------------------------------------------------------------------
// A host context made on device 1 is used, grown and destroyed while device 0 is current.
static void context_device()
{
    const int block4[8] = {2, 0, 0, (1 << 16) + 2, 2, 2, 4, (1 << 16) + 2}, idx[8] = {0, 1, 2, 3, 0, 1, 2, 3};
    const float val[8] = {1, 1, 1, 1, 1, 1, 1, 1};
    float x[4 * 64] = {}, y[4 * 64] = {};
    agcn_host_ctx *c = nullptr;
    cudaSetDevice(1);
    CHECK(agcn_host_ctx_create(&c) == AGCN_OK);
    CHECK(agcn_spmm_host(c, block4, 2, idx, val, x, y, 4, 4, 8, 16) == AGCN_OK);
    cudaSetDevice(0);
    CHECK(agcn_spmm_host(c, block4, 2, idx, val, x, y, 4, 4, 8, 64) == AGCN_OK);      // grows X and Y
    CHECK(agcn_host_set_graph(c, block4, 2, idx, val, 4, 4, 8) == AGCN_OK);
    CHECK(agcn_host_spmm(c, x, y, 33) == AGCN_OK);
    CHECK(t_device == 0);
    const int before = g_syncs[0];
    CHECK(agcn_host_ctx_destroy(c) == AGCN_OK);
    CHECK(t_device == 0);
    CHECK(g_syncs[0] == before);                         // the context's device was waited for, not this one
    CHECK(g_syncs[1] > 0);
    CHECK(g_wrong_device == 0);
    CHECK(g_block_device.empty());                       // and every buffer went back
    // a failing free is reported
    cudaSetDevice(1);
    CHECK(agcn_host_ctx_create(&c) == AGCN_OK);
    CHECK(agcn_spmm_host(c, block4, 2, idx, val, x, y, 4, 4, 8, 16) == AGCN_OK);
    g_fail_free = 1;
    CHECK(agcn_host_ctx_destroy(c) == AGCN_ERR_CUDA);
    g_fail_free = 0;
}

// A block allocated on a stream that is being captured would be the graph's: none is handed out.
static void pool_under_capture()
{
    void *p = nullptr;
    cudaSetDevice(0);
    g_capturing = true;
    CHECK(agcn::pool_alloc(&p, 64, nullptr) == cudaErrorStreamCaptureUnsupported);
    CHECK(p == nullptr && g_block_device.empty());
    g_capturing = false;
    CHECK(agcn::pool_alloc(&p, 64, nullptr) == cudaSuccess && p != nullptr);
    agcn::pool_free(p, nullptr);
    CHECK(g_block_device.empty());
}

// A copy that fails on one of several threads: the call fails, and by then nothing uses the shared buffers any more.
static void staged_copy_fails()
{
    std::vector<unsigned char> src(64 << 20, 7), dst(64 << 20, 0);
    const agcn::HostSegment seg = {dst.data(), src.data(), src.size()};
    for (const int k : {1, 9, 40}) {
        g_copies = 0; g_copies_waited_for = 0; g_fail_copy = k;
        CHECK(agcn::host_upload(&seg, 1, nullptr) == AGCN_ERR_CUDA);
        CHECK(g_copies >= k && g_copies_waited_for == g_copies);
    }
    g_fail_copy = 0;
    CHECK(agcn::host_upload(&seg, 1, nullptr) == AGCN_OK);
    CHECK(src == dst);
}

// No memory for the k-th thread: the call goes on with those that run, and no exception leaves it.
static void staged_copy_without_threads()
{
    std::vector<unsigned char> src(64 << 20, 9), dst(64 << 20), out(8 << 20, 1);
    const agcn::HostSegment seg = {dst.data(), src.data(), src.size()}, touched = {dst.data(), out.data(), out.size()};
    for (int k = 0; k < 18; k++) {
        std::memset(dst.data(), 0, dst.size());
        t_news_left = k;
        const int rc = agcn::host_upload(&seg, 1, nullptr, &touched, 1);
        t_news_left = -1;
        CHECK(rc == AGCN_OK && src == dst && out[12345] == 1);
    }
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "context_device") context_device();
    else if (what == "pool_under_capture") pool_under_capture();
    else if (what == "staged_copy_fails") staged_copy_fails();
    else if (what == "staged_copy_without_threads") staged_copy_without_threads();
    else { std::printf("unknown scenario\n"); return 2; }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
