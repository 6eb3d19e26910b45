// Copies between the device and ordinary (pageable) host arrays.
//
// Given pageable memory, cudaMemcpy moves it through the driver's own small buffer on one thread: 6-12 GB/s,
// and where the destination is a fresh array that thread also takes its page faults.  The host-array entry
// points (degree sort, partitioner: what a caller does with arrays read from files) spent 90 % of their time
// there.  Here several threads move 1 MiB pieces through pinned buffers, two per thread, so that the page
// faults and the host-side copies run in parallel and the copy engine stays busy.
#include "host_copy.h"

#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

namespace agcn {

constexpr size_t STAGE_PIECE = (size_t)1 << 20;
constexpr int STAGE_THREADS = 12;                  // the link needs about 6 at 8-10 GB/s each; fresh pages cost as much again
// Threads beside these that only fault in the pages of the output arrays while the upload keeps the link busy: a
// fresh array is zeroed by the kernel page by page at its first write, which took 2 ms of 120 MB of outputs.
constexpr int TOUCH_THREADS = 4;
constexpr size_t TOUCH_PIECE = (size_t)2 << 20;
constexpr size_t STAGE_MIN_BYTES = (size_t)2 << 20;    // below this, starting threads costs more than it saves

// The pinned buffers: 24 MiB, made at the first use, given back by agcn_release_scratch.  One call at a time
// uses them; another that comes meanwhile takes the driver's path.
struct StageBuffers {
    std::mutex busy;
    unsigned char *memory = nullptr;
};
static StageBuffers g_stage;

static bool is_pinned(const void *p)
{
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type != cudaMemoryTypeUnregistered;
}

static cudaError_t copy_piece(const HostSegment &g, size_t at, void *piece, size_t bytes, bool up, cudaStream_t s)
{
    unsigned char *d = static_cast<unsigned char *>(g.device) + at;
    return up ? cudaMemcpyAsync(d, piece, bytes, cudaMemcpyHostToDevice, s) : cudaMemcpyAsync(piece, d, bytes, cudaMemcpyDeviceToHost, s);
}

static cudaError_t copy_plain(const HostSegment &g, bool up, cudaStream_t s) { return g.bytes == 0 ? cudaSuccess : copy_piece(g, 0, g.host, g.bytes, up, s); }

struct StageJob {
    const HostSegment *seg;
    int n;
    bool up;
    cudaStream_t stream;
    int device;
    std::atomic<size_t> next{0}, next_touch{0};
    std::atomic<int> error{0};
    const HostSegment *touch;
    int n_touch;
    size_t first[HOST_SEGMENTS_MAX + 1];           // first piece of every segment

    // piece i: its segment, offset and size; false past the end
    bool piece(size_t i, const HostSegment **g, size_t *at, size_t *bytes) const
    {
        if (i >= first[n]) return false;
        int k = 0;
        while (i >= first[k + 1]) k++;
        *g = &seg[k];
        *at = (i - first[k]) * STAGE_PIECE;
        *bytes = seg[k].bytes - *at < STAGE_PIECE ? seg[k].bytes - *at : STAGE_PIECE;
        return true;
    }

    // Faults in output pages, TOUCH_PIECE at a time, until none are left.  Their contents stay: an output may be
    // the array that is being uploaded.
    void touch_outputs()
    {
        for (;;) {
            size_t i = next_touch.fetch_add(1);
            const HostSegment *g = nullptr;
            for (int k = 0; k < n_touch; k++) {
                const size_t pieces = (touch[k].bytes + TOUCH_PIECE - 1) / TOUCH_PIECE;
                if (i < pieces) { g = &touch[k]; break; }
                i -= pieces;
            }
            if (g == nullptr) return;
            unsigned char *p = static_cast<unsigned char *>(g->host) + i * TOUCH_PIECE;
            const size_t bytes = g->bytes - i * TOUCH_PIECE < TOUCH_PIECE ? g->bytes - i * TOUCH_PIECE : TOUCH_PIECE;
            for (size_t at = 0; at < bytes; at += 4096) __atomic_fetch_or(p + at, (unsigned char)0, __ATOMIC_RELAXED);
            __atomic_fetch_or(p + bytes - 1, (unsigned char)0, __ATOMIC_RELAXED);
        }
    }

    void work(unsigned char *buffers)
    {
        cudaError_t e = cudaSetDevice(device);
        cudaEvent_t done[2] = {nullptr, nullptr};
        for (int b = 0; b < 2 && e == cudaSuccess; b++) e = cudaEventCreateWithFlags(&done[b], cudaEventDisableTiming);
        struct { const HostSegment *g; size_t at, bytes; bool busy; } held[2] = {};
        // Buffer b is in flight while held[b].busy; settle() waits for it and, going down, hands it on to the host array.
        auto settle = [&](int b) {
            if (!held[b].busy || e != cudaSuccess) return;
            e = cudaEventSynchronize(done[b]);
            if (e == cudaSuccess && !up) memcpy(static_cast<unsigned char *>(held[b].g->host) + held[b].at, buffers + b * STAGE_PIECE, held[b].bytes);
            held[b].busy = false;
        };
        for (int b = 0; e == cudaSuccess && error.load() == 0; b ^= 1) {
            settle(b);
            const HostSegment *g;
            size_t at, bytes;
            if (e != cudaSuccess || !piece(next.fetch_add(1), &g, &at, &bytes)) break;
            unsigned char *mine = buffers + b * STAGE_PIECE;
            if (up) memcpy(mine, static_cast<const unsigned char *>(g->host) + at, bytes);
            e = copy_piece(*g, at, mine, bytes, up, stream);
            if (e == cudaSuccess) e = cudaEventRecord(done[b], stream);
            held[b] = {g, at, bytes, true};
        }
        settle(0);
        settle(1);
        for (cudaEvent_t ev : done) if (ev != nullptr) cudaEventDestroy(ev);
        if (e != cudaSuccess) error.store((int)e);
    }
};

static int host_copy(const HostSegment *seg, int n, bool up, cudaStream_t s, const HostSegment *outputs, int n_outputs)
{
    AGCN_REQUIRE(n >= 0 && n <= HOST_SEGMENTS_MAX, "host copy: too many segments");
    HostSegment staged[HOST_SEGMENTS_MAX];
    int m = 0;
    size_t total = 0;
    for (int i = 0; i < n; i++) {
        if (seg[i].bytes == 0) continue;
        if (is_pinned(seg[i].host)) { AGCN_CUDA(copy_plain(seg[i], up, s)); continue; }
        staged[m++] = seg[i];
        total += seg[i].bytes;
    }
    std::unique_lock<std::mutex> lock(g_stage.busy, std::defer_lock);
    bool fast = total >= STAGE_MIN_BYTES && lock.try_lock();
    if (fast && g_stage.memory == nullptr &&
        cudaHostAlloc(reinterpret_cast<void **>(&g_stage.memory), STAGE_THREADS * 2 * STAGE_PIECE, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_stage.memory = nullptr;
        fast = false;
    }
    if (!fast) {
        for (int i = 0; i < m; i++) AGCN_CUDA(copy_plain(staged[i], up, s));
        return AGCN_OK;
    }
    HostSegment touch[HOST_SEGMENTS_MAX];
    StageJob job;
    job.touch = touch; job.n_touch = 0;
    for (int i = 0; i < n_outputs && i < HOST_SEGMENTS_MAX; i++)
        if (outputs[i].bytes > 0 && !is_pinned(outputs[i].host)) touch[job.n_touch++] = outputs[i];
    job.seg = staged; job.n = m; job.up = up; job.stream = s;
    AGCN_CUDA(cudaGetDevice(&job.device));
    job.first[0] = 0;
    for (int i = 0; i < m; i++) job.first[i + 1] = job.first[i] + (staged[i].bytes + STAGE_PIECE - 1) / STAGE_PIECE;
    const unsigned cores = std::thread::hardware_concurrency();
    int threads = cores > 1 ? (int)(cores < STAGE_THREADS ? cores : STAGE_THREADS) : 1;
    if ((size_t)threads > job.first[m]) threads = (int)job.first[m];
    std::thread pool[STAGE_THREADS], touchers[TOUCH_THREADS];
    int started = 1, touching = 0;                  // the calling thread is one of them
    try {
        for (; job.n_touch > 0 && cores > TOUCH_THREADS && touching < TOUCH_THREADS; touching++) touchers[touching] = std::thread([&job] { job.touch_outputs(); });
        for (; started < threads; started++)
            pool[started] = std::thread([&job, started] { job.work(g_stage.memory + (size_t)started * 2 * STAGE_PIECE); job.touch_outputs(); });
    } catch (const std::exception &) {
        // fewer threads than asked for (no thread or no memory for one): the ones that run share the pieces
    }
    job.work(g_stage.memory);
    for (int t = 1; t < started; t++) pool[t].join();
    for (int t = 0; t < touching; t++) touchers[t].join();
    const cudaError_t e = (cudaError_t)job.error.load();
    if (e != cudaSuccess) cudaStreamSynchronize(s);      // copies of other threads may still use the buffers the next call gets
    AGCN_CUDA(e);
    return AGCN_OK;
}

int host_upload(const HostSegment *seg, int n, cudaStream_t s, const HostSegment *outputs, int n_outputs)
{
    return host_copy(seg, n, true, s, outputs, n_outputs);
}

int host_download(const HostSegment *seg, int n, cudaStream_t s)
{
    const int rc = host_copy(seg, n, false, s, nullptr, 0);
    if (rc != AGCN_OK) return rc;
    AGCN_CUDA(cudaStreamSynchronize(s));
    return AGCN_OK;
}

void host_copy_release()
{
    std::lock_guard<std::mutex> lock(g_stage.busy);
    if (g_stage.memory != nullptr) cudaFreeHost(g_stage.memory);
    g_stage.memory = nullptr;
}

}  // namespace agcn
