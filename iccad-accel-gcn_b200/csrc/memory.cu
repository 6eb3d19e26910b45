// Memory the entry points take for the length of a call, and the words kernels report to the host.
//
// A cudaMalloc / cudaFree pair costs 0.1 ms to several ms and stalls the whole device; the set-up calls
// (degree sort, partitioner, plan) used to make up to a dozen of them for kernels of a few microseconds.
// Scratch now comes from one stream-ordered pool per device (cudaMallocFromPoolAsync): safe for any number
// of threads and streams, because the driver orders a block's next use after its last one.  What the pool
// keeps between calls is bounded by POOL_KEEP_BYTES; agcn_release_scratch gives that back too.
#include "host_common.h"
#include "host_copy.h"

#include <mutex>

namespace agcn {

constexpr int POOL_MAX_DEVICES = 64;
// What the pool may hold, blocks in use counted, before it returns what is free at the next synchronisation: about 1 %
// of the GPU's memory, enough for the buffers of three host contexts of 500 000 rows of 30 at 96 columns.  (With 512 MiB
// a context made while another one lives had all its buffers mapped anew: 12.6 ms for its first call, 9.5 without.)
constexpr uint64_t POOL_KEEP_BYTES = (uint64_t)2 << 30;

static std::mutex g_pool_mutex;
static cudaMemPool_t g_pool_of[POOL_MAX_DEVICES] = {};

static cudaError_t pool_of_current_device(cudaMemPool_t *out)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= POOL_MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (g_pool_of[dev] == nullptr) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return e;
        uint64_t keep = POOL_KEEP_BYTES;
        e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) { cudaMemPoolDestroy(pool); return e; }
        g_pool_of[dev] = pool;
    }
    *out = g_pool_of[dev];
    return cudaSuccess;
}

cudaError_t pool_alloc(void **out, size_t bytes, cudaStream_t s)
{
    *out = nullptr;
    cudaMemPool_t pool = nullptr;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &capture);
    if (e != cudaSuccess) return e;
    if (capture != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
    e = pool_of_current_device(&pool);
    return e != cudaSuccess ? e : cudaMallocFromPoolAsync(out, bytes > 0 ? bytes : 16, pool, s);
}

void pool_free(void *p, cudaStream_t s)
{
    if (p != nullptr) cudaFreeAsync(p, s);
}

cudaError_t pool_free_waiting(void *p, int device)
{
    if (p == nullptr) return cudaSuccess;
    const DeviceOf on(device);           // the wait and the per-thread stream are those of the current device
    const cudaError_t waited = cudaDeviceSynchronize();      // what cudaFree did: whoever still uses the block is done
    const cudaError_t freed = cudaFreeAsync(p, cudaStreamPerThread);
    return waited != cudaSuccess ? waited : freed;
}

// ---------------------------------------------------------------------------
// Host words: pinned, mapped, 128 bytes each with their link, kept in a free list.  A kernel stores its result or error
// code straight into one and the host reads it after the stream synchronisation it needs anyway, in place
// of a device word, a memset and a device-to-host copy.
// ---------------------------------------------------------------------------
constexpr int HOST_WORDS_PER_CHUNK = 64;      // 8 KiB; more chunks only if more calls run at once

struct HostWordsNode {
    HostWords words;
    HostWordsNode *next;
    char pad[64 - (sizeof(HostWords) + sizeof(HostWordsNode *)) % 64];
};
static_assert(sizeof(HostWordsNode) == 128, "as the comments say");

static int g_words_chunks = 0;
int host_words_chunks() { return g_words_chunks; }

static std::mutex g_words_mutex;
static HostWordsNode *g_words_free = nullptr;

HostWordsLease::HostWordsLease(cudaStream_t s) : s_(s)
{
    std::lock_guard<std::mutex> lock(g_words_mutex);
    if (g_words_free == nullptr) {
        void *chunk = nullptr;
        if (cudaHostAlloc(&chunk, HOST_WORDS_PER_CHUNK * sizeof(HostWordsNode), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) return;
        g_words_chunks++;
        HostWordsNode *n = static_cast<HostWordsNode *>(chunk);
        for (int i = 0; i < HOST_WORDS_PER_CHUNK; i++) { n[i].next = g_words_free; g_words_free = &n[i]; }
    }
    HostWordsNode *n = g_words_free;
    g_words_free = n->next;
    words_ = &n->words;
    for (int i = 0; i < HostWords::COUNT; i++) words_->w[i] = 0;
}

HostWordsLease::~HostWordsLease()
{
    if (words_ == nullptr) return;
    if (pending_) cudaStreamSynchronize(s_);     // a call that gave up early: nothing may still write here
    std::lock_guard<std::mutex> lock(g_words_mutex);
    HostWordsNode *n = reinterpret_cast<HostWordsNode *>(words_);
    n->next = g_words_free;
    g_words_free = n;
}

}  // namespace agcn

extern "C" int agcn_release_scratch(void)
{
    using namespace agcn;
    clear_error();
    cudaMemPool_t pool = nullptr;
    AGCN_CUDA(pool_of_current_device(&pool));
    AGCN_CUDA(cudaDeviceSynchronize());
    AGCN_CUDA(cudaMemPoolTrimTo(pool, 0));
    host_copy_release();
    return AGCN_OK;
}
