// C-ABI entry points of the block-level partitioner
// (replaces block_level_partition.py:38-106).
#include "host_common.h"
#include "host_copy.h"
#include "internal.h"
#include "kernels/partition_kernels.cuh"

#include <atomic>
#include <mutex>
#include <new>

struct agcn_partition_run {
    agcn::PartitionRun run;
};

namespace agcn {

// Tile scratch of one partitioner call.  The regular entry points take it from the pool; the
// allocation-free one points it at a fixed array in the library's device image.
struct PartScratch {
    PartTileInfo *info;
    unsigned *arrived;             // for calls that find no counter free
    int *tile_head;
    int64_t *tile_offset;
    HostWords *words = nullptr;    // on the device: where the answer is stored instead of in leased host words
};

static PartScratch part_scratch(Carver &c, int64_t tiles)
{
    PartScratch sc;
    sc.info = c.take<PartTileInfo>(tiles);
    sc.arrived = c.take<unsigned>(1);
    sc.tile_offset = c.take<int64_t>(tiles);
    sc.tile_head = c.take<int>(tiles);
    return sc;
}

static int partition_check(const char *who, const int *d_indptr, int64_t n_rows, const int *d_block4, const void *result)
{
    AGCN_REQUIRE(d_indptr != nullptr && result != nullptr, "%s: null pointer", who);
    AGCN_REQUIRE(n_rows > 0, "%s: empty graph (n_rows = %lld); the reference script raises IndexError here", who, (long long)n_rows);
    AGCN_REQUIRE(n_rows < (int64_t)INT32_MAX, "%s: n_rows = %lld does not fit the int32 row ids of .block4", who, (long long)n_rows);
    AGCN_REQUIRE(d_block4 == nullptr || aligned16(d_block4), "%s: block4 output must be 16-byte aligned", who);
    return AGCN_OK;
}

static int partition_answer(const char *who, int64_t negative, int64_t total, int64_t *n_blocks)
{
    if (negative != 0) {
        set_error("%s: indptr decreases somewhere (negative degree); "
                  "the reference script prints 'cur_degree number is wrong' and stops", who);
        return AGCN_ERR_RANGE;
    }
    *n_blocks = total;
    return AGCN_OK;
}

// The arrival counter of one call, its own until the call has waited for its kernel.  All zero when they are handed out:
// the kernel leaves its counter so, and one whose kernel is not known to have ended is not handed out again.
class ArrivalCounter {
public:
    ArrivalCounter()
    {
        uint64_t free = free_.load();
        while (free != 0 && !free_.compare_exchange_weak(free, free & (free - 1))) {}
        number_ = free != 0 ? __builtin_ctzll(free) : -1;
    }
    ~ArrivalCounter() { if (number_ >= 0 && !launched_) free_.fetch_or((uint64_t)1 << number_); }
    ArrivalCounter(const ArrivalCounter &) = delete;
    ArrivalCounter &operator=(const ArrivalCounter &) = delete;
    int number() const { return number_; }          // -1: none was free
    void launched() { launched_ = true; }
    void ended() { launched_ = false; }
private:
    static_assert(PART_COUNTERS == 64, "a bit of free_ each");
    static std::atomic<uint64_t> free_;
    int number_;
    bool launched_ = false;
};
std::atomic<uint64_t> ArrivalCounter::free_{~(uint64_t)0};

// Phases A and B: how many tuples there are and where every tile's begin.  `who` names the entry point in error messages.
static int partition_launch_count(const int *d_indptr, int64_t n_rows, const PartScratch &sc, unsigned *own, int counter, HostWords *words,
                                  cudaStream_t s)
{
    AGCN_KERNEL(part_describe_kernel, (unsigned)ceil_div(n_rows, PART_TILE), PART_BLOCK, s, d_indptr, n_rows, sc.info, own, counter, sc.tile_head,
                sc.tile_offset, words);
    AGCN_LAUNCH_CHECK("part_describe_kernel");
    return AGCN_OK;
}

// The same, and the wait for the stream.
static int partition_count(const char *who, const int *d_indptr, int64_t n_rows, int64_t *n_blocks, const PartScratch &sc, cudaStream_t s)
{
    if (sc.words != nullptr) {
        HostWords words;
        AGCN_CUDA(cudaMemsetAsync(sc.words, 0, sizeof(words), s));
        unsigned *arrived = reinterpret_cast<unsigned *>(&sc.words->w[HostWords::COUNT - 1]);      // zeroed with the words
        const int rc = partition_launch_count(d_indptr, n_rows, sc, arrived, 0, sc.words, s);
        if (rc != AGCN_OK) return rc;
        AGCN_CUDA(cudaMemcpyAsync(&words, sc.words, sizeof(words), cudaMemcpyDeviceToHost, s));
        AGCN_CUDA(cudaStreamSynchronize(s));
        return partition_answer(who, words.w[PART_WORD_NEGATIVE], words.w[PART_WORD_TOTAL], n_blocks);
    }
    ArrivalCounter counter;            // given back after the words, which wait for a kernel that an early return leaves running
    const bool none = counter.number() < 0;
    if (none) AGCN_CUDA(cudaMemsetAsync(sc.arrived, 0, sizeof(unsigned), s));
    AGCN_HOST_WORDS(words, s);
    const int rc = partition_launch_count(d_indptr, n_rows, sc, none ? sc.arrived : nullptr, counter.number(), words.device(), s);
    if (rc != AGCN_OK) return rc;
    counter.launched();
    AGCN_CUDA(words.sync());
    counter.ended();
    return partition_answer(who, words[PART_WORD_NEGATIVE], words[PART_WORD_TOTAL], n_blocks);
}

// Phase C, asynchronous.
static int partition_emit(const int *d_indptr, int64_t n_rows, int64_t n_blocks, int *d_block4, const PartScratch &sc, cudaStream_t s)
{
    if (n_blocks == 0) return AGCN_OK;
    const int64_t tiles = ceil_div(n_rows, PART_TILE), chunks = ceil_div(n_blocks, PART_CHUNK);
    AGCN_KERNEL(part_emit_kernel, (unsigned)(chunks + tiles), PART_BLOCK, s, d_indptr, n_rows, (const int *)sc.tile_head,
                (const int64_t *)sc.tile_offset, (int)tiles, (int)chunks, n_blocks, reinterpret_cast<int4 *>(d_block4));
    AGCN_LAUNCH_CHECK("part_emit_kernel");
    return AGCN_OK;
}

// Count and, given room, emit: what the one-call entry points do.
static int partition_pipeline(const char *who, const int *d_indptr, int64_t n_rows, int *d_block4, int64_t cap_blocks,
                              int64_t *n_blocks, const PartScratch &sc, cudaStream_t s)
{
    int rc = partition_count(who, d_indptr, n_rows, n_blocks, sc, s);
    if (rc != AGCN_OK || d_block4 == nullptr || cap_blocks == 0) return rc;
    if (cap_blocks < *n_blocks) {
        set_error("%s: %lld blocks needed, capacity %lld", who, (long long)*n_blocks, (long long)cap_blocks);
        return AGCN_ERR_CAPACITY;
    }
    rc = partition_emit(d_indptr, n_rows, *n_blocks, d_block4, sc, s);
    if (rc != AGCN_OK) return rc;
    AGCN_CUDA(cudaStreamSynchronize(s));
    return AGCN_OK;
}

int partition_device(const int *d_indptr, int64_t n_rows, int *d_block4, int64_t cap_blocks,
                     int64_t *n_blocks, cudaStream_t s)
{
    int rc = partition_check("agcn_partition", d_indptr, n_rows, d_block4, n_blocks);
    if (rc != AGCN_OK) return rc;
    *n_blocks = 0;
    const int64_t tiles = ceil_div(n_rows, PART_TILE);
    Carver size;
    part_scratch(size, tiles);
    DeviceScratch scratch(s);
    AGCN_ALLOC(block, scratch, unsigned char, (int64_t)size.bytes());
    Carver c(block);
    return partition_pipeline("agcn_partition", d_indptr, n_rows, d_block4, cap_blocks, n_blocks, part_scratch(c, tiles), s);
}

int partition_begin(PartitionRun *run, const int *d_indptr, int64_t n_rows, cudaStream_t s)
{
    int rc = partition_check("agcn_partition", d_indptr, n_rows, nullptr, run);
    if (rc != AGCN_OK) return rc;
    const int64_t tiles = ceil_div(n_rows, PART_TILE);
    Carver size;
    part_scratch(size, tiles);
    run->indptr = d_indptr; run->n_rows = n_rows; run->n_blocks = 0; run->stream = s;
    const cudaError_t e = pool_alloc(&run->memory, size.bytes(), s);
    if (e != cudaSuccess) {
        set_error("agcn_partition: device allocation of %zu bytes: %s", size.bytes(), cudaGetErrorString(e));
        return AGCN_ERR_CUDA;
    }
    Carver c(run->memory);
    rc = partition_count("agcn_partition", d_indptr, n_rows, &run->n_blocks, part_scratch(c, tiles), s);
    if (rc != AGCN_OK) { pool_free(run->memory, s); run->memory = nullptr; }
    return rc;
}

int partition_finish(PartitionRun *run, int *d_block4)
{
    if (run->memory == nullptr) return AGCN_OK;
    int rc = AGCN_OK;
    if (d_block4 != nullptr && run->n_blocks > 0) {
        Carver c(run->memory);
        rc = partition_emit(run->indptr, run->n_rows, run->n_blocks, d_block4, part_scratch(c, ceil_div(run->n_rows, PART_TILE)), run->stream);
    }
    pool_free(run->memory, run->stream);
    run->memory = nullptr;
    return rc;
}

}  // namespace agcn

extern "C" int agcn_partition_device(const int32_t *d_indptr, int64_t n_rows, int32_t *d_block4,
                                     int64_t cap_blocks, int64_t *n_blocks, void *stream)
{
    agcn::clear_error();
    return agcn::partition_device(d_indptr, n_rows, d_block4, cap_blocks, n_blocks, static_cast<cudaStream_t>(stream));
}

// The two halves of a call whose output the caller allocates in between (agcn_partition_device does the
// first half twice then: once to count and once to fill).
extern "C" int agcn_partition_begin(const int32_t *d_indptr, int64_t n_rows, agcn_partition_run **run, int64_t *n_blocks, void *stream)
{
    using namespace agcn;
    clear_error();
    AGCN_REQUIRE(run != nullptr && n_blocks != nullptr, "agcn_partition_begin: null pointer");
    *run = nullptr;
    *n_blocks = 0;
    agcn_partition_run *r = new (std::nothrow) agcn_partition_run;
    AGCN_REQUIRE(r != nullptr, "agcn_partition_begin: out of host memory");
    const int rc = partition_begin(&r->run, d_indptr, n_rows, static_cast<cudaStream_t>(stream));
    if (rc != AGCN_OK) { delete r; return rc; }
    *n_blocks = r->run.n_blocks;
    *run = r;
    return AGCN_OK;
}

extern "C" int agcn_partition_finish(agcn_partition_run *run, int32_t *d_block4)
{
    using namespace agcn;
    clear_error();
    AGCN_REQUIRE(run != nullptr, "agcn_partition_finish: null run");
    const bool misaligned = d_block4 != nullptr && !aligned16(d_block4);
    const int rc = partition_finish(&run->run, misaligned ? nullptr : d_block4);
    delete run;
    AGCN_REQUIRE(!misaligned, "agcn_partition_finish: block4 output must be 16-byte aligned");
    return rc;
}

extern "C" int agcn_partition_host(const int32_t *h_indptr, int64_t n_rows, int32_t *h_block4,
                                   int64_t cap_blocks, int64_t *n_blocks)
{
    using namespace agcn;
    clear_error();
    AGCN_REQUIRE(h_indptr != nullptr && n_blocks != nullptr, "agcn_partition_host: null pointer");
    AGCN_REQUIRE(n_rows > 0, "agcn_partition_host: empty graph (n_rows = %lld); the reference script raises IndexError here",
                 (long long)n_rows);
    AGCN_REQUIRE(n_rows < (int64_t)INT32_MAX, "agcn_partition_host: n_rows = %lld does not fit the int32 row ids of .block4", (long long)n_rows);
    *n_blocks = 0;
    const cudaStream_t s = nullptr;
    DeviceScratch scratch(s);
    const WaitOnExit drain(s);
    AGCN_ALLOC(d_indptr, scratch, int, n_rows + 1);
    const HostSegment up = {d_indptr, const_cast<int *>(h_indptr), (size_t)(n_rows + 1) * sizeof(int)};
    int rc = host_upload(&up, 1, s);
    if (rc != AGCN_OK) return rc;
    PartitionRun run;
    rc = partition_begin(&run, d_indptr, n_rows, s);
    if (rc != AGCN_OK) return rc;
    *n_blocks = run.n_blocks;
    const bool wanted = h_block4 != nullptr && cap_blocks != 0;
    if (!wanted || run.n_blocks == 0 || cap_blocks < run.n_blocks) {
        partition_finish(&run, nullptr);
        if (!wanted || cap_blocks >= *n_blocks) return AGCN_OK;
        set_error("agcn_partition_host: %lld blocks needed, capacity %lld", (long long)*n_blocks, (long long)cap_blocks);
        return AGCN_ERR_CAPACITY;
    }
    int *d_block4 = scratch.alloc<int>(run.n_blocks * 4);
    rc = partition_finish(&run, d_block4);
    if (d_block4 == nullptr) return AGCN_ERR_CUDA;
    if (rc != AGCN_OK) return rc;
    const HostSegment down = {d_block4, h_block4, (size_t)*n_blocks * 16};
    return host_download(&down, 1, s);
}

// ---------------------------------------------------------------------------
// Partitioner for callers that must not allocate device memory.
//
// Some hosts of this library cannot let it call cudaMalloc: a process whose
// framework allocator has already claimed all of HBM (a raw cudaMalloc then
// fails or steals from its pool), a latency-critical loop that cannot afford
// the device-wide synchronisation cudaMalloc / cudaFree imply, or a plug-in
// host that forbids allocation calls after start-up.  For them the tile
// scratch of the partitioner (28 bytes per 2048 rows) and its result words live in a
// fixed array in the library's device image instead of a per-call allocation or leased
// host words (which are pinned when there are none free).  Every GPU that
// loads the library holds that array (about 224 KB) until the process exits,
// which is why it is sized for AGCN_PARTITION_NOALLOC_MAX_ROWS rows and no
// more.
//
// The array's name is only a host-side handle; its device address is looked
// up once per device with cudaGetSymbolAddress, on the first call made with
// that device current.  That first call should therefore happen before any
// stream capture is started.  All calls on a device share the array and it
// keeps what the previous call left: everything is overwritten before it is
// read.  Two calls that overlap on the same GPU (different streams or threads) race on it.
// ---------------------------------------------------------------------------
namespace agcn {

constexpr int64_t PART_NOALLOC_MAX_ROWS = AGCN_PARTITION_NOALLOC_MAX_ROWS;
constexpr int64_t PART_NOALLOC_MAX_TILES = (PART_NOALLOC_MAX_ROWS + PART_TILE - 1) / PART_TILE;
constexpr int PART_NOALLOC_MAX_DEVICES = 64;

constexpr size_t PART_STATIC_BYTES = (size_t)PART_NOALLOC_MAX_TILES * (sizeof(PartTileInfo) + sizeof(int64_t) + sizeof(int)) + 3 * 256 + 2 * 256;

}  // namespace agcn

static __device__ __align__(256) unsigned char g_part_static_scratch[agcn::PART_STATIC_BYTES];

namespace agcn {

static std::mutex g_part_static_mutex;
static void *g_part_static_addr[PART_NOALLOC_MAX_DEVICES] = {};

// device address of the static scratch on the current device (looked up once per device)
static int part_static_scratch(void **out)
{
    int dev = -1;
    AGCN_CUDA(cudaGetDevice(&dev));
    AGCN_REQUIRE(dev >= 0 && dev < PART_NOALLOC_MAX_DEVICES, "agcn_partition_device_noalloc: device ordinal %d not supported", dev);
    std::lock_guard<std::mutex> lock(g_part_static_mutex);
    if (g_part_static_addr[dev] == nullptr) {
        void *ptr = nullptr;
        AGCN_CUDA(cudaGetSymbolAddress(&ptr, g_part_static_scratch));
        AGCN_REQUIRE(ptr != nullptr, "agcn_partition_device_noalloc: cudaGetSymbolAddress returned a null address");
        g_part_static_addr[dev] = ptr;
    }
    *out = g_part_static_addr[dev];
    return AGCN_OK;
}

static int partition_device_noalloc(const int *d_indptr, int64_t n_rows, int *d_block4, int64_t cap_blocks,
                                    int64_t *n_blocks, cudaStream_t s)
{
    AGCN_REQUIRE(d_indptr != nullptr && n_blocks != nullptr, "agcn_partition_device_noalloc: null pointer");
    AGCN_REQUIRE(n_rows > 0, "agcn_partition_device_noalloc: empty graph (n_rows = %lld)", (long long)n_rows);
    AGCN_REQUIRE(n_rows <= PART_NOALLOC_MAX_ROWS,
                 "agcn_partition_device_noalloc: n_rows = %lld exceeds the %lld rows the static scratch is sized for; "
                 "use agcn_partition_device for larger graphs", (long long)n_rows, (long long)PART_NOALLOC_MAX_ROWS);
    AGCN_REQUIRE(d_block4 == nullptr || aligned16(d_block4), "agcn_partition_device_noalloc: block4 output must be 16-byte aligned");
    *n_blocks = 0;

    void *memory = nullptr;
    int rc = part_static_scratch(&memory);
    if (rc != AGCN_OK) return rc;
    Carver c(memory);
    HostWords *words = c.take<HostWords>(1);
    PartScratch sc = part_scratch(c, ceil_div(n_rows, PART_TILE));
    sc.words = words;
    return partition_pipeline("agcn_partition_device_noalloc", d_indptr, n_rows, d_block4, cap_blocks, n_blocks, sc, s);
}

}  // namespace agcn

extern "C" int agcn_partition_device_noalloc(const int32_t *d_indptr, int64_t n_rows, int32_t *d_block4,
                                             int64_t cap_blocks, int64_t *n_blocks, void *stream)
{
    agcn::clear_error();
    return agcn::partition_device_noalloc(d_indptr, n_rows, d_block4, cap_blocks, n_blocks,
                                          static_cast<cudaStream_t>(stream));
}
