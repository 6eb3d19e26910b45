// Degree sort: stable ascending LSD radix sort of the rows by degree, then the
// CSR permute (and optional symmetric column relabel) that produces the
// degree-ordered `.new_indptr / .new_indices` arrays the Accel-GCN SpMM and
// its partitioner consume (main.cu:62-63, block_level_partition.py:31-38).
//
// One kernel counts the digits of all passes at once, those of the first pass
// tile by tile; every pass is then one kernel that ranks a tile of keys, adds
// up what the tiles before it count (in three levels, so that a tile reads a
// few dozen rows of counters) and writes runs of equal digits from shared
// memory, counting them for the tiles of the next pass.  No tile waits for
// another one.  Passes whose
// digit is zero for every row find that out on the device and return, so the
// host does not wait for the maximum degree between launches.  Stability
// inside a tile comes from ranking keys in tile order: each warp owns a
// contiguous run of keys and ranks 32 consecutive keys at a time with a
// match-any vote.
#pragma once
#include "../host_common.h"
#include "primitives.cuh"
#include "ptx.cuh"

#include <cooperative_groups.h>

namespace agcn {

constexpr int RADIX_BITS = 8;
constexpr int RADIX_BINS = 1 << RADIX_BITS;
constexpr int RADIX_PASSES = 4;                      // degrees have at most 31 bits
constexpr int SORT_BLOCK = 256;
constexpr int SORT_WARPS = SORT_BLOCK / 32;
constexpr int SORT_ITEMS = 16;                       // rows per thread of degree_count_kernel
constexpr int SORT_TILE = SORT_BLOCK * SORT_ITEMS;   // and per block, the same as in a pass
constexpr int RADIX_BLOCK = 512;                     // a pass: twice the threads, so that more warps rank at once (thread d looks after digit d)
constexpr int RADIX_WARPS = RADIX_BLOCK / 32;
constexpr int RADIX_ITEMS = SORT_TILE / RADIX_BLOCK; // keys per thread
constexpr int RADIX_WARP_KEYS = 32 * RADIX_ITEMS;    // contiguous keys owned by one warp
constexpr int FINAL_ITEMS = 8;                       // rows per thread of the last kernel of the sort
constexpr int FINAL_TILE = SORT_BLOCK * FINAL_ITEMS;

constexpr int SORT_WORD_NEGATIVE = 0, SORT_WORD_NNZ = 1, SORT_WORD_COLUMN = 2, SORT_WORD_TIMEOUT = 3;   // host words
constexpr int SORT_BAD_INPUT = 1, SORT_BAD_TIMEOUT = 2;       // bits of SortControl::bad

// Zero at the start of a call.
struct SortControl {
    unsigned hist[RADIX_PASSES][RADIX_BINS];
    unsigned next_tile;                              // tiles of the last kernel are numbered in the order blocks start: a tile's predecessors are running or done
    int bad;
};

// Digit counts of a pass: a row of RADIX_BINS counters per tile, per group of tiles and per group of groups (zero at
// the start of a call).  A tile's digits go behind those of all tiles before it: with the sums of the groups it reads
// at most 15 + 31 rows and one per two million keys.  The rows of the first pass come from degree_count_kernel, those
// of the others from the pass before, which knows where it puts every key; digit 0 of these is left out and follows
// from the rest (nearly all rows of a sparse graph have it).
// (A chained scan over the tiles before: with 444 tiles started together a tile walked over up to 55 steps of an L2
// latency each.  2.4 M rows, the passes that move keys: 34 and 22 us with it, 25 and 18 us without.)
constexpr int COUNT_GROUP = 16, COUNT_SUPER = 32 * COUNT_GROUP;

struct SortCounts {
    unsigned *rows;           // [pass][tiles, then groups, then super groups][RADIX_BINS]
    int64_t tiles, groups, supers;
    __device__ __forceinline__ unsigned *tile(int pass, int64_t t) const { return rows + ((int64_t)pass * (tiles + groups + supers) + t) * RADIX_BINS; }
    __device__ __forceinline__ unsigned *group(int pass, int64_t g) const { return tile(pass, tiles + g); }
    __device__ __forceinline__ unsigned *super(int pass, int64_t g) const { return tile(pass, tiles + groups + g); }
};

// Sum of `rows` rows of counters, this thread's column.  Sixteen loads in flight, also where fewer rows are left.
__device__ __forceinline__ unsigned counts_sum(const unsigned *first, int64_t rows)
{
    constexpr int AHEAD = 16;
    unsigned sum = 0;
    for (int64_t r = 0; r < rows; r += AHEAD) {
        unsigned v[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) v[k] = r + k < rows ? __ldcg(first + (r + k) * RADIX_BINS) : 0u;
#pragma unroll
        for (int k = 0; k < AHEAD; k++) sum += v[k];
    }
    return sum;
}

// keys of digit d in the tiles before `t`
__device__ __forceinline__ unsigned counts_before(const SortCounts &c, int pass, int64_t t, int d)
{
    const int64_t s = t / COUNT_SUPER, g = t / COUNT_GROUP;
    return counts_sum(c.super(pass, 0) + d, s) + counts_sum(c.group(pass, s * (COUNT_SUPER / COUNT_GROUP)) + d, g - s * (COUNT_SUPER / COUNT_GROUP)) +
           counts_sum(c.tile(pass, g * COUNT_GROUP) + d, t - g * COUNT_GROUP);
}

// Chained scan of the last kernel: one word per tile holds a state and a value, so no fence is needed to publish it.
constexpr unsigned long long CHAIN_COUNT = 1ull << 62, CHAIN_PREFIX = 2ull << 62, CHAIN_VALUE = (1ull << 62) - 1;
// Polls before a tile gives up on a predecessor (each backs off; well over a second): predecessors only ever wait
// for their own predecessors, so the limit is there for a bug, not for load.
constexpr int CHAIN_SPIN_LIMIT = 1 << 22;

__device__ __forceinline__ unsigned long long chain_load(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void chain_store(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

// Sum of the values of all tiles before `tile`, by one warp; publishes nothing.  CHAIN_AHEAD * 32 predecessors are
// read at a time: most have only their count to say when many tiles start together, and the walk is a chain of L2
// latencies, by one thread and eight at a time 146 of them for 1172 tiles.
constexpr int CHAIN_AHEAD = 4;

__device__ __forceinline__ unsigned long long chain_look_back(const unsigned long long *state, int64_t tile, SortControl *ctl, HostWords *out)
{
    unsigned long long sum = 0;
    for (int64_t t = tile - 1 - lane_id();; t -= CHAIN_AHEAD * 32) {
        unsigned long long v[CHAIN_AHEAD];
#pragma unroll
        for (int k = 0; k < CHAIN_AHEAD; k++) v[k] = t - 32 * k >= 0 ? chain_load(state + t - 32 * k) : CHAIN_PREFIX;
#pragma unroll
        for (int k = 0; k < CHAIN_AHEAD; k++) {
            for (int spin = 0; (v[k] & ~CHAIN_VALUE) == 0; spin++) {
                if (spin >= CHAIN_SPIN_LIMIT || *reinterpret_cast<volatile int *>(&ctl->bad) == SORT_BAD_TIMEOUT) {
                    ctl->bad = SORT_BAD_TIMEOUT;
                    out->w[SORT_WORD_TIMEOUT] = 1;
                    v[k] = CHAIN_PREFIX;
                    break;
                }
                if (spin > 16) __nanosleep(200);
                v[k] = chain_load(state + t - 32 * k);
            }
            // lane 0 holds the nearest tile: up to the first prefix
            const unsigned prefixes = __ballot_sync(FULL_MASK, (v[k] & CHAIN_PREFIX) != 0);
            const int last = prefixes != 0 ? __ffs(prefixes) - 1 : 31;
            sum += warp_reduce(lane_id() <= last ? v[k] & CHAIN_VALUE : 0ull, OpAdd());
            if (prefixes != 0) return sum;
        }
    }
}

// Digit counts of all passes, those of the first also by tile.  Bound by HBM (4 bytes per row) for millions of rows.
__global__ void __launch_bounds__(SORT_BLOCK)
degree_count_kernel(const int *__restrict__ indptr, int64_t n_rows, int64_t nnz, int check_nnz, SortCounts counts, SortControl *__restrict__ ctl,
                    HostWords *out)
{
    __shared__ unsigned s_hist[RADIX_PASSES][RADIX_BINS];
    launch_dependents();
    for (int b = threadIdx.x; b < RADIX_PASSES * RADIX_BINS; b += SORT_BLOCK) (&s_hist[0][0])[b] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * SORT_TILE;
    bool negative = false;
    unsigned small[RADIX_PASSES] = {0, 0, 0, 0};       // rows whose digit of a higher pass is zero: most of them, counted without atomics
    int deg[SORT_ITEMS];                               // all loads before the first atomic: one HBM latency, not sixteen
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const int64_t i = base + (int64_t)k * SORT_BLOCK + threadIdx.x;
        deg[k] = i < n_rows ? indptr[i + 1] - indptr[i] : 0;
    }
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        if (base + (int64_t)k * SORT_BLOCK + threadIdx.x < n_rows) {
            int d = deg[k];
            if (d < 0) { negative = true; d = 0; }
            atomicAdd(&s_hist[0][d & (RADIX_BINS - 1)], 1u);
#pragma unroll
            for (int p = 1; p < RADIX_PASSES; p++) {
                const int digit = (d >> (p * RADIX_BITS)) & (RADIX_BINS - 1);
                if (digit == 0) small[p]++;
                else atomicAdd(&s_hist[p][digit], 1u);
            }
        }
    }
#pragma unroll
    for (int p = 1; p < RADIX_PASSES; p++) {
        const unsigned c = warp_reduce(small[p], OpAdd());
        if (lane_id() == 0) atomicAdd(&s_hist[p][0], c);
    }
    if (negative) { out->w[SORT_WORD_NEGATIVE] = 1; ctl->bad = SORT_BAD_INPUT; }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the caller's nnz sizes the grid of the CSR permute: it must be the matrix's own count
        const int64_t own = (int64_t)indptr[n_rows] - (int64_t)indptr[0];
        out->w[SORT_WORD_NNZ] = own;
        if (check_nnz && own != nnz) ctl->bad = SORT_BAD_INPUT;
    }
    __syncthreads();
    for (int b = threadIdx.x; b < RADIX_PASSES * RADIX_BINS; b += SORT_BLOCK) {
        const unsigned c = (&s_hist[0][0])[b];
        if (c != 0) atomicAdd(&ctl->hist[0][0] + b, c);
        if (b < RADIX_BINS) {
            counts.tile(0, blockIdx.x)[b] = c;
            if (c != 0) {
                atomicAdd(counts.group(0, blockIdx.x / COUNT_GROUP) + b, c);
                atomicAdd(counts.super(0, blockIdx.x / COUNT_SUPER) + b, c);
            }
        }
    }
}

struct SortBuffers {
    unsigned *keys[2];
    int *rows[2];
};

// How many of the passes before `pass` moved anything (the first always does): says which buffer holds their result.
__device__ __forceinline__ int sort_passes_done(const SortControl *ctl, int pass, int64_t n)
{
    int done = pass > 0 ? 1 : 0;
    for (int p = 1; p < pass; p++) done += ctl->hist[p][0] != (unsigned)n;
    return done;
}

// One pass.  8 bytes read and 8 written per row; the first pass takes the degrees from the row pointers.
// Bound by the rank votes (instruction issue).
__global__ void __launch_bounds__(RADIX_BLOCK, 3)
radix_pass_kernel(const int *__restrict__ indptr, int n, int pass, int passes, SortBuffers buf, const SortControl *ctl, SortCounts counts)
{
    __shared__ unsigned s_key[SORT_TILE];
    __shared__ int s_row[SORT_TILE];
    __shared__ unsigned short s_count[RADIX_WARPS][RADIX_BINS];     // keys of each digit seen by each warp, then their exclusive prefix
    __shared__ int s_out[RADIX_BINS];                              // output position of a digit's first key minus its place in the tile
    __shared__ unsigned long long s_scan[RADIX_WARPS + 1];
    __shared__ unsigned s_first[RADIX_BINS];
    wait_for_predecessor();      // every kernel of the sort is launched early behind the one before it
    launch_dependents();
    if (pass > 0 && ctl->hist[pass][0] == (unsigned)n) return;     // every digit is zero: nothing moves
    for (int b = threadIdx.x; b < RADIX_WARPS * RADIX_BINS / 2; b += RADIX_BLOCK) reinterpret_cast<unsigned *>(&s_count[0][0])[b] = 0;
    __syncthreads();
    const int tile = (int)blockIdx.x;
    int next = pass + 1;                        // the pass after this one that moves anything
    while (next < passes && ctl->hist[next][0] == (unsigned)n) next++;
    const int done = sort_passes_done(ctl, pass, n);
    const bool odd = (done & 1) != 0;           // pass k of those that move something writes buffer k mod 2
    // (not __restrict__: the pass before may still be writing them when this kernel starts)
    const unsigned *keys_in = odd ? buf.keys[0] : buf.keys[1];
    const int *rows_in = odd ? buf.rows[0] : buf.rows[1];
    unsigned *keys_out = odd ? buf.keys[1] : buf.keys[0];
    int *rows_out = odd ? buf.rows[1] : buf.rows[0];

    const int w = warp_id(), lane = lane_id(), shift = pass * RADIX_BITS;
    const unsigned warp_base = (unsigned)tile * SORT_TILE + w * RADIX_WARP_KEYS, un = (unsigned)n;      // may pass 2^31, not 2^32
    unsigned key[RADIX_ITEMS];
    unsigned short rank[RADIX_ITEMS];        // position of the key among the warp's keys of the same digit
#pragma unroll
    for (int k = 0; k < RADIX_ITEMS; k++) {
        const unsigned i = warp_base + k * 32 + lane;
        key[k] = 0xffffffffu;
        if (i < un) {
            if (pass == 0) { const int d = indptr[i + 1] - indptr[i]; key[k] = d < 0 ? 0u : (unsigned)d; }
            else key[k] = keys_in[i];
        }
    }
    // thread d: where the tile's keys of digit d go (none of this depends on the keys, which are still on their way)
    unsigned out_first = 0, before = 0;
    if (threadIdx.x < RADIX_BINS) { out_first = ctl->hist[pass][threadIdx.x]; before = counts_before(counts, pass, tile, threadIdx.x); }
    {
        unsigned long long all;
        if (pass > 0 && threadIdx.x == 0) before = 0;
        const unsigned long long ex = block_scan_exclusive<RADIX_BLOCK>((unsigned long long)out_first << 32 | before, OpAdd(), 0ull, all, s_scan);
        // digit 0 is not counted: the tiles before are full, what is no other digit is this one
        if (pass > 0 && threadIdx.x == 0) before = (unsigned)tile * SORT_TILE - (unsigned)all;
        out_first = (unsigned)(ex >> 32) + before;
    }
#pragma unroll
    for (int k = 0; k < RADIX_ITEMS; k++) {
        const bool live = warp_base + k * 32 + lane < un;
        // lanes past the end vote in a bin of their own and are never written
        const unsigned digit = live ? ((key[k] >> shift) & (RADIX_BINS - 1)) : (unsigned)RADIX_BINS;
        const unsigned peers = __match_any_sync(FULL_MASK, digit);
        const unsigned before = __popc(peers & ((1u << lane) - 1u));
        unsigned seen = 0;
        if (live) seen = s_count[w][digit];
        __syncwarp();
        if (live && before == 0) s_count[w][digit] = (unsigned short)(seen + __popc(peers));
        __syncwarp();
        rank[k] = (unsigned short)(seen + before);
    }
    int row[RADIX_ITEMS];
#pragma unroll
    for (int k = 0; k < RADIX_ITEMS; k++) {
        const unsigned i = warp_base + k * 32 + lane;
        row[k] = pass > 0 && i < un ? rows_in[i] : (int)i;
    }
    __syncthreads();
    {
        // thread d: the tile's keys of digit d, and where they begin in the tile
        const int d = threadIdx.x;
        unsigned total = 0;
        if (d < RADIX_BINS) {
#pragma unroll
            for (int ww = 0; ww < RADIX_WARPS; ww++) {
                const unsigned c = s_count[ww][d];
                s_count[ww][d] = (unsigned short)total;
                total += c;
            }
        }
        unsigned long long unused;
        const unsigned first = (unsigned)block_scan_exclusive<RADIX_BLOCK>((unsigned long long)total, OpAdd(), 0ull, unused, s_scan);
        if (d < RADIX_BINS) {
            s_first[d] = first;
            s_out[d] = (int)(out_first - first);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RADIX_ITEMS; k++) {
        if (warp_base + k * 32 + lane < un) {
            const unsigned digit = (key[k] >> shift) & (RADIX_BINS - 1);
            const unsigned at = s_first[digit] + s_count[w][digit] + rank[k];
            s_key[at] = key[k];
            s_row[at] = row[k];
        }
    }
    __syncthreads();
    const int live = min(n - tile * SORT_TILE, SORT_TILE);
#pragma unroll 4
    for (int j0 = 0; j0 < SORT_TILE; j0 += RADIX_BLOCK) {
        const int j = j0 + threadIdx.x;
        const unsigned k = j < live ? s_key[j] : 0u;
        const int pos = s_out[(k >> shift) & (RADIX_BINS - 1)] + j;
        const bool in = j < live && pos >= 0 && pos < n;          // j < live, unless the row pointers changed since they were counted
        if (in) {
            keys_out[pos] = k;
            rows_out[pos] = s_row[j];
        }
        if (next < passes) {
            const unsigned digit = in ? (k >> (next * RADIX_BITS)) & (RADIX_BINS - 1) : 0u;
            if (__any_sync(FULL_MASK, digit != 0)) {
                // neighbours go to neighbouring places: one atomic for those of a tile
                const unsigned to = (unsigned)pos / SORT_TILE, peers = __match_any_sync(FULL_MASK, digit != 0 ? to * RADIX_BINS + digit : 0u);
                if (digit != 0 && lane == __ffs(peers) - 1) {
                    const unsigned c = __popc(peers);
                    atomicAdd(counts.tile(next, to) + digit, c);
                    atomicAdd(counts.group(next, to / COUNT_GROUP) + digit, c);
                    atomicAdd(counts.super(next, to / COUNT_SUPER) + digit, c);
                }
            }
        }
    }
}

constexpr int PERMUTE_BLOCK = 256;
constexpr int PERMUTE_ITEMS = 8;                     // nonzeros per thread
constexpr int PERMUTE_TILE = 32 * PERMUTE_ITEMS;     // and per warp
constexpr int PERMUTE_WARPS = PERMUTE_BLOCK / 32;

// What the CSR permute needs to know of the order.
struct PermuteMap {
    int *new_id;       // new name of every column; null: columns keep their names
    int *delta;        // per new row: where it began among the old nonzeros minus where it begins now
    int *tile_row;     // the row that owns the first nonzero of every PERMUTE_TILE; null: no nonzeros
};

// After the passes: the permutation, the new row pointers (a chained scan of the sorted degrees), and for the CSR
// permute the inverse permutation and where every row comes from.
__global__ void __launch_bounds__(SORT_BLOCK)
sort_finish_kernel(const int *__restrict__ indptr, int64_t n, int passes, SortBuffers buf, SortControl *__restrict__ ctl,
                   unsigned long long *__restrict__ state, int *__restrict__ perm, int *__restrict__ new_indptr, PermuteMap map, HostWords *out)
{
    __shared__ unsigned s_scan[SORT_WARPS + 1];
    __shared__ unsigned s_deg[FINAL_TILE + FINAL_TILE / 32];       // degrees, then where the rows begin (sums below 2^31, or the input is bad)
    __shared__ unsigned s_tile;
    __shared__ unsigned long long s_before;
    wait_for_predecessor();
    launch_dependents();
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->next_tile, 1u);
    __syncthreads();
    const int64_t tile = s_tile, base = tile * FINAL_TILE;
    const bool odd = (sort_passes_done(ctl, passes, n) & 1) != 0;
    const int *rows = odd ? buf.rows[0] : buf.rows[1];          // written by the kernel before: not __restrict__
    const unsigned *keys = odd ? buf.keys[0] : buf.keys[1];
    int from[FINAL_ITEMS];                 // the old row, then where it begins
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = k * SORT_BLOCK + threadIdx.x;
        from[k] = base + j < n ? rows[base + j] : 0;
        if (new_indptr != nullptr) s_deg[j + (j >> 5)] = base + j < n ? keys[base + j] : 0u;
    }
    unsigned local[FINAL_ITEMS], sum = 0, total = 0, ex = 0;
    if (new_indptr != nullptr) {
        __syncthreads();
        // thread t scans rows t * FINAL_ITEMS ...
#pragma unroll
        for (int k = 0; k < FINAL_ITEMS; k++) {
            const int j = threadIdx.x * FINAL_ITEMS + k;
            local[k] = sum;
            sum += s_deg[j + (j >> 5)];
        }
        ex = block_scan_exclusive<SORT_BLOCK>(sum, OpAdd(), 0u, total, s_scan);
        if (threadIdx.x == 0 && tile > 0) chain_store(state + tile, CHAIN_COUNT | (unsigned long long)total);
    }
    // while the tiles before say what they have
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int64_t r = base + k * SORT_BLOCK + threadIdx.x;
        if (r < n) {
            perm[r] = from[k];
            if (map.new_id != nullptr) map.new_id[from[k]] = (int)r;
            if (map.delta != nullptr) from[k] = indptr[from[k]] - indptr[0];
        }
    }
    if (new_indptr == nullptr) return;
    if (threadIdx.x < 32) {
        const unsigned long long before = chain_look_back(state, tile, ctl, out);
        if (threadIdx.x == 0) {
            chain_store(state + tile, CHAIN_PREFIX | (before + (unsigned long long)total));
            s_before = before;
        }
    }
    __syncthreads();
    const unsigned start = (unsigned)s_before + ex;
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = threadIdx.x * FINAL_ITEMS + k;
        const unsigned b = start + local[k], e = k + 1 < FINAL_ITEMS ? start + local[k + 1] : start + sum;
        s_deg[j + (j >> 5)] = b;
        if (base + j == n - 1) new_indptr[n] = (int)e;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = k * SORT_BLOCK + threadIdx.x;
        if (base + j < n) {
            const int start = (int)s_deg[j + (j >> 5)];
            new_indptr[base + j] = start;
            if (map.delta != nullptr) map.delta[base + j] = from[k] - start;
        }
    }
}

// The row that owns the first nonzero of every PERMUTE_TILE: the last row that begins no later.  A thread per tile,
// which searches the row pointers (some 20 reads, most of them in L1 and L2).  (Where sort_finish_kernel marked the
// tiles row by row, the block of the hub rows, a third of all nonzeros, kept it for 60 us instead of 20.)
__global__ void __launch_bounds__(SORT_BLOCK)
tile_rows_kernel(const int *new_indptr, int n, int tiles, const SortControl *ctl, int *__restrict__ tile_row)
{
    wait_for_predecessor();
    launch_dependents();
    const int t = blockIdx.x * SORT_BLOCK + threadIdx.x;
    if (t >= tiles || ctl->bad != 0) return;
    const int first = t * PERMUTE_TILE;
    int lo = 0, hi = n;                    // row lo begins no later, row hi (if any) later
    while (hi - lo > 1) {
        const int mid = lo + ((hi - lo) >> 1);
        if (new_indptr[mid] <= first) lo = mid; else hi = mid;
    }
    tile_row[t] = lo;
}

// The whole sort of a small graph in one cluster of eight thread blocks: keys stay in registers, a pass exchanges
// them through the blocks' shared memory, and the results are those of the kernels above.  Five launches of a few
// thread blocks each are a chain of launch, load and scan latencies: 16 384 rows took 56 us on the GPU, one thread
// block of 16 rows per thread 35 us, this 17 us; 65 536 rows are as many as eight blocks hold.
constexpr int SMALL_CLUSTER = 8;
constexpr int SMALL_BLOCK = 1024;
constexpr int SMALL_WARPS = SMALL_BLOCK / 32;
constexpr int SMALL_ITEMS = 8;
constexpr int SMALL_MAX_ROWS = SMALL_CLUSTER * SMALL_BLOCK * SMALL_ITEMS;
constexpr unsigned SMALL_MARKS = 64;                 // tiles of a row that its thread marks by itself
constexpr int small_smem_bytes(int items) { return SMALL_BLOCK * items * 8 + SMALL_WARPS * RADIX_BINS * 2; }

// items = rows per thread: ceil(n / 8192), at most SMALL_ITEMS
__global__ void __cluster_dims__(SMALL_CLUSTER, 1, 1) __launch_bounds__(SMALL_BLOCK, 1)
sort_small_kernel(const int *__restrict__ indptr, int n, int items, int64_t nnz, int check_nnz, SortControl *__restrict__ ctl,
                  int *__restrict__ perm, int *__restrict__ new_indptr, PermuteMap map, HostWords *out)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    launch_dependents();         // the permute takes its place on the SMs that this leaves idle
    __shared__ unsigned s_total[RADIX_BINS], s_base[RADIX_BINS], s_scan[SMALL_WARPS + 1];
    __shared__ unsigned s_say[3];                // for the other blocks: largest degree, negative seen, sum of degrees
    __shared__ unsigned s_get[SMALL_CLUSTER][2];
    const int w = warp_id(), lane = lane_id(), block = (int)cluster.block_rank();
    const int per_block = SMALL_BLOCK * items, first = block * per_block + w * 32 * items + lane;       // item k of this thread is row first + 32 k
    extern __shared__ unsigned s_small[];        // small_smem_bytes(items): no more than there are rows, or the SM changes its carve-out
    unsigned *s_key = s_small;
    int *s_row = reinterpret_cast<int *>(s_small + per_block);
    unsigned short (*s_count)[RADIX_BINS] = reinterpret_cast<unsigned short (*)[RADIX_BINS]>(s_small + 2 * per_block);
    if (threadIdx.x < 3) s_say[threadIdx.x] = 0;
    __syncthreads();
    unsigned key[SMALL_ITEMS], top = 0;
    int row[SMALL_ITEMS];
#pragma unroll
    for (int k = 0; k < SMALL_ITEMS; k++) {
        const int i = first + k * 32;
        row[k] = i;
        key[k] = 0;
        if (k < items && i < n) {
            const int d = indptr[i + 1] - indptr[i];
            if (d < 0) s_say[1] = 1;
            else key[k] = (unsigned)d;
        }
        top = max(top, key[k]);
    }
    top = warp_reduce(top, OpMax());
    if (lane == 0) atomicMax(&s_say[0], top);
    bool bad = false;
    // the first pass says with its counts which other ones move anything
    for (int shift = 0; shift == 0 || (shift < 32 && (top >> shift) != 0); shift += RADIX_BITS) {
        for (int b = threadIdx.x; b < SMALL_WARPS * RADIX_BINS / 2; b += SMALL_BLOCK) reinterpret_cast<unsigned *>(&s_count[0][0])[b] = 0;
        __syncthreads();
        unsigned short rank[SMALL_ITEMS];
#pragma unroll
        for (int k = 0; k < SMALL_ITEMS; k++) {
            if (k >= items) break;
            const bool live = first + k * 32 < n;
            const unsigned digit = live ? ((key[k] >> shift) & (RADIX_BINS - 1)) : (unsigned)RADIX_BINS;
            const unsigned peers = __match_any_sync(FULL_MASK, digit);
            const unsigned before = __popc(peers & ((1u << lane) - 1u));
            unsigned seen = 0;
            if (live) seen = s_count[w][digit];
            __syncwarp();
            if (live && before == 0) s_count[w][digit] = (unsigned short)(seen + __popc(peers));
            __syncwarp();
            rank[k] = (unsigned short)(seen + before);
        }
        __syncthreads();
        if (threadIdx.x < RADIX_BINS) {
            unsigned total = 0;
#pragma unroll 8
            for (int ww = 0; ww < SMALL_WARPS; ww++) {
                const unsigned c = s_count[ww][threadIdx.x];
                s_count[ww][threadIdx.x] = (unsigned short)total;
                total += c;
            }
            s_total[threadIdx.x] = total;
        }
        cluster.sync();
        if (shift == 0 && threadIdx.x < 2 * SMALL_CLUSTER)
            s_get[threadIdx.x >> 1][threadIdx.x & 1] = *cluster.map_shared_rank(&s_say[threadIdx.x & 1], threadIdx.x >> 1);
        unsigned all = 0, before = 0, unused;
        if (threadIdx.x < RADIX_BINS) {
#pragma unroll
            for (int b = 0; b < SMALL_CLUSTER; b++) {
                const unsigned c = *cluster.map_shared_rank(&s_total[threadIdx.x], b);
                all += c;
                before += b < block ? c : 0u;
            }
        }
        const unsigned bin = block_scan_exclusive<SMALL_BLOCK>(all, OpAdd(), 0u, unused, s_scan);
        if (threadIdx.x < RADIX_BINS) s_base[threadIdx.x] = bin + before;
        __syncthreads();
        if (shift == 0) {
            bool negative = false;
#pragma unroll
            for (int b = 0; b < SMALL_CLUSTER; b++) { top = max(top, s_get[b][0]); negative |= s_get[b][1] != 0; }
            const int64_t own = (int64_t)indptr[n] - (int64_t)indptr[0];
            bad = negative || (check_nnz && own != nnz);
            if (block == 0 && threadIdx.x == 0) {
                out->w[SORT_WORD_NNZ] = own;
                if (negative) out->w[SORT_WORD_NEGATIVE] = 1;
                ctl->bad = bad ? SORT_BAD_INPUT : 0;
            }
        }
#pragma unroll
        for (int k = 0; k < SMALL_ITEMS; k++) {
            if (k < items && first + k * 32 < n) {
                const unsigned digit = (key[k] >> shift) & (RADIX_BINS - 1);
                const unsigned pos = s_base[digit] + s_count[w][digit] + rank[k], to = pos / (unsigned)per_block, at = pos - to * per_block;
                *cluster.map_shared_rank(&s_key[at], to) = key[k];
                *cluster.map_shared_rank(&s_row[at], to) = row[k];
            }
        }
        cluster.sync();
#pragma unroll
        for (int k = 0; k < SMALL_ITEMS; k++) {
            if (k < items && first + k * 32 < n) {
                const int at = first - block * per_block + k * 32;
                key[k] = s_key[at];
                row[k] = s_row[at];
            }
        }
    }
    // row pointers: the warp's rows in order, 32 at a time (their sum fits 31 bits, or the input is bad)
    unsigned sum = 0, total;
#pragma unroll
    for (int k = 0; k < SMALL_ITEMS; k++) sum += warp_reduce(key[k], OpAdd());
    const unsigned start = block_scan_exclusive<SMALL_BLOCK>(lane == 0 ? sum : 0u, OpAdd(), 0u, total, s_scan);
    if (threadIdx.x == 0) s_say[2] = total;
    cluster.sync();
    if (threadIdx.x < SMALL_CLUSTER) s_get[threadIdx.x][0] = *cluster.map_shared_rank(&s_say[2], threadIdx.x);
    __syncthreads();
    cluster.barrier_arrive();    // this block reads no other one's shared memory any more
    unsigned e = __shfl_sync(FULL_MASK, start, 0);
    for (int b = 0; b < block; b++) e += s_get[b][0];
    const bool mark = map.tile_row != nullptr && !bad, hubs = top > SMALL_MARKS * PERMUTE_TILE;
#pragma unroll
    for (int k = 0; k < SMALL_ITEMS; k++) {
        if (k >= items) break;
        const int i = first + k * 32;
        const unsigned incl = warp_scan_inclusive(key[k], OpAdd()), b = e + incl - key[k];
        e += __shfl_sync(FULL_MASK, incl, 31);
        if (i < n) {
            perm[i] = row[k];
            if (map.new_id != nullptr) map.new_id[row[k]] = i;
            if (new_indptr != nullptr) {
                new_indptr[i] = (int)b;
                if (map.delta != nullptr) map.delta[i] = indptr[row[k]] - indptr[0] - (int)b;
                if (i == n - 1) new_indptr[n] = (int)(b + key[k]);
            }
        }
        if (!mark) continue;
        // the tiles that begin in the row (none past the end: no nonzeros).  Those of a row of a great many are dealt out to the
        // warp, row after row: by one thread a hub row of 1e7 nonzeros made the sort of 60 000 rows of 25 take 313 us instead
        // of 131, 300 rows of 30 000 90 instead of 74.  (From 4 tiles on, or the tiles of 32 rows at once and a search for
        // whose each is, power-law graphs of up to 16 000 nonzeros per row lost up to 15 and 7 us of 190.)
        unsigned t = (b + PERMUTE_TILE - 1) / PERMUTE_TILE;
        const unsigned t_end = (b + key[k] + PERMUTE_TILE - 1) / PERMUTE_TILE;
        if (hubs) {
            for (unsigned many = __ballot_sync(FULL_MASK, t_end - t > SMALL_MARKS); many != 0; many &= many - 1) {
                const int from = __ffs(many) - 1;
                const unsigned last = __shfl_sync(FULL_MASK, t_end, from);
                for (unsigned q = __shfl_sync(FULL_MASK, t, from) + lane; q < last; q += 32) map.tile_row[q] = i - lane + from;
            }
            if (t_end - t > SMALL_MARKS) continue;
        }
        for (; t < t_end; t++) map.tile_row[t] = i;
    }
    cluster.barrier_wait();      // no block ends while another may read its shared memory
}

// CSR permute.  Each warp produces PERMUTE_TILE consecutive column ids or values by itself.  The rows it touches (all
// non-empty: degrees ascend) mark their first nonzero in a bit map; the row of a nonzero is the number of
// marks up to it, and its source is a per-row offset away.  Per thread all loads of column ids, then all
// lookups of new names are in flight together.  map.new_id == nullptr keeps column ids.
// Bound by the 4-byte lookups, a tag and a 32-byte sector each: 6e7 random ones into 2.4 M names take 257 us by
// themselves, through whichever cache path.  Column ids and values are moved by different thread
// blocks (of every pair, where both are wanted): a warp that moves one of them fits 32 registers, so that an SM holds 64
// of them, and a warp waits for tile, rows, ids and names in turn.  (By thread blocks of 2048 nonzeros, which synchronised
// three times: 392 us for 6e7 nonzeros, so 380.)
__global__ void __launch_bounds__(PERMUTE_BLOCK, 8)
csr_permute_kernel(const int *__restrict__ old_indices, const float *__restrict__ old_vals, const int *new_indptr, const PermuteMap map,
                   int64_t n_rows, int64_t nnz, int *__restrict__ new_indices, float *__restrict__ new_vals,
                   const SortControl *ctl, HostWords *out)
{
    // (what the sort makes is not __restrict__: no load of it may move above the wait)
    __shared__ int s_delta_of[PERMUTE_WARPS][PERMUTE_TILE + 1];       // per row of the tile
    __shared__ unsigned s_bits_of[PERMUTE_WARPS][PERMUTE_ITEMS];
    int *s_delta = s_delta_of[warp_id()];
    unsigned *s_bits = s_bits_of[warp_id()];
    const int lane = lane_id();
    if (lane < PERMUTE_ITEMS) s_bits[lane] = 0;
    __syncwarp();
    wait_for_predecessor();      // launched early: the order of the rows is there
    const bool both = new_vals != nullptr && new_indices != nullptr, move_vals = both ? (blockIdx.x & 1) != 0 : new_vals != nullptr;
    const int tile = (int)(both ? blockIdx.x >> 1 : blockIdx.x) * PERMUTE_WARPS + warp_id();
    const int64_t p0 = (int64_t)tile * PERMUTE_TILE;
    if (p0 >= nnz || ctl->bad != 0) return;
    const int count = (int)(nnz - p0 < PERMUTE_TILE ? nnz - p0 : PERMUTE_TILE);
    const int r_lo = map.tile_row[tile];
    const int r_hi = p0 + PERMUTE_TILE < nnz ? map.tile_row[tile + 1] : (int)n_rows - 1;
    for (int k = lane; k <= r_hi - r_lo && k <= PERMUTE_TILE; k += 32) {
        const int at = new_indptr[r_lo + k] - (int)p0, delta = map.delta[r_lo + k];
        if (at < count) {
            s_delta[k] = delta;
            if (k > 0) atomicOr(&s_bits[at >> 5], 1u << (at & 31));
        }
    }
    __syncwarp();
    const unsigned upto = 0xffffffffu >> (31 - lane);
    int src[PERMUTE_ITEMS], row = 0;
#pragma unroll
    for (int k = 0; k < PERMUTE_ITEMS; k++) {
        const unsigned marks = s_bits[k];
        src[k] = k * 32 + lane < count ? (int)p0 + k * 32 + lane + s_delta[row + __popc(marks & upto)] : -1;
        row += __popc(marks);
    }
    if (move_vals) {
        float v[PERMUTE_ITEMS];
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++) v[k] = src[k] >= 0 ? __ldcs(old_vals + src[k]) : 0.f;
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++)
            if (k * 32 + lane < count) __stcs(new_vals + p0 + k * 32 + lane, v[k]);
        return;
    }
    int c[PERMUTE_ITEMS];
#pragma unroll
    for (int k = 0; k < PERMUTE_ITEMS; k++) c[k] = src[k] >= 0 ? __ldcs(old_indices + src[k]) : 0;
    if (map.new_id != nullptr) {
        bool bad = false;
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++)
            if ((unsigned)c[k] >= (unsigned)n_rows) { bad = true; c[k] = 0; }
        if (bad) out->w[SORT_WORD_COLUMN] = 1;
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++) c[k] = map.new_id[c[k]];
    }
#pragma unroll
    for (int k = 0; k < PERMUTE_ITEMS; k++)
        if (k * 32 + lane < count) __stcs(new_indices + p0 + k * 32 + lane, c[k]);
}

}  // namespace agcn
