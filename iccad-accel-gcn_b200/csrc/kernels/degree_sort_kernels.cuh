// Degree sort: stable ascending LSD radix sort of the rows by degree, then the
// CSR permute (and optional symmetric column relabel) that produces the
// degree-ordered `.new_indptr / .new_indices` arrays the Accel-GCN SpMM and
// its partitioner consume (main.cu:62-63, block_level_partition.py:31-38).
//
// One kernel counts the digits of all passes at once; every pass is then one
// kernel that ranks a tile of keys, learns from the tiles before it where its
// digits go (a chained scan: each tile publishes its digit counts, then its
// prefix) and writes runs of equal digits from shared memory.  Passes whose
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
constexpr int SORT_BLOCK = 256;                      // = RADIX_BINS: thread d looks after digit d
constexpr int SORT_WARPS = SORT_BLOCK / 32;
constexpr int SORT_ITEMS = 16;                       // keys per thread
constexpr int SORT_TILE = SORT_BLOCK * SORT_ITEMS;   // keys per block
constexpr int SORT_WARP_KEYS = 32 * SORT_ITEMS;      // contiguous keys owned by one warp
constexpr int FINAL_ITEMS = 8;                       // rows per thread of the last kernel of the sort
constexpr int FINAL_TILE = SORT_BLOCK * FINAL_ITEMS;

constexpr int SORT_WORD_NEGATIVE = 0, SORT_WORD_NNZ = 1, SORT_WORD_COLUMN = 2, SORT_WORD_TIMEOUT = 3;   // host words
constexpr int SORT_BAD_INPUT = 1, SORT_BAD_TIMEOUT = 2;       // bits of SortControl::bad

// Zero at the start of a call.
struct SortControl {
    unsigned hist[RADIX_PASSES][RADIX_BINS];
    unsigned next_tile[RADIX_PASSES + 1];            // tiles are numbered in the order blocks start: a tile's predecessors are running or done
    int bad;
};

// Chained scans: one word per (tile, digit) holds a state and a value, so no fence is needed to publish it.
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

// Sum of the values of all tiles before `tile`; `stride` words between tiles.  Publishes nothing.  Eight
// predecessors are read at a time: most have only their count to say when many tiles start together, and one by
// one the walk is a chain of L2 latencies.
__device__ __forceinline__ unsigned long long chain_look_back(const unsigned long long *state, int64_t tile, int64_t stride,
                                                              SortControl *ctl, HostWords *out)
{
    constexpr int AHEAD = 8;
    unsigned long long sum = 0;
    for (int64_t t = tile - 1; t >= 0; t -= AHEAD) {
        unsigned long long v[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) v[k] = t - k >= 0 ? chain_load(state + (t - k) * stride) : CHAIN_PREFIX;
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            for (int spin = 0; (v[k] & ~CHAIN_VALUE) == 0; spin++) {
                if (spin >= CHAIN_SPIN_LIMIT || *reinterpret_cast<volatile int *>(&ctl->bad) == SORT_BAD_TIMEOUT) {
                    ctl->bad = SORT_BAD_TIMEOUT;
                    out->w[SORT_WORD_TIMEOUT] = 1;
                    return sum;
                }
                if (spin > 16) __nanosleep(200);
                v[k] = chain_load(state + (t - k) * stride);
            }
            sum += v[k] & CHAIN_VALUE;
            if (v[k] & CHAIN_PREFIX) return sum;
        }
    }
    return sum;
}

// Digit counts of all passes.  Bound by HBM (4 bytes per row) for millions of rows.
__global__ void __launch_bounds__(SORT_BLOCK)
degree_count_kernel(const int *__restrict__ indptr, int64_t n_rows, int64_t nnz, int check_nnz, SortControl *__restrict__ ctl, HostWords *out)
{
    __shared__ unsigned s_hist[RADIX_PASSES][RADIX_BINS];
    launch_dependents();
    for (int b = threadIdx.x; b < RADIX_PASSES * RADIX_BINS; b += SORT_BLOCK) (&s_hist[0][0])[b] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * SORT_TILE;
    bool negative = false;
    unsigned small[RADIX_PASSES] = {0, 0, 0, 0};       // rows whose digit of a higher pass is zero: most of them, counted without atomics
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const int64_t i = base + (int64_t)k * SORT_BLOCK + threadIdx.x;
        if (i < n_rows) {
            int d = indptr[i + 1] - indptr[i];
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
// Bound by the rank votes (instruction issue) and, per tile, by the latency of the chain.
__global__ void __launch_bounds__(SORT_BLOCK, 3)
radix_pass_kernel(const int *__restrict__ indptr, int64_t n, int pass, SortBuffers buf, SortControl *__restrict__ ctl,
                  unsigned long long *__restrict__ state, HostWords *out)
{
    __shared__ unsigned s_key[SORT_TILE];
    __shared__ int s_row[SORT_TILE];
    __shared__ unsigned short s_count[SORT_WARPS][RADIX_BINS];     // keys of each digit seen by each warp, then their exclusive prefix
    __shared__ int64_t s_out[RADIX_BINS];                          // output position of a digit's first key minus its place in the tile
    __shared__ unsigned s_scan[SORT_WARPS + 1];
    __shared__ unsigned s_first[RADIX_BINS];
    __shared__ unsigned s_tile;
    wait_for_predecessor();      // every kernel of the sort is launched early behind the one before it
    launch_dependents();
    if (pass > 0 && ctl->hist[pass][0] == (unsigned)n) return;     // every digit is zero: nothing moves
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->next_tile[pass], 1u);
    for (int b = threadIdx.x; b < SORT_WARPS * RADIX_BINS / 2; b += SORT_BLOCK) reinterpret_cast<unsigned *>(&s_count[0][0])[b] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const int done = sort_passes_done(ctl, pass, n);
    const bool odd = (done & 1) != 0;           // pass k of those that move something writes buffer k mod 2
    // (not __restrict__: the pass before may still be writing them when this kernel starts)
    const unsigned *keys_in = odd ? buf.keys[0] : buf.keys[1];
    const int *rows_in = odd ? buf.rows[0] : buf.rows[1];
    unsigned *keys_out = odd ? buf.keys[1] : buf.keys[0];
    int *rows_out = odd ? buf.rows[1] : buf.rows[0];

    const int w = warp_id(), lane = lane_id(), shift = pass * RADIX_BITS;
    const int64_t warp_base = tile * SORT_TILE + (int64_t)w * SORT_WARP_KEYS;
    unsigned key[SORT_ITEMS];
    int row[SORT_ITEMS];
    unsigned short rank[SORT_ITEMS];        // position of the key among the warp's keys of the same digit
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const int64_t i = warp_base + k * 32 + lane;
        key[k] = 0xffffffffu;
        row[k] = (int)i;
        if (i < n) {
            if (pass == 0) { const int d = indptr[i + 1] - indptr[i]; key[k] = d < 0 ? 0u : (unsigned)d; }
            else { key[k] = keys_in[i]; row[k] = rows_in[i]; }
        }
    }
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const bool live = warp_base + k * 32 + lane < n;
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
    __syncthreads();
    {
        // thread d: the tile's keys of digit d, where they begin in the tile and in the output
        const int d = threadIdx.x;
        unsigned total = 0;
#pragma unroll
        for (int ww = 0; ww < SORT_WARPS; ww++) {
            const unsigned c = s_count[ww][d];
            s_count[ww][d] = (unsigned short)total;
            total += c;
        }
        unsigned long long *mine = state + tile * RADIX_BINS + d;
        if (tile > 0) chain_store(mine, CHAIN_COUNT | total);
        unsigned unused;
        const unsigned first = block_scan_exclusive<SORT_BLOCK>(total, OpAdd(), 0u, unused, s_scan);
        const unsigned bin = block_scan_exclusive<SORT_BLOCK>(ctl->hist[pass][d], OpAdd(), 0u, unused, s_scan);
        const unsigned long long before = chain_look_back(state + d, tile, RADIX_BINS, ctl, out);
        chain_store(mine, CHAIN_PREFIX | (before + total));
        s_first[d] = first;
        s_out[d] = (int64_t)bin + (int64_t)before - (int64_t)first;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        if (warp_base + k * 32 + lane < n) {
            const unsigned digit = (key[k] >> shift) & (RADIX_BINS - 1);
            const unsigned at = s_first[digit] + s_count[w][digit] + rank[k];
            s_key[at] = key[k];
            s_row[at] = row[k];
        }
    }
    __syncthreads();
    const int live = (int)(n - tile * SORT_TILE < SORT_TILE ? n - tile * SORT_TILE : SORT_TILE);
#pragma unroll 4
    for (int j = threadIdx.x; j < live; j += SORT_BLOCK) {
        const unsigned k = s_key[j];
        const int64_t pos = s_out[(k >> shift) & (RADIX_BINS - 1)] + j;
        if (pos >= 0 && pos < n) {          // always, unless the chain gave up
            keys_out[pos] = k;
            rows_out[pos] = s_row[j];
        }
    }
}

constexpr int PERMUTE_BLOCK = 256;
constexpr int PERMUTE_ITEMS = 8;
constexpr int PERMUTE_TILE = PERMUTE_BLOCK * PERMUTE_ITEMS;

// After the passes: the permutation, the new row pointers (a chained scan of the sorted degrees), the inverse
// permutation, and for the CSR permute the row that owns the first nonzero of each of its tiles.
__global__ void __launch_bounds__(SORT_BLOCK)
sort_finish_kernel(int64_t n, int passes, SortBuffers buf, SortControl *__restrict__ ctl, unsigned long long *__restrict__ state,
                   int *__restrict__ perm, int *__restrict__ new_indptr, int *__restrict__ new_id, int *__restrict__ tile_row,
                   HostWords *out)
{
    __shared__ int64_t s_scan[SORT_WARPS + 1];
    __shared__ int64_t s_deg[FINAL_TILE + FINAL_TILE / 32];
    __shared__ unsigned s_tile;
    __shared__ unsigned long long s_before;
    wait_for_predecessor();
    launch_dependents();
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->next_tile[RADIX_PASSES], 1u);
    __syncthreads();
    const int64_t tile = s_tile, base = tile * FINAL_TILE;
    const bool odd = (sort_passes_done(ctl, passes, n) & 1) != 0;
    const int *rows = odd ? buf.rows[0] : buf.rows[1];          // written by the kernel before: not __restrict__
    const unsigned *keys = odd ? buf.keys[0] : buf.keys[1];
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = k * SORT_BLOCK + threadIdx.x;
        const int64_t r = base + j;
        if (r < n) {
            const int old = rows[r];
            perm[r] = old;
            if (new_id != nullptr) new_id[old] = (int)r;
        }
        if (new_indptr != nullptr) s_deg[j + (j >> 5)] = r < n ? (int64_t)keys[r] : 0;
    }
    if (new_indptr == nullptr) return;
    __syncthreads();
    // thread t scans rows t * FINAL_ITEMS ...
    int64_t local[FINAL_ITEMS], sum = 0;
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = threadIdx.x * FINAL_ITEMS + k;
        local[k] = sum;
        sum += s_deg[j + (j >> 5)];
    }
    int64_t total;
    const int64_t ex = block_scan_exclusive<SORT_BLOCK>(sum, OpAdd(), (int64_t)0, total, s_scan);
    if (threadIdx.x == 0) {
        if (tile > 0) chain_store(state + tile, CHAIN_COUNT | (unsigned long long)total);
        const unsigned long long before = chain_look_back(state, tile, 1, ctl, out);
        chain_store(state + tile, CHAIN_PREFIX | (before + (unsigned long long)total));
        s_before = before;
    }
    __syncthreads();
    const int64_t start = (int64_t)s_before + ex;
    const bool mark = tile_row != nullptr && *reinterpret_cast<volatile int *>(&ctl->bad) == 0;
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = threadIdx.x * FINAL_ITEMS + k;
        const int64_t b = start + local[k], e = k + 1 < FINAL_ITEMS ? start + local[k + 1] : start + sum;
        s_deg[j + (j >> 5)] = b;
        if (base + j < n && mark)
            for (int64_t t = (b + PERMUTE_TILE - 1) / PERMUTE_TILE; t * PERMUTE_TILE < e; t++) tile_row[t] = (int)(base + j);
        if (base + j == n - 1) new_indptr[n] = (int)e;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < FINAL_ITEMS; k++) {
        const int j = k * SORT_BLOCK + threadIdx.x;
        if (base + j < n) new_indptr[base + j] = (int)s_deg[j + (j >> 5)];
    }
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
constexpr int SMALL_SMEM_BYTES = SMALL_BLOCK * SMALL_ITEMS * 8 + SMALL_WARPS * RADIX_BINS * 2;

// items = rows per thread: ceil(n / 8192), at most SMALL_ITEMS
__global__ void __cluster_dims__(SMALL_CLUSTER, 1, 1) __launch_bounds__(SMALL_BLOCK, 1)
sort_small_kernel(const int *__restrict__ indptr, int n, int items, int64_t nnz, int check_nnz, SortControl *__restrict__ ctl,
                  int *__restrict__ perm, int *__restrict__ new_indptr, int *__restrict__ new_id, int *__restrict__ tile_row,
                  HostWords *out)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    launch_dependents();         // the permute takes its place on the SMs that this leaves idle
    extern __shared__ unsigned s_small[];
    unsigned *s_key = s_small;
    int *s_row = reinterpret_cast<int *>(s_small + SMALL_BLOCK * SMALL_ITEMS);
    unsigned short (*s_count)[RADIX_BINS] = reinterpret_cast<unsigned short (*)[RADIX_BINS]>(s_small + 2 * SMALL_BLOCK * SMALL_ITEMS);
    __shared__ unsigned s_total[RADIX_BINS], s_base[RADIX_BINS], s_scan[SMALL_WARPS + 1];
    __shared__ unsigned s_say[3];                // for the other blocks: largest degree, negative seen, sum of degrees
    __shared__ unsigned s_get[SMALL_CLUSTER][2];
    const int w = warp_id(), lane = lane_id(), block = (int)cluster.block_rank();
    const int per_block = SMALL_BLOCK * items, first = block * per_block + w * 32 * items + lane;       // item k of this thread is row first + 32 k
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
    cluster.sync();
    if (threadIdx.x < 2 * SMALL_CLUSTER) s_get[threadIdx.x >> 1][threadIdx.x & 1] = *cluster.map_shared_rank(&s_say[threadIdx.x & 1], threadIdx.x >> 1);
    __syncthreads();
    bool negative = false;
#pragma unroll
    for (int b = 0; b < SMALL_CLUSTER; b++) { top = max(top, s_get[b][0]); negative |= s_get[b][1] != 0; }
    const int64_t own = (int64_t)indptr[n] - (int64_t)indptr[0];
    const bool bad = negative || (check_nnz && own != nnz);
    if (block == 0 && threadIdx.x == 0) {
        out->w[SORT_WORD_NNZ] = own;
        if (negative) out->w[SORT_WORD_NEGATIVE] = 1;
        ctl->bad = bad ? SORT_BAD_INPUT : 0;
    }
    for (int shift = 0; shift < 32 && (top >> shift) != 0; shift += RADIX_BITS) {
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
    unsigned e = __shfl_sync(FULL_MASK, start, 0);
    for (int b = 0; b < block; b++) e += s_get[b][0];
#pragma unroll
    for (int k = 0; k < SMALL_ITEMS; k++) {
        if (k >= items) break;
        const int i = first + k * 32;
        const unsigned incl = warp_scan_inclusive(key[k], OpAdd()), b = e + incl - key[k];
        e += __shfl_sync(FULL_MASK, incl, 31);
        if (i >= n) continue;
        perm[i] = row[k];
        if (new_id != nullptr) new_id[row[k]] = i;
        if (new_indptr == nullptr) continue;
        new_indptr[i] = (int)b;
        if (i == n - 1) new_indptr[n] = (int)(b + key[k]);
        if (tile_row != nullptr && !bad)
            for (unsigned t = (b + PERMUTE_TILE - 1) / PERMUTE_TILE; t * PERMUTE_TILE < b + key[k]; t++) tile_row[t] = i;
    }
    cluster.sync();              // no block ends while another may read its shared memory
}

// CSR permute.  Each block produces PERMUTE_TILE consecutive output nonzeros.  The rows it touches (all
// non-empty: degrees ascend) mark their first nonzero in a bit map; the row of a nonzero is the number of
// marks up to it, and its source is a per-row offset away.  Per thread all loads of column ids, then all
// lookups of new names, then all values are in flight together.  new_id == nullptr keeps column ids.
// Bound by the 4-byte lookups (a 32-byte sector of L2 each) and HBM.
__global__ void __launch_bounds__(PERMUTE_BLOCK)
csr_permute_kernel(const int *__restrict__ old_indptr, const int *__restrict__ old_indices,
                   const float *__restrict__ old_vals, const int *perm, const int *new_indptr, const int *new_id,
                   const int *tile_row, int64_t n_rows, int64_t nnz, int *__restrict__ new_indices, float *__restrict__ new_vals,
                   const SortControl *ctl, HostWords *out)
{
    // (what the sort makes is not __restrict__: no load of it may move above the wait)
    constexpr int WORDS = PERMUTE_TILE / 32;
    __shared__ int s_delta[PERMUTE_TILE + 1];     // per row of the tile: old start - new start
    __shared__ unsigned s_bits[WORDS];
    __shared__ int s_rank[WORDS];                 // marks before a word
    static_assert(WORDS <= PERMUTE_BLOCK && WORDS == 64, "one warp scans the words, two per lane");
    wait_for_predecessor();      // launched early: the order of the rows is there
    if (ctl->bad != 0) return;
    const int64_t p0 = (int64_t)blockIdx.x * PERMUTE_TILE;
    const int count = (int)(nnz - p0 < PERMUTE_TILE ? nnz - p0 : PERMUTE_TILE);
    const int64_t r_lo = tile_row[blockIdx.x];
    const int64_t r_hi = blockIdx.x + 1 < gridDim.x ? tile_row[blockIdx.x + 1] : n_rows - 1;
    const int ip0 = old_indptr[0];
    if (threadIdx.x < WORDS) s_bits[threadIdx.x] = 0;
    __syncthreads();
    for (int k = threadIdx.x; k <= (int)(r_hi - r_lo); k += PERMUTE_BLOCK) {
        const int start = new_indptr[r_lo + k];
        const int64_t at = (int64_t)start - p0;
        if (at < count) {
            s_delta[k] = old_indptr[perm[r_lo + k]] - ip0 - start;
            if (k > 0) atomicOr(&s_bits[at >> 5], 1u << (at & 31));
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int a = __popc(s_bits[2 * threadIdx.x]), b = __popc(s_bits[2 * threadIdx.x + 1]);
        const int before = warp_scan_inclusive(a + b, OpAdd()) - a - b;
        s_rank[2 * threadIdx.x] = before;
        s_rank[2 * threadIdx.x + 1] = before + a;
    }
    __syncthreads();
    const unsigned upto = 0xffffffffu >> (31 - lane_id());
    int src[PERMUTE_ITEMS], c[PERMUTE_ITEMS];
    float v[PERMUTE_ITEMS];
#pragma unroll
    for (int k = 0; k < PERMUTE_ITEMS; k++) {
        const int q = k * PERMUTE_BLOCK + threadIdx.x;
        const int row = s_rank[q >> 5] + __popc(s_bits[q >> 5] & upto);
        src[k] = q < count ? (int)p0 + q + s_delta[row] : -1;
    }
#pragma unroll
    for (int k = 0; k < PERMUTE_ITEMS; k++) c[k] = src[k] >= 0 ? __ldcs(old_indices + src[k]) : 0;
    if (new_vals != nullptr) {
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++) v[k] = src[k] >= 0 ? __ldcs(old_vals + src[k]) : 0.f;
    }
    if (new_id != nullptr) {
        bool bad = false;
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++)
            if (c[k] < 0 || c[k] >= n_rows) { bad = true; c[k] = 0; }
        if (bad) out->w[SORT_WORD_COLUMN] = 1;
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++) c[k] = new_id[c[k]];
    }
#pragma unroll
    for (int k = 0; k < PERMUTE_ITEMS; k++)
        if (src[k] >= 0) __stcs(new_indices + p0 + k * PERMUTE_BLOCK + threadIdx.x, c[k]);
    if (new_vals != nullptr) {
#pragma unroll
        for (int k = 0; k < PERMUTE_ITEMS; k++)
            if (src[k] >= 0) __stcs(new_vals + p0 + k * PERMUTE_BLOCK + threadIdx.x, v[k]);
    }
}

}  // namespace agcn
