// Block-level partitioner: degree-ordered CSR row pointers -> `.block4`
// metadata, bit-exact with the sequential walk of the reference script
// (block_level_partition.py:48-103) for ANY degree sequence, sorted or not.
//
// The walk is a state machine over rows, but its output has a closed form per
// row once the start of the row's run of equal consecutive degrees is known:
//   degree 0            -> no tuple
//   1 <= D <= 384       -> the row opens a tuple iff (row - run_start) % R(D) == 0;
//                          the tuple covers j = min(R(D), rows left in the run) rows
//   D > 384             -> ceil(D / 384) tuples of <= 384 nonzeros each
// with R(D), w(D) the pattern tables of block_level_partition.py:7-21 and the
// fall-backs of :56-63.  Two launches over tiles of PART_TILE rows staged
// through shared memory: (A) every tile describes itself -- its last run start,
// its leading rows that belong to a run begun earlier, the tuples all other rows
// open -- and (B) the thread block that is done last scans the descriptions, which
// closes the open runs, and leaves every tile its incoming run start and its first
// output position; (C) every row writes its own tuples.  The host waits between (B) and (C), for
// the number of tuples it has to find room for, and not behind (C).
// Bound: launches and the wait up to some 100 000 rows; above, instruction issue and a tile's chain of loads, scans and
// stores (2.4 M rows of 25: 16 and 19 us, of which HBM needs 4).
#pragma once
#include "../host_common.h"
#include "primitives.cuh"
#include "ptx.cuh"

namespace agcn {

constexpr int PART_DEG_BOUND = 384;   // 12 warps x 32 nonzeros: a format constant of .block4
constexpr int PART_BLOCK = 256;
constexpr int PART_ITEMS = 8;
constexpr int PART_TILE = PART_BLOCK * PART_ITEMS;
constexpr int PART_MAX_ROWS_PER_TUPLE = 12;
constexpr int PART_HALO = PART_MAX_ROWS_PER_TUPLE + 1;   // rows looked at past a tile
constexpr int PART_WORD_TOTAL = 0, PART_WORD_NEGATIVE = 1;    // host words

// rows per tuple R(D) and nonzeros per virtual warp w(D), 1 <= D <= 384
__device__ __forceinline__ int part_rows_per_tuple(int d)
{
    return d <= 32 ? 12 : d <= 64 ? 6 : d <= 96 ? 4 : d <= 128 ? 3 : d <= 191 ? 2 : 1;
}
__device__ __forceinline__ int part_warp_nz(int d)
{
    if (d >= 192) return 32;
    const int f = 12 / part_rows_per_tuple(d);
    return (d + f - 1) / f;
}

// x mod R(d), with the division by a constant in every case
__device__ __forceinline__ unsigned part_mod_rows(unsigned x, int d)
{
    return d <= 32 ? x % 12u : d <= 64 ? x % 6u : d <= 96 ? x & 3u : d <= 128 ? x % 3u : d <= 191 ? x & 1u : 0u;
}

// Shared-memory view of indptr[tile_first - 1 .. tile_first + PART_TILE + PART_HALO]
// (indices clamped to [0, n_rows]); deg(i) is valid for tile_first-1 <= i and
// i < tile_first + PART_TILE + PART_HALO, and returns -1 for rows that do not exist.
// Every thread walks PART_ITEMS consecutive rows, so the threads of a warp read words PART_ITEMS
// apart: one pad word per 32 keeps those reads on different banks (unpadded they collide 8 ways).
__device__ __forceinline__ int part_pad(int k) { return k + (k >> 5); }

struct PartTile {
    int *s_ip;
    int64_t first;    // first row of the tile
    int64_t n_rows;
    __device__ __forceinline__ int ip(int64_t i) const { return s_ip[part_pad((int)(i - first + 1))]; }
    __device__ __forceinline__ int deg(int64_t i) const
    {
        if (i < 0 || i >= n_rows) return -1;
        return ip(i + 1) - ip(i);
    }
};

constexpr int PART_TILE_INTS = PART_TILE + PART_HALO + 2;                  // row pointers a tile looks at
constexpr int PART_SMEM_INTS = PART_TILE_INTS + PART_TILE_INTS / 32 + 1;   // the same, padded

// All loads of a thread are in flight together (one by one, nine L2 or HBM latencies were half of the kernel's time).
__device__ __forceinline__ PartTile part_load_tile(const int *__restrict__ indptr, int64_t n_rows, int64_t tile, int *s_ip)
{
    constexpr int LOADS = (PART_TILE_INTS + PART_BLOCK - 1) / PART_BLOCK;
    PartTile t;
    t.s_ip = s_ip;
    t.first = tile * PART_TILE;
    t.n_rows = n_rows;
    int v[LOADS];
#pragma unroll
    for (int k = 0; k < LOADS; k++) {
        int64_t i = t.first - 1 + k * PART_BLOCK + threadIdx.x;
        i = i < 0 ? 0 : (i > n_rows ? n_rows : i);
        v[k] = indptr[i];
    }
#pragma unroll
    for (int k = 0; k < LOADS; k++)
        if (k * PART_BLOCK + (int)threadIdx.x < PART_TILE_INTS) s_ip[part_pad(k * PART_BLOCK + threadIdx.x)] = v[k];
    __syncthreads();
    return t;
}

// What a tile says about itself.
struct PartTileInfo {         // read as an int4
    int last_head;    // last row of the tile that starts a run, -1 if none
    int lead;         // rows before the tile's first run start, where their tuples depend on where that run began
    int lead_deg;     // ... and their degree (1 .. 384; lead is 0 for any other degree)
    int rest;         // tuples opened by all other rows
};

// Number of tuples each of this thread's PART_ITEMS rows opens.
// incoming_head = start of the run that is open when the tile begins; -1: not known, rows of that run
// that need it count in `lead` instead.  Returns the last run start of this thread's rows, -1 if none; `heads` has
// a bit for every one of its rows that starts a run.
__device__ __forceinline__ int part_row_counts(const PartTile &t, int incoming_head, int *s_scan, int (&deg)[PART_ITEMS],
                                               int (&cnt)[PART_ITEMS], unsigned &heads, int &lead, int &lead_deg, bool &negative)
{
    const int64_t my_first = t.first + (int64_t)threadIdx.x * PART_ITEMS;
    // last run head among this thread's rows, then an exclusive max-scan over the block
    int head_local = -1;
    int prev = my_first > 0 && my_first < t.n_rows ? t.deg(my_first - 1) : -1;
    heads = 0;
    int at = t.ip(my_first);
#pragma unroll
    for (int k = 0; k < PART_ITEMS; k++) {
        const int64_t i = my_first + k;
        const int next = t.ip(i + 1);
        deg[k] = next - at;
        at = next;
        if (i < t.n_rows) {
            negative |= deg[k] < 0;
            if (i == 0 || deg[k] != prev) { head_local = (int)i; heads |= 1u << k; }
        }
        prev = deg[k];
    }
    int unused_total;
    int run_head = block_scan_exclusive<PART_BLOCK>(head_local, OpMax(), -1, unused_total, s_scan);
    run_head = run_head > incoming_head ? run_head : incoming_head;
    lead = 0;
    lead_deg = 0;
#pragma unroll
    for (int k = 0; k < PART_ITEMS; k++) {
        const int64_t i = my_first + k;
        int c = 0;
        if (i < t.n_rows) {
            const int d = deg[k];
            if (heads & (1u << k)) run_head = (int)i;
            if (d > PART_DEG_BOUND) c = (d + PART_DEG_BOUND - 1) / PART_DEG_BOUND;
            else if (d >= 1) {
                if (run_head < 0) { lead++; lead_deg = d; }
                else c = part_mod_rows((unsigned)((int)i - run_head), d) == 0 ? 1 : 0;
            }
        }
        cnt[k] = c;
    }
    return head_local;
}

// Tuples opened by the leading rows of tile b, once the start of their run is known.
__device__ __forceinline__ int64_t part_lead_tuples(const PartTileInfo &info, int64_t b, int head)
{
    if (info.lead <= 0) return 0;
    // rows o .. o + lead - 1 of their run open a tuple where their number is a multiple of R
    const int64_t o = b * PART_TILE - head;
    const int r = part_rows_per_tuple(info.lead_deg);
    return (o + info.lead + r - 1) / r - (o + r - 1) / r;
}

// How many thread blocks of a call have described their tile: a counter for each of the calls under way (partition.cu
// hands them out).  Zero when the library is loaded, and after every call: the block that arrives last resets it.
constexpr int PART_COUNTERS = 64;
static __device__ unsigned g_part_arrived[PART_COUNTERS];

// (A) the description of every tile, and (B) by the block that arrives last, whichever that is, the run start that is
// open when every tile begins and every tile's first output position.  (As a launch of its own, one block, (B) cost the
// host 3 us and the GPU 6 more.)  `own`: a zeroed word to count arrivals in; null: counter number `counter` does.
__global__ void __launch_bounds__(PART_BLOCK)
part_describe_kernel(const int *__restrict__ indptr, int64_t n_rows, PartTileInfo *tiles, unsigned *own, int counter, int *__restrict__ tile_head,
                     int64_t *__restrict__ tile_offset, HostWords *out)
{
    __shared__ int s_ip[PART_SMEM_INTS];
    __shared__ int s_scan[PART_BLOCK / 32 + 1];
    __shared__ int64_t s_scan64[PART_BLOCK / 32 + 1];
    __shared__ int s_red[4][PART_BLOCK / 32];
    __shared__ bool s_last;
    const PartTile t = part_load_tile(indptr, n_rows, blockIdx.x, s_ip);
    int deg[PART_ITEMS], cnt[PART_ITEMS], lead, lead_deg;
    unsigned heads;
    bool negative = false;
    int head = part_row_counts(t, -1, s_scan, deg, cnt, heads, lead, lead_deg, negative);
    if (negative) out->w[PART_WORD_NEGATIVE] = 1;
    int rest = 0;
#pragma unroll
    for (int k = 0; k < PART_ITEMS; k++) rest += cnt[k];
    head = warp_reduce(head, OpMax());
    lead = warp_reduce(lead, OpAdd());
    lead_deg = warp_reduce(lead_deg, OpMax());
    rest = warp_reduce(rest, OpAdd());
    if (lane_id() == 0) { s_red[0][warp_id()] = head; s_red[1][warp_id()] = lead; s_red[2][warp_id()] = lead_deg; s_red[3][warp_id()] = rest; }
    __syncthreads();
    if (threadIdx.x == 0) {
        PartTileInfo info = {-1, 0, 0, 0};
        for (int w = 0; w < PART_BLOCK / 32; w++) {
            info.last_head = max(info.last_head, s_red[0][w]);
            info.lead += s_red[1][w];
            info.lead_deg = max(info.lead_deg, s_red[2][w]);
            info.rest += s_red[3][w];
        }
        tiles[blockIdx.x] = info;
        unsigned *arrived = own != nullptr ? own : g_part_arrived + counter;
        __threadfence();
        s_last = atomicAdd(arrived, 1u) == gridDim.x - 1;
        if (s_last) *arrived = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();                 // all descriptions are there
    int carry_head = -1;
    int64_t carry = 0;
    for (int64_t base = 0; base < gridDim.x; base += PART_BLOCK) {
        const int64_t b = base + threadIdx.x;
        PartTileInfo info = {-1, 0, 0, 0};
        if (b < gridDim.x) {
            const int4 v = __ldcg(reinterpret_cast<const int4 *>(tiles) + b);
            info = {v.x, v.y, v.z, v.w};
        }
        int head_total;
        int head_in = block_scan_exclusive<PART_BLOCK>(info.last_head, OpMax(), -1, head_total, s_scan);
        head_in = max(head_in, carry_head);
        const int64_t count = info.rest + part_lead_tuples(info, b, head_in);
        int64_t total;
        const int64_t ex = block_scan_exclusive<PART_BLOCK>(count, OpAdd(), (int64_t)0, total, s_scan64);
        if (b < gridDim.x) { tile_head[b] = head_in; tile_offset[b] = carry + ex; }
        carry += total;
        carry_head = max(carry_head, head_total);
    }
    if (threadIdx.x == 0) out->w[PART_WORD_TOTAL] = carry;
}

// (C) every row that opens tuples writes them at its scanned offset.  A row of degree D > 384 owns ceil(D / 384) of
// them, so the tiles of a graph's hub rows have many times the tuples of the others: tuples are then dealt out one per
// thread, which looks its row up in the scanned offsets, and a tile of more than PART_CHUNK is shared by the blocks
// before the tile blocks, PART_CHUNK output positions each.  (Row by row the last of 1172 tiles, 2.4 M rows of 25,
// kept the kernel for 44 us; 19 now.)
constexpr int PART_CHUNK = 4096;

// The tuples of one tile that lie at output positions [lo, hi), hi <= first_out + their number.
struct PartEmitShared {
    int ip[PART_SMEM_INTS];
    int scan[PART_BLOCK / 32 + 1];
    int pos[PART_TILE];                        // tuples of the tile before each of its rows
    unsigned char heads[PART_BLOCK + 2];       // a bit per row that starts a run (or lies past the end), a byte per thread
};

// Tuple c of row i (row r of its tile)
__device__ __forceinline__ int4 part_tuple(const PartEmitShared &sh, int64_t i, int r, int d, int loc, int c)
{
    if (d > PART_DEG_BOUND) {
        const int done = c * PART_DEG_BOUND;
        return make_int4(d, (int)i, loc + done, d - done < PART_DEG_BOUND ? d - done : PART_DEG_BOUND);
    }
    // up to R(D) rows, as far as the run goes
    const int at = r >> 3;
    const unsigned window = sh.heads[at] | sh.heads[at + 1] << 8 | sh.heads[at + 2] << 16;
    const int run = __ffs((window >> ((r & 7) + 1)) | 1u << (PART_MAX_ROWS_PER_TUPLE - 1));
    return make_int4(d, (int)i, loc, (part_warp_nz(d) << 16) + min(part_rows_per_tuple(d), run));
}

__device__ __forceinline__ void part_emit_tile(const PartTile &t, PartEmitShared &sh, int incoming, int64_t first_out, int64_t lo, int64_t hi,
                                               int64_t cap, int ip0, int4 *__restrict__ block4)
{
    static_assert(PART_ITEMS == 8, "a byte of run starts per thread");
    int deg[PART_ITEMS], cnt[PART_ITEMS], lead, lead_deg;
    unsigned heads;
    bool negative;
    part_row_counts(t, incoming, sh.scan, deg, cnt, heads, lead, lead_deg, negative);
    const int64_t my_first = t.first + (int64_t)threadIdx.x * PART_ITEMS;
    int sum = 0;
    bool several = false;
#pragma unroll
    for (int k = 0; k < PART_ITEMS; k++) {
        sum += cnt[k];
        several |= cnt[k] > 1;
        if (my_first + k >= t.n_rows) heads |= 1u << k;
    }
    sh.heads[threadIdx.x] = (unsigned char)heads;
    if (threadIdx.x < 2) {               // the rows a tuple of this tile may reach into
        unsigned m = 0;
        for (int k = 0; k < 8; k++) {
            const int64_t i = t.first + PART_TILE + threadIdx.x * 8 + k;
            if (i >= t.n_rows || threadIdx.x * 8 + k >= PART_MAX_ROWS_PER_TUPLE || t.deg(i) != t.deg(i - 1)) m |= 1u << k;
        }
        sh.heads[PART_BLOCK + threadIdx.x] = (unsigned char)m;
    }
    int tile_total;
    int at = block_scan_exclusive<PART_BLOCK>(sum, OpAdd(), 0, tile_total, sh.scan);      // synchronises: heads is complete
    if (!__syncthreads_or(several)) {
#pragma unroll
        for (int k = 0; k < PART_ITEMS; k++) {
            if (cnt[k] == 0) continue;
            const int64_t out = first_out + at++;
            if (out >= lo && out < hi && (uint64_t)out < (uint64_t)cap)
                block4[out] = part_tuple(sh, my_first + k, threadIdx.x * PART_ITEMS + k, deg[k], t.ip(my_first + k) - ip0, 0);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < PART_ITEMS; k++) { sh.pos[threadIdx.x * PART_ITEMS + k] = at; at += cnt[k]; }
    __syncthreads();
    const int64_t end = first_out + tile_total < hi ? first_out + tile_total : hi;
    for (int64_t out = (first_out > lo ? first_out : lo) + threadIdx.x; out < end; out += PART_BLOCK) {
        const int o = (int)(out - first_out);
        int r = 0;                       // the last row with no more than o tuples before it
#pragma unroll
        for (int step = PART_TILE / 2; step > 0; step >>= 1)
            if (sh.pos[r + step] <= o) r += step;
        const int64_t i = t.first + r;
        if ((uint64_t)out < (uint64_t)cap) block4[out] = part_tuple(sh, i, r, t.deg(i), t.ip(i) - ip0, o - sh.pos[r]);
    }
}

// `cap` is the number of tuples; nothing is written outside of them, whatever became of indptr since they were counted.
// The first `chunks` blocks: PART_CHUNK output positions each; the others: a tile each.
__global__ void __launch_bounds__(PART_BLOCK, 4)
part_emit_kernel(const int *__restrict__ indptr, int64_t n_rows, const int *__restrict__ tile_incoming_head, const int64_t *__restrict__ tile_offset,
                 int tiles, int chunks, int64_t cap, int4 *__restrict__ block4)
{
    __shared__ PartEmitShared sh;
    __shared__ int s_list[2], s_listed;
    const int of_tile = (int)blockIdx.x - chunks;
    const int ip0 = indptr[0];
    auto offset = [&](int b) { return b < tiles ? tile_offset[b] : cap; };
    if (of_tile >= 0) {
        const int64_t first_out = offset(of_tile), end = offset(of_tile + 1);
        if (end - first_out <= PART_CHUNK)
            part_emit_tile(part_load_tile(indptr, n_rows, of_tile, sh.ip), sh, tile_incoming_head[of_tile], first_out, first_out, end, cap, ip0, block4);
        return;
    }
    // tiles of more than PART_CHUNK tuples that reach into this block's positions: two at most
    const int64_t lo = (int64_t)blockIdx.x * PART_CHUNK, hi = lo + PART_CHUNK;
    auto tiles_before = [&](int64_t x) {           // how many tiles begin before position x: a step by all threads leaves 1/256
        int a = 0, z = tiles;
        while (a < z) {
            const int step = (z - a + PART_BLOCK - 1) / PART_BLOCK, mine = a + (int)threadIdx.x * step;
            const int before = __syncthreads_count(mine < z && offset(mine) < x);      // samples a, a + step, ... that begin before x
            if (before == 0) return a;
            z = min(z, a + before * step);
            a = a + (before - 1) * step + 1;
        }
        return a;
    };
    const int b1 = tiles_before(hi), b0 = tiles_before(lo + 1);
    if (threadIdx.x == 0) s_listed = 0;
    __syncthreads();
    for (int b = (b0 > 0 ? b0 - 1 : 0) + threadIdx.x; b < b1; b += PART_BLOCK)
        if (offset(b + 1) - offset(b) > PART_CHUNK) {
            const int q = atomicAdd(&s_listed, 1);
            if (q < 2) s_list[q] = b;
        }
    __syncthreads();
    for (int q = 0; q < min(s_listed, 2); q++) {
        const int b = s_list[q];
        __syncthreads();                 // the tile before is done with
        part_emit_tile(part_load_tile(indptr, n_rows, b, sh.ip), sh, tile_incoming_head[b], offset(b), lo, hi, cap, ip0, block4);
    }
}

}  // namespace agcn
