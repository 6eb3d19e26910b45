// Block-level-partitioned CSR SpMM for sm_100a:  Y[n_rows x dim] = A * X,
// A given as the degree-ordered (idx, val) arrays plus `.block4` metadata
// (one tuple {degree, row_begin, loc_begin, info} per block of <= 384
// nonzeros; decode rules of spmm_accel.cu:18-34).
//
// Work decomposition.  A thread block ("unit") takes SPMM_WARPS consecutive
// tuples, one per warp.
// A warp first stages its tuple's (col, val) slice -- at most 384 pairs -- into
// shared memory with coalesced loads, then walks it.
// The columns of one dense row are covered by a "slot" of S lanes, each lane
// holding a float4 (the counterpart of the reference's combined warp,
// spmm_accel.cu:36-53, with 16-byte instead of 4-byte lanes); a warp therefore
// works on 32/S nonzeros at a time.  Rows of degree <= 32 are given whole to a
// slot, longer rows are split over the slots of the warp and folded with
// butterfly shuffles.  Accumulators live in registers.
//
// Heavy rows (degree > 384) span several tuples.  Their per-tuple partial sums
// meet in shared memory and are added in tuple order; a row that is contained
// in one unit is then stored directly.  A row that crosses a unit boundary
// leaves one partial per unit in a small "carry" array (at most two per unit),
// and these are added in unit order: in a launch of few units by the unit that
// arrives last at the row's counter, otherwise by spmm_carry_kernel.  (Waiting
// for a counter keeps a thread block's registers for 1-2 us, 2 % of a product
// of 50 000 units; a second launch costs 3 us, a third of a product of 2 048 rows.)
// Every element of Y is thus written exactly once with a plain store, in a
// fixed order of additions: no floating-point atomics, no dependence on what Y
// held before, bit-identical from run to run.
// Rows no tuple covers (degree 0) are zero-filled by extra blocks of the same
// launch.
#pragma once
#include "../host_common.h"
#include "primitives.cuh"
#include "ptx.cuh"
#include "../spmm_rules.h"

namespace agcn {

constexpr int PLAN_MADE_UNITS = 0, PLAN_MADE_ZERO = 1, PLAN_MADE_WORDS = 2;

constexpr int SPMM_DEG_BOUND = 384;    // format constant of .block4 (spmm_accel.cu:11)
// tuples per unit, one per warp (4, 6 and 12 were measured within 2 % of 8; override to experiment)
#ifndef AGCN_SPMM_WARPS
#define AGCN_SPMM_WARPS 8
#endif
constexpr int SPMM_WARPS = AGCN_SPMM_WARPS;
constexpr int SPMM_THREADS = SPMM_WARPS * 32;
constexpr int SPMM_PANEL = 128;        // dense columns covered by one launch
constexpr int SPMM_ZERO_ROWS_PER_BLOCK = 64;
// Gathers a lane keeps in flight, and thread blocks per SM the register budget is capped for.
// Seven gathers at 4 blocks (32 warps per SM, 64 registers) are 1-8 % faster than four at 5 blocks (48 registers)
// for widths up to 16 and above 32, six or eight 2-8 % slower than seven; at 17..32 columns, where a warp takes four
// nonzeros at a time, the 40 warps are 2-5 % faster.  (2.4 M rows of 25, B200, us: dim 16 601 -> 555, dim 64 1490 ->
// 1447, dim 128 2983 -> 2875; 700 000 rows of 15, dim 64: 235 -> 221.  More gathers at fewer blocks lose 5-30 %.)
constexpr int SPMM_GATHER_BATCH = 7, SPMM_MIN_BLOCKS = 4;
constexpr int SPMM_WIDE_GATHER_BATCH = 4, SPMM_WIDE_MIN_BLOCKS = 5;
// With 32-byte loads: large launches, others, others with five blocks per SM (three, six gathers: 1-9 %, 14 % slower)
constexpr int SPMM_OCTET_BATCH = 4, SPMM_OCTET_FEW = 3;
// Small products (no more tuples than the GPU has room for warps) cannot hide latency with occupancy, and what they
// wait for is the warp that walks 384 nonzeros alone.  Their plan cuts the tuples into pieces of fewer nonzeros
// (plan_small_kernel), and where they fit two blocks per SM the kernel keeps more gathers in flight per lane
// (16 384 rows of 8, dim 60: 9.0 -> 8.6 us).
constexpr int SPMM_DEEP_GATHER_BATCH = 16, SPMM_DEEP_MIN_BLOCKS = 2;
// Between those and the others: three blocks per SM (spmm_few_form).
constexpr int SPMM_THREE_GATHER_BATCH = 8, SPMM_THREE_MIN_BLOCKS = 3;

struct SpmmParams {
    const int4 *tuples;       // the plan's: `.block4`, or its pieces
    int64_t n_tuples;
    int64_t n_units;          // units of this launch (thread blocks beyond them zero-fill uncovered rows)
    int light_every;          // order of the units: from the heavy end, but every light_every-th (0: none) from the light end
    int64_t unit_base;        // first unit of this launch: a product may be launched as several unit ranges
    const int *abort_flag;    // optional: a nonzero word makes every thread block return at once
    const int *idx;
    const float *val;
    const float *x;     // first column of the panel
    int64_t ldx;        // floats between consecutive rows of X
    float *y;
    int64_t ldy;
    int dim;            // columns in this panel, 1..SPMM_PANEL
    const int2 *unit_carry;   // per unit: carry slot of a row entering / leaving the unit, or -1
    float *carry;             // [n_carry][SPMM_PANEL]
    const int2 *carry_span;   // per slot: the first slot of its row, and how many the row has
    int *carry_count;         // per slot (a row's first): units of the row that have arrived, zero between products;
                              // null: spmm_carry_kernel follows
    const int *zero_rows;     // rows no tuple covers
    int64_t n_zero_rows;
    int hot_column;           // HOT kernels: rows of X from this column on are kept in L2; 0: no such choice
    const int *made;          // ONCE kernels: where the plan kernel before this launch left its numbers of units and of rows without a
                              // tuple (PLAN_MADE_*), of which n_units and n_zero_rows are the most there can be
    int early;                // host only: launched so that it overlaps the kernel before it
    int wait_first;           // ... which may be any kernel: idx and val, too, are read behind the wait for it
    int relu;                 // nonzero: Y = max(A * X, 0) (fused GCN activation)
    // The fields below are read only by the general (PLAIN = false) kernel flavour.
    int accumulate;           // nonzero: Y += A * X (later column ranges of a column-tiled product)
    int y_vec;                // nonzero: rows of Y are 16-byte aligned and dim_store % 4 == 0
    int dim_store;            // columns of Y written (dim rounded up to 4 is what is gathered)
};

struct TupleView {
    int row0, loc, n_rows, row_nz;
    bool valid, small;
};

// What the plan's kernel wrote.  A product launched behind that kernel (ONCE) is resident while it is written: such data
// must not be read as read-only, not even behind the wait.
template <bool ONCE, typename T>
__device__ __forceinline__ T ld_plan(const T *p)
{
    if constexpr (ONCE) return *p;
    else return __ldg(p);
}

template <bool ONCE>
__device__ __forceinline__ TupleView decode_tuple(const int4 *tuples, int64_t e, int64_t n_tuples)
{
    TupleView t;
    t.valid = e < n_tuples;
    const int4 b = t.valid ? ld_plan<ONCE>(tuples + e) : make_int4(0, 0, 0, 0);
    t.small = b.x <= SPMM_DEG_BOUND;
    t.row0 = b.y;
    t.loc = b.z;
    t.n_rows = t.small ? (b.w & 0xffff) : 1;
    t.row_nz = t.small ? b.x : b.w;
    if (!t.valid) { t.n_rows = 0; t.row_nz = 0; }
    return t;
}

// ---------------------------------------------------------------------------
// gather-accumulate over the staged pairs  first, first+step, ... < count
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 relu4(const float4 &v, int on)
{
    return on ? make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f)) : v;
}
__device__ __forceinline__ float relu1(float v, int on) { return on ? fmaxf(v, 0.f) : v; }

// LOOSE: lanes that share a row which have columns LOOSE apart, yr + col being the first one's place.
// Otherwise writes columns col .. col+3 of one result row.  PLAIN: one 16-byte store.  Otherwise the row may
// be unaligned or end inside the four columns (dim not a multiple of 4: narrower stores), and
// the product may be added to what the row holds (column-tiled products).
template <bool PLAIN, int LOOSE = 0>
__device__ __forceinline__ void emit_row4(const SpmmParams &p, float *yr, int col, float4 v, int act, uint64_t policy)
{
    if (LOOSE > 0) {
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float *d = yr + col + k * LOOSE;
            if (col + k * LOOSE < p.dim_store) st_y1(d, relu1(p.accumulate ? e[k] + *d : e[k], act), policy);
        }
    } else if (PLAIN) {
        st_y4(yr + col, relu4(v, act), policy);
    } else if (p.y_vec) {
        if (p.accumulate) {
            const float4 o = *reinterpret_cast<const float4 *>(yr + col);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        st_y4(yr + col, relu4(v, act), policy);
    } else {
        float *d = yr + col;
        float e[4] = {v.x, v.y, v.z, v.w};
        if (col + 3 < p.dim_store) {
            // as wide as the row's alignment allows: element by element, the four stores of a row touched every
            // sector four times (500 000 x 61: 27 us of a product)
#pragma unroll
            for (int k = 0; k < 4; k++) e[k] = relu1(p.accumulate ? e[k] + d[k] : e[k], act);
            const unsigned at = (unsigned)reinterpret_cast<uintptr_t>(d) & 15u;
            if (at == 0) st_y4(d, make_float4(e[0], e[1], e[2], e[3]), policy);
            else if (at == 8) { st_y2(d, e[0], e[1], policy); st_y2(d + 2, e[2], e[3], policy); }
            else { st_y1(d, e[0], policy); st_y2(d + 1, e[1], e[2], policy); st_y1(d + 3, e[3], policy); }
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (col + k < p.dim_store) st_y1(d + k, relu1(p.accumulate ? e[k] + d[k] : e[k], act), policy);
        }
    }
}
template <bool PLAIN>
__device__ __forceinline__ void emit_row1(const SpmmParams &p, float *y, float v, int act, uint64_t policy)
{
    st_y1(y, relu1(!PLAIN && p.accumulate ? v + *y : v, act), policy);
}

__device__ __forceinline__ void fma4(float4 &acc, float a, const float4 &v)
{
    acc.x = fmaf(a, v.x, acc.x);
    acc.y = fmaf(a, v.y, acc.y);
    acc.z = fmaf(a, v.z, acc.z);
    acc.w = fmaf(a, v.w, acc.w);
}

// UNROLL independent 16-byte loads are issued per lane before the first FMA needs one.
template <int UNROLL, bool HOT, int LOOSE>
__device__ __forceinline__ float4 gather_vec4(const int2 *pairs, int count, int first, int step,
                                              const float *__restrict__ x, int64_t ldx, bool active, const L2Policies &pol)
{
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!active) return acc;
    int i = first;
    for (; i + (UNROLL - 1) * step < count; i += UNROLL * step) {
        int2 p[UNROLL];
        float4 v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) p[u] = pairs[i + u * step];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) v[u] = ld_x<HOT, LOOSE>(x + (int64_t)p[u].x * ldx, pol, p[u].x);
#pragma unroll
        for (int u = 0; u < UNROLL; u++) fma4(acc, __int_as_float(p[u].y), v[u]);
    }
    if (i < count) {
        // tail: the same batch with the loads past the end switched off
        int2 p[UNROLL - 1];
        float4 v[UNROLL - 1];
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++) {
            const bool live = i + u * step < count;
            p[u] = live ? pairs[i + u * step] : make_int2(0, 0);
            v[u] = live ? ld_x<HOT, LOOSE>(x + (int64_t)p[u].x * ldx, pol, p[u].x) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++)
            if (i + u * step < count) fma4(acc, __int_as_float(p[u].y), v[u]);
    }
    return acc;
}

// `rows` consecutive rows of row_nz nonzeros each, whole rows for this lane: one stream of gathers, UNROLL in
// flight across row boundaries.  (Row by row, rows of three nonzeros keep three gathers in flight and a slot with
// six of them waits six times.)
template <int UNROLL, bool PLAIN, bool HOT, int LOOSE>
__device__ __forceinline__ void gather_rows4(const SpmmParams &p, const int2 *pairs, int rows, int row_nz, const float *__restrict__ x,
                                             float *yr, int col, const L2Policies &pol)
{
    const int count = rows * row_nz;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    int left = row_nz;
    auto take = [&](float a, const float4 &v) {
        fma4(acc, a, v);
        if (--left == 0) {
            emit_row4<PLAIN, LOOSE>(p, yr, col, acc, p.relu, pol.stream);
            acc = make_float4(0.f, 0.f, 0.f, 0.f);
            left = row_nz;
            yr += p.ldy;
        }
    };
    int i = 0;
    for (; i + UNROLL <= count; i += UNROLL) {
        int2 q[UNROLL];
        float4 v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) q[u] = pairs[i + u];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) v[u] = ld_x<HOT, LOOSE>(x + (int64_t)q[u].x * p.ldx, pol, q[u].x);
#pragma unroll
        for (int u = 0; u < UNROLL; u++) take(__int_as_float(q[u].y), v[u]);
    }
    if (i < count) {
        int2 q[UNROLL - 1];
        float4 v[UNROLL - 1];
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++) {
            const bool live = i + u < count;
            q[u] = live ? pairs[i + u] : make_int2(0, 0);
            v[u] = live ? ld_x<HOT, LOOSE>(x + (int64_t)q[u].x * p.ldx, pol, q[u].x) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++)
            if (i + u < count) take(__int_as_float(q[u].y), v[u]);
    }
}

// The same with 8 columns per lane, 32 bytes per load.  (Functions of their own: written as one for either width they
// cost the 16-byte forms registers, and small products 1-5 %.)
struct Octet {
    float4 a, b;
};
__device__ __forceinline__ Octet zero_octet() { return {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)}; }
__device__ __forceinline__ void fma8(Octet &acc, float a, const Octet &v) { fma4(acc.a, a, v.a); fma4(acc.b, a, v.b); }
template <bool HOT>
__device__ __forceinline__ Octet ld_octet(const float *p, const L2Policies &pol, int column)
{
    Octet v;
    ld_x8(p, x_policy<HOT>(pol, column), v.a, v.b);
    return v;
}
template <bool PLAIN>
__device__ __forceinline__ void emit_row8(const SpmmParams &p, float *yr, int col, const Octet &v, uint64_t policy)
{
    if (PLAIN) st_y8(yr + col, relu4(v.a, p.relu), relu4(v.b, p.relu), policy);
    else { emit_row4<false>(p, yr, col, v.a, p.relu, policy); emit_row4<false>(p, yr, col + 4, v.b, p.relu, policy); }
}

template <int UNROLL, bool HOT>
__device__ __forceinline__ Octet gather_vec8(const int2 *pairs, int count, int first, int step, const float *__restrict__ x, int64_t ldx, bool active,
                                             const L2Policies &pol)
{
    Octet acc = zero_octet();
    if (!active) return acc;
    int i = first;
    for (; i + (UNROLL - 1) * step < count; i += UNROLL * step) {
        int2 p[UNROLL];
        Octet v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) p[u] = pairs[i + u * step];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) v[u] = ld_octet<HOT>(x + (int64_t)p[u].x * ldx, pol, p[u].x);
#pragma unroll
        for (int u = 0; u < UNROLL; u++) fma8(acc, __int_as_float(p[u].y), v[u]);
    }
    if (i < count) {
        int2 p[UNROLL - 1];
        Octet v[UNROLL - 1];
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++) {
            const bool live = i + u * step < count;
            p[u] = live ? pairs[i + u * step] : make_int2(0, 0);
            v[u] = live ? ld_octet<HOT>(x + (int64_t)p[u].x * ldx, pol, p[u].x) : zero_octet();
        }
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++)
            if (i + u * step < count) fma8(acc, __int_as_float(p[u].y), v[u]);
    }
    return acc;
}

template <int UNROLL, bool PLAIN, bool HOT>
__device__ __forceinline__ void gather_rows8(const SpmmParams &p, const int2 *pairs, int rows, int row_nz, const float *__restrict__ x, float *yr, int col,
                                             const L2Policies &pol)
{
    const int count = rows * row_nz;
    Octet acc = zero_octet();
    int left = row_nz;
    auto take = [&](float a, const Octet &v) {
        fma8(acc, a, v);
        if (--left == 0) {
            emit_row8<PLAIN>(p, yr, col, acc, pol.stream);
            acc = zero_octet();
            left = row_nz;
            yr += p.ldy;
        }
    };
    int i = 0;
    for (; i + UNROLL <= count; i += UNROLL) {
        int2 q[UNROLL];
        Octet v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) q[u] = pairs[i + u];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) v[u] = ld_octet<HOT>(x + (int64_t)q[u].x * p.ldx, pol, q[u].x);
#pragma unroll
        for (int u = 0; u < UNROLL; u++) take(__int_as_float(q[u].y), v[u]);
    }
    if (i < count) {
        int2 q[UNROLL - 1];
        Octet v[UNROLL - 1];
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++) {
            const bool live = i + u < count;
            q[u] = live ? pairs[i + u] : make_int2(0, 0);
            v[u] = live ? ld_octet<HOT>(x + (int64_t)q[u].x * p.ldx, pol, q[u].x) : zero_octet();
        }
#pragma unroll
        for (int u = 0; u < UNROLL - 1; u++)
            if (i + u < count) take(__int_as_float(q[u].y), v[u]);
    }
}

__device__ __forceinline__ float4 fold4(float4 v, int off)
{
    v.x += __shfl_xor_sync(FULL_MASK, v.x, off);
    v.y += __shfl_xor_sync(FULL_MASK, v.y, off);
    v.z += __shfl_xor_sync(FULL_MASK, v.z, off);
    v.w += __shfl_xor_sync(FULL_MASK, v.w, off);
    return v;
}

constexpr int SPMM_SCALAR_COLS = SPMM_PANEL / 32;   // columns per lane in scalar mode

// Scalar mode: lane l owns columns l, l+32, ... (K = ceil(dim / 32) of them), every load instruction
// of the warp reads 128 contiguous bytes of one X row.  Nonzeros are taken in batches so that about
// 8 loads per lane are in flight, as in the float4 mode.
template <int K>
__device__ __forceinline__ void gather_strided(const int2 *pairs, int count, const float *__restrict__ x,
                                               int64_t ldx, int dim, float (&acc)[SPMM_SCALAR_COLS], uint64_t keep)
{
    constexpr int U = K <= 2 ? 4 : 2;        // nonzeros per batch
    const int lane = lane_id();
    bool live[K];
#pragma unroll
    for (int k = 0; k < K; k++) live[k] = lane + 32 * k < dim;
#pragma unroll
    for (int k = 0; k < SPMM_SCALAR_COLS; k++) acc[k] = 0.f;
    int i = 0;
    for (; i + U <= count; i += U) {
        int2 p[U];
        float v[U][K];
#pragma unroll
        for (int u = 0; u < U; u++) p[u] = pairs[i + u];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float *xr = x + (int64_t)p[u].x * ldx + lane;
#pragma unroll
            for (int k = 0; k < K; k++) v[u][k] = live[k] ? ld_x1(xr + 32 * k, keep) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int k = 0; k < K; k++) acc[k] = fmaf(__int_as_float(p[u].y), v[u][k], acc[k]);
    }
    for (; i < count; i++) {
        const int2 p0 = pairs[i];
        const float *xr = x + (int64_t)p0.x * ldx + lane;
#pragma unroll
        for (int k = 0; k < K; k++)
            if (live[k]) acc[k] = fmaf(__int_as_float(p0.y), ld_x1(xr + 32 * k, keep), acc[k]);
    }
}

__device__ __forceinline__ void gather_scalar(const int2 *pairs, int count, const float *__restrict__ x,
                                              int64_t ldx, int dim, float (&acc)[SPMM_SCALAR_COLS], uint64_t keep)
{
    switch ((dim + 31) >> 5) {            // uniform over the launch
    case 1: gather_strided<1>(pairs, count, x, ldx, dim, acc, keep); break;
    case 2: gather_strided<2>(pairs, count, x, ldx, dim, acc, keep); break;
    case 3: gather_strided<3>(pairs, count, x, ldx, dim, acc, keep); break;
    default: gather_strided<4>(pairs, count, x, ldx, dim, acc, keep); break;
    }
}

// the partials warps w .. w_end - 1 left in shared memory, added in warp order
__device__ __forceinline__ float4 sum_parts4(const float (*part)[SPMM_PANEL], int w, int w_end, int col)
{
    float4 sum = *reinterpret_cast<const float4 *>(&part[w][col]);
    for (int ww = w + 1; ww < w_end; ww++) {
        const float4 v = *reinterpret_cast<const float4 *>(&part[ww][col]);
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    return sum;
}
__device__ __forceinline__ float sum_parts1(const float (*part)[SPMM_PANEL], int w, int w_end, int c)
{
    float sum = part[w][c];
    for (int ww = w + 1; ww < w_end; ww++) sum += part[ww][c];
    return sum;
}

// Stores a row whose partials lie in carry slots span.x .. span.x + span.y - 1, adding them in slot order.
// VEC: `first` is the place of the first of the four columns of this lane (SPMM_PANEL: it has none); otherwise the lane
// takes columns first, first + 32, ...
template <bool VEC, bool PLAIN, int LOOSE = 0>
__device__ __forceinline__ void finish_carried_row(const SpmmParams &p, int2 span, int row, int first, uint64_t policy)
{
    const float *parts = p.carry + (int64_t)span.x * SPMM_PANEL;
    float *yr = p.y + (int64_t)row * p.ldy;
    if (VEC) {
        if (first >= (LOOSE > 0 ? SPMM_PANEL : p.dim)) return;
        float4 sum = __ldcg(reinterpret_cast<const float4 *>(parts + first));
#pragma unroll 8
        for (int q = 1; q < span.y; q++) {
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(parts + (int64_t)q * SPMM_PANEL + first));
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        emit_row4<PLAIN, LOOSE>(p, yr, LOOSE > 0 ? first / 4 : first, sum, p.relu, policy);
    } else {
        for (int c = first; c < p.dim; c += 32) {
            float sum = __ldcg(parts + c);
#pragma unroll 8
            for (int q = 1; q < span.y; q++) sum += __ldcg(parts + (int64_t)q * SPMM_PANEL + c);
            emit_row1<PLAIN>(p, yr + c, sum, p.relu, policy);
        }
    }
}

// ---------------------------------------------------------------------------
// main kernel.  S = lanes per slot in float4 mode (4, 8, 16 or 32; needs
// dim % 4 == 0, dim <= 4*S and 16-byte aligned rows); S = 0 is the scalar
// mode for every other dim (lane l owns columns l, l+32, l+64, l+96).
// ONCE: the plan's kernel was launched before, and only it knows how many units and rows without a tuple there are (p.made).
// Q = columns per lane / 4: with 2, a lane has 8 columns (S = 8 or 16 for up to 64 or 128 of them), loaded 32 bytes at a time:
// rows of X on 32-byte boundaries, dim % 8 == 0; for what products, see spmm_octets.
// FINISH: rows that cross units are finished here (in launches of few units);
// a template parameter because the code costs registers the large launches
// do not have (two more spills, 3 % of a product of 500 000 rows).
// HOT: rows of X the L2 is to keep are told from the others.
// ANY_ROWS: as float4 mode, with the same additions in the same order, but rows of X and Y of any alignment: lane l of a
// slot has columns l, l + S, l + 2 S, l + 3 S (consecutive ones cost four times the wavefronts).
// ---------------------------------------------------------------------------
template <int S, int Q, int BATCH, int MIN_BLOCKS, bool PLAIN, bool FINISH, bool HOT, bool ANY_ROWS, bool ONCE = false>
__global__ void __launch_bounds__(SPMM_THREADS, MIN_BLOCKS)
spmm_units_kernel(const SpmmParams p)
{
    __shared__ int2 s_pair[SPMM_WARPS][SPMM_DEG_BOUND];
    __shared__ __align__(16) float s_part[SPMM_WARPS][SPMM_PANEL];
    __shared__ int s_row[SPMM_WARPS];
    __shared__ int s_big[SPMM_WARPS];               // the warp left a partial sum of row s_row in s_part

    constexpr bool VEC = S > 0;
    constexpr int LANES = VEC ? S : 32;
    constexpr int NS = 32 / LANES;          // nonzeros a warp works on at a time
    const int w = warp_id(), lane = lane_id();
    const int slot = lane / LANES, sl = lane % LANES;
    constexpr int LOOSE = ANY_ROWS ? S : 0;
    const int col = VEC ? sl * 4 * Q : sl;              // place of the lane's sums among the partials
    const int ycol = ANY_ROWS ? sl : col;           // and of the first of them in a row of X and Y
    const bool active = ycol < (ANY_ROWS ? p.dim_store : p.dim);
    L2Policies pol = make_l2_policies();
    if (HOT) pol.hot = p.hot_column;
    if constexpr (ANY_ROWS) pol.cols = (p.dim_store - sl + S - 1) / S;

    if constexpr (ONCE) wait_for_predecessor();                // launched early behind the plan's kernel, or the copy of X behind it
    if (!p.wait_first) launch_dependents();     // a dense transform of this product's result may lay out its weights meanwhile
    if (p.abort_flag != nullptr && *p.abort_flag != 0) return;     // input rejected by a check earlier in the stream
    if constexpr (ONCE) {
        if ((int64_t)blockIdx.x < p.n_units && blockIdx.x >= (unsigned)p.made[PLAN_MADE_UNITS]) return;
    }
    if ((int64_t)blockIdx.x >= p.n_units) {
        wait_for_predecessor();
        // zero-fill rows that no tuple covers
        // (when accumulating, these rows keep their value and only the activation is applied)
        int64_t zb = ((int64_t)blockIdx.x - p.n_units) * SPMM_ZERO_ROWS_PER_BLOCK;
        const int64_t n_zero_rows = ONCE ? (int64_t)p.made[PLAN_MADE_ZERO] : p.n_zero_rows;
        do {
            for (int k = w * NS + slot; k < SPMM_ZERO_ROWS_PER_BLOCK; k += SPMM_WARPS * NS) {
                if (zb + k >= n_zero_rows) break;
                float *yr = p.y + (int64_t)p.zero_rows[zb + k] * p.ldy;
                if (VEC) {
                    if constexpr (Q == 2) {
                        if (active) emit_row8<PLAIN>(p, yr, ycol, zero_octet(), pol.stream);
                    } else if (active) emit_row4<PLAIN, LOOSE>(p, yr, ycol, make_float4(0.f, 0.f, 0.f, 0.f), p.relu, pol.stream);
                } else {
                    for (int c = lane; c < p.dim; c += 32) emit_row1<PLAIN>(p, yr + c, 0.f, p.relu, pol.stream);
                }
            }
            zb += ((int64_t)gridDim.x - p.n_units) * SPMM_ZERO_ROWS_PER_BLOCK;       // ONCE: as many blocks as there may be rows would be a great many
        } while (ONCE && zb < n_zero_rows);
        return;
    }

    const unsigned b = blockIdx.x, k = p.light_every, n = ONCE ? (unsigned)p.made[PLAN_MADE_UNITS] : (unsigned)p.n_units;
    const int64_t unit = p.unit_base + (k != 0 && b % k == k - 1 ? b / k : n - 1 - (k != 0 ? b - b / k : b));
    const int64_t e = unit * SPMM_WARPS + w;
    const TupleView t = decode_tuple<ONCE>(p.tuples, e, p.n_tuples);
    const bool big = t.valid && !t.small;
    const int total = t.n_rows * t.row_nz;
    if (p.wait_first) {                 // tuples are the plan's and do not change
        wait_for_predecessor();
        launch_dependents();            // not above the wait: then whoever comes next finds that one finished, too
    }

    // stage the tuple's (col, val) pairs
    {
        const int *__restrict__ gi = p.idx + t.loc;
        const float *__restrict__ gv = p.val + t.loc;
#pragma unroll 4
        for (int k = lane; k < total; k += 32)
            s_pair[w][k] = make_int2(ld_a(gi + k, pol.stream), __float_as_int(ld_a(gv + k, pol.stream)));
    }
    __syncwarp();

    const int2 *pairs = s_pair[w];
    wait_for_predecessor();             // X may be what the launch before this one makes

    if constexpr (Q == 2) {
        const float *xc = p.x + ycol;
        if (t.small && t.row_nz <= 32) {
            const int each = (t.n_rows + NS - 1) / NS, r0 = slot * each;
            const int rows = r0 < t.n_rows ? (r0 + each < t.n_rows ? each : t.n_rows - r0) : 0;
            if (active) gather_rows8<BATCH, PLAIN, HOT>(p, pairs + r0 * t.row_nz, rows, t.row_nz, xc, p.y + (int64_t)(t.row0 + r0) * p.ldy, ycol, pol);
        } else {
            for (int r = 0; r < t.n_rows; r++) {
                Octet acc = gather_vec8<BATCH, HOT>(pairs + r * t.row_nz, t.row_nz, slot, NS, xc, p.ldx, active, pol);
#pragma unroll
                for (int off = LANES; off < 32; off <<= 1) { acc.a = fold4(acc.a, off); acc.b = fold4(acc.b, off); }
                if (slot == 0 && active) {
                    if (t.small) emit_row8<PLAIN>(p, p.y + (int64_t)(t.row0 + r) * p.ldy, ycol, acc, pol.stream);
                    else {
                        *reinterpret_cast<float4 *>(&s_part[w][col]) = acc.a;
                        *reinterpret_cast<float4 *>(&s_part[w][col + 4]) = acc.b;
                    }
                }
            }
        }
    } else if (VEC) {
        const float *xc = p.x + ycol;
        if (t.small && t.row_nz <= 32) {
            // whole rows for every slot, consecutive ones
            const int each = (t.n_rows + NS - 1) / NS, r0 = slot * each;
            const int rows = r0 < t.n_rows ? (r0 + each < t.n_rows ? each : t.n_rows - r0) : 0;
            if (active)
                gather_rows4<BATCH, PLAIN, HOT, LOOSE>(p, pairs + r0 * t.row_nz, rows, t.row_nz, xc, p.y + (int64_t)(t.row0 + r0) * p.ldy, ycol, pol);
        } else {
            // the slots of the warp share each row
            for (int r = 0; r < t.n_rows; r++) {
                float4 acc = gather_vec4<BATCH, HOT, LOOSE>(pairs + r * t.row_nz, t.row_nz, slot, NS, xc, p.ldx, active, pol);
#pragma unroll
                for (int off = LANES; off < 32; off <<= 1) {
                    acc.x += __shfl_xor_sync(FULL_MASK, acc.x, off);
                    acc.y += __shfl_xor_sync(FULL_MASK, acc.y, off);
                    acc.z += __shfl_xor_sync(FULL_MASK, acc.z, off);
                    acc.w += __shfl_xor_sync(FULL_MASK, acc.w, off);
                }
                if (slot == 0 && active) {
                    if (t.small) emit_row4<PLAIN, LOOSE>(p, p.y + (int64_t)(t.row0 + r) * p.ldy, ycol, acc, p.relu, pol.stream);
                    else *reinterpret_cast<float4 *>(&s_part[w][col]) = acc;
                }
            }
        }
    } else {
        for (int r = 0; r < t.n_rows; r++) {
            float acc[SPMM_SCALAR_COLS];
            gather_scalar(pairs + r * t.row_nz, t.row_nz, p.x, p.ldx, p.dim, acc, pol.keep);
#pragma unroll
            for (int k = 0; k < SPMM_SCALAR_COLS; k++) {
                const int c = lane + 32 * k;
                if (c < p.dim) {
                    if (t.small) emit_row1<PLAIN>(p, p.y + (int64_t)(t.row0 + r) * p.ldy + c, acc[k], p.relu, pol.stream);
                    else s_part[w][c] = acc[k];
                }
            }
        }
    }

    // heavy rows: add the per-tuple partials of a row in tuple order
    if (lane == 0) { s_row[w] = t.row0; s_big[w] = big ? 1 : 0; }
    __syncthreads();
    if (!big) return;
    if (w > 0 && s_big[w - 1] && s_row[w - 1] == t.row0) return;   // not the first tuple of its row here
    int w_end = w + 1;
    while (w_end < SPMM_WARPS && s_big[w_end] && s_row[w_end] == t.row0) w_end++;
    const int64_t left = p.n_tuples - unit * SPMM_WARPS;
    const int w_last = left < SPMM_WARPS ? (int)left - 1 : SPMM_WARPS - 1;
    const int2 uc = ld_plan<ONCE>(p.unit_carry + unit);
    const bool enters = w == 0 && uc.x >= 0;            // the row began in an earlier unit
    const bool leaves = w_end - 1 == w_last && uc.y >= 0;   // the row goes on in the next unit
    const bool partial = enters || leaves;     // other units hold the rest of the row
    float *yr = p.y + (int64_t)t.row0 * p.ldy;
    if (!partial) {
        if (VEC) {
            if constexpr (Q == 2) {
                if (slot == 0 && active) emit_row8<PLAIN>(p, yr, ycol, {sum_parts4(s_part, w, w_end, col), sum_parts4(s_part, w, w_end, col + 4)}, pol.stream);
            } else if (slot == 0 && active) emit_row4<PLAIN, LOOSE>(p, yr, ycol, sum_parts4(s_part, w, w_end, col), p.relu, pol.stream);
        } else {
            for (int c = lane; c < p.dim; c += 32) emit_row1<PLAIN>(p, yr + c, sum_parts1(s_part, w, w_end, c), p.relu, pol.stream);
        }
        return;
    }
    const int my_slot = enters ? uc.x : uc.y;
    float *mine = p.carry + (int64_t)my_slot * SPMM_PANEL;
    if (VEC) {
        if (slot == 0 && active) *reinterpret_cast<float4 *>(mine + col) = sum_parts4(s_part, w, w_end, col);
        if constexpr (Q == 2)
            if (slot == 0 && active) *reinterpret_cast<float4 *>(mine + col + 4) = sum_parts4(s_part, w, w_end, col + 4);
    } else {
        for (int c = lane; c < p.dim; c += 32) mine[c] = sum_parts1(s_part, w, w_end, c);
    }
    if (!FINISH) return;                            // spmm_carry_kernel follows
    // the row's last unit to arrive adds the partials
    const int2 span = ld_plan<ONCE>(p.carry_span + my_slot);
    __threadfence();
    __syncwarp();
    int arrived = 0;
    if (lane == 0) arrived = atomicAdd(p.carry_count + span.x, 1);
    arrived = __shfl_sync(FULL_MASK, arrived, 0);
    if (arrived != span.y - 1) return;
    if (lane == 0) p.carry_count[span.x] = 0;       // ready for the next product
    __threadfence();
    finish_carried_row<VEC, PLAIN, LOOSE>(p, span, t.row0, VEC ? (slot == 0 && active ? col : SPMM_PANEL) : lane, pol.stream);
    if constexpr (Q == 2) finish_carried_row<VEC, PLAIN, LOOSE>(p, span, t.row0, slot == 0 && active ? col + 4 : SPMM_PANEL, pol.stream);
}

// Adds the carried partials of every row that crosses unit boundaries.  One warp per carry slot; the warp of
// the first slot of a row does the work.  Bound by latency: the partials of a row are loaded eight at a time
// (a hub row of 90 000 nonzeros has 30; loaded one by one they took 12 us).
template <bool VEC>
__global__ void __launch_bounds__(SPMM_THREADS)
spmm_carry_kernel(const SpmmParams p, const int *__restrict__ carry_row, int64_t n_carry)
{
    const int64_t s = (int64_t)blockIdx.x * SPMM_WARPS + warp_id();
    wait_for_predecessor();         // launched early behind the units
    launch_dependents();
    if (s >= n_carry) return;
    const int2 span = p.carry_span[s];
    if (span.x != s) return;
    finish_carried_row<VEC, false>(p, span, carry_row[s], VEC ? lane_id() * 4 : lane_id(), make_l2_policies().stream);
}

// X[n_rows x dim] with row stride ldx  ->  XP[n_rows x ldp], ldp = dim rounded up to 4, tail zero:
// the 16-byte-aligned copy of a dense operand whose rows are not (dim % 4 != 0 or an unaligned base).
// Every thread writes PAD_ITEMS times 16 bytes; a 64-bit division for each of them was as much work as the
// memory traffic (500 000 x 61: 40 us).  It lets the product that follows begin at once: that one waits
// before it reads X.
constexpr int PAD_BLOCK = 256, PAD_ITEMS = 4;

__global__ void __launch_bounds__(PAD_BLOCK)
spmm_pad_rows_kernel(const float *x, int64_t ldx, int dim, float *xp, int ldp, int64_t n_rows)      // not __restrict__: X is read behind the wait
{
    wait_for_predecessor();         // launched early behind whatever makes X
    launch_dependents();            // not above the wait: the product reads column ids and values before it waits for this kernel
    const unsigned quads = (unsigned)ldp >> 2, per_quad = ((1u << 20) + quads - 1) / quads;      // n / quads = n * per_quad >> 20 for n * quads < 2^20
    const int64_t first = (int64_t)blockIdx.x * (PAD_BLOCK * PAD_ITEMS);
    const int64_t row0 = first / quads;
    const unsigned rest = (unsigned)(first - row0 * quads);
    float4 v[PAD_ITEMS];
#pragma unroll
    for (int k = 0; k < PAD_ITEMS; k++) {
        const unsigned at = rest + k * PAD_BLOCK + threadIdx.x;
        const unsigned r = quads <= 512 ? at * per_quad >> 20 : at / quads;
        const int64_t row = row0 + r;
        const int c = (int)(at - r * quads) * 4;
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n_rows) {
            const float *src = x + row * ldx + c;
            if (c + 0 < dim) v[k].x = src[0];
            if (c + 1 < dim) v[k].y = src[1];
            if (c + 2 < dim) v[k].z = src[2];
            if (c + 3 < dim) v[k].w = src[3];
        }
    }
#pragma unroll
    for (int k = 0; k < PAD_ITEMS; k++) {
        const int64_t at = first + k * PAD_BLOCK + threadIdx.x;
        if (at < n_rows * quads) *reinterpret_cast<float4 *>(xp + at * 4) = v[k];
    }
}

// ---------------------------------------------------------------------------
// plan: built once per `.block4` array
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool tuple_is_big(const int4 &b) { return b.x > SPMM_DEG_BOUND; }
__device__ __forceinline__ int tuple_rows(const int4 &b) { return tuple_is_big(b) ? 1 : (b.w & 0xffff); }

constexpr int PLAN_FULL_NZ = 192;
constexpr int PLAN_BLOCK = 256;      // units per thread block, one per thread

__device__ __forceinline__ void plan_report(HostWords *out, int err, int *bad = nullptr)
{
    if (bad != nullptr) *bad = 1;
#pragma unroll
    for (int k = 0; k < PLAN_ERR_BITS; k++)
        if (err & (1 << k)) out->w[PLAN_WORD_ERR + k] = 1;
}

__device__ __forceinline__ int64_t tuple_nz(const int4 &b) { return tuple_is_big(b) ? (int64_t)b.w : (int64_t)tuple_rows(b) * b.x; }

// rows that lie between tuples a and b (a == nullptr: before the first); negative: out of order or overlapping
__device__ __forceinline__ int64_t tuple_gap(bool has_prev, const int4 &a, const int4 &b)
{
    if (!has_prev) return b.y;
    if (tuple_is_big(b) && tuple_is_big(a) && a.y == b.y) return 0;       // a later chunk of the same heavy row
    return (int64_t)b.y - ((int64_t)a.y + tuple_rows(a));
}

__device__ __forceinline__ int tuple_errors(bool has_prev, const int4 &a, const int4 &b, int64_t n_rows, int64_t nnz)
{
    const int rows = tuple_rows(b);
    const int64_t nz = tuple_nz(b);
    const int64_t prev_loc_end = has_prev ? (int64_t)a.z + tuple_nz(a) : 0;
    int err = 0;
    if (b.x < 1 || rows < 1 || nz < 1 || nz > SPMM_DEG_BOUND) err |= SPMM_ERR_TUPLE;
    // tuples take their nonzeros in order and without overlap (what lets A be uploaded and multiplied
    // range by range: a tuple never reaches into a range that has not arrived)
    if (b.z < 0 || (int64_t)b.z + nz > nnz || (int64_t)b.z < prev_loc_end) err |= SPMM_ERR_LOC;
    if (b.y < 0 || (int64_t)b.y + rows > n_rows || tuple_gap(has_prev, a, b) < 0) err |= SPMM_ERR_ROW;
    return err;
}

// How a tuple is cut into pieces of at most `most` nonzeros: whole rows where they fit, otherwise every row by itself.
// A piece has the form of a tuple; one that is part of a row says so by a degree above the bound.
struct TupleCut {
    int pieces, rows_each, row_pieces, nz_each;
};
__device__ __forceinline__ TupleCut tuple_cut(const int4 &b, int most)
{
    const int rows = tuple_rows(b), row_nz = tuple_is_big(b) ? b.w : b.x;
    TupleCut c;
    if (row_nz <= most && !tuple_is_big(b)) {
        const int fit = most / row_nz;
        c.pieces = (rows + fit - 1) / fit;
        c.rows_each = (rows + c.pieces - 1) / c.pieces;
        c.pieces = (rows + c.rows_each - 1) / c.rows_each;
        c.row_pieces = 0; c.nz_each = 0;
    } else {
        c.row_pieces = (row_nz + most - 1) / most;
        c.nz_each = (row_nz + c.row_pieces - 1) / c.row_pieces;
        c.row_pieces = (row_nz + c.nz_each - 1) / c.nz_each;
        c.pieces = rows * c.row_pieces;
        c.rows_each = 0;
    }
    return c;
}

// Does a heavy row enter unit u from the left / leave it to the right?
__device__ __forceinline__ void unit_crossings(const int4 *__restrict__ block4, int64_t n_blocks, int64_t u,
                                               bool &enters, bool &leaves, bool &same_row, int &row_in, int &row_out)
{
    const int64_t e0 = u * SPMM_WARPS;
    const int64_t e1 = e0 + SPMM_WARPS < n_blocks ? e0 + SPMM_WARPS : n_blocks;   // one past the unit
    const int4 first = block4[e0], last = block4[e1 - 1];
    enters = false; leaves = false;
    if (e0 > 0 && tuple_is_big(first)) {
        const int4 a = block4[e0 - 1];
        enters = tuple_is_big(a) && a.y == first.y;
    }
    if (e1 < n_blocks && tuple_is_big(last)) {
        const int4 c = block4[e1];
        leaves = tuple_is_big(c) && c.y == last.y;
    }
    row_in = first.y; row_out = last.y;
    same_row = enters && leaves && first.y == last.y;
}

// Is any of the column ids idx[0 .. n_idx) outside [0, n_cols)?  The part of thread `first` of `stride`.  16 bytes per
// load (one id per load and 64-bit comparisons: 54 us for 6e7 ids, of which HBM needs 37) but for the ends that are not
// aligned.
__device__ __forceinline__ bool ids_outside(const int *__restrict__ idx, int64_t n_idx, int64_t n_cols, int64_t first, int64_t stride)
{
    const unsigned n = (unsigned)n_cols;                       // below 2^31: negative ids compare as larger ones
    int64_t head = (int64_t)((16 - (reinterpret_cast<uintptr_t>(idx) & 15)) & 15) / 4;
    if (head > n_idx) head = n_idx;
    const int4 *quads = reinterpret_cast<const int4 *>(idx + head);
    const int64_t n_quads = (n_idx - head) / 4, tail = head + n_quads * 4;
    bool bad = false;
#pragma unroll 4
    for (int64_t i = first; i < n_quads; i += stride) {
        const int4 c = __ldcs(quads + i);
        bad |= (unsigned)c.x >= n || (unsigned)c.y >= n || (unsigned)c.z >= n || (unsigned)c.w >= n;
    }
    if (first < head) bad |= (unsigned)idx[first] >= n;        // at most three ids at either end; there are as many threads
    if (first < n_idx - tail) bad |= (unsigned)idx[tail + first] >= n;
    return bad;
}

// Column ids, by `blocks` thread blocks of which this is number `block`.
__device__ __forceinline__ void plan_check_ids(const int *__restrict__ idx, int64_t n_idx, int64_t n_cols, unsigned block, unsigned blocks, HostWords *out,
                                               int *bad = nullptr)
{
    if (ids_outside(idx, n_idx, n_cols, (int64_t)block * blockDim.x + threadIdx.x, (int64_t)blocks * blockDim.x)) plan_report(out, SPMM_ERR_COL, bad);
}

// How many of PLAN_SAMPLES column ids, one from every PLAN_SAMPLES-th part of the nonzeros, are at least `first` (anywhere
// in its part: at even distances it could always be the last, largest id of a row).  By one thread block.
constexpr int PLAN_SAMPLE_ITEMS = 16, PLAN_SAMPLES = PLAN_BLOCK * PLAN_SAMPLE_ITEMS;

__device__ __forceinline__ void plan_tail_share(const int *__restrict__ idx, int64_t n_idx, int64_t first, HostWords *out)
{
    const int64_t part = n_idx / PLAN_SAMPLES;
    int count = 0;
#pragma unroll
    for (int k = 0; k < PLAN_SAMPLE_ITEMS; k++) {
        const unsigned n = k * PLAN_BLOCK + threadIdx.x;
        const int64_t within = part * (int64_t)(n * 2654435769u >> 8) >> 24;
        count += n_idx > 0 && __ldg(idx + n * part + within) >= first;
    }
    __shared__ int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    count = warp_reduce(count, OpAdd());
    if (lane_id() == 0) atomicAdd(&s_sum, count);
    __syncthreads();
    if (threadIdx.x == 0) out->w[PLAN_WORD_TAIL] = s_sum;
}

// First pass over a `.block4` array: validates every tuple (and, in the blocks behind the tuple blocks,
// every column id), and counts per PLAN_BLOCK units the rows no tuple covers and the carry slots.  One
// launch and one read of 16 bytes per tuple and 4 per nonzero: bound by HBM for large graphs, by launch
// latency for small ones.  ctl[0..2]: totals (the third: tuples of at least PLAN_FULL_NZ nonzeros), ctl[3]: blocks
// done (zero at launch).  tail_first >= 0: the first block behind the tuple blocks samples the column ids from there on.
__global__ void __launch_bounds__(PLAN_BLOCK)
plan_check_kernel(const int4 *__restrict__ block4, int64_t n_blocks, int64_t n_units, int64_t n_rows, int64_t nnz,
                  const int *__restrict__ idx, int64_t n_idx, int64_t n_cols, unsigned unit_grid, int64_t tail_first,
                  int64_t *__restrict__ tile_zero, int *__restrict__ tile_carry, unsigned long long *__restrict__ ctl,
                  HostWords *out)
{
    if (blockIdx.x >= unit_grid) {
        const unsigned asked = tail_first >= 0 ? 1 : 0;
        if (blockIdx.x - unit_grid < asked) plan_tail_share(idx, n_idx, tail_first, out);
        else plan_check_ids(idx, n_idx, n_cols, blockIdx.x - unit_grid - asked, gridDim.x - unit_grid - asked, out);
        return;
    }
    __shared__ int64_t s_zero[PLAN_BLOCK / 32];
    __shared__ int s_carry[PLAN_BLOCK / 32], s_full[PLAN_BLOCK / 32];
    const int64_t u = (int64_t)blockIdx.x * PLAN_BLOCK + threadIdx.x;
    int64_t zero = 0;
    int carry = 0, err = 0, full = 0;
    if (u < n_units || (n_units == 0 && u == 0)) {          // without any tuple, one thread counts the rows
        const int64_t e0 = u * SPMM_WARPS;
        const int64_t e1 = e0 + SPMM_WARPS < n_blocks ? e0 + SPMM_WARPS : n_blocks;
        int4 a = e0 > 0 ? block4[e0 - 1] : make_int4(0, 0, 0, 0);
        for (int64_t e = e0; e < e1; e++) {
            const int4 b = block4[e];
            err |= tuple_errors(e > 0, a, b, n_rows, nnz);
            full += tuple_nz(b) >= PLAN_FULL_NZ;
            const int64_t g = tuple_gap(e > 0, a, b);
            zero += g > 0 ? g : 0;
            a = b;
        }
        if (e1 == n_blocks) {                 // rows after the last tuple
            const int64_t g = n_rows - ((int64_t)a.y + tuple_rows(a));
            zero += g > 0 ? g : 0;
        }
        bool en = false, lv = false, same = false; int ri, ro;
        if (u < n_units) unit_crossings(block4, n_blocks, u, en, lv, same, ri, ro);
        carry = (en ? 1 : 0) + (lv ? 1 : 0) - (same ? 1 : 0);
    }
    if (err) plan_report(out, err);
    zero = warp_reduce(zero, OpAdd());
    carry = warp_reduce(carry, OpAdd());
    full = warp_reduce(full, OpAdd());
    if (lane_id() == 0) { s_zero[warp_id()] = zero; s_carry[warp_id()] = carry; s_full[warp_id()] = full; }
    __syncthreads();
    if (threadIdx.x == 0) {
        zero = 0; carry = 0; full = 0;
        for (int w = 0; w < PLAN_BLOCK / 32; w++) { zero += s_zero[w]; carry += s_carry[w]; full += s_full[w]; }
        tile_zero[blockIdx.x] = zero;
        tile_carry[blockIdx.x] = carry;
        atomicAdd(ctl + 0, (unsigned long long)zero);
        atomicAdd(ctl + 1, (unsigned long long)carry);
        atomicAdd(ctl + 2, (unsigned long long)full);
        __threadfence();
        if (atomicAdd(ctl + 3, 1ull) == unit_grid - 1) {
            __threadfence();
            out->w[PLAN_WORD_ZERO] = (int64_t)__ldcg(ctl + 0);
            out->w[PLAN_WORD_CARRY] = (int64_t)__ldcg(ctl + 1);
            out->w[PLAN_WORD_FULL] = (int64_t)__ldcg(ctl + 2);
        }
    }
}

// column ids of a range that has just been uploaded, for products that are streamed: raises a device flag
__global__ void __launch_bounds__(256)
plan_check_cols_kernel(const int *__restrict__ idx, int64_t nnz, int64_t n_cols, int *__restrict__ err_flag)
{
    if (ids_outside(idx, nnz, n_cols, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x)) atomicOr(err_flag, SPMM_ERR_COL);
}

// First and last tuple of the row that tuple e belongs to (tuples are in ascending row order).  In steps that double,
// then halve: a row of few tuples is two or three loads away, where a search of all tuples is a chain of 18.
__device__ __forceinline__ int64_t tuple_row_first(const int4 *__restrict__ block4, int64_t e)
{
    const int row = block4[e].y;
    int64_t step = 1;
    while (e - step >= 0 && block4[e - step].y == row) { e -= step; step *= 2; }
    for (step >>= 1; step > 0; step >>= 1)
        if (e - step >= 0 && block4[e - step].y == row) e -= step;
    return e;
}
__device__ __forceinline__ int64_t tuple_row_last(const int4 *__restrict__ block4, int64_t n_blocks, int64_t e)
{
    const int row = block4[e].y;
    int64_t step = 1;
    while (e + step < n_blocks && block4[e + step].y == row) { e += step; step *= 2; }
    for (step >>= 1; step > 0; step >>= 1)
        if (e + step < n_blocks && block4[e + step].y == row) e += step;
    return e;
}

// Second pass: carry slots in unit order, and the list of rows no tuple covers.  A block adds up the counts
// of the tiles before it itself (a few thousand words at most) -- no scan launches between the passes.
// Gaps of many rows (the degree-0 rows of an ordered graph are one gap) are written by the whole block.
constexpr int PLAN_INLINE_GAP = 16, PLAN_GAP_QUEUE = 64;

__global__ void __launch_bounds__(PLAN_BLOCK)
plan_assign_kernel(const int4 *__restrict__ block4, int64_t n_blocks, int64_t n_units, int64_t n_rows,
                   const int64_t *__restrict__ tile_zero, const int *__restrict__ tile_carry,
                   int2 *__restrict__ unit_carry, int2 *__restrict__ carry_span, int *__restrict__ carry_row,
                   int *__restrict__ zero_rows)
{
    __shared__ int64_t s_scan64[PLAN_BLOCK / 32 + 1];
    __shared__ int64_t s_gap_out[PLAN_GAP_QUEUE], s_gap_row[PLAN_GAP_QUEUE], s_gap_len[PLAN_GAP_QUEUE];
    __shared__ int s_gaps;
    if (threadIdx.x == 0) s_gaps = 0;
    int64_t zb = 0, cb = 0;
    for (int64_t k = threadIdx.x; k < blockIdx.x; k += PLAN_BLOCK) { zb += tile_zero[k]; cb += tile_carry[k]; }
    int64_t zero_base, carry_base, total;
    block_scan_exclusive<PLAN_BLOCK>(zb, OpAdd(), (int64_t)0, zero_base, s_scan64);
    block_scan_exclusive<PLAN_BLOCK>(cb, OpAdd(), (int64_t)0, carry_base, s_scan64);

    const int64_t u = (int64_t)blockIdx.x * PLAN_BLOCK + threadIdx.x;
    const int64_t e0 = u * SPMM_WARPS;
    const int64_t e1 = e0 + SPMM_WARPS < n_blocks ? e0 + SPMM_WARPS : n_blocks;
    bool en = false, lv = false, same = false;
    int ri = 0, ro = 0;
    int64_t zero = 0;
    const bool mine = u < n_units || (n_units == 0 && u == 0);
    if (mine) {
        if (u < n_units) unit_crossings(block4, n_blocks, u, en, lv, same, ri, ro);
        if (zero_rows != nullptr) {
            int4 a = e0 > 0 ? block4[e0 - 1] : make_int4(0, 0, 0, 0);
            for (int64_t e = e0; e < e1; e++) { const int4 b = block4[e]; zero += tuple_gap(e > 0, a, b); a = b; }
            if (e1 == n_blocks) zero += n_rows - ((int64_t)a.y + tuple_rows(a));
        }
    }
    const int64_t slot = carry_base + block_scan_exclusive<PLAN_BLOCK>((int64_t)((en ? 1 : 0) + (lv ? 1 : 0) - (same ? 1 : 0)),
                                                                       OpAdd(), (int64_t)0, total, s_scan64);
    int64_t out = zero_base + block_scan_exclusive<PLAN_BLOCK>(zero, OpAdd(), (int64_t)0, total, s_scan64);
    if (mine) {
        int2 uc = make_int2(-1, -1);
        if (en) uc.x = (int)slot;
        if (lv) uc.y = same ? (int)slot : (int)slot + (en ? 1 : 0);
        if (u < n_units) unit_carry[u] = uc;
        // a row has one slot in every unit it touches, and these are consecutive
        for (int side = 0; side < 2; side++) {
            const int s = side == 0 ? uc.x : uc.y;
            if (s < 0 || (side == 1 && same)) continue;
            const int row = side == 0 ? ri : ro;
            const int64_t e = side == 0 ? e0 : e1 - 1;
            const int64_t u0 = tuple_row_first(block4, e) / SPMM_WARPS;
            const int64_t u1 = tuple_row_last(block4, n_blocks, e) / SPMM_WARPS;
            carry_span[s] = make_int2(s - (int)(u - u0), (int)(u1 - u0 + 1));
            carry_row[s] = row;
        }
        if (zero_rows != nullptr && zero > 0) {
            int4 a = e0 > 0 ? block4[e0 - 1] : make_int4(0, 0, 0, 0);
            for (int64_t e = e0; e <= e1; e++) {
                if (e == e1 && e1 != n_blocks) break;
                const int4 b = e < e1 ? block4[e] : make_int4(0, 0, 0, 0);
                const int64_t first = e > 0 ? (int64_t)a.y + tuple_rows(a) : 0;
                const int64_t g = e < e1 ? tuple_gap(e > 0, a, b) : n_rows - first;
                int q = PLAN_GAP_QUEUE;
                if (g > PLAN_INLINE_GAP) q = atomicAdd(&s_gaps, 1);
                if (q < PLAN_GAP_QUEUE) { s_gap_out[q] = out; s_gap_row[q] = first; s_gap_len[q] = g; }
                else for (int64_t k = 0; k < g; k++) zero_rows[out + k] = (int)(first + k);
                out += g;
                a = b;
            }
        }
    }
    __syncthreads();
    const int gaps = s_gaps < PLAN_GAP_QUEUE ? s_gaps : PLAN_GAP_QUEUE;
    for (int q = 0; q < gaps; q++)
        for (int64_t k = threadIdx.x; k < s_gap_len[q]; k += PLAN_BLOCK) zero_rows[s_gap_out[q] + k] = (int)(s_gap_row[q] + k);
}

// How the tuples of a small graph are cut: into pieces of at most `most` nonzeros where that makes no more than `fit` of
// them (`fit_uneven` where the rows are of very different lengths), else of at most `otherwise`.
struct PieceChoice {
    int most, otherwise;
    int fit, fit_uneven;
};

// The whole plan of a small graph in one launch: block 0 validates the tuples, cuts them into pieces
// (cap_pieces of them fit), lists the rows no tuple covers and hands out the carry slots; the next
// clear_blocks zero the arrival counters of the slots, the other blocks check the column ids.  Every array has its final place already, sized by bounds the host knows, so the
// host waits once.  (Two kernels with a wait between them before, the cutting 8 tuples per thread: a plan of 16 384
// rows took 70 us; 26 now, 12 of them on the GPU.)  Bound by latency: a chain of scans over about ten tuples per thread.
constexpr int PLAN_SMALL_BLOCK = 1024;

__global__ void __launch_bounds__(PLAN_SMALL_BLOCK)
plan_small_kernel(const int4 *__restrict__ block4, int n_blocks, int64_t n_rows, int64_t nnz, const int *__restrict__ idx, int64_t n_idx,
                  int64_t n_cols, const PieceChoice choice, int4 *pieces, int cap_pieces, int2 *unit_carry, int2 *carry_span, int *carry_row, int *zero_rows,
                  int *made, int *bad, int *counters, int64_t n_counters, unsigned clear_blocks, HostWords *out)
{
    // made, bad: null, or for a product launched behind this kernel: the numbers it needs, and a word that is zero unless something is wrong
    launch_dependents();
    if (blockIdx.x > clear_blocks) {
        plan_check_ids(idx, n_idx, n_cols, blockIdx.x - 1 - clear_blocks, gridDim.x - 1 - clear_blocks, out, bad);
        return;
    }
    if (blockIdx.x > 0) {
        // 32 for every slot there may be: past 2^31 of them where the pieces are forced to be few nonzeros each
        for (int64_t k = (int64_t)(blockIdx.x - 1) * PLAN_SMALL_BLOCK + threadIdx.x; k < n_counters; k += (int64_t)clear_blocks * PLAN_SMALL_BLOCK) counters[k] = 0;
        return;
    }
    __shared__ int s_scan[PLAN_SMALL_BLOCK / 32 + 1];
    __shared__ int s_gap_out[PLAN_GAP_QUEUE], s_gap_row[PLAN_GAP_QUEUE], s_gap_len[PLAN_GAP_QUEUE];
    __shared__ int s_gaps;
    if (threadIdx.x == 0) s_gaps = 0;
    const int longest = block4[n_blocks - 1].x;            // of rows in degree order
    const int each = (n_blocks + PLAN_SMALL_BLOCK - 1) / PLAN_SMALL_BLOCK;
    const int e0 = min((int)threadIdx.x * each, n_blocks), e1 = min(e0 + each, n_blocks);
    const int4 before = e0 > 0 ? block4[e0 - 1] : make_int4(0, 0, 0, 0);
    int4 a = before;
    int err = 0, mine = 0, most = choice.most;
    int64_t zero = 0;
    for (int e = e0; e < e1; e++) {
        const int4 b = block4[e];
        err |= tuple_errors(e > 0, a, b, n_rows, nnz);
        if (err == 0) { mine += tuple_cut(b, most).pieces; zero += tuple_gap(e > 0, a, b); }
        a = b;
    }
    const bool last = e0 < e1 && e1 == n_blocks;
    if (last && err == 0) zero += n_rows - ((int64_t)a.y + tuple_rows(a));
    if (err) plan_report(out, err, bad);
    if (__syncthreads_or(err)) return;
    int n_pieces, n_zero;
    int piece = block_scan_exclusive<PLAN_SMALL_BLOCK>(mine, OpAdd(), 0, n_pieces, s_scan);
    if (choice.otherwise != most) {
        // rows of an even graph that are longer than a piece would cross thread blocks all of them: three of them fit a piece
        const bool uneven = longest > 2 * most && longest * n_rows > 4 * nnz;
        if (n_pieces > (uneven ? choice.fit_uneven : choice.fit) || (!uneven && 3 * nnz > most * n_rows)) {
            most = choice.otherwise;
            mine = 0;
            for (int e = e0; e < e1; e++) mine += tuple_cut(block4[e], most).pieces;
            piece = block_scan_exclusive<PLAN_SMALL_BLOCK>(mine, OpAdd(), 0, n_pieces, s_scan);
        }
    }
    int zero_out = block_scan_exclusive<PLAN_SMALL_BLOCK>((int)zero, OpAdd(), 0, n_zero, s_scan);
    if (threadIdx.x == 0) { out->w[PLAN_WORD_ZERO] = n_zero; out->w[PLAN_WORD_PIECES] = n_pieces; out->w[PLAN_WORD_LONGEST] = longest; }
    if (n_pieces > cap_pieces) {                    // cannot be: valid tuples do not overlap
        if (threadIdx.x == 0 && bad != nullptr) *bad = 1;
        return;
    }
    if (made != nullptr) {
        if (threadIdx.x == 0) { made[PLAN_MADE_UNITS] = (n_pieces + SPMM_WARPS - 1) / SPMM_WARPS; made[PLAN_MADE_ZERO] = n_zero; }
        // the product counts on cap_pieces of them: the last unit's missing ones are empty
        const int at = n_pieces + threadIdx.x;
        if (threadIdx.x < SPMM_WARPS && at < cap_pieces) pieces[at] = make_int4(0, 0, 0, 0);
    }
    a = before;
    for (int e = e0; e < e1; e++) {
        const int4 b = block4[e];
        const TupleCut c = tuple_cut(b, most);
        const int rows = tuple_rows(b), row_nz = tuple_is_big(b) ? b.w : b.x;
        if (c.row_pieces == 0) {
            for (int r = 0; r < rows; r += c.rows_each)
                pieces[piece++] = make_int4(b.x, b.y + r, b.z + r * row_nz, rows - r < c.rows_each ? rows - r : c.rows_each);
        } else {
            for (int r = 0; r < rows; r++)
                for (int k = 0; k < row_nz; k += c.nz_each)
                    pieces[piece++] = make_int4(SPMM_DEG_BOUND + 1, b.y + r, b.z + r * row_nz + k, row_nz - k < c.nz_each ? row_nz - k : c.nz_each);
        }
        a = b;
    }
    if (zero > 0) {
        a = before;
        for (int e = e0; e < e1 + (last ? 1 : 0); e++) {
            const int4 b = e < e1 ? block4[e] : make_int4(0, 0, 0, 0);
            const int first = e > 0 ? a.y + tuple_rows(a) : 0;
            const int g = e < e1 ? (int)tuple_gap(e > 0, a, b) : (int)(n_rows - first);
            int q = PLAN_GAP_QUEUE;
            if (g > PLAN_INLINE_GAP) q = atomicAdd(&s_gaps, 1);
            if (q < PLAN_GAP_QUEUE) { s_gap_out[q] = zero_out; s_gap_row[q] = first; s_gap_len[q] = g; }
            else for (int k = 0; k < g; k++) zero_rows[zero_out + k] = first + k;
            zero_out += g;
            a = b;
        }
    }
    __syncthreads();                // the pieces are there, and the queue of gaps
    for (int q = 0; q < min(s_gaps, PLAN_GAP_QUEUE); q++)
        for (int k = threadIdx.x; k < s_gap_len[q]; k += PLAN_SMALL_BLOCK) zero_rows[s_gap_out[q] + k] = s_gap_row[q] + k;

    // Carry slots: a row that crosses units has one in every unit it touches, consecutive ones.  `chain` = first slot
    // of the row that is open when a unit begins.
    const int n_units = (n_pieces + SPMM_WARPS - 1) / SPMM_WARPS;
    int slot_base = 0, chain_base = -1;
    for (int u0 = 0; u0 < n_units; u0 += PLAN_SMALL_BLOCK) {
        const int u = u0 + threadIdx.x;
        bool en = false, lv = false;
        int row_in = 0;
        if (u < n_units) {
            const int p0 = u * SPMM_WARPS, p1 = min(p0 + SPMM_WARPS, n_pieces);
            const int4 head = __ldcg(pieces + p0), tail = __ldcg(pieces + p1 - 1);
            row_in = head.y;
            if (p0 > 0 && tuple_is_big(head)) {
                const int4 x = __ldcg(pieces + p0 - 1);
                en = tuple_is_big(x) && x.y == head.y;
            }
            if (p1 < n_pieces && tuple_is_big(tail)) {
                const int4 x = __ldcg(pieces + p1);
                lv = tuple_is_big(x) && x.y == tail.y;
            }
        }
        const bool same = en && lv && u < n_units && __ldcg(pieces + min((u + 1) * SPMM_WARPS, n_pieces) - 1).y == row_in;
        const bool opens = lv && !same;
        int slots, chain_last;
        const int slot = slot_base + block_scan_exclusive<PLAN_SMALL_BLOCK>((en ? 1 : 0) + (opens ? 1 : 0), OpAdd(), 0, slots, s_scan);
        const int out_slot = slot + (en ? 1 : 0);
        int chain = block_scan_exclusive<PLAN_SMALL_BLOCK>(opens ? out_slot : -1, OpMax(), -1, chain_last, s_scan);
        chain = max(chain, chain_base);
        if (u < n_units) {
            unit_carry[u] = make_int2(en ? slot : -1, lv ? (same ? slot : out_slot) : -1);
            if (en && !same)             // the row ends here: its slots are chain .. slot
                for (int q = chain; q <= slot; q++) { carry_span[q] = make_int2(chain, slot - chain + 1); carry_row[q] = row_in; }
        }
        slot_base += slots;
        chain_base = max(chain_base, chain_last);
    }
}

}  // namespace agcn
