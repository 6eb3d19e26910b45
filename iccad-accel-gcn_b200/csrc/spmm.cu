// C-ABI entry points of the SpMM plug-in (replaces SPMM_ACCEL,
// spmm_accel.cu:104-139) and of the host-buffer call.
#include "host_common.h"
#include "internal.h"
#include "kernels/spmm_kernels.cuh"
#include "spmm_rules.h"

#include <atomic>
#include <cstdlib>
#include <new>

namespace agcn {

int env_int(const char *name, int dflt)
{
    const char *v = getenv(name);
    return v != nullptr && *v ? atoi(v) : dflt;
}

static cudaError_t pad_free(agcn_spmm_plan *p)
{
    float *x_pad = p->x_pad;
    p->x_pad = nullptr; p->x_pad_bytes = 0;
    return p->x_pad_malloc ? cudaFree(x_pad) : pool_free_waiting(x_pad, p->device);
}

void plan_free(agcn_spmm_plan *p)
{
    if (p == nullptr) return;
    pool_free_waiting(p->memory, p->device);
    pad_free(p);
    delete p;
}

// The same memory, of a plan that has only been used on `s`: in that stream's order, without a wait for the device.
static void plan_give_back(agcn_spmm_plan *p, cudaStream_t s)
{
    pool_free(p->memory, s);
    if (p->x_pad_malloc) cudaFree(p->x_pad); else pool_free(p->x_pad, s);
}

// Up to this many thread blocks a cut plan's products keep 16 gathers in flight per lane.
static int spmm_deep_units(int sm_count) { return 8 * sm_count / 3; }

// Nonzeros per piece when the tuples of a plan are to be cut into pieces, 0 when they are not.  A product ends with
// its longest warp, so pieces are as small as the nonzeros that an SM has to go through allow; beyond 7 500 of them
// (20 full tuples; the SM holds 32 to 40 warps) the extra warps cost more than they balance, unless there are few
// tuples for them.  us per product (before launches overlapped), uncut / 192 / 128 / 64, B200, nonzeros per SM in brackets:
// 16 384 rows of 8 [900], dim 60: 17.7 / 9.4 / 8.3 / 7.3;  80 000 rows of 4 [2 100], dim 64: - / 12.4 / 11.2 / 10.3;
// 80 000 of 7 [3 900]: - / 15.1 / 13.5 / 15.2, dim 128: - / 25 / 23 / 25;  135 000 of 4 [3 400]: 50 / 34 / 31 / -;
// 165 000 of 6 [6 300], dim 32: 17.4 / 13.4 / 14.2 / -, dim 128: 54 / 45 / 47 / -;  200 000 of 6 [7 700], dim 64:
// 29.2 / 30.0 / 31.4 / -;  100 000 of 25 [17 000], dim 32: 25 / 33 / - / -.
// Two ranges (pieces of 64 leave SMs idle; they are just too many for two blocks per SM) have a second size, which the
// kernel that cuts takes where its thread blocks fit: the form with 16 gathers
// in flight has two per SM, and a second wave of equal blocks is as long as the first.  Blocks of graphs with hub rows are
// not equal, the heavy ones go first, and up to 8/3 per SM are faster in that form.  Rows of an even graph that do not
// fit a piece would have to meet across blocks, all of them, which costs more than short warps give.  us, one size / 64,
// nonzeros per SM in brackets, dim 60 unless stated:
// 32, taken: 8 192 rows of 8 [440]: 3.4 / 4.9;  power law, 2 048 of 14 [200], dim 60, 128: 5.6 / 6.3, 5.7 / 6.8;  4 500 of 4
// [130], dim 16: 5.4 / 4.9;  not taken: rows of 20 [140], dim 32: 5.3 / 3.7;  of 100 [340], dim 16: 4.9 / 3.3;
// 96, taken: 8 192 of 20 [1 110], 256 blocks: 6.3 / 9.6;  power law, 20 000 of 8 [1 140], 348: 8.1 / 9.2, 9 500 of 20 [1 360],
// 338, dim 128 (the largest loss): 13.6 / 11.1;  skewed, 20 000 of 10 [1 300], 392: 9.1 / 10.9;  not taken: 1 000 of 200 [1 350],
// 375: 12.2 / 6.6;  16 384 of 14 [1 550], 342: 10.4 / 6.3;  30 000 of 6 [1 220], 313, dim 32: 7.4 / 4.4;  4 096 of 40 [1 110], 256:
// 6.2 / 4.9.
// Beyond 80 tuples per SM one thread block takes so long to cut them that a plan used once loses (150 000 rows of 5:
// 236 -> 244 us from the graph to Y).
static PieceChoice spmm_piece(int64_t n_blocks, int64_t nnz, int sm_count)
{
    const int64_t per_sm = nnz / sm_count;
    const auto always = [](int most) { return PieceChoice{most, most, 0, 0}; };
    const auto where_it_fits = [&](int most) {
        const PieceChoice c = {most, 64, SPMM_WARPS * SPMM_DEEP_MIN_BLOCKS * sm_count, SPMM_WARPS * spmm_deep_units(sm_count)};
        return n_blocks > c.fit_uneven || nnz > (int64_t)most * c.fit_uneven ? always(64) : c;       // more pieces than fit for certain
    };
    if (n_blocks > (int64_t)80 * sm_count) return always(0);
    if (per_sm <= 500) return where_it_fits(32);
    if (per_sm > 1050 && per_sm <= 1575) return where_it_fits(96);
    if (per_sm <= 1900) return always(64);
    if (per_sm <= 2700) return always(96);
    if (per_sm <= 4000) return always(128);
    return always(per_sm <= 7500 || n_blocks + nnz / SPMM_DEG_BOUND <= (int64_t)80 * sm_count ? 192 : 0);
}

// A cut plan keeps room for a list of all rows: not where there are a great many without any nonzero.
static PieceChoice spmm_piece_choice(int64_t n_blocks, int64_t n_rows, int64_t nnz, int sm_count)
{
    if (n_blocks == 0 || n_rows > ((int64_t)1 << 20)) return PieceChoice{0, 0, 0, 0};
    const int forced = env_int("AGCN_SPMM_PIECE", INT32_MIN);
    return forced != INT32_MIN ? PieceChoice{forced, forced, 0, 0} : spmm_piece(n_blocks, nnz, sm_count);
}

// The thread blocks of (half) full tuples take about equally long and are started first.  Where there are a few more
// than 4 blocks per SM hold at once, the second round is a tail in which most of the GPU waits, and 5 blocks per SM
// avoid it: dim 128, skewed rows, full blocks per SM and us at 4 / 5 blocks: 3.7: 52 / 57, 4.0: 78 / 63, 4.3: 79 / 63,
// 4.5: 91 / 70, 4.9: 87 / 84, 5.1: 96 / 106, 6.1: 105 / 127.
// Narrower passes gain as much or lose nothing, full blocks per SM and time at 5 / 4 blocks: 4.6 skewed, dim 16, 48, 64:
// -10, -19, -19 %; 4.7 power law: -4, 0, 0 %; 4.8 skewed: -7, -9, -11 %; 4.9 skewed: -3, -3, -5 % (dim 96, 128: +2, +1 %);
// 5.3 dense: +3, -2, -1 %; 5.7 skewed: +21, +18, +20 %; 5.8 dense: +12, +9, +10 %.
// Also where all tuples are full and little more than half of a slot's 32 lanes have a column (139 000 rows of 456, dims
// 68 and 80: 2 % faster, dim 96 already 3 % slower).
static bool spmm_wide_form(const agcn_spmm_plan *p, int width)
{
    if (p->nnz >= 250 * p->n_blocks && width > 64 && width <= 80) return true;
    return p->n_full > (int64_t)SPMM_MIN_BLOCKS * SPMM_WARPS * p->sm_count && 10 * p->n_full <= (int64_t)49 * SPMM_WARPS * p->sm_count;
}

// Columns whose rows of X are to stay in L2 when X is many times larger: the last ones, 45 % of L2 (each half of the
// GPU keeps its own copy of what it reads), where they are named often enough: in a symmetric graph with columns in
// degree order they are.  0 = all alike.  Dim 128, time with / without:
// degree order, X / L2 = 9, 19: window named by 50, 42 % of the nonzeros: -3, -3 %; dim 64..96, X / L2 = 4.6, 5.8,
// 6.2, 6.9: +0.7, +0.5, +0.2, +0.2 %, hence the 6x;
// popular rows anywhere: window named by 3, 13, 23, 32, 42, 52 %: +18, +9, +3, -0.2, -2, -3 %, hence the share of a
// third; uniform columns: 5, 14, 24, 33, 43 %: +4, -3, -8, -12, -13 %;
// row blocks of 2, 4, 8 ranks, whose last rows are the middle of the degree order: 14, 6, 5 %: +7, +12, +11 %.
// (Passes of up to 32 columns were not measured and have no such kernel.)
constexpr double SPMM_HOT_X = 6.0, SPMM_HOT_L2 = 0.45, SPMM_HOT_SHARE = 0.33;

static UncutPlan spmm_uncut(const agcn_spmm_plan *p, int width)
{
    return UncutPlan{p->n_units, p->n_blocks, p->nnz, spmm_wide_form(p, width), p->sm_count};
}
static bool spmm_many_units(const agcn_spmm_plan *p) { return !p->split && spmm_many_units(p->n_units, p->sm_count); }
static bool spmm_octets(const agcn_spmm_plan *p, int width, int columns)
{
    return !p->split && p->panel_override == 0 && spmm_octets(spmm_uncut(p, width), width, columns);
}

static int64_t hot_rows(const agcn_spmm_plan *p, int width) { return (int64_t)(SPMM_HOT_L2 * p->l2_bytes / (width * 4.0)); }

int64_t spmm_hot_column(const agcn_spmm_plan *p, int width)
{
    if (!p->hot_tail || width <= 32 || (double)p->n_cols * width * 4.0 < SPMM_HOT_X * p->l2_bytes) return 0;
    return p->n_cols - hot_rows(p, width);
}

bool spmm_plan_splits(int64_t n_blocks, int64_t n_rows, int64_t nnz)
{
    int device = 0, sm_count = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return true;
    return spmm_piece_choice(n_blocks, n_rows, nnz, sm_count).most > 0;
}

// Order of the units, which are in ascending degree.  Starting at the heavy end leaves light units for the end of
// the launch (500 000 rows of 12, dim 64: 159 -> 144 us).  Where nearly all tuples are full there is nothing to
// balance, and units from both ends in turn are faster by 4-10 % (250 000 rows of 490, dim 32: 934 -> 872 us;
// 20 000 rows of 400: 82 -> 72 us).  In between, with X in L2 and many waves, every fourth unit from the light end
// is (500 000 skewed rows of 29, dim 32: 152 -> 146 us); with X beyond L2 it is not (5 M rows, dim 128: 5.59 -> 5.68 ms).
static int spmm_light_every(const agcn_spmm_plan *p, int width)
{
    if (p->split) return 0;
    if (p->nnz >= 250 * p->n_blocks) return 2;
    const double x_bytes = (double)p->n_cols * width * 4.0;
    return p->n_units > (int64_t)28 * p->sm_count && x_bytes <= 0.6 * p->l2_bytes ? 4 : 0;
}

// most_pieces: as for plan_faults
static int plan_errors(const HostWordsLease &words, int64_t most_pieces)
{
    const int err = plan_faults(words, most_pieces);
    if (err == 0) return AGCN_OK;
    AGCN_REQUIRE((err & SPMM_ERR_PIECES) == 0, "agcn_spmm_create: more pieces than the tuples can have");
    set_error("agcn_spmm_create: invalid input:%s%s%s%s",
              (err & SPMM_ERR_TUPLE) ? " malformed .block4 tuple;" : "",
              (err & SPMM_ERR_ROW) ? " tuple rows out of range or not ascending;" : "",
              (err & SPMM_ERR_LOC) ? " tuple nonzero range outside [0, nnz) or out of order;" : "",
              (err & SPMM_ERR_COL) ? " column index outside [0, n_cols);" : "");
    return AGCN_ERR_RANGE;
}

// The plan's arrays, in one pool block: n_pieces tuples of its own (0: it walks the caller's), bookkeeping of its
// units, n_carry slots, n_zero rows, n_numbers words for the plan kernel to leave numbers in.
static int plan_memory(agcn_spmm_plan *p, int64_t n_pieces, int64_t n_numbers, int4 **pieces, int **numbers, cudaStream_t s)
{
    for (int pass = 0; pass < 2; pass++) {
        Carver m(p->memory);
        *pieces = m.take<int4>(n_pieces);
        p->unit_carry = m.take<int2>(p->n_units);
        p->carry_span = m.take<int2>(p->n_carry);
        p->carry_row = m.take<int>(p->n_carry);
        p->carry = m.take<unsigned char>((int64_t)spmm_carry_bytes(p->n_carry));
        p->zero_rows = m.take<int>(p->n_zero);
        *numbers = m.take<int>(n_numbers);
        if (pass == 1 || m.bytes() == 0) break;
        const cudaError_t e = pool_alloc(&p->memory, m.bytes(), s);
        if (e != cudaSuccess) {
            set_error("agcn_spmm_create: allocation of %zu bytes of plan scratch: %s", m.bytes(), cudaGetErrorString(e));
            return AGCN_ERR_CUDA;
        }
    }
    return AGCN_OK;
}

// One launch: the memory is sized by what the pieces can be at most (a piece that is not the last of its tuple or row
// holds more than half of the nonzeros that a piece may have).  made, bad: as for the kernel.
static int plan_launch_small(agcn_spmm_plan *p, const PieceChoice &choice, const int *d_indices, int64_t n_idx, int *bad, const int **made,
                             HostWordsLease &words, cudaStream_t s)
{
    const int64_t cap = p->n_blocks + 2 * p->nnz / (choice.most < choice.otherwise ? choice.most : choice.otherwise) + 8;
    AGCN_REQUIRE(cap < (int64_t)INT32_MAX / 4, "agcn_spmm_create: too many pieces");
    p->split = true;
    p->n_tuples = cap;
    p->n_units = ceil_div(cap, SPMM_WARPS);
    p->n_carry = 2 * p->n_units;
    p->n_zero = p->n_rows;
    int4 *pieces = nullptr;
    int *numbers = nullptr;
    const int rc = plan_memory(p, cap, made != nullptr ? PLAN_MADE_WORDS : 0, &pieces, &numbers, s);
    if (rc != AGCN_OK) return rc;
    if (made != nullptr) *made = numbers;
    p->tuples = pieces;
    const int64_t col_blocks = ceil_div(n_idx, PLAN_SMALL_BLOCK * 16), counters = p->n_carry * SPMM_CARRY_PASSES;
    const int64_t clear_blocks = ceil_div(counters, PLAN_SMALL_BLOCK * 16);
    AGCN_KERNEL(plan_small_kernel, (unsigned)(1 + clear_blocks + (col_blocks < 2368 ? col_blocks : 2368)), PLAN_SMALL_BLOCK, s, p->block4,
                (int)p->n_blocks, p->n_rows, p->nnz, d_indices, n_idx, p->n_cols, choice, pieces, (int)cap, p->unit_carry, p->carry_span, p->carry_row,
                p->zero_rows, made != nullptr ? numbers : nullptr, bad, spmm_carry_counters(p->carry, p->n_carry), counters, (unsigned)clear_blocks,
                words.device());
    AGCN_LAUNCH_CHECK("plan_small_kernel");
    return AGCN_OK;
}

// The same, and one wait.
static int plan_fill_small(agcn_spmm_plan *p, const PieceChoice &choice, const int *d_indices, int64_t n_idx, cudaStream_t s)
{
    AGCN_HOST_WORDS(words, s);
    int rc = plan_launch_small(p, choice, d_indices, n_idx, nullptr, nullptr, words, s);
    if (rc != AGCN_OK) return rc;
    AGCN_CUDA(words.sync());
    rc = plan_errors(words, p->n_tuples);
    if (rc != AGCN_OK) return rc;
    p->n_tuples = words[PLAN_WORD_PIECES];
    p->n_units = ceil_div(p->n_tuples, SPMM_WARPS);
    p->n_zero = words[PLAN_WORD_ZERO];
    p->longest = words[PLAN_WORD_LONGEST];
    return AGCN_OK;
}

// Two launches: the first pass counts and validates, the host sizes the plan's one pool block from its
// answer, the second pass fills it.  (Six cudaMalloc / cudaFree pairs and nine launches before.)
static int plan_fill(agcn_spmm_plan *p, const int *d_indices, int64_t n_idx, cudaStream_t s)
{
    p->tuples = p->block4;
    p->n_tuples = p->n_blocks;
    p->n_units = ceil_div(p->n_blocks, SPMM_WARPS);
    const int64_t tiles = p->n_units > 0 ? ceil_div(p->n_units, PLAN_BLOCK) : 1;
    DeviceScratch scratch(s);
    Carver size;
    size.take<unsigned long long>(4); size.take<int64_t>(tiles); size.take<int>(tiles);
    AGCN_ALLOC(block, scratch, unsigned char, (int64_t)size.bytes());
    Carver c(block);
    unsigned long long *ctl = c.take<unsigned long long>(4);
    int64_t *tile_zero = c.take<int64_t>(tiles);
    int *tile_carry = c.take<int>(tiles);
    AGCN_HOST_WORDS(words, s);
    AGCN_CUDA(cudaMemsetAsync(ctl, 0, 4 * sizeof(*ctl), s));
    // 16 column ids per thread, at most 64 thread blocks per SM's worth of them
    const int64_t col_grid = n_idx > 0 ? ceil_div(n_idx, PLAN_BLOCK * 16) : 0;
    // the widest pass has the narrowest window: where that one is named often enough, so are the others
    const bool ask_tail = n_idx > 0 && (double)p->n_cols * SPMM_PANEL * 4.0 >= SPMM_HOT_X * p->l2_bytes;
    const unsigned grid = (unsigned)(tiles + (ask_tail ? 1 : 0) + (col_grid < 9472 ? col_grid : 9472));
    AGCN_KERNEL(plan_check_kernel, grid, PLAN_BLOCK, s, p->block4, p->n_blocks, p->n_units, p->n_rows, p->nnz, d_indices, n_idx, p->n_cols,
                (unsigned)tiles, ask_tail ? p->n_cols - hot_rows(p, SPMM_PANEL) : (int64_t)-1, tile_zero, tile_carry, ctl, words.device());
    AGCN_LAUNCH_CHECK("plan_check_kernel");
    AGCN_CUDA(words.sync());
    int rc = plan_errors(words, INT64_MAX);
    if (rc != AGCN_OK) return rc;
    p->n_zero = words[PLAN_WORD_ZERO];
    p->n_carry = words[PLAN_WORD_CARRY];
    p->n_full = words[PLAN_WORD_FULL];
    p->hot_tail = ask_tail && (double)words[PLAN_WORD_TAIL] >= SPMM_HOT_SHARE * PLAN_SAMPLES;
    int4 *pieces = nullptr;
    int *numbers = nullptr;
    rc = plan_memory(p, 0, 0, &pieces, &numbers, s);
    if (rc != AGCN_OK) return rc;
    if (p->n_carry > 0)
        AGCN_CUDA(cudaMemsetAsync(spmm_carry_counters(p->carry, p->n_carry), 0, (size_t)p->n_carry * SPMM_CARRY_PASSES * sizeof(int), s));
    if (p->n_carry > 0 || p->n_zero > 0) {
        AGCN_KERNEL(plan_assign_kernel, (unsigned)tiles, PLAN_BLOCK, s, p->tuples, p->n_tuples, p->n_units, p->n_rows, (const int64_t *)tile_zero,
                    (const int *)tile_carry, p->unit_carry, p->carry_span, p->carry_row, p->n_zero > 0 ? p->zero_rows : nullptr);
        AGCN_LAUNCH_CHECK("plan_assign_kernel");
    } else if (p->n_units > 0) {
        AGCN_CUDA(cudaMemsetAsync(p->unit_carry, 0xff, (size_t)p->n_units * sizeof(int2), s));      // no row crosses units
    }
    AGCN_CUDA(cudaStreamSynchronize(s));          // products may run on any stream
    return AGCN_OK;
}

static int spmm_check_graph(const int *d_block4, int64_t n_blocks, int64_t n_rows, int64_t n_cols, int64_t nnz)
{
    AGCN_REQUIRE(n_blocks >= 0 && (n_blocks == 0 || d_block4 != nullptr), "agcn_spmm_create: null block4");
    AGCN_REQUIRE(aligned16(d_block4), "agcn_spmm_create: block4 must be 16-byte aligned");
    AGCN_REQUIRE(n_rows > 0 && n_rows < (int64_t)INT32_MAX && n_cols > 0 && n_cols < (int64_t)INT32_MAX,
                 "agcn_spmm_create: n_rows / n_cols out of range");
    AGCN_REQUIRE(nnz >= 0 && nnz <= (int64_t)INT32_MAX, "agcn_spmm_create: nnz out of range");
    AGCN_REQUIRE(n_blocks < (int64_t)INT32_MAX, "agcn_spmm_create: too many blocks");
    return AGCN_OK;
}

// What a plan knows before it looks at the tuples.
static int spmm_begin(agcn_spmm_plan *p, const int *d_block4, int64_t n_blocks, int64_t n_rows, int64_t n_cols, int64_t nnz)
{
    AGCN_CUDA(cudaGetDevice(&p->device));
    AGCN_CUDA(cudaDeviceGetAttribute(&p->sm_count, cudaDevAttrMultiProcessorCount, p->device));
    AGCN_CUDA(cudaDeviceGetAttribute(&p->l2_bytes, cudaDevAttrL2CacheSize, p->device));
    p->block4 = reinterpret_cast<const int4 *>(d_block4);
    p->n_blocks = n_blocks; p->n_rows = n_rows; p->n_cols = n_cols; p->nnz = nnz;
    p->panel_override = env_int("AGCN_SPMM_PANEL", 0);
    p->pad_unaligned = env_int("AGCN_SPMM_PAD", 1);
    return AGCN_OK;
}

int spmm_create(agcn_spmm_plan **out, const int *d_block4, int64_t n_blocks, const int *d_indices,
                       int64_t n_rows, int64_t n_cols, int64_t nnz, cudaStream_t s)
{
    AGCN_REQUIRE(out != nullptr, "agcn_spmm_create: null plan pointer");
    *out = nullptr;
    int rc = spmm_check_graph(d_block4, n_blocks, n_rows, n_cols, nnz);
    if (rc != AGCN_OK) return rc;

    agcn_spmm_plan *p = new (std::nothrow) agcn_spmm_plan;
    AGCN_REQUIRE(p != nullptr, "agcn_spmm_create: out of host memory");
    struct Guard { agcn_spmm_plan *p; ~Guard() { plan_free(p); } } guard{p};       // frees the half-built plan on every early return
    rc = spmm_begin(p, d_block4, n_blocks, n_rows, n_cols, nnz);
    if (rc != AGCN_OK) return rc;
    const int64_t n_idx = d_indices != nullptr ? nnz : 0;
    const PieceChoice choice = spmm_piece_choice(n_blocks, n_rows, nnz, p->sm_count);
    rc = choice.most > 0 ? plan_fill_small(p, choice, d_indices, n_idx, s) : plan_fill(p, d_indices, n_idx, s);
    if (rc != AGCN_OK) return rc;
    guard.p = nullptr;
    *out = p;
    return AGCN_OK;
}

// Column ids idx[0 .. count) against [0, n_cols): ORs SPMM_ERR_COL into *d_flag when one is outside.
int spmm_check_cols(const int *d_idx, int64_t count, int64_t n_cols, int *d_flag, cudaStream_t s)
{
    if (count <= 0) return AGCN_OK;
    const int64_t blocks = ceil_div(count, 256 * 16);
    AGCN_KERNEL(plan_check_cols_kernel, (unsigned)(blocks < 65535 ? blocks : 65535), 256, s, d_idx, count, n_cols, d_flag);
    AGCN_LAUNCH_CHECK("plan_check_cols_kernel");
    return AGCN_OK;
}

template <int S, int BATCH, int MIN_BLOCKS, bool FINISH, bool HOT = false, int Q = 1>
static void launch_units(const SpmmParams &prm, unsigned grid, bool plain, cudaStream_t s)
{
    auto k = plain ? spmm_units_kernel<S, Q, BATCH, MIN_BLOCKS, true, FINISH, HOT, false> : spmm_units_kernel<S, Q, BATCH, MIN_BLOCKS, false, FINISH, HOT, false>;
    launch_early(prm.early != 0, k, grid, SPMM_THREADS, 0, s, prm);
}

// Which of the kernel's forms a launch uses.
struct SpmmForm {
    bool plain;      // Y overwritten with 16-byte stores
    bool finish;     // rows that cross units are finished in the launch
    bool deep;       // few thread blocks, many gathers per lane
    bool wide;       // more thread blocks per SM, fewer gathers per lane
    bool loose;      // rows of X of any alignment, 4 bytes at a time (spmm_loose)
    int few;         // thread blocks per SM of a launch of few, more than the deep ones: 3, 4 (17 to 32 columns) or 0: as ever
    bool octets;     // 32-byte loads (spmm_octets), of a plan of many units or not
    bool many;
};

// S = lanes of 8 columns
template <int S>
static void launch_octets(const SpmmParams &prm, unsigned grid, const SpmmForm &f, cudaStream_t s)
{
    if (f.many) {
        if (f.finish) launch_units<S, SPMM_OCTET_BATCH, SPMM_MIN_BLOCKS, true, false, 2>(prm, grid, f.plain, s);
        else if (prm.hot_column > 0) launch_units<S, SPMM_OCTET_BATCH, SPMM_MIN_BLOCKS, false, true, 2>(prm, grid, f.plain, s);
        else launch_units<S, SPMM_OCTET_BATCH, SPMM_MIN_BLOCKS, false, false, 2>(prm, grid, f.plain, s);
    } else if constexpr (S == 16) {                      // (spmm_octets: none of up to 64 columns)
        if (f.wide) launch_units<S, SPMM_OCTET_FEW, SPMM_WIDE_MIN_BLOCKS, true, false, 2>(prm, grid, f.plain, s);
        else launch_units<S, SPMM_OCTET_FEW, SPMM_MIN_BLOCKS, true, false, 2>(prm, grid, f.plain, s);
    }
}

template <int S>
static void launch_units_for(const SpmmParams &prm, unsigned grid, const SpmmForm &f, cudaStream_t s)
{
    if constexpr (S > 0) {
        if (f.loose) {
            auto k = f.deep ? spmm_units_kernel<S, 1, SPMM_DEEP_GATHER_BATCH, SPMM_DEEP_MIN_BLOCKS, false, true, false, true>
                            : spmm_units_kernel<S, 1, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, false, true, false, true>;
            launch_early(prm.early != 0, k, grid, SPMM_THREADS, 0, s, prm);
            return;
        }
    }
    if (f.deep) { launch_units<S, SPMM_DEEP_GATHER_BATCH, SPMM_DEEP_MIN_BLOCKS, true>(prm, grid, f.plain, s); return; }
    // 17..32 columns, and the 4-byte mode, always take the 5-block form, but for launches of few blocks
    constexpr bool ALWAYS_WIDE = S == 8 || S == 0;
    if (f.finish) {
        if constexpr (S > 0) {
            if (f.few == 3) { launch_units<S, SPMM_THREE_GATHER_BATCH, SPMM_THREE_MIN_BLOCKS, true>(prm, grid, f.plain, s); return; }
        }
        if constexpr (S == 8) {
            if (f.few == 4) { launch_units<S, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, true>(prm, grid, f.plain, s); return; }
        }
        if (ALWAYS_WIDE || f.wide) launch_units<S, SPMM_WIDE_GATHER_BATCH, SPMM_WIDE_MIN_BLOCKS, true>(prm, grid, f.plain, s);
        else if constexpr (!ALWAYS_WIDE) launch_units<S, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, true>(prm, grid, f.plain, s);
        return;
    }
    if constexpr (ALWAYS_WIDE) {
        launch_units<S, SPMM_WIDE_GATHER_BATCH, SPMM_WIDE_MIN_BLOCKS, false>(prm, grid, f.plain, s);
    } else {
        // launches of many blocks: the 5-block form above 64 columns only (constexpr: no other one is built)
        if constexpr (S == 32) {
            if (f.wide) { launch_units<S, SPMM_WIDE_GATHER_BATCH, SPMM_WIDE_MIN_BLOCKS, false>(prm, grid, f.plain, s); return; }
        }
        if constexpr (S >= 16) {
            if (prm.hot_column > 0) { launch_units<S, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, false, true>(prm, grid, f.plain, s); return; }
        }
        launch_units<S, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, false>(prm, grid, f.plain, s);
    }
}

// Behind the plan's kernel (ONCE): the general flavour, deep or not, whatever the widths and blocks.
template <int S>
static void launch_once(const SpmmParams &prm, unsigned grid, const SpmmForm &f, cudaStream_t s)
{
    auto go = [&](auto k) { launch_early(prm.early != 0, k, grid, SPMM_THREADS, 0, s, prm); };
    if constexpr (S == 0) go(spmm_units_kernel<0, 1, SPMM_WIDE_GATHER_BATCH, SPMM_WIDE_MIN_BLOCKS, false, true, false, false, true>);
    else if (f.loose) {
        if (f.deep) go(spmm_units_kernel<S, 1, SPMM_DEEP_GATHER_BATCH, SPMM_DEEP_MIN_BLOCKS, false, true, false, true, true>);
        else go(spmm_units_kernel<S, 1, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, false, true, false, true, true>);
    } else if (f.deep) go(spmm_units_kernel<S, 1, SPMM_DEEP_GATHER_BATCH, SPMM_DEEP_MIN_BLOCKS, false, true, false, false, true>);
    else go(spmm_units_kernel<S, 1, SPMM_GATHER_BATCH, SPMM_MIN_BLOCKS, false, true, false, false, true>);
}

static void launch_units_for_width(int width, bool vec, const SpmmParams &prm, unsigned grid, const SpmmForm &f, cudaStream_t s)
{
    if (prm.made != nullptr) {
        if (!vec) launch_once<0>(prm, grid, f, s);
        else if (width <= 16) launch_once<4>(prm, grid, f, s);
        else if (width <= 32) launch_once<8>(prm, grid, f, s);
        else if (width <= 64) launch_once<16>(prm, grid, f, s);
        else launch_once<32>(prm, grid, f, s);
    } else if (f.octets) width <= 64 ? launch_octets<8>(prm, grid, f, s) : launch_octets<16>(prm, grid, f, s);
    else if (!vec) launch_units_for<0>(prm, grid, f, s);
    else if (width <= 16) launch_units_for<4>(prm, grid, f, s);
    else if (width <= 32) launch_units_for<8>(prm, grid, f, s);
    else if (width <= 64) launch_units_for<16>(prm, grid, f, s);
    else launch_units_for<32>(prm, grid, f, s);
}

int spmm_pad_rows(const float *d_x, int64_t ldx, int dim, float *d_xp, int64_t n_rows, cudaStream_t s)
{
    const int ldp = (dim + 3) & ~3;
    const int64_t blocks = ceil_div(n_rows * (ldp >> 2), PAD_BLOCK * PAD_ITEMS);
    AGCN_REQUIRE(blocks < (int64_t)INT32_MAX, "agcn_spmm_run: operand too large to pad");
    // Early: it is resident when the operation before it ends.  135 small graphs, dims 17 to 127, not early / early: in a
    // stream 1.02 on average, up to 1.4 (4 096 rows of 40, dim 17: 8.3 / 5.8 us), 500 000 of 12, dim 17: 84.1 / 81.0;  in a
    // replayed graph, where launches are closer, 0.97, at worst 16.9 / 18.8 (100 000 of 10, dim 17).
    AGCN_CUDA(launch_early(true, spmm_pad_rows_kernel, (unsigned)blocks, PAD_BLOCK, 0, s, d_x, ldx, dim, d_xp, ldp, n_rows));
    AGCN_LAUNCH_CHECK("spmm_pad_rows_kernel");
    return AGCN_OK;
}

static bool x_rows_aligned(const float *d_x, int64_t ldx, int dim) { return dim % 4 == 0 && ldx % 4 == 0 && aligned16(d_x); }

static int spmm_few_form(const agcn_spmm_plan *p, int width)
{
    return p->split ? spmm_few_form(CutPlan{p->n_units, p->n_rows, p->nnz, p->longest, p->sm_count}, width) : 0;
}

static bool spmm_deep(const agcn_spmm_plan *p)
{
    return p->split && (p->likely_units > 0 ? p->likely_units : p->n_units) <= spmm_deep_units(p->sm_count);
}

// Small products gather 4 bytes at a time from X as it is instead, with the additions of the 16-byte path in its order:
// to a chain of latencies the copy adds a kernel, and where a row of X is named a few times the copy of it is a good part
// of the work.  us with the copy / without, nonzeros per SM and per row of X in brackets, dims 17, 61, 127:
// 2 048 rows of 4 [70, 5]: 7.9 / 6.7 (17);  500 dense rows of 100 [340, 100]: 7.7 / 7.1, 7.9 / 7.1, 9.2 / 7.3;
// 16 384 of 8 [1 000, 9]: 10.1 / 7.8, 14.1 / 11.0, 19.2 / 15.4;  30 000 of 12 [2 600, 13]: 13.2 / 10.6, 16.0 / 14.6, 24.1 / 22.6;
// 80 000 of 4 [2 700, 5]: - , 20.4 / 14.3, 37.0 / 26.8;  but
// 1 000 dense of 150 [1 000, 150]: 9.5 / 9.5, 11.4 / 11.9, 14.2 / 15.6;  30 000 skewed of 16 [3 200, 16]: 14.9 / 12.2, 16.6 / 17.6,
// 26.7 / 26.7;  100 000 skewed of 10 [6 800, 10]: 17.8 / 20.7, 29.7 / 32.4, 62.0 / 64.8.
// The widths turn the balance both ways (rows named 13 to 16 times gain at 17 columns and lose at 61), so the limits leave
// gains: they are where no width of the graphs above loses.  Over 68 graphs inside them, dims 17, 61, 127: 0.82 of the time
// with the copy; slower: 30 000 rows of exactly 12 and 16 384 of exactly 10, dim 17 (12 and 7 %), 500 of 100, dim 127 (3 to 7 %).
// (Its sums take 4 S places of a carry slot where the columns may be fewer: forced passes might not leave them.)
// Large products of an X whose rows are named a few times and that is a good part of L2 or more do, too: there the copy is two
// passes of HBM over X, and the gather reads rows of the copy as often from HBM as it would those of X.  Time without the copy /
// with, nonzeros per row of X and X of 61 columns / L2 in brackets, dims 30, 39, 54, 61, 78, 99, 127:
// power law, 1.5 M of 4 [3.9, 2.8]: .86 .80 .78 .80 .78 .76 .76;  500 000 of 5 [4.9, 0.9]: .84 .80 .81 .81 .82 .79 .78;  2.4 M of 7 [6.8, 4.4]: .98 .90 .91 .96
// .88 .87 .92;  900 000 of 8 [7.8, 1.7]: .99 .91 .91 .94 .91 .90 .93;  350 000 of 8 [7.7, 0.65]: .95 .88 .88 .89 .91 .88 .87;  skewed, 500 000 of
// 8 [7.8, 0.9]: 1.16 .94 .93 .98 .91 .88 .91;  300 000 of 6 [5.9, 0.55]: - - .92 .96 .88 .88 .87;  not taken: power law, 160 000 of 6 [5.7, 0.30]: 1.03
// - .94 .89 1.02 .90 .87;  2 M of 10 [9.8, 3.7]: 1.04 - .97 1.03 .96 .95 .98;  500 000 of 12 [11.6, 0.9]: 1.06 - .98 1.00 .99 .98 1.00;  500 000 of 18
// [17.3, 0.9]: 1.18 - 1.06 1.10 1.07 1.07 1.09.
constexpr double SPMM_LOOSE_L2 = 0.4;

static bool spmm_loose(const agcn_spmm_plan *p, int dim)
{
    if (!p->pad_unaligned || p->panel_override != 0) return false;
    if (!p->split) {
        // rows of whole eights keep the order of additions that the same columns have where they are aligned
        if (dim > SPMM_PANEL || p->nnz > (dim > 32 ? 8 : 6) * p->n_cols || (double)p->n_cols * dim * 4.0 < SPMM_LOOSE_L2 * p->l2_bytes) return false;
        return dim % 8 != 0 || !spmm_octets(p, dim, dim);
    }
    return (spmm_deep(p) && p->nnz <= (int64_t)500 * p->sm_count) || (p->nnz <= 13 * p->n_cols && p->nnz <= (int64_t)2700 * p->sm_count);
}

// Rows of X that are not 16-byte aligned (dim % 4 != 0 with the reference's ld = dim, an odd
// stride or base) would force 4-byte gathers: 1.2-1.6x the time of the 16-byte path.  Instead X
// is copied once into plan-owned rows padded to a multiple of 4 floats (2 * n_cols * dim * 4
// bytes of streaming traffic against nnz * dim * 4 bytes of gather) and the 16-byte path runs
// on the copy; Y keeps the caller's layout and gets stores as wide as each row's alignment allows.
// On return *x_use / *ldx_use name the operand to gather from and *x_vec says whether its rows
// are 16-byte aligned.
int spmm_prepare_x(agcn_spmm_plan *p, const float *d_x, int64_t ldx, int dim, cudaStream_t s,
                   const float **x_use, int64_t *ldx_use, bool *x_vec)
{
    const bool x_aligned = x_rows_aligned(d_x, ldx, dim);
    *x_use = d_x;
    *ldx_use = ldx;
    *x_vec = x_aligned;
    if (x_aligned || !p->pad_unaligned || p->nnz == 0) return AGCN_OK;
    const int ldp = (dim + 3) & ~3;
    const size_t need = (size_t)p->n_cols * ldp * sizeof(float);
    if (need > p->x_pad_bytes) {
        // growing the scratch synchronises the device once per plan and width; steady state allocates nothing
        // (Under stream capture a pool block would be the graph's own and gone outside of it; cudaMalloc is refused
        // there, or in relaxed capture gives memory that outlives the graph.)
        AGCN_CUDA(pad_free(p));
        cudaError_t e = pool_alloc(reinterpret_cast<void **>(&p->x_pad), need, s);
        p->x_pad_malloc = e == cudaErrorStreamCaptureUnsupported;
        if (p->x_pad_malloc) e = cudaMalloc(reinterpret_cast<void **>(&p->x_pad), need);
        if (e != cudaSuccess) {
            cudaGetLastError();
            p->x_pad = nullptr;
            set_error("agcn_spmm_run: %zu bytes for the aligned copy of X: %s", need, cudaGetErrorString(e));
            return AGCN_ERR_CUDA;
        }
        p->x_pad_bytes = need;
    }
    const int rc = spmm_pad_rows(d_x, ldx, dim, p->x_pad, p->n_cols, s);
    if (rc != AGCN_OK) return rc;
    p->launches_last_run++;
    *x_use = p->x_pad;
    *ldx_use = ldp;
    *x_vec = true;
    return AGCN_OK;
}

int spmm_check_run_args(const agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *d_x, int64_t ldx,
                        const float *d_y, int64_t ldy, int dim, int activation)
{
    AGCN_REQUIRE(activation == 0 || activation == 1, "agcn_spmm_run_act: activation must be AGCN_ACT_NONE or AGCN_ACT_RELU");
    AGCN_REQUIRE(p != nullptr, "agcn_spmm_run: null plan");
    AGCN_REQUIRE(d_x != nullptr && d_y != nullptr, "agcn_spmm_run: null X or Y");
    AGCN_REQUIRE(p->nnz == 0 || (d_indices != nullptr && d_vals != nullptr), "agcn_spmm_run: null indices or values");
    AGCN_REQUIRE(dim >= 1, "agcn_spmm_run: dim = %d", dim);
    AGCN_REQUIRE(ldx >= dim && ldy >= dim, "agcn_spmm_run: row stride smaller than dim");
    return AGCN_OK;
}

// One product on one set of tuples, X already prepared.  accumulate: Y += A * X (a later column
// range of a column-tiled product; rows no tuple covers then keep their value, and only get the
// activation).
int spmm_run_prepared(agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *x_use, int64_t ldx_use,
                      bool x_vec, float *d_y, int64_t ldy, int dim, cudaStream_t s, int activation, int accumulate,
                      const SpmmLaunchPart &part)
{
    const int64_t unit0 = part.unit0, unit1 = part.unit1 < 0 ? p->n_units : part.unit1;
    AGCN_REQUIRE(unit0 >= 0 && unit0 <= unit1 && unit1 <= p->n_units, "agcn_spmm_run: unit range outside the plan");
    // rows no tuple covers: zero-filled -- or, when accumulating, left alone unless an activation is due
    int64_t zero_blocks = !part.zero_fill || (accumulate && !activation) ? 0 : ceil_div(p->n_zero, SPMM_ZERO_ROWS_PER_BLOCK);
    if (part.made != nullptr && zero_blocks > 2 * p->sm_count) zero_blocks = 2 * p->sm_count;         // n_zero is all rows then; the blocks take turns
    const int64_t grid = (unit1 - unit0) + zero_blocks;
    AGCN_REQUIRE(grid < (int64_t)INT32_MAX, "agcn_spmm_run: grid too large");

    // Column panels.  The gather re-reads a row of X once per nonzero of that column, so it runs
    // at L2 speed only while the X columns of a pass stay L2-resident.  When dim > 64 and the
    // operand is somewhat larger than what L2 keeps, two 64-column passes (each re-streaming the
    // 8 bytes per nonzero of A) beat one 128-column pass that spills to HBM (measured on B200:
    // 3.8 ms against 4.2-4.7 ms at N = 250 000, dim 128; 0.77 against 0.86 ms at N = 500 000).
    // When X is many times larger than L2 neither pass fits and one pass is as fast or faster
    // (6.3 against 6.5 ms at N = 5 000 000), so the split is limited to operands up to 4x L2.
    // Passes stay multiples of 32 columns so that every row segment is whole 128-byte lines.
    // AGCN_SPMM_PANEL (read when the plan is created) overrides the choice.  (A product whose A is
    // column-tiled -- agcn_spmm_tiled_* -- keeps its X slab in L2 by construction and never splits.)
    const bool whole = unit0 == 0 && unit1 == p->n_units;
    const bool loose = !x_vec && whole && spmm_loose(p, dim);
    const int64_t ldx_panel = loose ? (dim + 3) & ~3 : ldx_use;         // the passes, hence the sums, that the aligned copy would get
    int panel = SPMM_PANEL;
    if (dim > 64 && dim % 32 == 0 && ldx_panel % 32 == 0 && !accumulate && !p->never_split) {
        const int full = dim < SPMM_PANEL ? dim : SPMM_PANEL;
        const double x_bytes = (double)p->n_cols * full * 4.0;
        if (x_bytes > 0.75 * (double)p->l2_bytes && x_bytes <= 4.0 * (double)p->l2_bytes) panel = 64;
    }
    if (p->panel_override > 0) panel = p->panel_override;
    const bool carry_inside = !whole || loose || !spmm_many_units(p);        // parts of a product, and that form, always finish their rows
    // A carry slot holds SPMM_PANEL floats and every column pass uses its own columns (and arrival
    // counters) of it, so a product of up to SPMM_PANEL columns can be issued in parts whatever its
    // passes are -- with the same passes, hence the same bits, as a whole run.
    if (!whole) AGCN_REQUIRE(dim <= SPMM_PANEL, "agcn_spmm_run: a product issued in unit ranges is limited to %d columns", SPMM_PANEL);
    AGCN_REQUIRE(panel >= 1 && panel <= SPMM_PANEL, "agcn_spmm_run: AGCN_SPMM_PANEL must be 1..%d", SPMM_PANEL);
    if ((x_vec || loose) && panel % 4 != 0) panel = (panel + 3) & ~3;         // keep every panel's first column 16-byte aligned
    if (panel > SPMM_PANEL) panel = SPMM_PANEL;
    for (int col0 = 0, width = 0; col0 < dim; col0 += width) {
        // a pass ends where the carry slot does: behind the last slot lie the arrival counters
        const int slot_left = SPMM_PANEL - col0 % SPMM_PANEL;
        width = dim - col0 < panel ? dim - col0 : panel;
        if (width > slot_left) width = slot_left;
        SpmmParams prm;
        prm.tuples = p->tuples; prm.n_tuples = p->n_tuples;
        prm.n_units = unit1 - unit0; prm.unit_base = unit0; prm.abort_flag = part.abort_flag; prm.made = part.made;
        // a later pass follows the one before it, which waits for what came before
        prm.early = part.early == SpmmLaunchPart::ANY || (part.early == SpmmLaunchPart::ONLY_X && col0 == 0) ? 1 : 0;
        prm.wait_first = part.early == SpmmLaunchPart::ANY ? 1 : 0;
        prm.light_every = spmm_light_every(p, width);
        prm.hot_column = (int)spmm_hot_column(p, width);
        prm.idx = d_indices; prm.val = d_vals;
        prm.x = x_use + col0; prm.ldx = ldx_use;
        prm.y = d_y + col0; prm.ldy = ldy;
        prm.unit_carry = p->unit_carry;
        void *carry = part.carry != nullptr ? part.carry : p->carry;
        prm.carry = static_cast<float *>(carry) + col0 % SPMM_PANEL;
        prm.carry_span = p->carry_span;
        prm.carry_count = spmm_carry_counters(carry, p->n_carry) + (int64_t)(col0 % SPMM_PANEL / 4) * p->n_carry;
        prm.zero_rows = p->zero_rows; prm.n_zero_rows = p->n_zero;
        prm.relu = activation;
        prm.accumulate = accumulate;
        const bool vec = loose || (x_vec && aligned16(prm.x));
        const bool y_vec = width % 4 == 0 && ldy % 4 == 0 && aligned16(prm.y);
        prm.y_vec = y_vec ? 1 : 0;
        prm.dim_store = width;
        prm.dim = vec ? (width + 3) & ~3 : width;       // columns gathered (the padded copy holds zeros past dim)
        // (not for the copy of an X that a whole product reads as it is: one issued in parts has the same bits)
        const bool octets = vec && !loose && prm.dim % 8 == 0 && ldx_use % 8 == 0 && aligned32(prm.x) && spmm_octets(p, prm.dim, width) &&
                            (dim % 4 == 0 || p->never_split || !spmm_loose(p, dim));
        const bool plain = !accumulate && !loose && (vec ? y_vec : true) && (!octets || (width % 8 == 0 && ldy % 8 == 0 && aligned32(prm.y)));
        if (grid > 0) {
            const SpmmForm form = {plain, carry_inside, spmm_deep(p), spmm_wide_form(p, width), loose, spmm_few_form(p, width), octets, spmm_many_units(p)};
            launch_units_for_width(prm.dim, vec, prm, (unsigned)grid, form, s);
            AGCN_LAUNCH_CHECK("spmm_units_kernel");
            p->launches_last_run++;
        }
        if (p->n_carry > 0 && !carry_inside) {
            auto k = vec ? spmm_carry_kernel<true> : spmm_carry_kernel<false>;
            AGCN_CUDA(launch_early(true, k, (unsigned)ceil_div(p->n_carry, SPMM_WARPS), SPMM_THREADS, 0, s, prm, (const int *)p->carry_row, p->n_carry));
            AGCN_LAUNCH_CHECK("spmm_carry_kernel");
            p->launches_last_run++;
        }
    }
    return AGCN_OK;
}

// made, bad: null, or of a plan whose kernel was launched before on the stream: SpmmLaunchPart::made and abort_flag
static int spmm_run_whole(agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *d_x, int64_t ldx,
                          float *d_y, int64_t ldy, int dim, cudaStream_t s, int activation, int accumulate, const int *made, const int *bad)
{
    p->launches_last_run = 0;
    const float *x_use = d_x;
    int64_t ldx_use = ldx;
    bool x_vec = x_rows_aligned(d_x, ldx, dim);
    const int rc = spmm_loose(p, dim) ? AGCN_OK : spmm_prepare_x(p, d_x, ldx, dim, s, &x_use, &ldx_use, &x_vec);
    if (rc != AGCN_OK) return rc;
    SpmmLaunchPart part;
    // A product is launched while the operation before it still runs and waits for it on the GPU, so that launch, first
    // instructions and tuples are no longer paid one after the other by a row of small products.  us per call, B200, before
    // and after: 2 048 rows of 4, dim 16: 6.1, 4.6; 16 384 rows of 8, dim 60: 10.2, 7.4; from 300 us on no difference.
    part.early = x_use != d_x ? SpmmLaunchPart::ONLY_X : SpmmLaunchPart::ANY;       // behind the copy of X, or the caller's work
    part.made = made;
    part.abort_flag = bad;
    return spmm_run_prepared(p, d_indices, d_vals, x_use, ldx_use, x_vec, d_y, ldy, dim, s, activation, accumulate, part);
}

int spmm_run(agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *d_x, int64_t ldx,
             float *d_y, int64_t ldy, int dim, cudaStream_t s, int activation, int accumulate)
{
    const int rc = spmm_check_run_args(p, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, activation);
    if (rc != AGCN_OK) return rc;
    const DeviceOf on(p->device);
    return spmm_run_whole(p, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, s, activation, accumulate, nullptr, nullptr);
}

// The words that say "something is wrong" to products launched behind the plan of their graph: one for each of the calls
// under way, zero when the library is loaded and when they are handed out.
constexpr int PLAN_BAD_WORDS = 64;
static __device__ int g_plan_bad[PLAN_BAD_WORDS];
static std::atomic<uint64_t> g_plan_bad_free{~(uint64_t)0};

class BadWord {
public:
    BadWord()
    {
        uint64_t free = g_plan_bad_free.load();
        while (free != 0 && !g_plan_bad_free.compare_exchange_weak(free, free & (free - 1))) {}
        number_ = free != 0 ? __builtin_ctzll(free) : -1;
    }
    ~BadWord() { if (number_ >= 0 && zero_) g_plan_bad_free.fetch_or((uint64_t)1 << number_); }     // else it stays out of use
    BadWord(const BadWord &) = delete;
    BadWord &operator=(const BadWord &) = delete;
    bool none() const { return number_ < 0; }
    cudaError_t address(int **out) const
    {
        void *base = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&base, g_plan_bad);
        *out = e == cudaSuccess ? static_cast<int *>(base) + number_ : nullptr;
        return e;
    }
    void launched() { zero_ = false; }
    void zero() { zero_ = true; }
private:
    int number_;
    bool zero_ = true;
};

// Plan, product and the end of the plan in one call, which returns when Y is there (or untouched, and something was wrong); it waits
// for its own stream only.  The product of a small graph is launched behind the plan's kernel, without a wait between them: it finds on the device how many
// thread blocks it has (PLAN_MADE_*), and whether anything is wrong.  (As create, run and destroy: a wait for the plan, one
// for the device, and the launch of the product between.  From the graph, degree sort and partitioner included, to Y, us, B200, before / so:
// 2 048 rows of 4: 114 / 102;  16 384 of 8: 122 / 112;  60 000 of 8: 176 / 160;  140 000 of 6: 181 / 177.)
static int spmm_once(const int *d_block4, int64_t n_blocks, const int *d_indices, const float *d_vals, int64_t n_rows, int64_t n_cols, int64_t nnz,
                     const float *d_x, int64_t ldx, float *d_y, int64_t ldy, int dim, cudaStream_t s)
{
    int rc = spmm_check_graph(d_block4, n_blocks, n_rows, n_cols, nnz);
    if (rc != AGCN_OK) return rc;
    agcn_spmm_plan plan;
    rc = spmm_begin(&plan, d_block4, n_blocks, n_rows, n_cols, nnz);
    if (rc != AGCN_OK) return rc;
    const PieceChoice choice = spmm_piece_choice(n_blocks, n_rows, nnz, plan.sm_count);
    BadWord word;
    if (choice.most <= 0 || word.none()) {
        agcn_spmm_plan *p = nullptr;
        rc = spmm_create(&p, d_block4, n_blocks, d_indices, n_rows, n_cols, nnz, s);
        if (rc != AGCN_OK) return rc;
        rc = spmm_run(p, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, s);
        const cudaError_t waited = cudaStreamSynchronize(s);
        plan_give_back(p, s);
        delete p;
        if (rc == AGCN_OK) AGCN_CUDA(waited);
        return rc;
    }
    int *bad = nullptr;
    AGCN_CUDA(word.address(&bad));
    // what is wrong with the graph is said before what is wrong with the operands
    const int run_rc = spmm_check_run_args(&plan, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, 0);
    struct Memory {
        agcn_spmm_plan *p;
        cudaStream_t s;
        ~Memory() { plan_give_back(p, s); }
    } memory{&plan, s};
    AGCN_HOST_WORDS(words, s);
    const int *made = nullptr;
    rc = plan_launch_small(&plan, choice, d_indices, d_indices != nullptr ? nnz : 0, bad, &made, words, s);
    if (rc != AGCN_OK) return rc;
    word.launched();
    if (run_rc == AGCN_OK) {
        // the bound on the number of pieces says nothing of how many gathers pay: about three quarters of a piece's nonzeros are there
        const int64_t likely = ceil_div(4 * nnz, 3 * (int64_t)choice.most);
        plan.likely_units = ceil_div(choice.otherwise != choice.most && likely > choice.fit ? ceil_div(4 * nnz, 3 * (int64_t)choice.otherwise) : likely, SPMM_WARPS);
        rc = spmm_run_whole(&plan, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, s, 0, 0, made, bad);
    }
    AGCN_CUDA(words.sync());
    const int plan_rc = plan_errors(words, plan.n_tuples);        // whatever sets *bad is an error here, too: the word is handed out again
    if (plan_rc != AGCN_OK) {
        AGCN_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s));
        AGCN_CUDA(cudaStreamSynchronize(s));
    }
    word.zero();
    if (plan_rc != AGCN_OK) return plan_rc;
    if (run_rc != AGCN_OK) return spmm_check_run_args(&plan, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, 0);
    return rc;
}

}  // namespace agcn

extern "C" int agcn_spmm_create(agcn_spmm_plan **plan, const int32_t *d_block4, int64_t n_blocks,
                                const int32_t *d_indices, int64_t n_rows, int64_t n_cols, int64_t nnz, void *stream)
{
    agcn::clear_error();
    return agcn::spmm_create(plan, d_block4, n_blocks, d_indices, n_rows, n_cols, nnz, static_cast<cudaStream_t>(stream));
}

extern "C" int agcn_spmm_run(agcn_spmm_plan *plan, const int32_t *d_indices, const float *d_vals,
                             const float *d_x, int64_t ldx, float *d_y, int64_t ldy, int dim, void *stream)
{
    agcn::clear_error();
    return agcn::spmm_run(plan, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, static_cast<cudaStream_t>(stream));
}

extern "C" int agcn_spmm_run_act(agcn_spmm_plan *plan, const int32_t *d_indices, const float *d_vals,
                                 const float *d_x, int64_t ldx, float *d_y, int64_t ldy, int dim, int activation,
                                 void *stream)
{
    agcn::clear_error();
    return agcn::spmm_run(plan, d_indices, d_vals, d_x, ldx, d_y, ldy, dim, static_cast<cudaStream_t>(stream), activation);
}

extern "C" int agcn_spmm_once(const int32_t *d_block4, int64_t n_blocks, const int32_t *d_indices, const float *d_vals, int64_t n_rows,
                              int64_t n_cols, int64_t nnz, const float *d_x, int64_t ldx, float *d_y, int64_t ldy, int dim, void *stream)
{
    agcn::clear_error();
    return agcn::spmm_once(d_block4, n_blocks, d_indices, d_vals, n_rows, n_cols, nnz, d_x, ldx, d_y, ldy, dim, static_cast<cudaStream_t>(stream));
}

extern "C" int agcn_spmm_destroy(agcn_spmm_plan *plan)
{
    agcn::clear_error();
    agcn::plan_free(plan);
    return AGCN_OK;
}

extern "C" int agcn_spmm_plan_info(const agcn_spmm_plan *plan, int64_t *n_units, int64_t *n_carry,
                                   int64_t *n_zero_rows, int *launches_last_run)
{
    agcn::clear_error();
    AGCN_REQUIRE(plan != nullptr, "agcn_spmm_plan_info: null plan");
    if (n_units) *n_units = plan->n_units;
    if (n_carry) *n_carry = plan->n_carry;
    if (n_zero_rows) *n_zero_rows = plan->n_zero;
    if (launches_last_run) *launches_last_run = plan->launches_last_run;
    return AGCN_OK;
}

extern "C" int agcn_spmm_plan_hot_column(const agcn_spmm_plan *plan, int width, int64_t *column)
{
    agcn::clear_error();
    AGCN_REQUIRE(plan != nullptr && column != nullptr && width >= 1 && width <= agcn::SPMM_PANEL, "agcn_spmm_plan_hot_column: null argument, or width outside 1..128");
    *column = agcn::spmm_hot_column(plan, width);
    return AGCN_OK;
}
