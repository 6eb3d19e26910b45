// Declarations shared between the translation units of the library (not part of the C ABI).
#pragma once
#include "host_common.h"

struct agcn_spmm_plan {
    const int4 *block4 = nullptr;     // borrowed
    const int4 *tuples = nullptr;     // what the kernels walk: block4, or the plan's own pieces of it (small plans)
    bool split = false;
    int64_t n_blocks = 0, n_tuples = 0, n_units = 0, n_rows = 0, n_cols = 0, nnz = 0;
    int device = -1;
    void *memory = nullptr;           // one pool block that holds the arrays below
    int2 *unit_carry = nullptr;       // [n_units]
    int2 *carry_span = nullptr;       // [n_carry]
    int *carry_row = nullptr;         // [n_carry]
    void *carry = nullptr;            // spmm_carry_bytes(n_carry): partial sums and arrival counters
    int *zero_rows = nullptr;         // [n_zero]
    int64_t n_carry = 0, n_zero = 0;
    int64_t likely_units = 0;         // about how many units there are, where n_units is only a bound
    int64_t longest = 0;              // degree of the last tuple (cut plans)
    int64_t n_full = 0;               // tuples of at least 192 nonzeros (uncut plans)
    int launches_last_run = 0;
    int l2_bytes = 0, sm_count = 0;   // of the device the plan was created on
    int panel_override = 0;           // AGCN_SPMM_PANEL at creation (0 = choose automatically)
    bool never_split = false;         // set for the ranges of a column-tiled product
    bool hot_tail = false;            // the last rows of X are named so often that L2 is better kept for them (uncut plans)
    int pad_unaligned = 1;            // AGCN_SPMM_PAD at creation: copy unaligned X into 16-byte-aligned rows
    float *x_pad = nullptr;           // [n_cols][dim rounded up to 4], grown on demand
    size_t x_pad_bytes = 0;
    bool x_pad_malloc = false;        // from cudaMalloc, not from the pool
};

namespace agcn {

int env_int(const char *name, int dflt);

// partition.cu
int partition_device(const int *d_indptr, int64_t n_rows, int *d_block4, int64_t cap_blocks, int64_t *n_blocks, cudaStream_t s);
// The same in two halves: begin counts (and waits for the stream), finish fills n_blocks tuples asynchronously, from the
// row pointers, and gives the scratch back (d_block4 == nullptr: only that).
struct PartitionRun {
    const int *indptr = nullptr;
    int64_t n_rows = 0, n_blocks = 0;
    void *memory = nullptr;
    cudaStream_t stream = nullptr;
};
int partition_begin(PartitionRun *run, const int *d_indptr, int64_t n_rows, cudaStream_t s);
int partition_finish(PartitionRun *run, int *d_block4);

// spmm.cu
int spmm_create(agcn_spmm_plan **out, const int *d_block4, int64_t n_blocks, const int *d_indices,
                int64_t n_rows, int64_t n_cols, int64_t nnz, cudaStream_t s);
int spmm_run(agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *d_x, int64_t ldx,
             float *d_y, int64_t ldy, int dim, cudaStream_t s, int activation = 0, int accumulate = 0);
// First row of X that a pass of `width` columns keeps in L2 before the others; 0: all rows alike
int64_t spmm_hot_column(const agcn_spmm_plan *p, int width);
int spmm_check_run_args(const agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *d_x, int64_t ldx,
                        const float *d_y, int64_t ldy, int dim, int activation);
int spmm_prepare_x(agcn_spmm_plan *p, const float *d_x, int64_t ldx, int dim, cudaStream_t s,
                   const float **x_use, int64_t *ldx_use, bool *x_vec);
// Partial sums of the rows that cross unit boundaries: 128 floats per carry slot, and per slot one arrival
// counter for every column pass a product of up to 128 columns can be cut into (products issued in unit
// ranges have several passes under way).  The counters must be zero before a product and are zero after it.
constexpr int SPMM_CARRY_PASSES = 32;
inline size_t spmm_carry_bytes(int64_t n_carry) { return (size_t)n_carry * (128 * sizeof(float) + SPMM_CARRY_PASSES * sizeof(int)); }
inline int *spmm_carry_counters(void *carry, int64_t n_carry) { return reinterpret_cast<int *>(static_cast<float *>(carry) + n_carry * 128); }

// Which part of a product one call of spmm_run_prepared launches.  A product may be issued as
// several unit ranges (a unit = 8 consecutive tuples = one thread block); the zero-fill of uncovered
// rows goes with one of them.  A heavy row that crosses into the next range is stored by that range.
struct SpmmLaunchPart {
    int64_t unit0 = 0, unit1 = -1;      // units [unit0, unit1); -1 = to the end
    bool zero_fill = true;
    // Start while the launch before this one on the stream still runs: ONLY_X: that one makes X and nothing else that
    // is read here, and was itself launched behind all it follows; ANY: it may be any operation.
    enum Early { NO, ONLY_X, ANY } early = NO;
    const int *made = nullptr;          // with abort_flag: of a plan whose kernel was launched before, its numbers (SpmmParams::made)
    const int *abort_flag = nullptr;    // optional device word: nonzero makes the kernels return at once
    void *carry = nullptr;              // optional carry scratch to use instead of the plan's (products in flight together)
};
int spmm_run_prepared(agcn_spmm_plan *p, const int *d_indices, const float *d_vals, const float *x_use, int64_t ldx_use,
                      bool x_vec, float *d_y, int64_t ldy, int dim, cudaStream_t s, int activation, int accumulate,
                      const SpmmLaunchPart &part);
// Aligned copy of X: rows of dim floats padded with zeros to a multiple of four
int spmm_pad_rows(const float *d_x, int64_t ldx, int dim, float *d_xp, int64_t n_rows, cudaStream_t s);
// Whether spmm_create would cut the tuples of a graph of that size on the current device
bool spmm_plan_splits(int64_t n_blocks, int64_t n_rows, int64_t nnz);
int spmm_check_cols(const int *d_idx, int64_t count, int64_t n_cols, int *d_flag, cudaStream_t s);
void plan_free(agcn_spmm_plan *p);


// gemm.cu: Z = H * W (128 x 128, TF32) enqueued on `s`; nothing allocated, nothing synchronised.  keep_status: *d_status
// is not zeroed first; early: the launch before it on the stream makes H; d_stamp: when it began and ended, in ns, the
// end zero before the first launch (all optional)
int gemm_tf32_async(const float *d_h, int64_t ldh, const float *d_w, float *d_z, int64_t ldz, int64_t m_rows,
                    int *d_status, cudaStream_t s, bool keep_status = false, bool early = false, unsigned long long *d_stamp = nullptr);
// Z = relu(P * W1) * W2, all of 128 columns, started while the launch before it, which makes P, still runs; *d_status is not
// zeroed, and d_stamp is as above
int gemm_pair_async(const float *d_p, const float *d_w1, const float *d_w2, float *d_z, int64_t m_rows, int *d_status, cudaStream_t s,
                    unsigned long long *d_stamp);
// Z2[r] = relu(A[r, :] * Z1) * W for the first m_rows rows of a CSR block, all of at most
// fused_layer_max_degree() nonzeros (gemm.cu)
int fused_layer_async(const int *d_indptr, const int *d_indices, const float *d_vals, const float *d_z_in, const float *d_w,
                      float *d_z_out, int64_t m_rows, int64_t n_cols, int *d_status, cudaStream_t s);
int fused_layer_max_degree();

// layout.cu
int balanced_blocks(const int *h_indptr, int64_t n_rows, int world, int64_t *h_ranges, int64_t *rows_per_block);

}  // namespace agcn
