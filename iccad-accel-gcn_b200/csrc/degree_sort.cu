// C-ABI entry points of the degree sort (the ordering the reference assumes
// of its <graph>.new_indptr / .new_indices inputs, main.cu:62-63).
#include "host_common.h"
#include "host_copy.h"
#include "kernels/degree_sort_kernels.cuh"

namespace agcn {

// Two launches up to 65 536 rows, a memset and five to eight above; one synchronisation at the end (15 to 25 launches, eight allocations and
// two synchronisations before: 0.9 ms for 16 384 rows, most of it in the allocator).
static int degree_sort_device(const int *d_indptr, const int *d_indices, const float *d_vals,
                              int64_t n_rows, int64_t nnz, int relabel_cols,
                              int *d_perm, int *d_new_indptr, int *d_new_indices, float *d_new_vals,
                              cudaStream_t s)
{
    AGCN_REQUIRE(d_indptr != nullptr && d_perm != nullptr, "agcn_degree_sort: null indptr or perm");
    AGCN_REQUIRE(n_rows > 0 && n_rows < (int64_t)INT32_MAX, "agcn_degree_sort: n_rows = %lld out of range", (long long)n_rows);
    AGCN_REQUIRE(nnz >= 0 && nnz <= (int64_t)INT32_MAX, "agcn_degree_sort: nnz = %lld out of range", (long long)nnz);
    AGCN_REQUIRE(d_new_indices == nullptr || d_indices != nullptr, "agcn_degree_sort: new_indices wanted but indices is null");
    AGCN_REQUIRE(d_new_vals == nullptr || (d_vals != nullptr && d_new_indices != nullptr),
                 "agcn_degree_sort: new_vals needs vals and new_indices");
    AGCN_REQUIRE(d_new_indices == nullptr || d_new_indptr != nullptr, "agcn_degree_sort: new_indices needs new_indptr");

    const bool permute = d_new_indices != nullptr;
    const int64_t tiles = ceil_div(n_rows, SORT_TILE), final_tiles = ceil_div(n_rows, FINAL_TILE);
    const int64_t permute_tiles = permute && nnz > 0 ? ceil_div(nnz, PERMUTE_TILE) : 0;
    // a degree has no more bits than the number of nonzeros; without the CSR arrays nnz is not checked and says nothing
    int passes = RADIX_PASSES;
    if (permute) {
        passes = 1;
        while (passes < RADIX_PASSES && (nnz >> (passes * RADIX_BITS)) != 0) passes++;
    }
    const bool small = n_rows <= SMALL_MAX_ROWS;
    DeviceScratch scratch(s);
    SortBuffers buf;
    SortControl *ctl = nullptr;
    unsigned long long *final_state = nullptr;
    SortCounts counts = {nullptr, tiles, ceil_div(tiles, COUNT_GROUP), ceil_div(tiles, COUNT_SUPER)};
    PermuteMap map = {nullptr, nullptr, nullptr};
    size_t cleared = 0;
    void *block = nullptr;
    for (int round = 0; round < 2; round++) {
        Carver c(block);
        ctl = c.take<SortControl>(1);
        final_state = c.take<unsigned long long>(small ? 0 : final_tiles);
        counts.rows = c.take<unsigned>(small ? 0 : passes * (counts.tiles + counts.groups + counts.supers) * RADIX_BINS);
        cleared = c.bytes();
        for (int k = 0; k < 2; k++) { buf.keys[k] = c.take<unsigned>(small ? 0 : n_rows); buf.rows[k] = c.take<int>(small ? 0 : n_rows); }
        map.new_id = permute && relabel_cols ? c.take<int>(n_rows) : nullptr;
        map.delta = permute_tiles > 0 ? c.take<int>(n_rows) : nullptr;
        map.tile_row = permute_tiles > 0 ? c.take<int>(permute_tiles) : nullptr;
        if (round == 0 && (block = scratch.alloc<unsigned char>((int64_t)c.bytes())) == nullptr) return AGCN_ERR_CUDA;
    }
    AGCN_HOST_WORDS(words, s);
    if (small) {
        const int items = (int)ceil_div(n_rows, SMALL_CLUSTER * SMALL_BLOCK), smem = small_smem_bytes(items);
        if (smem > 40 << 10) AGCN_CUDA(cudaFuncSetAttribute(sort_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, small_smem_bytes(SMALL_ITEMS)));
        sort_small_kernel<<<SMALL_CLUSTER, SMALL_BLOCK, smem, s>>>(d_indptr, (int)n_rows, items, nnz, permute ? 1 : 0, ctl, d_perm, d_new_indptr, map,
                                                                   words.device());
        AGCN_LAUNCH_CHECK("sort_small_kernel");
    } else {
        AGCN_CUDA(cudaMemsetAsync(ctl, 0, cleared, s));
        AGCN_KERNEL(degree_count_kernel, (unsigned)tiles, SORT_BLOCK, s, d_indptr, n_rows, nnz, permute ? 1 : 0, counts, ctl, words.device());
        AGCN_LAUNCH_CHECK("degree_count_kernel");
        for (int pass = 0; pass < passes; pass++) {
            AGCN_CUDA(launch_early(true, radix_pass_kernel, (unsigned)tiles, RADIX_BLOCK, 0, s, d_indptr, (int)n_rows, pass, passes, buf,
                                   (const SortControl *)ctl, counts));
            AGCN_LAUNCH_CHECK("radix_pass_kernel");
        }
        AGCN_CUDA(launch_early(true, sort_finish_kernel, (unsigned)final_tiles, SORT_BLOCK, 0, s, d_indptr, n_rows, passes, buf, ctl, final_state, d_perm,
                               d_new_indptr, map, words.device()));
        AGCN_LAUNCH_CHECK("sort_finish_kernel");
        if (permute_tiles > 0) {
            AGCN_CUDA(launch_early(true, tile_rows_kernel, (unsigned)ceil_div(permute_tiles, SORT_BLOCK), SORT_BLOCK, 0, s, (const int *)d_new_indptr,
                                   (int)n_rows, (int)permute_tiles, (const SortControl *)ctl, map.tile_row));
            AGCN_LAUNCH_CHECK("tile_rows_kernel");
        }
    }
    if (permute_tiles > 0) {
        AGCN_CUDA(launch_early(true, csr_permute_kernel, (unsigned)(ceil_div(permute_tiles, PERMUTE_WARPS) * (d_new_vals != nullptr ? 2 : 1)), PERMUTE_BLOCK, 0, s, d_indices,
                               d_new_vals != nullptr ? d_vals : (const float *)nullptr, (const int *)d_new_indptr, map, n_rows, nnz, d_new_indices,
                               d_new_vals, (const SortControl *)ctl, words.device()));
        AGCN_LAUNCH_CHECK("csr_permute_kernel");
    }
    AGCN_CUDA(words.sync());
    if (words[SORT_WORD_NEGATIVE] != 0) {
        set_error("agcn_degree_sort: indptr decreases somewhere (negative degree)");
        return AGCN_ERR_RANGE;
    }
    if (permute && words[SORT_WORD_NNZ] != nnz) {
        set_error("agcn_degree_sort: nnz = %lld but indptr[n_rows] - indptr[0] = %lld", (long long)nnz, (long long)words[SORT_WORD_NNZ]);
        return AGCN_ERR_INVALID;
    }
    if (words[SORT_WORD_TIMEOUT] != 0) {
        set_error("agcn_degree_sort: a wait between tiles ran out; the outputs are incomplete");
        return AGCN_ERR_CUDA;
    }
    if (words[SORT_WORD_COLUMN] != 0) {
        set_error("agcn_degree_sort: a column id lies outside [0, n_rows) and cannot be relabelled");
        return AGCN_ERR_RANGE;
    }
    return AGCN_OK;
}

}  // namespace agcn

extern "C" int agcn_degree_sort_device(const int32_t *d_indptr, const int32_t *d_indices, const float *d_vals,
                                       int64_t n_rows, int64_t nnz, int relabel_cols,
                                       int32_t *d_perm, int32_t *d_new_indptr,
                                       int32_t *d_new_indices, float *d_new_vals, void *stream)
{
    agcn::clear_error();
    return agcn::degree_sort_device(d_indptr, d_indices, d_vals, n_rows, nnz, relabel_cols, d_perm, d_new_indptr,
                                    d_new_indices, d_new_vals, static_cast<cudaStream_t>(stream));
}

extern "C" int agcn_degree_sort_host(const int32_t *h_indptr, const int32_t *h_indices, const float *h_vals,
                                     int64_t n_rows, int64_t nnz, int relabel_cols,
                                     int32_t *h_perm, int32_t *h_new_indptr,
                                     int32_t *h_new_indices, float *h_new_vals)
{
    using namespace agcn;
    clear_error();
    AGCN_REQUIRE(h_indptr != nullptr && h_perm != nullptr, "agcn_degree_sort_host: null indptr or perm");
    AGCN_REQUIRE(n_rows > 0 && n_rows < (int64_t)INT32_MAX && nnz >= 0 && nnz <= (int64_t)INT32_MAX, "agcn_degree_sort_host: bad sizes");
    const bool want_idx = h_new_indices != nullptr, want_val = h_new_vals != nullptr;
    AGCN_REQUIRE(!want_idx || (h_indices != nullptr && h_new_indptr != nullptr), "agcn_degree_sort_host: new_indices needs indices and new_indptr");
    AGCN_REQUIRE(!want_val || (h_vals != nullptr && want_idx), "agcn_degree_sort_host: new_vals needs vals and new_indices");
    const cudaStream_t s = nullptr;
    DeviceScratch scratch(s);
    const WaitOnExit drain(s);
    unsigned char *block = nullptr;
    int *d_indptr = nullptr, *d_perm = nullptr, *d_new_indptr = nullptr, *d_indices = nullptr, *d_new_indices = nullptr;
    float *d_vals = nullptr, *d_new_vals = nullptr;
    for (int round = 0; round < 2; round++) {
        Carver c(block);
        d_indptr = c.take<int>(n_rows + 1);
        d_perm = c.take<int>(n_rows);
        d_new_indptr = c.take<int>(n_rows + 1);
        d_indices = want_idx ? c.take<int>(nnz) : nullptr;
        d_new_indices = want_idx ? c.take<int>(nnz) : nullptr;
        d_vals = want_val ? c.take<float>(nnz) : nullptr;
        d_new_vals = want_val ? c.take<float>(nnz) : nullptr;
        if (round == 0 && (block = scratch.alloc<unsigned char>((int64_t)c.bytes())) == nullptr) return AGCN_ERR_CUDA;
    }
    const size_t row_bytes = (size_t)n_rows * sizeof(int), nz_bytes = (size_t)nnz * 4;
    const HostSegment up[] = {{d_indptr, const_cast<int *>(h_indptr), row_bytes + sizeof(int)},
                              {d_indices, const_cast<int *>(h_indices), want_idx ? nz_bytes : 0},
                              {d_vals, const_cast<float *>(h_vals), want_val ? nz_bytes : 0}};
    const HostSegment down[] = {{d_perm, h_perm, row_bytes},
                                {d_new_indptr, h_new_indptr, h_new_indptr != nullptr ? row_bytes + sizeof(int) : 0},
                                {d_new_indices, h_new_indices, want_idx ? nz_bytes : 0},
                                {d_new_vals, h_new_vals, want_val ? nz_bytes : 0}};
    int rc = host_upload(up, 3, s, down, 4);
    if (rc != AGCN_OK) return rc;
    rc = degree_sort_device(d_indptr, d_indices, d_vals, n_rows, nnz, relabel_cols, d_perm, d_new_indptr, d_new_indices, d_new_vals, s);
    if (rc != AGCN_OK) return rc;
    return host_download(down, 4, s);
}
