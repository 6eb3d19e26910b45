// Both dense transforms of a two-layer GCN in one kernel,  Z[M x 128] = relu(P[M x 128] * W1) * W2  for P = A * X: where
// A is applied to X before W1 (A * (X * W1) = (A * X) * W1) the layers' transforms follow one another, and what lies between
// them never leaves the SM.  TF32 multiply with fp32 accumulation; the parts are those of gemm_tf32_128_kernel:
//
//   warp 0 (one lane)  TMA producer: a tile's 128 rows of P as four boxes of 128 rows x 32 floats;
//   warp 1 (one lane)  MMA issuer: P * W1 of a tile into one of two accumulators, then, one tile behind, H * W2 into one of
//                      two others; H, the first operand of that product, is read from tensor memory;
//   warps 2-5          H = relu(P * W1), written back in the place of the accumulator;
//   warps 6-9          epilogue: rows of Z from the second accumulator.
//
// The four accumulators are all of the tensor memory (512 columns).  Both W take 128 KiB of shared memory and leave four
// stages of 16 KiB for P, one tile; the 64 KiB in flight per SM are twice what HBM needs.  Bound by HBM: 1 KiB per row, where
// two launches of gemm_tf32_128_kernel move 2: a forward over 5 M rows of 20 takes 11.09 ms instead of 11.95.
//
// The tensor core cuts the low 13 bits of a TF32 operand off, which shrinks each product by 3.6e-4 on average.  H passes
// through registers and is rounded to nearest there: relative error of a forward over 100 000 to 1 M rows against 64 bits 1.13e-3 to 1.17e-3, where the separate calls give 1.45e-3
// to 1.50e-3.
// (With both W rounded as well it is 4.7e-4, but then 1.2e-3 from what the separate calls give.)
//
// Every wait is bounded as in gemm_tf32_128_kernel.
#pragma once
#include "gemm_tf32_kernels.cuh"
#include "ptx.cuh"

namespace agcn {

constexpr int PAIR_STAGES = GEMM_KBLKS;                               // one tile
constexpr int PAIR_THREADS = 32 * (2 + 2 * GEMM_EPI_WARPS);
constexpr int PAIR_TMEM_COLS = 4 * GEMM_DIM;                          // two accumulators of either product
constexpr int PAIR_SMEM_BYTES = 1024 /* alignment slack */ + 2 * GEMM_W_BYTES + PAIR_STAGES * GEMM_STAGE_BYTES + GEMM_EPI_WARPS * GEMM_PATCH_BYTES +
                                256 /* barriers */;

// D[tmem] (+)= A[tmem] * B[smem], one elected thread: row i of A in lane i, K along the columns
__device__ __forceinline__ void mma_tf32_from_tmem(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// 32 registers per thread -> 32 lanes x 32 consecutive columns of tensor memory
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const float (&v)[32])
{
    uint32_t r[32];
#pragma unroll
    for (int i = 0; i < 32; i++) r[i] = __float_as_uint(v[i]);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
                 :: "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                    "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                    "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                    "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The nearest TF32 number to a v >= 0, ties upwards; above the largest one v itself, which the tensor core cuts (a finite number
// does not become infinite)
__device__ __forceinline__ float to_tf32(float v)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return v < 0x1.ffep127f ? __uint_as_float(r) : v;
}

__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_tf32_pair_kernel(const __grid_constant__ CUtensorMap map_p, const float *__restrict__ w1, const float *__restrict__ w2, float *__restrict__ z,
                      int64_t m_rows, int n_tiles, int *__restrict__ err_flag, uint32_t spin_limit, int skip_first_load, unsigned long long *stamp)
{
    // err_flag, spin_limit, skip_first_load, stamp: as in gemm_tf32_128_kernel
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *s_w1 = smem, *s_w2 = smem + GEMM_W_BYTES;             // 64 KiB each, K-major, swizzled
    uint8_t *s_ring = smem + 2 * GEMM_W_BYTES;                     // PAIR_STAGES x 16 KiB
    float *s_patch = reinterpret_cast<float *>(s_ring + PAIR_STAGES * GEMM_STAGE_BYTES);
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(s_patch) + GEMM_EPI_WARPS * GEMM_PATCH_BYTES);
    uint64_t *bar_full = s_bar;                                    // [PAIR_STAGES] TMA -> MMA
    uint64_t *bar_empty = s_bar + PAIR_STAGES;                     // [PAIR_STAGES] MMA -> TMA
    uint64_t *bar_sum_full = s_bar + 2 * PAIR_STAGES;              // [2] P * W1 is there
    uint64_t *bar_h_full = bar_sum_full + 2;                       // [2] H is there, in its place
    uint64_t *bar_h_empty = bar_sum_full + 4;                      // [2] ... and has been multiplied
    uint64_t *bar_acc_full = bar_sum_full + 6;                     // [2] H * W2 is there
    uint64_t *bar_acc_empty = bar_sum_full + 8;                    // [2] ... and has been read
    uint64_t *bar_end = bar_sum_full + 10;                         // all products of the thread block are done
    uint32_t *s_tmem_base = reinterpret_cast<uint32_t *>(bar_sum_full + 11);
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem_base + 1);
    volatile int *s_never = s_abort + 1;       // stays 0: for waits that must not be cut short by the abort flag

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // ---- prologue ----------------------------------------------------------------------------
    if (threadIdx.x == 0) {
        for (int i = 0; i < PAIR_STAGES; i++) { mbar_init(smem_u32(&bar_full[i]), 1); mbar_init(smem_u32(&bar_empty[i]), 1); }
        for (int i = 0; i < 2; i++) {
            mbar_init(smem_u32(&bar_sum_full[i]), 1); mbar_init(smem_u32(&bar_h_full[i]), GEMM_EPI_WARPS); mbar_init(smem_u32(&bar_h_empty[i]), 1);
            mbar_init(smem_u32(&bar_acc_full[i]), 1); mbar_init(smem_u32(&bar_acc_empty[i]), GEMM_EPI_WARPS);
        }
        mbar_init(smem_u32(bar_end), 1);
        *s_abort = 0;
        *s_never = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(s_tmem_base), PAIR_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem_base;
    if (warp != 0) {
        // while the producer's first loads are under way
        gemm_load_w<PAIR_THREADS - 32>(w1, s_w1, threadIdx.x - 32);
        gemm_load_w<PAIR_THREADS - 32>(w2, s_w2, threadIdx.x - 32);
        fence_proxy_async();             // generic-proxy writes of W must be visible to the tensor core's reads
        asm volatile("bar.sync 1, %0;" :: "n"(PAIR_THREADS - 32) : "memory");
    }

    const int my_tiles = n_tiles > (int)blockIdx.x ? (n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const auto give_up = [&](int code) {
        if (!*s_abort) { atomicExch(err_flag, code); *s_abort = 1; }
    };

    if (warp == 0) {
        // ---- TMA producer ---------------------------------------------------------------------
        if (lane == 0) {
            uint32_t g = 0;      // K-blocks issued so far
            wait_for_predecessor();          // P is what the launch before this one makes
            if (stamp != nullptr && blockIdx.x == 0) stamp[0] = global_time_ns();
            for (int it = 0; it < my_tiles && !*s_abort; it++) {
                const int tile = (int)blockIdx.x + it * (int)gridDim.x;
                for (int kb = 0; kb < GEMM_KBLKS; kb++, g++) {
                    const uint32_t s = g % PAIR_STAGES, ph = (g / PAIR_STAGES) & 1;
                    if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1, s_abort, spin_limit)) { give_up(GEMM_ERR_TIMEOUT_PRODUCER); break; }
                    if (skip_first_load && g == 0) continue;      // self-test: this stage never fills
                    mbar_arrive_expect_tx(smem_u32(&bar_full[s]), GEMM_STAGE_BYTES);
                    tma_load_2d(smem_u32(s_ring + s * GEMM_STAGE_BYTES), &map_p, kb * GEMM_KBLK, tile * GEMM_TILE_M, smem_u32(&bar_full[s]));
                }
            }
            if (*s_abort) {
                // copies already issued still land in shared memory: give each stage a bounded chance to finish
                for (uint32_t back = 0; back < PAIR_STAGES && back < g; back++) {
                    const uint32_t gg = g - 1 - back;
                    mbar_wait(smem_u32(&bar_full[gg % PAIR_STAGES]), (gg / PAIR_STAGES) & 1, s_never, spin_limit);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the first product of tile `it`, then the second one of the tile before it ----------------
        if (lane == 0) {
            uint32_t g = 0;
            for (int it = 0; it <= my_tiles && !*s_abort; it++) {
                bool ok = true;
                if (it < my_tiles) {
                    const uint32_t b = it & 1, ph_tile = (it >> 1) & 1, d_tmem = tmem_base + b * GEMM_DIM;
                    ok = mbar_wait(smem_u32(&bar_h_empty[b]), ph_tile ^ 1, s_abort, spin_limit);
                    tc_fence_after();
                    for (int kb = 0; kb < GEMM_KBLKS && ok; kb++, g++) {
                        const uint32_t s = g % PAIR_STAGES, ph = (g / PAIR_STAGES) & 1;
                        if (!(ok = mbar_wait(smem_u32(&bar_full[s]), ph, s_abort, spin_limit))) break;
                        tc_fence_after();
                        const uint32_t a_addr = smem_u32(s_ring + s * GEMM_STAGE_BYTES), b_addr = smem_u32(s_w1 + kb * GEMM_STAGE_BYTES);
#pragma unroll
                        for (int k8 = 0; k8 < GEMM_KBLK / 8; k8++)
                            mma_tf32(d_tmem, make_kmajor_sw128_desc(a_addr + k8 * 32), make_kmajor_sw128_desc(b_addr + k8 * 32), GEMM_IDESC,
                                     (uint32_t)((kb | k8) != 0));
                        mma_commit(smem_u32(&bar_empty[s]));
                    }
                    if (ok) mma_commit(smem_u32(&bar_sum_full[b]));
                }
                if (ok && it > 0) {
                    const uint32_t b = (it - 1) & 1, ph_tile = ((it - 1) >> 1) & 1;
                    const uint32_t a_tmem = tmem_base + b * GEMM_DIM, d_tmem = tmem_base + (2 + b) * GEMM_DIM;
                    ok = mbar_wait(smem_u32(&bar_h_full[b]), ph_tile, s_abort, spin_limit) &&
                         mbar_wait(smem_u32(&bar_acc_empty[b]), ph_tile ^ 1, s_abort, spin_limit);
                    if (ok) {
                        tc_fence_after();
#pragma unroll
                        for (int k = 0; k < GEMM_DIM / 8; k++)
                            mma_tf32_from_tmem(d_tmem, a_tmem + k * 8,
                                               make_kmajor_sw128_desc(smem_u32(s_w2 + (k / 4) * GEMM_STAGE_BYTES) + (k % 4) * 32), GEMM_IDESC,
                                               (uint32_t)(k != 0));
                        mma_commit(smem_u32(&bar_h_empty[b]));
                        mma_commit(smem_u32(&bar_acc_full[b]));
                    }
                }
                if (!ok) { give_up(GEMM_ERR_TIMEOUT_MMA); break; }
            }
            // shared and tensor memory are given up only behind the products that read them
            mma_commit(smem_u32(bar_end));
            mbar_wait(smem_u32(bar_end), 0, s_never, spin_limit);
        }
    } else if (warp < 2 + GEMM_EPI_WARPS) {
        // ---- the activation ---------------------------------------------------------------------
        const uint32_t quarter = (uint32_t)((warp & 3) * 32) << 16;                 // TMEM lane quarter this warp may use
        for (int it = 0; it < my_tiles; it++) {
            const uint32_t b = it & 1;
            if (!mbar_wait_warp(smem_u32(&bar_sum_full[b]), (it >> 1) & 1, s_abort, spin_limit)) { give_up(GEMM_ERR_TIMEOUT_EPILOGUE); break; }
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < GEMM_DIM / 32; c++) {
                float v[32];
                const uint32_t at = tmem_base + quarter + b * GEMM_DIM + c * 32;
                tmem_ld_32x32(at, v);
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = to_tf32(fmaxf(v[j], 0.f));
                tmem_st_32x32(at, v);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_h_full[b]));
        }
    } else {
        // ---- epilogue: as in gemm_tf32_128_kernel -----------------------------------------------
        const int q = warp & 3;
        float *patch = s_patch + (warp - 2 - GEMM_EPI_WARPS) * (GEMM_PATCH_BYTES / 4);
        for (int it = 0; it < my_tiles; it++) {
            const int tile = (int)blockIdx.x + it * (int)gridDim.x;
            const uint32_t b = it & 1;
            if (!mbar_wait_warp(smem_u32(&bar_acc_full[b]), (it >> 1) & 1, s_abort, spin_limit)) { give_up(GEMM_ERR_TIMEOUT_EPILOGUE); break; }
            tc_fence_after();
            const int64_t row0 = (int64_t)tile * GEMM_TILE_M + q * 32;
#pragma unroll 1
            for (int c = 0; c < GEMM_DIM / 32; c++) {
                float v[32];
                tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + (2 + b) * GEMM_DIM + c * 32, v);
                gemm_store_patch(v, patch, lane, z, (int64_t)GEMM_DIM, row0, m_rows, c);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_acc_empty[b]));
        }
    }

    // ---- teardown: everyone is done (or gave up); free the tensor memory ------------------------
    tc_fence_before();
    __syncthreads();
    if (stamp != nullptr && threadIdx.x == 0) atomicMax(stamp + 1, global_time_ns());
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, PAIR_TMEM_COLS);
    }
}

}  // namespace agcn
