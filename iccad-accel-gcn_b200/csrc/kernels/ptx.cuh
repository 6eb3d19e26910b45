// Memory-access wrappers of the SpMM kernels (sm_100a inline PTX).
//
// The gather is bound by what L2 can deliver, so what stays in L2 matters:
//  - the dense operand X is re-read once per nonzero of its column and should
//    stay resident: loads carry an L2 evict_last policy;
//  - the sparse operand (column ids, values) and the .block4 tuples are read
//    exactly once per launch: loads bypass L1 allocation and carry an L2
//    evict_first policy, so that streaming 8 bytes per nonzero does not push X
//    rows out of L2;
//  - result rows are written once and not read again by the kernel: stores
//    carry evict_first as well.
#ifndef AGCN_PTX_CUH
#define AGCN_PTX_CUH
#include <stdint.h>

namespace agcn {

struct L2Policies {
    uint64_t keep;     // evict_last
    uint64_t stream;   // evict_first
    int hot;           // first column whose row of X is to be kept
    int cols;          // how many columns this lane has, where rows of X are read 4 bytes at a time
};

// Rows of X from column `hot` on are to stay in L2, the others are to leave first (HOT: X many times larger than L2).
template <bool HOT>
__device__ __forceinline__ uint64_t x_policy(const L2Policies &p, int column) { return !HOT || column >= p.hot ? p.keep : p.stream; }

__device__ __forceinline__ L2Policies make_l2_policies()
{
    L2Policies p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p.keep));
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p.stream));
    p.hot = 0; p.cols = 4;
    return p;
}

// dense operand X: 16 bytes per lane, keep in L2.  Not the read-only path (.nc): the launch before may still be
// making X while the reader is already resident and waits for it.  (A load needs a column id, staged in shared memory
// and read behind that wait, for its address: it cannot move above it.)
__device__ __forceinline__ float4 ld_x4(const float *p, uint64_t policy)
{
    float4 v;
    asm("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "l"(policy));
    return v;
}
// the same, 32 bytes per lane
__device__ __forceinline__ void ld_x8(const float *p, uint64_t policy, float4 &a, float4 &b)
{
    asm("ld.global.L2::cache_hint.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(p), "l"(policy));
}
__device__ __forceinline__ float ld_x1(const float *p, uint64_t policy)
{
    float v;
    asm("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(policy));
    return v;
}

// Four columns of row `column` of X for this lane: the 16 bytes at p, or (LOOSE lanes per row: rows of any alignment)
// p[0], p[LOOSE], p[2 LOOSE], p[3 LOOSE] as far as the row goes.
template <bool HOT, int LOOSE>
__device__ __forceinline__ float4 ld_x(const float *p, const L2Policies &pol, int column)
{
    if (LOOSE == 0) return ld_x4(p, x_policy<HOT>(pol, column));
    float4 v = make_float4(ld_x1(p, pol.keep), 0.f, 0.f, 0.f);
    if (pol.cols > 1) v.y = ld_x1(p + LOOSE, pol.keep);
    if (pol.cols > 2) v.z = ld_x1(p + 2 * LOOSE, pol.keep);
    if (pol.cols > 3) v.w = ld_x1(p + 3 * LOOSE, pol.keep);
    return v;
}

// sparse operand (col ids / values): streamed once per launch.  Not .nc and volatile: where the launch before may be
// anything it may also be what makes them, and no load of them moves above the wait for it.
__device__ __forceinline__ int ld_a(const int *p, uint64_t policy)
{
    int v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(policy));
    return v;
}
__device__ __forceinline__ float ld_a(const float *p, uint64_t policy)
{
    float v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(policy));
    return v;
}

// result rows: written once
__device__ __forceinline__ void st_y4(float *p, const float4 &v, uint64_t policy)
{
    asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;"
                 :: "l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "l"(policy) : "memory");
}
__device__ __forceinline__ void st_y8(float *p, const float4 &a, const float4 &b, uint64_t policy)
{
    asm volatile("st.global.L2::cache_hint.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8}, %9;"
                 :: "l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(policy) : "memory");
}
__device__ __forceinline__ void st_y2(float *p, float a, float b, uint64_t policy)
{
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" :: "l"(p), "f"(a), "f"(b), "l"(policy) : "memory");
}
__device__ __forceinline__ void st_y1(float *p, float v, uint64_t policy)
{
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" :: "l"(p), "f"(v), "l"(policy) : "memory");
}

__device__ __forceinline__ unsigned long long global_time_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Programmatic dependent launch: the launch after this one may start; this one's predecessor has finished and what
// it wrote is visible.  Both do nothing in launches without that attribute.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace agcn
#endif
