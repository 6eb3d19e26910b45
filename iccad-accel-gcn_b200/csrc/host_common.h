// Host-side helpers shared by the C-ABI translation units: error reporting,
// checked CUDA calls, scratch buffers and the device-wide prefix sum.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <cstdarg>
#include <cstdio>
#include <vector>

#include "../../include/accelgcn.h"

namespace agcn {

void set_error(const char *fmt, ...);
void clear_error();

#define AGCN_CUDA(call)                                                                          \
    do {                                                                                         \
        cudaError_t agcn_e_ = (call);                                                            \
        if (agcn_e_ != cudaSuccess) {                                                            \
            ::agcn::set_error("%s: %s (%s:%d)", #call, cudaGetErrorString(agcn_e_), __FILE__, __LINE__); \
            return AGCN_ERR_CUDA;                                                                \
        }                                                                                        \
    } while (0)

// kernel launch: `kernel` is a function name or a pointer to an instantiated template
#ifndef AGCN_KERNEL
#define AGCN_KERNEL(kernel, grid, block, stream, ...) kernel<<<(grid), (block), 0, (stream)>>>(__VA_ARGS__)
#endif

#define AGCN_LAUNCH_CHECK(name)                                                                  \
    do {                                                                                         \
        cudaError_t agcn_e_ = cudaGetLastError();                                                \
        if (agcn_e_ != cudaSuccess) {                                                            \
            ::agcn::set_error("launch of %s: %s (%s:%d)", name, cudaGetErrorString(agcn_e_), __FILE__, __LINE__); \
            return AGCN_ERR_CUDA;                                                                \
        }                                                                                        \
    } while (0)

#define AGCN_REQUIRE(cond, ...)                                                                  \
    do {                                                                                         \
        if (!(cond)) { ::agcn::set_error(__VA_ARGS__); return AGCN_ERR_INVALID; }                \
    } while (0)

// Kernel launch that, if `early`, may start while the launch before it on the stream still runs (the kernel waits
// for that one itself before it uses what it makes).
template <typename... Params, typename... Args>
inline cudaError_t launch_early(bool early, void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cfg.attrs = &attr; cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// Makes a device current for a scope; nothing is done where it already is.
class DeviceOf {
public:
    explicit DeviceOf(int device)
    {
        if (cudaGetDevice(&before_) != cudaSuccess || before_ == device || device < 0) before_ = -1;
        else cudaSetDevice(device);
    }
    ~DeviceOf() { if (before_ >= 0) cudaSetDevice(before_); }
    DeviceOf(const DeviceOf &) = delete;
    DeviceOf &operator=(const DeviceOf &) = delete;
private:
    int before_ = -1;
};

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool aligned32(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }
inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Stream-ordered memory of the current device's pool (memory.cu).  Refused (cudaErrorStreamCaptureUnsupported) while
// `s` is being captured: the block would belong to the graph.
cudaError_t pool_alloc(void **out, size_t bytes, cudaStream_t s);
void pool_free(void *p, cudaStream_t s);
// for blocks that work on any stream may still use: waits for `device`, whose pool the block is from, as cudaFree does
cudaError_t pool_free_waiting(void *p, int device);

// Pool memory for the length of a call, used and given back on one stream.
class DeviceScratch {
public:
    explicit DeviceScratch(cudaStream_t s) : s_(s) {}
    DeviceScratch(const DeviceScratch &) = delete;
    DeviceScratch &operator=(const DeviceScratch &) = delete;
    ~DeviceScratch() { for (void *p : ptrs_) pool_free(p, s_); }
    // returns nullptr (and records the error) on failure
    template <typename T> T *alloc(int64_t count)
    {
        void *p = nullptr;
        const size_t bytes = (size_t)(count > 0 ? count : 1) * sizeof(T);
        cudaError_t e = pool_alloc(&p, bytes, s_);
        if (e != cudaSuccess) {
            set_error("device allocation of %zu bytes: %s", bytes, cudaGetErrorString(e));
            return nullptr;
        }
        ptrs_.push_back(p);
        return static_cast<T *>(p);
    }
private:
    cudaStream_t s_;
    std::vector<void *> ptrs_;
};

// Lays several arrays out in one allocation, each on a 256-byte boundary: take() every array first with a
// null base to get the size, then again with the block.
class Carver {
public:
    explicit Carver(void *base = nullptr) : base_(static_cast<unsigned char *>(base)) {}
    template <typename T> T *take(int64_t count)
    {
        T *p = base_ != nullptr ? reinterpret_cast<T *>(base_ + used_) : nullptr;
        used_ += ((size_t)(count > 0 ? count : 0) * sizeof(T) + 255) & ~(size_t)255;
        return p;
    }
    size_t bytes() const { return used_; }
private:
    unsigned char *base_;
    size_t used_ = 0;
};

// Words in pinned host memory that kernels store results and error codes into (memory.cu).
struct HostWords {
    enum { COUNT = 8 };
    int64_t w[COUNT];
};

int host_words_chunks();          // how many pinned chunks of them there are

class HostWordsLease {
public:
    explicit HostWordsLease(cudaStream_t s);
    ~HostWordsLease();
    HostWordsLease(const HostWordsLease &) = delete;
    HostWordsLease &operator=(const HostWordsLease &) = delete;
    HostWords *device() { pending_ = true; return words_; }      // to hand to a kernel (null: no pinned memory)
    cudaError_t sync() { pending_ = false; return cudaStreamSynchronize(s_); }
    int64_t operator[](int i) const { return const_cast<const volatile HostWords *>(words_)->w[i]; }
private:
    HostWords *words_ = nullptr;
    cudaStream_t s_;
    bool pending_ = false;
};

#define AGCN_HOST_WORDS(var, stream)                                                      \
    HostWordsLease var(stream);                                                           \
    do {                                                                                  \
        if ((var).device() == nullptr) {                                                  \
            ::agcn::set_error("no pinned host memory for the result words");              \
            return AGCN_ERR_CUDA;                                                         \
        }                                                                                 \
    } while (0)

#define AGCN_ALLOC(var, scratch, type, count)                  \
    type *var = (scratch).alloc<type>(count);                  \
    if (var == nullptr) return AGCN_ERR_CUDA

// Exclusive prefix sum of a whole array (defined in common.cu).
// tile_sums must hold ceil(n / 2048) elements.  total_out may be null.
int exclusive_scan_i32_i64(const int *in, int64_t *out, int64_t n, int64_t *tile_sums, int64_t *total_out, cudaStream_t s);
int64_t scan_tiles(int64_t n);

}  // namespace agcn
