// Copies between the device and host arrays of any kind (host_copy.cu).
#pragma once
#include "host_common.h"

namespace agcn {

struct HostSegment {
    void *device;
    void *host;
    size_t bytes;
};
constexpr int HOST_SEGMENTS_MAX = 4;

// Pageable arrays may be reused when host_upload returns, pinned ones when `s` has been waited for (WaitOnExit); the
// device side is ordered on `s`.  Downloads are complete.
// `outputs`: arrays a later host_download fills, whose pages may be faulted in meanwhile.
int host_upload(const HostSegment *seg, int n, cudaStream_t s, const HostSegment *outputs = nullptr, int n_outputs = 0);
int host_download(const HostSegment *seg, int n, cudaStream_t s);
// Waits for `s` when a call that uploads ends, however it ends: the caller's arrays are the caller's again.
class WaitOnExit {
public:
    explicit WaitOnExit(cudaStream_t s) : s_(s) {}
    ~WaitOnExit() { cudaStreamSynchronize(s_); }
    WaitOnExit(const WaitOnExit &) = delete;
    WaitOnExit &operator=(const WaitOnExit &) = delete;
private:
    cudaStream_t s_;
};

// gives the pinned buffers back
void host_copy_release();

}  // namespace agcn
