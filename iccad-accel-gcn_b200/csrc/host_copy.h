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

// Host arrays may be reused when these return; the device side is ordered on `s`.  Downloads are complete.
// `outputs`: arrays a later host_download fills, whose pages may be faulted in meanwhile.
int host_upload(const HostSegment *seg, int n, cudaStream_t s, const HostSegment *outputs = nullptr, int n_outputs = 0);
int host_download(const HostSegment *seg, int n, cudaStream_t s);
// gives the pinned buffers back
void host_copy_release();

}  // namespace agcn
