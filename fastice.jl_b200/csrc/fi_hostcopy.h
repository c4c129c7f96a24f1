// fi_hostcopy.h -- device -> pageable host copies of whole fields (fi_hostcopy.cu).
#pragma once

#include <cuda_runtime.h>

#include <mutex>

namespace fi {

// Pinned staging of one object, made on its first large copy to pageable memory.
struct HostStage {
    static constexpr int kLanes = 8;
    static constexpr size_t kBytes = 2 << 20;  // a lane's buffer
    char *buf = nullptr;
    cudaEvent_t done[kLanes] = {};
    bool failed = false;  // no room for it: plain copies
    std::mutex busy;      // one copy at a time
};
void host_stage_release(HostStage *s);

// The device -> host 3D copy p (from one pitched box to contiguous host rows) on the stream,
// complete on return.
cudaError_t host_download(const cudaMemcpy3DParms &p, int device, cudaStream_t stream, HostStage *s);

}  // namespace fi
