// fi_hostcopy.cu -- reading a field back into ordinary (pageable) host memory.
//
// A caller's fresh array has no pages yet: one thread of the driver staging and writing it is
// bound by that core (page faults and copy), 36.5 ms for the 133 MB of a 255^3 FP64 field.
// Here a few lanes take the planes in turn: each copies its next slab into its own pinned
// buffer on the stream and writes it out while the other lanes' slabs arrive (14.6 ms with two
// lanes, 8.5 with four, 6.6 with eight).  Pinned destinations keep the plain copy, and so do
// fields whose first copy would lose more to the buffers' allocation (some 6 ms, once per
// model) than it gains.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <system_error>
#include <thread>

#include "fi_hostcopy.h"

namespace fi {

namespace {

constexpr size_t kStagedMin = 64 << 20;

bool ready(HostStage *s) {
    if (s->failed || s->buf) return !s->failed;
    bool ok = cudaMallocHost(&s->buf, HostStage::kLanes * HostStage::kBytes) == cudaSuccess;
    for (cudaEvent_t &e : s->done) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        host_stage_release(s);
        s->failed = true;
    }
    return ok;
}

bool pageable(const void *host) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t plain(const cudaMemcpy3DParms &p, cudaStream_t stream) {
    cudaError_t e = cudaMemcpy3DAsync(&p, stream);
    return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
}

}  // namespace

void host_stage_release(HostStage *s) {
    if (s->buf) cudaFreeHost(s->buf);
    s->buf = nullptr;
    for (cudaEvent_t &e : s->done) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
}

cudaError_t host_download(const cudaMemcpy3DParms &p, int device, cudaStream_t stream, HostStage *s) {
    const size_t row = p.extent.width, rows = p.extent.height, plane = row * rows, planes = p.extent.depth;
    if (plane * planes < kStagedMin || row > HostStage::kBytes || !pageable(p.dstPtr.ptr)) return plain(p, stream);
    std::lock_guard<std::mutex> lock(s->busy);
    if (!ready(s)) return plain(p, stream);
    // a slab: whole planes, or rows of one where a plane does not fit
    const size_t dz = std::max<size_t>(HostStage::kBytes / plane, 1), dy = std::min(rows, HostStage::kBytes / row);
    const size_t ny = (rows + dy - 1) / dy, slabs = ny * ((planes + dz - 1) / dz);
    std::atomic<int> err{(int)cudaSuccess};
    auto lane = [&](int l) {
        char *buf = s->buf + l * HostStage::kBytes;
        cudaError_t e = cudaSetDevice(device);
        for (size_t k = l; k < slabs && e == cudaSuccess && err.load() == (int)cudaSuccess; k += HostStage::kLanes) {
            const size_t z0 = k / ny * dz, y0 = k % ny * dy, cz = std::min(dz, planes - z0), cy = std::min(dy, rows - y0);
            cudaMemcpy3DParms q = p;
            q.srcPos.y += y0;
            q.srcPos.z += z0;
            q.dstPtr = make_cudaPitchedPtr(buf, row, row, cy);
            q.extent.height = cy;
            q.extent.depth = cz;
            e = cudaMemcpy3DAsync(&q, stream);
            if (e == cudaSuccess) e = cudaEventRecord(s->done[l], stream);
            if (e == cudaSuccess) e = cudaEventSynchronize(s->done[l]);
            if (e == cudaSuccess) std::memcpy((char *)p.dstPtr.ptr + z0 * plane + y0 * row, buf, cz * cy * row);
        }
        if (e != cudaSuccess) err.store((int)e);
    };
    std::thread others[HostStage::kLanes - 1];
    bool all = true;
    for (int l = 1; l < HostStage::kLanes; l++) {
        try {
            others[l - 1] = std::thread(lane, l);
        } catch (const std::system_error &) {
            all = false;
            break;
        }
    }
    lane(0);
    for (std::thread &t : others)
        if (t.joinable()) t.join();
    const cudaError_t e = (cudaError_t)err.load(), w = cudaStreamSynchronize(stream);
    if (!all && e == cudaSuccess && w == cudaSuccess) return plain(p, stream);
    return e != cudaSuccess ? e : w;
}

}  // namespace fi
