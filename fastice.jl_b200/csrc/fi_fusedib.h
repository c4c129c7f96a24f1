// fi_fusedib.h -- host interface of the fused immersed-boundary sweep (fi_fusedib.cu).
#pragma once

#include <vector>

#include "fi_internal.h"

namespace fi {

// planes [k0, k1) of the 32x8 column (x, y) that an iteration touches
struct IbRun {
    int x, y, k0, k1;
};

// one model of a batched launch: f[e] is read and f[2 + e] written when the roles of its
// buffers are e (0: as when the table was built, 1: swapped)
template <typename T>
struct IbFusedHead {
    Geom g;
    KParams p;
    TConst<T> q;
    Ptrs<T> f[4];
    int *err;
};
template <typename T>
struct alignas(128) IbFusedMember {
    unsigned char maps[2][11][128];  // tensor maps of what is read under either role
    IbFusedHead<T> head;
};

// the runs of a model from its activity bytes (waits for the stream)
cudaError_t ib_runs(const Geom &g, const unsigned char *flags, std::vector<IbRun> *runs, cudaStream_t s);
// the z-block depth for the runs of the models of one launch, and their jobs
int ib_job_depth(const std::vector<const std::vector<IbRun> *> &all);
void ib_make_jobs(const std::vector<IbRun> &runs, int zb, int member, std::vector<int4> *jobs);

// (chained: right after another of these launches on the stream)
template <typename T>
cudaError_t launch_fusedib(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, const void *maps11,
                           const int4 *jobs, int njobs, int *err, cudaStream_t s, bool chained);
template <typename T>
cudaError_t launch_fusedib_batched(const IbFusedMember<T> *members, const int4 *jobs, int njobs, int e, cudaStream_t s, bool chained);

}  // namespace fi
