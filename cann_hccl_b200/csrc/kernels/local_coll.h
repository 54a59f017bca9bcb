// Launch interface of the direct collectives (kernels/local_coll.cuh, local_coll.cu): communicators whose ranks all live in
// this process on one GPU, a single rank included.  Every rank's buffers are addressable by every thread, so a collective
// is one pass over memory: each input byte is read once and each output byte written once, in one launch whose CTAs wait
// for nothing.  (With one process per GPU the caller's buffers are not mapped on the peers; those communicators stage.)
//
// Bound: HBM for messages beyond L2, launch and one memory round trip below.  Measured on a B200 against the staged kernels
// (push, reduce and copy-out through staging buffers, CTAs of all ranks resident together): AllReduce of 64 MiB fp32 over
// eight ranks 655 -> 164 us (6.56 TB/s), ReduceScatter of 4 MiB bf16 blocks over eight ranks 286 -> 55 us, AlltoAllV of 1024
// rows of 7168 bf16 from each of eight ranks 138 -> 37 us, AllGather of 1 MiB over four ranks 31 -> 8.5 us, the copy of a
// single rank's 64 MiB 28.8 -> 21.8 us (6.2 TB/s).
#pragma once
#include "algo/plan.h"

namespace hcclb {

constexpr int kLocalMaxJobs = kMaxRanks * kMaxRanks;  // AlltoAllV: one per ordered pair of ranks

// dst rank d in `mask`: out[d] + doff receives `bytes` from src
struct LocalCopyJob {
    const uint8_t *src;
    uint64_t doff, bytes;
    uint32_t tile0;  // first tile of this job (filled by the launcher)
    uint32_t mask;
};
struct LocalCopy {
    uint8_t *out[kMaxRanks];
    int njobs;
    LocalCopyJob job[kLocalMaxJobs];
};
// Job j: out[d] (d in mask[j]) = reduction over the p ranks, in rank order, of count[j] elements at in[q] + off[j].
struct LocalReduce {
    const uint8_t *in[kMaxRanks];
    uint8_t *out[kMaxRanks];
    uint64_t off[kMaxRanks], count[kMaxRanks];
    uint32_t tile0[kMaxRanks + 1];  // first tile of a job (filled by the launcher)
    uint32_t mask[kMaxRanks];
    int p, njobs;
    uint32_t tile_vecs;
};

// Both take and change the caller's description (tile tables).
HcclResult launch_local_copy(LocalCopy &c, void *stream);
HcclResult launch_local_reduce(LocalReduce &r, int dtype, int redop, void *stream);

}  // namespace hcclb
