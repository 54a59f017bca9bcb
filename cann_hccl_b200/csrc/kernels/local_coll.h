// Launch interface of the direct collectives (kernels/local_coll.cuh, local_coll.cu): communicators whose ranks all live in
// this process on one GPU, a single rank included.  Every rank's buffers are addressable by every thread, so a collective
// is one pass over memory: each input byte is read once and each output byte written once, in one launch whose CTAs wait
// for nothing.  (With one process per GPU the caller's buffers are not mapped on the peers; those communicators stage.)
//
// Bound: HBM for messages beyond L2, launch and one memory round trip below.  Measured on a B200 against the staged kernels
// (push, reduce and copy-out through staging buffers, CTAs of all ranks resident together): AllReduce of 64 MiB fp32 over
// eight ranks 655 -> 159 us (6.8 TB/s), ReduceScatter of 4 MiB bf16 blocks over eight ranks 286 -> 46 us (6.6 TB/s), AlltoAllV
// of 1024 rows of 7168 bf16 from each of eight ranks 138 -> 36 us, the copy of a single rank's 64 MiB 28.8 -> 21.4 us.
// What the last steps gave (ReduceScatter case): how a job lies over vectors worked out by the launcher instead of by every
// CTA, 55 -> 50 us; 32-byte instead of 16-byte vectors, 50 -> 46 us.
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
// Job: out[d] (d in mask) = reduction over the p ranks, in rank order, of `count` elements at in[q] + off.  The launcher fills
// in how the job is laid over vectors, so that a CTA loads a few words and starts.
enum LocalLayout : uint32_t { LOCAL_ALIGNED = 0, LOCAL_SHIFTED = 1, LOCAL_SCALAR = 2 };
struct LocalReduceJob {
    uint64_t off, count;
    uint32_t mask, layout;
    uint64_t nvec;       // vectors of the outputs
    uint32_t head;       // elements before the first vector
    uint32_t tile0;      // first tile; the job's last tile holds the elements outside the vectors when there are any
};
struct LocalReduce {
    const uint8_t *in[kMaxRanks];
    uint8_t *out[kMaxRanks];
    LocalReduceJob job[kMaxRanks];
    int p, njobs;
    uint32_t tile_vecs, tile_elems;  // of a tile; tile_elems: where a job goes one by one
    uint32_t uniform;                // tiles per job when all jobs have the same number, else 0
};

// Both take and change the caller's description (tile tables).
HcclResult launch_local_copy(LocalCopy &c, void *stream);
HcclResult launch_local_reduce(LocalReduce &r, int dtype, int redop, void *stream);

}  // namespace hcclb
