// Direct path of communicators whose ranks all live in this process on one GPU (virtual ranks, or a single rank): every
// rank's buffers are addressable here, so a collective needs no staging, no flags and no plan.  The call is turned into a job
// table that travels as a kernel argument (kernels/local_coll.*), one ordinary launch per collective.
#include <cstring>
#include "common/env.h"
#include "common/log.h"
#include "core/communicator.h"
#include "kernels/local_coll.h"

namespace hcclb {

// The choice for such communicators where nothing else is asked for.  Another algorithm (that of the parametric AlltoAll and of
// the peers' registered buffers included), a CTA count or an execution mode that the caller or the environment asks for keeps
// the staged kernels, which is how those are tested on one GPU; so do in-kernel timestamps (HCCL_KERNEL_TRACE), which only those write.
bool Communicator::direct_applies(const OpRequest &rq) const
{
    if (calibrating_) return false;  // measures the staged kernels, which requests of those kinds choose among
    if (rq.algo == ALGO_LOCAL) return settings_.transport == TR_DEVICE && nlocal() == nranks_;
    return rq.algo == ALGO_AUTO && rq.nchan <= 0 && direct_default(rq.coll);
}

bool Communicator::direct_default(int coll) const
{
    const EnvConfig &env = env_config();
    if (settings_.transport != TR_DEVICE || nlocal() != nranks_ || env.channels > 0 || dev_trace_) return false;
    if ((settings_.expansion_mode ? settings_.expansion_mode : env.expansion_mode) == 1) return false;
    return env.algo.empty() || forced_algo_for(env, coll).empty();
}

HcclResult Communicator::run_direct(const OpRequest &rq)
{
    const int p = nranks_;
    const uint64_t es = (uint64_t)dtype_size(rq.dtype), n = rq.count;
    const uint32_t all = (1u << p) - 1u;
    if (rq.coll == COLL_BARRIER) return HCCL_SUCCESS;  // one stream carries every rank: stream order is the barrier
    stats_.launches++;

    const bool reduces = rq.coll == COLL_ALLREDUCE || rq.coll == COLL_REDUCE || rq.coll == COLL_REDUCE_SCATTER || rq.coll == COLL_REDUCE_SCATTER_V;
    if (reduces && p > 1) {
        LocalReduce r;
        for (int q = 0; q < p; ++q) { r.in[q] = (const uint8_t *)rq.in[q]; r.out[q] = (uint8_t *)rq.out[q]; }
        r.p = p;
        if (rq.coll == COLL_ALLREDUCE || rq.coll == COLL_REDUCE) {
            r.njobs = 1;
            r.job[0].off = 0; r.job[0].count = n; r.job[0].mask = rq.coll == COLL_ALLREDUCE ? all : 1u << rq.root;
        } else {
            r.njobs = p;
            for (int j = 0; j < p; ++j) {
                const bool v = rq.coll == COLL_REDUCE_SCATTER_V;
                r.job[j].off = (v ? rq.displs[j] : (uint64_t)j * n) * es;
                r.job[j].count = v ? rq.counts[j] : n;
                r.job[j].mask = 1u << j;
            }
        }
        return launch_local_reduce(r, rq.dtype, rq.redop, rq.stream);
    }

    LocalCopy c;
    c.njobs = 0;
    for (int q = 0; q < p; ++q) c.out[q] = (uint8_t *)rq.out[q];
    // ranks of `mask` that already hold the block where it belongs (in-place forms) drop out; destinations whose 32-byte
    // alignments differ become jobs of their own
    auto add = [&](const void *src, uint64_t doff, uint64_t bytes, uint32_t mask) {
        if (!bytes) return;
        for (int d = 0; d < p; ++d)
            if (((mask >> d) & 1u) && c.out[d] + doff == (const uint8_t *)src) mask &= ~(1u << d);
        while (mask) {
            const int first = __builtin_ctz(mask);
            uint32_t same = 0;
            for (int d = first; d < p; ++d)
                if (((mask >> d) & 1u) && ((((uintptr_t)c.out[d]) ^ ((uintptr_t)c.out[first])) & 31) == 0) same |= 1u << d;
            c.job[c.njobs++] = LocalCopyJob{(const uint8_t *)src, doff, bytes, 0, same};
            mask &= ~same;
        }
    };
    switch (rq.coll) {
        case COLL_BROADCAST: add(rq.in[rq.root], 0, n * es, all & ~(1u << rq.root)); break;
        case COLL_SCATTER:
            for (int d = 0; d < p; ++d) add((const uint8_t *)rq.in[rq.root] + (uint64_t)d * n * es, 0, n * es, 1u << d);
            break;
        case COLL_GATHER:
            for (int q = 0; q < p; ++q) add(rq.in[q], (uint64_t)q * n * es, n * es, 1u << rq.root);
            break;
        case COLL_ALLGATHER:
            for (int q = 0; q < p; ++q) add(rq.in[q], (uint64_t)q * n * es, n * es, all);
            break;
        case COLL_ALLGATHER_V:
            for (int q = 0; q < p; ++q) add(rq.in[q], rq.displs[q] * es, rq.counts[q] * es, all);
            break;
        case COLL_ALLTOALL:
            for (int q = 0; q < p; ++q)
                for (int d = 0; d < p; ++d) add((const uint8_t *)rq.in[q] + (uint64_t)d * n * es, (uint64_t)q * n * es, n * es, 1u << d);
            break;
        case COLL_ALLTOALLV: case COLL_ALLTOALLVC:
            for (int q = 0; q < p; ++q)
                for (int d = 0; d < p; ++d)
                    add((const uint8_t *)rq.in[q] + rq.send_displs[(size_t)q * p + d] * es, rq.recv_displs[(size_t)d * p + q] * es,
                        rq.send_counts[(size_t)q * p + d] * es, 1u << d);
            break;
        case COLL_REDUCE_SCATTER_V: add((const uint8_t *)rq.in[0] + rq.displs[0] * es, 0, rq.counts[0] * es, 1u); break;  // one rank
        default: add(rq.in[0], 0, n * es, 1u); break;  // AllReduce, Reduce, ReduceScatter of one rank
    }
    return launch_local_copy(c, rq.stream);
}

}  // namespace hcclb
