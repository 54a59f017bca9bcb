// MoE dispatch / combine kernels (kernels/moe_a2a.cu).  All pointers are device pointers; peer tables are host arrays
// of p device pointers (rank q's buffer as mapped on this rank).
#pragma once
#include <algorithm>
#include "common/base.h"
#include "hccl/hccl_b200.h"
namespace hcclb {
HcclResult moe_count(const int32_t *topk_idx, int64_t npairs, int n_experts, int32_t *hist, int32_t *pos, void *stream);
HcclResult moe_offsets(const int32_t *counts, int p, int n_experts, int me, int32_t *base, int32_t *expert_offsets, int32_t *recv_rows,
                       int64_t capacity_rows, int32_t *overflow, void *stream);
HcclResult moe_dispatch(const void *x, const int32_t *topk_idx, const int32_t *pos, const int32_t *base, int64_t tokens, int topk, int hidden,
                        int n_experts, int p, int me, int pairwise, void *const *recv_peers, int32_t *dst_row, int64_t capacity_rows, void *stream);
HcclResult moe_combine(void *const *y_peers, const int32_t *topk_idx, const float *gates, const int32_t *dst_row, int64_t tokens, int topk,
                       int hidden, int n_experts, int p, int me, int pairwise, void *out, int64_t capacity_rows, void *stream);

// ---- all ranks in this process on one GPU (kernels/moe_local.cu)
constexpr int kMoeLocalMaxExperts = 4096;  // two shared-memory words each
struct MoeLocalLayer {
    int64_t tokens, capacity;  // tokens of a rank; rows of a receive buffer
    int p, topk, hidden, n_experts;
    int32_t *const *pos, *const *dst_row, *const *expert_offsets, *const *recv_rows, *const *overflow;  // [p] device pointers
    int32_t *scratch;          // moe_local_scratch_words() words, zero before the first call
};
// The count kernel cuts a rank's pairs into chunks: one CTA numbers a chunk in shared memory.  At most 64 chunks: the CTA that
// turns the histograms into row bases reads all of them.
inline void moe_local_chunks(int64_t npairs, int *chunk, int *nchunk)
{
    const int64_t c = std::max<int64_t>(1024, (npairs + 63) / 64);
    *chunk = (int)c;
    *nchunk = (int)std::max<int64_t>(1, (npairs + c - 1) / c);
}
inline int64_t moe_local_scratch_words(int p, int64_t tokens, int topk, int n_experts)
{
    int chunk, nchunk;
    moe_local_chunks(tokens * topk, &chunk, &nchunk);
    return 4 + (int64_t)p * nchunk * n_experts;
}
HcclResult moe_local_dispatch(const MoeLocalLayer &l, void *const *recv, const void *const *x, const int32_t *const *idx, void *stream);
HcclResult moe_local_combine(const MoeLocalLayer &l, void *const *rows, const int32_t *const *idx, const float *const *gates, void *const *out, void *stream);
}  // namespace hcclb
