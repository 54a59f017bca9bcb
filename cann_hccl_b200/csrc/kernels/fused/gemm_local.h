// Launch interface of the tcgen05 GEMM that needs no communication (kernels/fused/gemm_local.cu): the plain product, and the
// tensor-parallel layers of communicators whose ranks all live in this process on one GPU, where a "peer's" operand is just
// another pointer.  All of them are one tile space:
//   plain      C[M,N] = A * B^T
//   all-gather rank r's output = (row shards A_0..A_{p-1} stacked) * B_r^T: A by row shard, B and C by column shard
//   reduce     rank r's output = rows of shard r of sum_q A_q * B_q^T: A and B by K segment (the sum over the ranks stays in
//              the fp32 accumulator), C by row shard
#pragma once
#include "common/base.h"

namespace hcclb {

constexpr int kGemmShards = 4;  // ranks of a tensor-parallel layer
enum GemmAct : int { GEMM_ACT_NONE = 0, GEMM_ACT_SILU = 1, GEMM_ACT_GELU = 2 };
enum GemmForm : int { GEMM_PLAIN = 0, GEMM_GATHER = 1, GEMM_REDUCE = 2 };

struct GemmCall {
    int form = GEMM_PLAIN, act = GEMM_ACT_NONE, p = 1;
    int M = 0, N = 0, K = 0;               // gathered rows, columns of one B, depth of one B
    const void *A[kGemmShards] = {};       // gather: [M/p, K] each; reduce: [M, K] each
    const void *B[kGemmShards] = {};       // [N, K] each
    void *C[kGemmShards] = {};             // plain [M, N]; gather [M, N] each; reduce [M/p, N] each
};
// status: host-mapped block that records a wait that ran out (may be null).
HcclResult launch_gemm_local(const GemmCall &c, DevStatus *status, void *stream);
// Launches so far: tiles of 128 rows on single CTAs, tiles of 256 rows on pairs (64 to 256 columns either way).
void gemm_local_launch_counts(uint64_t *single, uint64_t *pair);

}  // namespace hcclb
