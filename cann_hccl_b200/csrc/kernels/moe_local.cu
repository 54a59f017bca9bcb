// MoE exchange where every rank is in this process on one GPU (a single rank included): three launches for a dispatch and a
// combine of all ranks, ordered by their stream (no barrier, no all-gather of counts), each a programmatic dependent launch.
//
//   count     every CTA numbers the (token, k) pairs of its chunk inside their experts with shared-memory counters; the CTA
//             that finishes last turns all histograms into row bases, so nothing waits and no counter needs clearing first;
//   dispatch  a CTA takes one token's row (or a part of it when tokens are few), reads it ONCE and stores it to its top-k
//             receive rows: tokens x (1 + k) rows of traffic, the least the exchange can do;
//   combine   the same split over the output rows: eight expert rows in flight per thread, fp32 sum in k order, one rounding.
//
// Bound: HBM for prefill batches, launches and latency for decode batches.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include "common/log.h"
#include "kernels/moe_a2a.h"
#include "kernels/pdl.cuh"

namespace hcclb {

namespace {

constexpr int kCountThreads = 512, kRowThreads = 256, kRowBatch = 8;

struct MoeTables {
    const __nv_bfloat16 *x[kMaxRanks];
    const int32_t *idx[kMaxRanks];
    int32_t *pos[kMaxRanks], *dst_row[kMaxRanks], *expert_offsets[kMaxRanks], *recv_rows[kMaxRanks], *overflow[kMaxRanks];
    __nv_bfloat16 *rows[kMaxRanks];  // receive buffers (dispatch) or expert outputs (combine) by owner
    const float *gates[kMaxRanks];
    __nv_bfloat16 *out[kMaxRanks];
    int32_t *hist;       // [rank][chunk][expert]: pairs, then the first row of that group
    uint32_t *arrived;   // zero between calls
    int64_t tokens, capacity;
    int p, topk, nvec, n_experts, chunk, nchunk, nseg;
};

// grid (chunks, ranks)
__global__ void __launch_bounds__(kCountThreads) moe_local_count_kernel(const __grid_constant__ MoeTables a)
{
    extern __shared__ int32_t sh[];  // [experts]
    __shared__ int s_last;
    pdl_trigger();
    const int E = a.n_experts, r = blockIdx.y;
    const int64_t npairs = a.tokens * a.topk, i0 = (int64_t)blockIdx.x * a.chunk, i1 = min(i0 + a.chunk, npairs);
    for (int e = threadIdx.x; e < E; e += kCountThreads) sh[e] = 0;
    __syncthreads();
    pdl_wait();
    for (int64_t i = i0 + threadIdx.x; i < i1; i += kCountThreads) {
        const int e = a.idx[r][i];
        a.pos[r][i] = e >= 0 && e < E ? atomicAdd(&sh[e], 1) : -1;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += kCountThreads) a.hist[((int64_t)r * a.nchunk + blockIdx.x) * E + e] = sh[e];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.arrived, 1u) == gridDim.x * gridDim.y - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // rows of an owner are grouped [local expert][source rank][chunk]
    const int groups = a.p * a.nchunk, El = E / a.p;
    for (int e = threadIdx.x; e < E; e += kCountThreads) {
        int t = 0;
#pragma unroll 8
        for (int g = 0; g < groups; ++g) t += __ldcg(a.hist + (int64_t)g * E + e);
        sh[e] = t;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive prefix over all experts
        int carry = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + threadIdx.x, t = e < E ? sh[e] : 0;
            int v = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int w = __shfl_up_sync(0xffffffffu, v, o);
                if ((int)threadIdx.x >= o) v += w;
            }
            if (e < E) sh[e] = carry + v - t;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (threadIdx.x == 0) { sh[E] = carry; *a.arrived = 0; }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += kCountThreads) {
        const int q = e / El, first = sh[q * El];
        int row = sh[e] - first;
        a.expert_offsets[q][e - q * El] = row;
        if (e == q * El + El - 1) {
            const int total = sh[e + 1] - first;
            a.expert_offsets[q][El] = total;
            *a.recv_rows[q] = total;
            if (total > a.capacity) *a.overflow[q] = 1;
        }
#pragma unroll 8
        for (int g = 0; g < groups; ++g) {
            int32_t *h = a.hist + (int64_t)g * E + e;
            const int n = __ldcg(h);
            *h = row;
            row += n;
        }
    }
}

// grid (tokens x segments, ranks)
__global__ void __launch_bounds__(kRowThreads) moe_local_dispatch_kernel(const __grid_constant__ MoeTables a)
{
    __shared__ uint4 *s_dst[kRowBatch];
    pdl_trigger();
    const int r = blockIdx.y, k = a.topk;
    const int64_t t = blockIdx.x / a.nseg;
    const int seg = (int)(blockIdx.x - t * a.nseg), per = (a.nvec + a.nseg - 1) / a.nseg, v1 = min(a.nvec, (seg + 1) * per);
    const uint4 *src = (const uint4 *)a.x[r] + t * a.nvec;
    pdl_wait();
    for (int k0 = 0; k0 < k; k0 += kRowBatch) {
        if (k0) __syncthreads();
        if (threadIdx.x < kRowBatch) {
            uint4 *d = nullptr;
            if (k0 + (int)threadIdx.x < k) {
                const int64_t i = t * k + k0 + threadIdx.x;
                const int e = a.idx[r][i];
                if (e >= 0 && e < a.n_experts) {
                    const int64_t row = (int64_t)a.hist[((int64_t)r * a.nchunk + i / a.chunk) * a.n_experts + e] + a.pos[r][i];
                    if (seg == 0) a.dst_row[r][i] = (int32_t)row;
                    if (row < a.capacity) d = (uint4 *)a.rows[e / (a.n_experts / a.p)] + row * a.nvec;
                }
            }
            s_dst[threadIdx.x] = d;
        }
        uint4 x[4];
        const int v0 = seg * per + threadIdx.x;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * kRowThreads < v1) x[u] = src[v0 + u * kRowThreads];
        __syncthreads();
        for (int vb = v0;;) {
#pragma unroll
            for (int j = 0; j < kRowBatch; ++j) {
                uint4 *d = s_dst[j];
                if (!d) continue;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (vb + u * kRowThreads < v1) d[vb + u * kRowThreads] = x[u];
            }
            vb += 4 * kRowThreads;
            if (vb >= v1) break;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (vb + u * kRowThreads < v1) x[u] = src[vb + u * kRowThreads];
        }
    }
}

// grid (tokens x segments, ranks)
__global__ void __launch_bounds__(kRowThreads) moe_local_combine_kernel(const __grid_constant__ MoeTables a)
{
    __shared__ const uint4 *s_src[kRowBatch];
    __shared__ float s_gate[kRowBatch];
    pdl_trigger();
    const int r = blockIdx.y, k = a.topk;
    const int64_t t = blockIdx.x / a.nseg;
    const int seg = (int)(blockIdx.x - t * a.nseg), per = (a.nvec + a.nseg - 1) / a.nseg, v1 = min(a.nvec, (seg + 1) * per);
    uint4 *out = (uint4 *)a.out[r] + t * a.nvec;
    pdl_wait();
    const bool one = k <= kRowBatch;
    auto batch = [&](int k0) {
        if (threadIdx.x < kRowBatch) {
            const uint4 *s = nullptr;
            float g = 0.f;
            if (k0 + (int)threadIdx.x < k) {
                const int64_t i = t * k + k0 + threadIdx.x;
                const int e = a.idx[r][i];
                const int64_t row = a.dst_row[r][i];
                if (e >= 0 && e < a.n_experts && row >= 0 && row < a.capacity) {
                    s = (const uint4 *)a.rows[e / (a.n_experts / a.p)] + row * a.nvec;
                    g = a.gates[r][i];
                }
            }
            s_src[threadIdx.x] = s;
            s_gate[threadIdx.x] = g;
        }
        __syncthreads();
    };
    if (one) batch(0);
    for (int vb = seg * per; vb < v1; vb += kRowThreads) {  // uniform trip count: the batches synchronise
        const int v = vb + threadIdx.x;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < k; k0 += kRowBatch) {
            if (!one) { __syncthreads(); batch(k0); }
            if (v < v1) {
                uint4 x[kRowBatch];
#pragma unroll
                for (int j = 0; j < kRowBatch; ++j)
                    if (s_src[j]) x[j] = s_src[j][v];
#pragma unroll
                for (int j = 0; j < kRowBatch; ++j) {
                    if (!s_src[j]) continue;
                    const float g = s_gate[j];
                    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&x[j];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(h[i]);
                        acc[2 * i] += g * f.x;
                        acc[2 * i + 1] += g * f.y;
                    }
                }
            }
        }
        if (v < v1) {
            uint4 o;
            __nv_bfloat162 *h = (__nv_bfloat162 *)&o;
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
            out[v] = o;
        }
    }
}

// Parts of a row per CTA row: whole rows once there is a CTA for every SM several times over.
int segments(int64_t units, int nvec)
{
    int s = 1;
    while (s < 4 && units * s < 4 * 148 && nvec / (2 * s) >= kRowThreads) s *= 2;
    return s;
}

void fill(MoeTables &t, const MoeLocalLayer &l)
{
    t.p = l.p; t.topk = l.topk; t.nvec = l.hidden / 8; t.n_experts = l.n_experts; t.tokens = l.tokens; t.capacity = l.capacity;
    moe_local_chunks(l.tokens * l.topk, &t.chunk, &t.nchunk);
    t.hist = l.scratch + 4;
    t.arrived = (uint32_t *)l.scratch;
    t.nseg = segments(l.tokens * l.p, t.nvec);
    for (int q = 0; q < l.p; ++q) { t.pos[q] = l.pos[q]; t.dst_row[q] = l.dst_row[q]; }
}

bool bad(const MoeLocalLayer &l)
{
    return l.p < 1 || l.p > kMaxRanks || l.tokens < 0 || l.topk < 1 || l.hidden < 8 || l.hidden % 8 || l.n_experts < l.p || l.n_experts % l.p ||
           l.n_experts > kMoeLocalMaxExperts || !l.scratch || l.tokens * l.topk > 0x7fffffff || l.tokens * 4 > 0x7fffffff;
}

}  // namespace

HcclResult moe_local_dispatch(const MoeLocalLayer &l, void *const *recv, const void *const *x, const int32_t *const *idx, void *stream)
{
    if (bad(l)) return HCCL_E_PARA;
    if (l.tokens == 0) return HCCL_SUCCESS;
    MoeTables t;
    fill(t, l);
    for (int q = 0; q < l.p; ++q) {
        t.x[q] = (const __nv_bfloat16 *)x[q]; t.idx[q] = idx[q]; t.rows[q] = (__nv_bfloat16 *)recv[q];
        t.expert_offsets[q] = l.expert_offsets[q]; t.recv_rows[q] = l.recv_rows[q]; t.overflow[q] = l.overflow[q];
    }
    HcclResult rc = launch_pdl((const void *)moe_local_count_kernel, dim3((unsigned)t.nchunk, (unsigned)l.p), kCountThreads,
                               sizeof(int32_t) * (l.n_experts + 1), &t, stream, "moe count");
    if (rc != HCCL_SUCCESS) return rc;
    return launch_pdl((const void *)moe_local_dispatch_kernel, dim3((unsigned)(l.tokens * t.nseg), (unsigned)l.p), kRowThreads, 0, &t, stream, "moe dispatch");
}

HcclResult moe_local_combine(const MoeLocalLayer &l, void *const *rows, const int32_t *const *idx, const float *const *gates, void *const *out, void *stream)
{
    if (bad(l)) return HCCL_E_PARA;
    if (l.tokens == 0) return HCCL_SUCCESS;
    MoeTables t;
    fill(t, l);
    for (int q = 0; q < l.p; ++q) { t.idx[q] = idx[q]; t.rows[q] = (__nv_bfloat16 *)rows[q]; t.gates[q] = gates[q]; t.out[q] = (__nv_bfloat16 *)out[q]; }
    return launch_pdl((const void *)moe_local_combine_kernel, dim3((unsigned)(l.tokens * t.nseg), (unsigned)l.p), kRowThreads, 0, &t, stream, "moe combine");
}

}  // namespace hcclb
