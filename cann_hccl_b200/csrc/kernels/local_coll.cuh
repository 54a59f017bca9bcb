// Direct collectives on one GPU: see local_coll.h.  Reduction kernel, one per (element type, operator, source batch).
#pragma once
#include "kernels/exec_plan_impl.cuh"
#include "kernels/local_coll.h"
#include "kernels/pdl.cuh"

namespace hcclb {

constexpr int kLocalThreads = 256;

// 16 bytes at v0 + s (0 < s < 16), v0 and v1 being the two aligned vectors that hold them.  s is uniform in a job.
__device__ __forceinline__ uint4 merge16(uint4 v0, uint4 v1, uint32_t s)
{
    const uint32_t b = (s & 3) * 8;
    const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint4 r;
    switch (s >> 2) {
        case 0: r = make_uint4(__funnelshift_r(w[0], w[1], b), __funnelshift_r(w[1], w[2], b), __funnelshift_r(w[2], w[3], b), __funnelshift_r(w[3], w[4], b)); break;
        case 1: r = make_uint4(__funnelshift_r(w[1], w[2], b), __funnelshift_r(w[2], w[3], b), __funnelshift_r(w[3], w[4], b), __funnelshift_r(w[4], w[5], b)); break;
        case 2: r = make_uint4(__funnelshift_r(w[2], w[3], b), __funnelshift_r(w[3], w[4], b), __funnelshift_r(w[4], w[5], b), __funnelshift_r(w[5], w[6], b)); break;
        default: r = make_uint4(__funnelshift_r(w[3], w[4], b), __funnelshift_r(w[4], w[5], b), __funnelshift_r(w[5], w[6], b), __funnelshift_r(w[6], w[7], b)); break;
    }
    return r;
}
// The aligned vectors touched here each hold at least one byte of the range, so no load leaves the caller's 16-byte granules.
__device__ __forceinline__ uint4 ld_shifted(const uint8_t *a)
{
    const uint32_t s = (uint32_t)((uintptr_t)a & 15);
    const uint4 *b = (const uint4 *)(a - s);
    return s ? merge16(b[0], b[1], s) : b[0];
}

// One tile of a job: U vectors of every source in flight per thread.  SHIFT: some source is not aligned like the outputs.
template <class T, int OP, int NP, int U, bool SHIFT>
__device__ __forceinline__ void local_reduce_tile(const uint8_t *const (&in)[kMaxRanks], uint8_t *const (&out)[kMaxRanks], uint32_t mask, uint64_t soff,
                                                  uint64_t doff, int p, uint64_t v0, uint64_t v1)
{
    using N = DNum<T>;
    using Acc = typename N::Acc;
    constexpr int E = 16 / sizeof(T);
    for (uint64_t i = v0 + threadIdx.x; i < v1; i += (uint64_t)U * kLocalThreads) {
        Acc acc[U][E];
        for (int q0 = 0; q0 < p; q0 += NP) {
            uint4 x[U][NP];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const uint64_t v = i + (uint64_t)u * kLocalThreads;
                    if (q0 + q < p && v < v1) {
                        const uint8_t *a = in[q0 + q] + soff + (v << 4);
                        x[u][q] = SHIFT ? ld_shifted(a) : ld_stream((const uint4 *)a);
                    }
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    if (q0 + q < p) {
                        Pack16<T> t;
                        t.u = x[u][q];
#pragma unroll
                        for (int k = 0; k < E; ++k) acc[u][k] = q == 0 && q0 == 0 ? N::up(t.e[k]) : red_op<OP>(acc[u][k], N::up(t.e[k]));
                    }
            if (NP < 8) break;  // the launcher takes the batch of eight for five and more ranks
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t v = i + (uint64_t)u * kLocalThreads;
            if (v < v1) {
                Pack16<T> z;
#pragma unroll
                for (int k = 0; k < E; ++k) z.e[k] = N::down(acc[u][k]);
#pragma unroll
                for (int d = 0; d < kMaxRanks; ++d)
                    if ((mask >> d) & 1u) *(uint4 *)(out[d] + doff + (v << 4)) = z.u;
            }
        }
    }
}

template <class T, int OP, int NP>
__global__ void __launch_bounds__(kLocalThreads) local_reduce_kernel(const __grid_constant__ LocalReduce a)
{
    using N = DNum<T>;
    using Acc = typename N::Acc;
    constexpr int E = 16 / sizeof(T), U = NP == 2 ? 4 : (NP == 4 ? 2 : 1);
    pdl_trigger();
    int j = 0;
    while (blockIdx.x >= a.tile0[j + 1]) ++j;  // the launcher's table ends with the grid's size
    const uint64_t n = a.count[j], soff = a.off[j];
    const uint32_t mask = a.mask[j], tile = blockIdx.x - a.tile0[j];
    // vectors are laid over the outputs' 16-byte granules; the elements before the first and after the last go one by one
    const uint8_t *d0 = a.out[__ffs(mask) - 1];
    uint32_t differ = 0, shift = 0;
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d)
        if ((mask >> d) & 1u) differ |= (uint32_t)((uintptr_t)a.out[d] ^ (uintptr_t)d0) & 15;
    uint64_t head = ((16 - ((uintptr_t)d0 & 15)) & 15) / sizeof(T);
    if (head > n || differ) head = n;
    const uint64_t nvec = (n - head) / E, hb = head * sizeof(T);
    for (int q = 0; q < a.p; ++q) shift |= (uint32_t)((uintptr_t)a.in[q] + soff + hb) & 15;
    pdl_wait();
    const uint64_t v0 = (uint64_t)tile * a.tile_vecs, v1 = v0 + a.tile_vecs < nvec ? v0 + a.tile_vecs : nvec;
    if (v0 < nvec) {
        if (!shift) local_reduce_tile<T, OP, NP, U, false>(a.in, a.out, mask, soff + hb, hb, a.p, v0, v1);
        else local_reduce_tile<T, OP, NP, 1, true>(a.in, a.out, mask, soff + hb, hb, a.p, v0, v1);
    }
    // leftovers: at most a vector at either end, or everything when the outputs do not share an alignment
    const uint64_t left = n - nvec * E, step = differ ? (uint64_t)(a.tile0[j + 1] - a.tile0[j]) * kLocalThreads : kLocalThreads;
    if (tile != 0 && !differ) return;
    for (uint64_t l = (uint64_t)(differ ? tile : 0) * kLocalThreads + threadIdx.x; l < left; l += step) {
        const uint64_t e = l < head ? l : nvec * E + l;
        Acc acc = N::up(((const T *)(a.in[0] + soff))[e]);
        for (int q = 1; q < a.p; ++q) acc = red_op<OP>(acc, N::up(((const T *)(a.in[q] + soff))[e]));
        const T r = N::down(acc);
        for (int d = 0; d < kMaxRanks; ++d)
            if ((mask >> d) & 1u) ((T *)a.out[d])[e] = r;
    }
}

// Defines local_kernel_<name>(op, p): the reduction kernel for element type T.
#define HCCLB_LOCAL_BATCH(T, OP) \
    (p <= 2 ? (const void *)local_reduce_kernel<T, OP, 2> : p <= 4 ? (const void *)local_reduce_kernel<T, OP, 4> : (const void *)local_reduce_kernel<T, OP, 8>)
#define HCCLB_INSTANTIATE_LOCAL(T, name)                                              \
    const void *local_kernel_##name(int op, int p)                                    \
    {                                                                                 \
        switch (op) {                                                                 \
            case HCCL_REDUCE_SUM: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_SUM);       \
            case HCCL_REDUCE_PROD: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_PROD);     \
            case HCCL_REDUCE_MAX: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_MAX);       \
            default: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_MIN);                    \
        }                                                                             \
    }

}  // namespace hcclb
