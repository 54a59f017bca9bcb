// Direct collectives on one GPU: see local_coll.h.  Reduction kernel, one per (element type, operator, source batch).
#pragma once
#include "kernels/exec_plan_impl.cuh"
#include "kernels/local_coll.h"
#include "kernels/pdl.cuh"

namespace hcclb {

constexpr int kLocalThreads = 128;

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

// A vector is one load per source: 32 bytes where every address allows it, else 16.
template <int VB> union Vec;
template <> union Vec<16> { uint4 u; uint32_t w[4]; };
template <> union Vec<32> { uint4 u[2]; uint32_t w[8]; };
__device__ __forceinline__ Vec<16> ld_vec(const uint8_t *p, Vec<16> *) { Vec<16> v; v.u = ld_stream((const uint4 *)p); return v; }
__device__ __forceinline__ Vec<32> ld_vec(const uint8_t *p, Vec<32> *)
{
    Vec<32> v;
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_vec(uint8_t *p, const Vec<16> &v) { *(uint4 *)p = v.u; }
__device__ __forceinline__ void st_vec(uint8_t *p, const Vec<32> &v)
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7]) : "memory");
}

// Vectors per thread of a full tile: 128 bytes of loads in flight per thread for two sources, 128 to 256 for more.
template <int NP, int VB> constexpr int kReduceVecs = NP == 2 ? 64 / VB : (NP == 4 ? 32 / VB : 1);

// One tile of a job.  SHIFT: some source is not aligned like the outputs.
template <class T, int OP, int NP, int VB, int U, bool SHIFT>
__device__ __forceinline__ void local_reduce_tile(const LocalReduce &a, const LocalReduceJob &j, uint32_t tile)
{
    using N = DNum<T>;
    using Acc = typename N::Acc;
    constexpr int E = VB / sizeof(T);
    union Elems { Vec<VB> v; T e[E]; __device__ Elems() {} };
    const uint64_t first = (uint64_t)tile * a.tile_vecs + threadIdx.x, soff = j.off + j.head * sizeof(T), doff = j.head * sizeof(T);
    const uint64_t end = min(j.nvec, (uint64_t)(tile + 1) * a.tile_vecs);
#pragma unroll 1
    for (uint64_t i = first; i < end; i += (uint64_t)U * kLocalThreads) {
        Acc acc[U][E];
#pragma unroll 1
        for (int q0 = 0; q0 < a.p; q0 += NP) {
            Elems x[U][NP];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const uint64_t v = i + (uint64_t)u * kLocalThreads;
                    if (q0 + q < a.p && v < end) {
                        const uint8_t *s = a.in[q0 + q] + soff + v * VB;
                        if constexpr (SHIFT) x[u][q].v.u = ld_shifted(s);
                        else x[u][q].v = ld_vec(s, (Vec<VB> *)nullptr);
                    }
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    if (q0 + q < a.p) {
#pragma unroll
                        for (int k = 0; k < E; ++k) acc[u][k] = q == 0 && q0 == 0 ? N::up(x[u][q].e[k]) : red_op<OP>(acc[u][k], N::up(x[u][q].e[k]));
                    }
            if (NP < 8) break;  // the launcher takes the batch of eight for five and more ranks
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t v = i + (uint64_t)u * kLocalThreads;
            if (v < end) {
                Elems z;
#pragma unroll
                for (int k = 0; k < E; ++k) z.e[k] = N::down(acc[u][k]);
                for (uint32_t m = j.mask; m; m &= m - 1) st_vec(a.out[__ffs(m) - 1] + doff + v * VB, z.v);
            }
        }
    }
}

template <class T, int OP, int NP, int VB>
__global__ void __launch_bounds__(kLocalThreads) local_reduce_kernel(const __grid_constant__ LocalReduce a)
{
    using N = DNum<T>;
    using Acc = typename N::Acc;
    constexpr int E = VB / sizeof(T);
    pdl_trigger();
    int ji = 0;
    if (a.uniform) ji = blockIdx.x / a.uniform;
    else
        while (ji + 1 < a.njobs && blockIdx.x >= a.job[ji + 1].tile0) ++ji;
    const LocalReduceJob &j = a.job[ji];
    const uint32_t tile = blockIdx.x - j.tile0;
    pdl_wait();
    if (j.layout != LOCAL_SCALAR && (uint64_t)tile * a.tile_vecs < j.nvec) {
        if (VB == 32 || j.layout == LOCAL_ALIGNED) local_reduce_tile<T, OP, NP, VB, kReduceVecs<NP, VB>, false>(a, j, tile);
        else if constexpr (VB == 16) local_reduce_tile<T, OP, NP, 16, 1, true>(a, j, tile);
        return;
    }
    // one by one: what lies outside the vectors (a tile of its own), or everything when the outputs do not share an alignment
    const bool scalar = j.layout == LOCAL_SCALAR;
    const uint64_t vecs = scalar ? 0 : j.nvec, left = j.count - vecs * E;
    const uint64_t l0 = scalar ? (uint64_t)tile * a.tile_elems : 0, l1 = scalar ? min(left, l0 + a.tile_elems) : left;
    for (uint64_t l = l0 + threadIdx.x; l < l1; l += kLocalThreads) {
        const uint64_t e = l < j.head ? l : vecs * E + l;
        Acc acc = N::up(((const T *)(a.in[0] + j.off))[e]);
        for (int q = 1; q < a.p; ++q) acc = red_op<OP>(acc, N::up(((const T *)(a.in[q] + j.off))[e]));
        const T r = N::down(acc);
        for (uint32_t m = j.mask; m; m &= m - 1) ((T *)a.out[__ffs(m) - 1])[e] = r;
    }
}

// Some buffer starts inside an element: no vectors, every element byte by byte.  A kernel of its own, because the byte accesses
// cost the one above registers (bf16, sources merged from aligned vectors: 349 us became 400 us for ReduceScatter of 16 MiB blocks
// over eight ranks).
template <class T> union ElemBytes { T e; uint8_t b[sizeof(T)]; __device__ ElemBytes() {} };
template <class T> __device__ __forceinline__ T ld_bytes(const uint8_t *p)
{
    ElemBytes<T> v;
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); ++i) v.b[i] = p[i];
    return v.e;
}
template <class T, int OP>
__global__ void __launch_bounds__(kLocalThreads) local_reduce_bytes_kernel(const __grid_constant__ LocalReduce a)
{
    using N = DNum<T>;
    pdl_trigger();
    int ji = 0;
    while (ji + 1 < a.njobs && blockIdx.x >= a.job[ji + 1].tile0) ++ji;
    const LocalReduceJob &j = a.job[ji];
    const uint64_t e0 = (uint64_t)(blockIdx.x - j.tile0) * a.tile_elems, e1 = min(j.count, e0 + a.tile_elems);
    pdl_wait();
    for (uint64_t e = e0 + threadIdx.x; e < e1; e += kLocalThreads) {
        const uint64_t b = e * sizeof(T);
        typename N::Acc acc = N::up(ld_bytes<T>(a.in[0] + j.off + b));
        for (int q = 1; q < a.p; ++q) acc = red_op<OP>(acc, N::up(ld_bytes<T>(a.in[q] + j.off + b)));
        ElemBytes<T> r;
        r.e = N::down(acc);
        for (uint32_t m = j.mask; m; m &= m - 1) {
            uint8_t *d = a.out[__ffs(m) - 1] + b;
#pragma unroll
            for (int i = 0; i < (int)sizeof(T); ++i) d[i] = r.b[i];
        }
    }
}

// Defines local_kernel_<name>(op, p, wide, bytes): the reduction kernel for element type T; wide: vectors of 32 bytes; bytes: some
// buffer starts inside an element.
#define HCCLB_LOCAL_BATCH(T, OP)                                                                                                            \
    (bytes ? (const void *)local_reduce_bytes_kernel<T, OP>                                                                                 \
     : wide ? (p <= 2 ? (const void *)local_reduce_kernel<T, OP, 2, 32> : p <= 4 ? (const void *)local_reduce_kernel<T, OP, 4, 32>           \
                                                                               : (const void *)local_reduce_kernel<T, OP, 8, 32>)          \
          : (p <= 2 ? (const void *)local_reduce_kernel<T, OP, 2, 16> : p <= 4 ? (const void *)local_reduce_kernel<T, OP, 4, 16>           \
                                                                               : (const void *)local_reduce_kernel<T, OP, 8, 16>))
#define HCCLB_INSTANTIATE_LOCAL(T, name)                                              \
    const void *local_kernel_##name(int op, int p, bool wide, bool bytes)             \
    {                                                                                 \
        switch (op) {                                                                 \
            case HCCL_REDUCE_SUM: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_SUM);       \
            case HCCL_REDUCE_PROD: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_PROD);     \
            case HCCL_REDUCE_MAX: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_MAX);       \
            default: return HCCLB_LOCAL_BATCH(T, HCCL_REDUCE_MIN);                    \
        }                                                                             \
    }

}  // namespace hcclb
