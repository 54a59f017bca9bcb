// Direct collectives on one GPU (see local_coll.h): the copy kernel (AllGather, Broadcast, Scatter, Gather, AlltoAll, every
// collective of a single rank) and the launchers of both kernels.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include "kernels/local_coll.cuh"

namespace hcclb {

const void *local_kernel_i8(int op, int p);
const void *local_kernel_u8(int op, int p);
const void *local_kernel_i16(int op, int p);
const void *local_kernel_u16(int op, int p);
const void *local_kernel_i32(int op, int p);
const void *local_kernel_u32(int op, int p);
const void *local_kernel_i64(int op, int p);
const void *local_kernel_u64(int op, int p);
const void *local_kernel_f32(int op, int p);
const void *local_kernel_f64(int op, int p);
const void *local_kernel_f16(int op, int p);
const void *local_kernel_bf16(int op, int p);

static const void *local_kernel_for(int dtype, int op, int p)
{
    switch (dtype) {
        case HCCL_DATA_TYPE_INT8: return local_kernel_i8(op, p);
        case HCCL_DATA_TYPE_UINT8: return local_kernel_u8(op, p);
        case HCCL_DATA_TYPE_INT16: return local_kernel_i16(op, p);
        case HCCL_DATA_TYPE_UINT16: return local_kernel_u16(op, p);
        case HCCL_DATA_TYPE_INT32: return local_kernel_i32(op, p);
        case HCCL_DATA_TYPE_UINT32: return local_kernel_u32(op, p);
        case HCCL_DATA_TYPE_INT64: return local_kernel_i64(op, p);
        case HCCL_DATA_TYPE_UINT64: return local_kernel_u64(op, p);
        case HCCL_DATA_TYPE_FP32: return local_kernel_f32(op, p);
        case HCCL_DATA_TYPE_FP64: return local_kernel_f64(op, p);
        case HCCL_DATA_TYPE_FP16: return local_kernel_f16(op, p);
        case HCCL_DATA_TYPE_BFP16: return local_kernel_bf16(op, p);
        default: return nullptr;
    }
}

namespace {

constexpr int kCopyVecs = 8;  // 16-byte vectors per thread and tile

template <int JOBS> struct LocalCopyArgs {
    uint8_t *out[kMaxRanks];
    LocalCopyJob job[JOBS];
    int njobs;
    uint32_t tile_vecs;
};

template <int U, bool SHIFT>
__device__ __forceinline__ void local_copy_tile(const uint8_t *src, uint8_t *const (&out)[kMaxRanks], uint32_t mask, uint64_t doff, uint64_t v0, uint64_t v1)
{
    for (uint64_t i = v0 + threadIdx.x; i < v1; i += (uint64_t)U * kLocalThreads) {
        uint4 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t v = i + (uint64_t)u * kLocalThreads;
            if (v < v1) x[u] = SHIFT ? ld_shifted(src + (v << 4)) : ld_stream((const uint4 *)(src + (v << 4)));
        }
        for (uint32_t m = mask; m; m &= m - 1) {
            uint8_t *d = out[__ffs(m) - 1] + doff;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t v = i + (uint64_t)u * kLocalThreads;
                if (v < v1) *(uint4 *)(d + (v << 4)) = x[u];
            }
        }
    }
}

template <int JOBS>
__global__ void __launch_bounds__(kLocalThreads) local_copy_kernel(const __grid_constant__ LocalCopyArgs<JOBS> a)
{
    pdl_trigger();
    int lo = 0;  // the last job that starts at or before this tile
    for (int hi = a.njobs; hi - lo > 1;) {
        const int mid = (lo + hi) >> 1;
        if (a.job[mid].tile0 <= blockIdx.x) lo = mid; else hi = mid;
    }
    const LocalCopyJob &j = a.job[lo];
    const uint32_t tile = blockIdx.x - j.tile0, mask = j.mask;
    const uint64_t n = j.bytes, doff = j.doff;
    const uint8_t *src = j.src;
    // the launcher gives a job only destinations that share their alignment
    uint64_t head = (16 - (((uintptr_t)a.out[__ffs(mask) - 1] + doff) & 15)) & 15;
    if (head > n) head = n;
    const uint64_t nvec = (n - head) >> 4;
    pdl_wait();
    const uint64_t v0 = (uint64_t)tile * a.tile_vecs, v1 = v0 + a.tile_vecs < nvec ? v0 + a.tile_vecs : nvec;
    if (v0 < nvec) {
        if ((((uintptr_t)src + head) & 15) == 0) local_copy_tile<kCopyVecs, false>(src + head, a.out, mask, doff + head, v0, v1);
        else local_copy_tile<kCopyVecs / 2, true>(src + head, a.out, mask, doff + head, v0, v1);
    }
    if (tile == 0) {
        const uint32_t left = (uint32_t)(n - (nvec << 4));  // below 31 bytes
        if (threadIdx.x < left) {
            const uint64_t b = threadIdx.x < head ? threadIdx.x : (nvec << 4) + threadIdx.x;
            const uint8_t v = src[b];
            for (uint32_t m = mask; m; m &= m - 1) (a.out[__ffs(m) - 1] + doff)[b] = v;
        }
    }
}

// Vectors per tile: full unrolling where that still leaves a few CTAs for every SM, one vector per thread where it does not
// (a small message is latency-bound: more CTAs with one load each finish sooner than fewer with many).
uint32_t tile_vecs_for(uint64_t total_vecs, uint32_t full)
{
    uint32_t t = full * kLocalThreads;
    while (t > kLocalThreads && total_vecs / t < 4 * 148) t >>= 1;
    return t;
}

template <int JOBS> HcclResult launch_copy(LocalCopy &c, uint32_t tile_vecs, unsigned tiles, void *stream)
{
    LocalCopyArgs<JOBS> a;
    memcpy(a.out, c.out, sizeof(a.out));
    memcpy(a.job, c.job, sizeof(LocalCopyJob) * c.njobs);
    a.njobs = c.njobs;
    a.tile_vecs = tile_vecs;
    return launch_pdl((const void *)local_copy_kernel<JOBS>, dim3(tiles), kLocalThreads, 0, &a, stream, "direct copy");
}

}  // namespace

HcclResult launch_local_copy(LocalCopy &c, void *stream)
{
    if (c.njobs < 0 || c.njobs > kLocalMaxJobs) return HCCL_E_PARA;
    uint64_t vecs = 0;
    for (int j = 0; j < c.njobs; ++j) vecs += c.job[j].bytes >> 4;
    const uint32_t tv = tile_vecs_for(vecs, kCopyVecs);
    uint64_t tiles = 0;
    int n = 0;
    for (int j = 0; j < c.njobs; ++j) {
        if (!c.job[j].bytes || !c.job[j].mask) continue;
        c.job[n] = c.job[j];
        c.job[n++].tile0 = (uint32_t)tiles;
        tiles += std::max<uint64_t>(1, ceil_div_u64(c.job[j].bytes >> 4, tv));
    }
    c.njobs = n;
    if (tiles == 0) return HCCL_SUCCESS;
    if (tiles > 0x7fffffffu) return HCCL_E_PARA;
    // the job table travels as a kernel argument: the smaller forms keep the launch of the common cases cheap
    if (n <= kMaxRanks) return launch_copy<kMaxRanks>(c, tv, (unsigned)tiles, stream);
    if (n <= 4 * kMaxRanks) return launch_copy<4 * kMaxRanks>(c, tv, (unsigned)tiles, stream);
    return launch_copy<kLocalMaxJobs>(c, tv, (unsigned)tiles, stream);
}

HcclResult launch_local_reduce(LocalReduce &r, int dtype, int redop, void *stream)
{
    const int es = dtype_size(dtype);
    const void *fn = local_kernel_for(dtype, redop, r.p);
    if (!fn || r.p < 1 || r.p > kMaxRanks || r.njobs < 1 || r.njobs > kMaxRanks) return HCCL_E_PARA;
    uint64_t vecs = 0;
    for (int j = 0; j < r.njobs; ++j) vecs += r.count[j] * es >> 4;
    const uint32_t tv = r.tile_vecs = tile_vecs_for(vecs, r.p <= 2 ? 4 : (r.p <= 4 ? 2 : 1));
    uint64_t tiles = 0;
    int n = 0;
    for (int j = 0; j < r.njobs; ++j) {
        if (!r.count[j] || !r.mask[j]) continue;
        r.off[n] = r.off[j]; r.count[n] = r.count[j]; r.mask[n] = r.mask[j];
        r.tile0[n++] = (uint32_t)tiles;
        tiles += std::max<uint64_t>(1, ceil_div_u64(r.count[j] * es >> 4, tv));
    }
    r.tile0[n] = (uint32_t)tiles;
    r.njobs = n;
    if (tiles == 0) return HCCL_SUCCESS;
    if (tiles > 0x7fffffffu) return HCCL_E_PARA;
    return launch_pdl(fn, dim3((unsigned)tiles), kLocalThreads, 0, &r, stream, "direct reduction");
}

}  // namespace hcclb
