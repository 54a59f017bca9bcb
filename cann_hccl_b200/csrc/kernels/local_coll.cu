// Direct collectives on one GPU (see local_coll.h): the copy kernel (AllGather, Broadcast, Scatter, Gather, AlltoAll, every
// collective of a single rank) and the launchers of both kernels.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include "kernels/local_coll.cuh"

namespace hcclb {

const void *local_kernel_i8(int op, int p, bool wide, bool bytes);
const void *local_kernel_u8(int op, int p, bool wide, bool bytes);
const void *local_kernel_i16(int op, int p, bool wide, bool bytes);
const void *local_kernel_u16(int op, int p, bool wide, bool bytes);
const void *local_kernel_i32(int op, int p, bool wide, bool bytes);
const void *local_kernel_u32(int op, int p, bool wide, bool bytes);
const void *local_kernel_i64(int op, int p, bool wide, bool bytes);
const void *local_kernel_u64(int op, int p, bool wide, bool bytes);
const void *local_kernel_f32(int op, int p, bool wide, bool bytes);
const void *local_kernel_f64(int op, int p, bool wide, bool bytes);
const void *local_kernel_f16(int op, int p, bool wide, bool bytes);
const void *local_kernel_bf16(int op, int p, bool wide, bool bytes);

static const void *local_kernel_for(int dtype, int op, int p, bool wide, bool bytes)
{
    switch (dtype) {
        case HCCL_DATA_TYPE_INT8: return local_kernel_i8(op, p, wide, bytes);
        case HCCL_DATA_TYPE_UINT8: return local_kernel_u8(op, p, wide, bytes);
        case HCCL_DATA_TYPE_INT16: return local_kernel_i16(op, p, wide, bytes);
        case HCCL_DATA_TYPE_UINT16: return local_kernel_u16(op, p, wide, bytes);
        case HCCL_DATA_TYPE_INT32: return local_kernel_i32(op, p, wide, bytes);
        case HCCL_DATA_TYPE_UINT32: return local_kernel_u32(op, p, wide, bytes);
        case HCCL_DATA_TYPE_INT64: return local_kernel_i64(op, p, wide, bytes);
        case HCCL_DATA_TYPE_UINT64: return local_kernel_u64(op, p, wide, bytes);
        case HCCL_DATA_TYPE_FP32: return local_kernel_f32(op, p, wide, bytes);
        case HCCL_DATA_TYPE_FP64: return local_kernel_f64(op, p, wide, bytes);
        case HCCL_DATA_TYPE_FP16: return local_kernel_f16(op, p, wide, bytes);
        case HCCL_DATA_TYPE_BFP16: return local_kernel_bf16(op, p, wide, bytes);
        default: return nullptr;
    }
}

namespace {

constexpr int kCopyBytes = 128;  // per thread and tile, in one round of loads

template <int JOBS> struct LocalCopyArgs {
    uint8_t *out[kMaxRanks];
    LocalCopyJob job[JOBS];
    int njobs;
    uint32_t tile_bytes;
};

template <int VB, bool SHIFT>
__device__ __forceinline__ void local_copy_tile(const uint8_t *src, uint8_t *const (&out)[kMaxRanks], uint32_t mask, uint64_t doff, uint64_t v0, uint64_t v1)
{
    constexpr int U = kCopyBytes / VB / (SHIFT ? 2 : 1);
#pragma unroll 1
    for (uint64_t i = v0 + threadIdx.x; i < v1; i += (uint64_t)U * kLocalThreads) {
        Vec<VB> x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t v = i + (uint64_t)u * kLocalThreads;
            if (v < v1) {
                if constexpr (SHIFT) x[u].u = ld_shifted(src + v * VB);
                else x[u] = ld_vec(src + v * VB, (Vec<VB> *)nullptr);
            }
        }
        for (uint32_t m = mask; m; m &= m - 1) {
            uint8_t *d = out[__ffs(m) - 1] + doff;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t v = i + (uint64_t)u * kLocalThreads;
                if (v < v1) st_vec(d + v * VB, x[u]);
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
    // the launcher gives a job only destinations that share their alignment (of 32 bytes)
    const uint8_t *d0 = a.out[__ffs(mask) - 1] + doff;
    uint64_t head = (32 - ((uintptr_t)d0 & 31)) & 31;
    if (head > n) head = n;
    const uint64_t body = (n - head) & ~31ull;
    pdl_wait();
    const uint64_t b0 = (uint64_t)tile * a.tile_bytes, b1 = b0 + a.tile_bytes < body ? b0 + a.tile_bytes : body;
    if (b0 < body) {
        const uint32_t s = (uint32_t)((uintptr_t)src + head) & 31;
        if (s == 0) local_copy_tile<32, false>(src + head, a.out, mask, doff + head, b0 / 32, b1 / 32);
        else if (s == 16) local_copy_tile<16, false>(src + head, a.out, mask, doff + head, b0 / 16, b1 / 16);
        else local_copy_tile<16, true>(src + head, a.out, mask, doff + head, b0 / 16, b1 / 16);
    } else {  // the job's last tile: what lies outside the body, below 64 bytes
        const uint32_t left = (uint32_t)(n - body);
        if (threadIdx.x < left) {
            const uint64_t b = threadIdx.x < head ? threadIdx.x : body + threadIdx.x;
            const uint8_t v = src[b];
            for (uint32_t m = mask; m; m &= m - 1) (a.out[__ffs(m) - 1] + doff)[b] = v;
        }
    }
}

// Bytes per tile: `full` where that still leaves a few CTAs for every SM, down to one load per thread where it does not (a small
// message is latency-bound: more CTAs with one load each finish sooner; 8 MiB copied with four loads per thread takes 4.6 us,
// with one 2.6 us).
uint32_t tile_bytes_for(uint64_t total, uint32_t full, uint32_t least)
{
    uint32_t t = full;
    while (t > least && total / t < 8 * 148) t >>= 1;
    return t;
}

template <int JOBS> HcclResult launch_copy(LocalCopy &c, uint32_t tile_bytes, unsigned tiles, void *stream)
{
    LocalCopyArgs<JOBS> a;
    memcpy(a.out, c.out, sizeof(a.out));
    memcpy(a.job, c.job, sizeof(LocalCopyJob) * c.njobs);
    a.njobs = c.njobs;
    a.tile_bytes = tile_bytes;
    return launch_pdl((const void *)local_copy_kernel<JOBS>, dim3(tiles), kLocalThreads, 0, &a, stream, "direct copy");
}

}  // namespace

HcclResult launch_local_copy(LocalCopy &c, void *stream)
{
    if (c.njobs < 0 || c.njobs > kLocalMaxJobs) return HCCL_E_PARA;
    uint64_t total = 0;
    for (int j = 0; j < c.njobs; ++j) total += c.job[j].bytes;
    const uint32_t tb = tile_bytes_for(total, kCopyBytes * kLocalThreads, 32 * kLocalThreads);
    uint64_t tiles = 0;
    int n = 0;
    for (int j = 0; j < c.njobs; ++j) {
        LocalCopyJob &job = c.job[j];
        if (!job.bytes || !job.mask) continue;
        const uint64_t head = std::min<uint64_t>(job.bytes, (32 - (((uintptr_t)c.out[__builtin_ctz(job.mask)] + job.doff) & 31)) & 31);
        const uint64_t body = (job.bytes - head) & ~31ull;
        job.tile0 = (uint32_t)tiles;
        tiles += ceil_div_u64(body, tb) + (body < job.bytes ? 1 : 0);
        c.job[n++] = job;
    }
    c.njobs = n;
    if (tiles == 0) return HCCL_SUCCESS;
    if (tiles > 0x7fffffffu) return HCCL_E_PARA;
    // the job table travels as a kernel argument: the smaller forms keep the launch of the common cases cheap
    if (n <= kMaxRanks) return launch_copy<kMaxRanks>(c, tb, (unsigned)tiles, stream);
    if (n <= 4 * kMaxRanks) return launch_copy<4 * kMaxRanks>(c, tb, (unsigned)tiles, stream);
    return launch_copy<kLocalMaxJobs>(c, tb, (unsigned)tiles, stream);
}

// How a job lies over vectors of vb bytes: outputs first, the sources as they then come.
static uint32_t layout_of(const LocalReduce &r, LocalReduceJob &j, uint32_t es, uint32_t vb)
{
    uint32_t differ = 0, shift = 0;
    const uintptr_t d0 = (uintptr_t)r.out[__builtin_ctz(j.mask)];
    for (uint32_t m = j.mask; m; m &= m - 1) differ |= (uint32_t)((uintptr_t)r.out[__builtin_ctz(m)] ^ d0) & (vb - 1);
    j.head = (uint32_t)std::min<uint64_t>(j.count, ((vb - (d0 & (vb - 1))) & (vb - 1)) / es);
    j.nvec = (j.count - j.head) * es / vb;
    for (int q = 0; q < r.p; ++q) shift |= (uint32_t)((uintptr_t)r.in[q] + j.off + (uint64_t)j.head * es) & (vb - 1);
    return differ ? LOCAL_SCALAR : (shift ? LOCAL_SHIFTED : LOCAL_ALIGNED);
}

HcclResult launch_local_reduce(LocalReduce &r, int dtype, int redop, void *stream)
{
    const uint32_t es = (uint32_t)dtype_size(dtype);
    if (!es || r.p < 1 || r.p > kMaxRanks || r.njobs < 1 || r.njobs > kMaxRanks) return HCCL_E_PARA;
    int n = 0;
    for (int j = 0; j < r.njobs; ++j)
        if (r.job[j].count && r.job[j].mask) r.job[n++] = r.job[j];
    r.njobs = n;
    if (n == 0) return HCCL_SUCCESS;
    // 32-byte vectors where every address of every job allows them (ReduceScatter of 4 MiB blocks over eight ranks: 43.7 us with
    // them, 46.2 us with 16 bytes), and one width for the whole launch
    uintptr_t bits = 0;  // of all addresses, to see whether each is a multiple of the element's size
    for (int q = 0; q < r.p; ++q) {
        bits |= (uintptr_t)r.in[q];
        for (int j = 0; j < n; ++j)
            if ((r.job[j].mask >> q) & 1u) bits |= (uintptr_t)r.out[q];
    }
    const bool bytes = (bits & (es - 1)) != 0;
    bool wide = !bytes;
    for (int j = 0; j < n && wide; ++j) wide = (r.job[j].layout = layout_of(r, r.job[j], es, 32)) == LOCAL_ALIGNED;
    const uint32_t vb = wide ? 32 : 16;
    uint64_t total = 0;
    for (int j = 0; j < n; ++j) {
        if (!wide) r.job[j].layout = bytes ? LOCAL_SCALAR : layout_of(r, r.job[j], es, 16);
        total += r.job[j].count * es;
    }
    const uint32_t full = r.p <= 2 ? 64 : (r.p <= 4 ? 32 : vb);  // bytes per thread (kReduceVecs)
    r.tile_vecs = tile_bytes_for(total, full * kLocalThreads, vb * kLocalThreads) / vb;
    // one by one: as many elements as the vectors of a tile hold, down to one per thread while that is not two CTAs for every SM
    // (2 KiB of int8 over eight ranks, outputs of different alignments: 16 elements per thread 17.9 us, one 4.7 us; 1 MiB over two
    // ranks, 512 CTAs of 16 elements per thread 7.9 us, 2048 CTAs of four 8.9 us)
    r.tile_elems = r.tile_vecs * (vb / es);
    while (r.tile_elems > kLocalThreads && total / es / r.tile_elems < 2 * 148) r.tile_elems >>= 1;
    uint64_t tiles = 0, same = 0;
    bool uniform = true;
    for (int j = 0; j < n; ++j) {
        LocalReduceJob &job = r.job[j];
        job.tile0 = (uint32_t)tiles;
        const uint64_t t = job.layout == LOCAL_SCALAR ? ceil_div_u64(job.count, r.tile_elems)
                                                      : ceil_div_u64(job.nvec, r.tile_vecs) + (job.nvec * (vb / es) < job.count ? 1 : 0);
        if (j == 0) same = t;
        uniform = uniform && t == same;
        tiles += t;
    }
    r.uniform = uniform ? (uint32_t)same : 0;
    if (tiles > 0x7fffffffu) return HCCL_E_PARA;
    const void *fn = local_kernel_for(dtype, redop, r.p, wide, bytes);
    if (!fn) return HCCL_E_PARA;
    return launch_pdl(fn, dim3((unsigned)tiles), kLocalThreads, 0, &r, stream, "direct reduction");
}

}  // namespace hcclb
