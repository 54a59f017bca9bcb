// tcgen05 GEMM without communication (see gemm_local.h): bf16 operands, fp32 accumulation in TMEM, bf16 results, optional
// activation on the fp32 sums.  One persistent CTA per SM:
//   warp 0     TMA producer: 128-byte-swizzled stages of A and B (cp.async.bulk.tensor, never multicast);
//   warp 1     one thread issues tcgen05.mma into one of two 256-column accumulators;
//   warps 2-9  drain the other accumulator: two warps per TMEM lane quarter, 128 columns each, full 32-byte sectors per store.
// Pair form: a cluster of two CTAs shares a 256 x 256 tile (cta_group::2), each CTA loading its 128 rows of A and half of the
// tile's B rows; single form: one CTA per 128 x 256 tile, where the rows are an odd number of 128-row blocks.
//
// Few tiles (a decode batch: one row block, deep K): a cluster of S units shares a tile along K (kSplit = S).  Each unit leaves
// its fp32 sums in its shared memory, the cluster meets, and unit s adds columns [256 s / S, 256 (s + 1) / S) over the S copies
// through distributed shared memory, in K order.  No scratch, no atomics, the same bits every time.
//
// Bound: tensor cores at the clock that the power cap leaves (prefill), HBM (decode: the weights are read once).  Measured on a
// B200, MLP block hidden 8192, FFN 28672, SiLU, against the communicating kernels with the activation as three passes over
// fp32 copies: 8192 tokens on one rank 8002 -> 6004 us; 2048 tokens over four ranks in one process 2270 -> 1633 us; 128 tokens
// 287 -> 189 us (down projection, 32 tiles split in four: 178 -> 93 us).  Tried and left out: cutting the last wave along K
// over all units with fp32 shares in global memory (512 x 8192 x 28672: 210 -> 268 us; units at different k share nothing in
// L2, and under the power cap an idle last wave costs little).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include "common/env.h"
#include "common/log.h"
#include "core/device_api.h"
#include "kernels/fused/gemm_local.h"
#include "kernels/fused/tc05.cuh"
#include "kernels/fused/tp_gemm.h"
#include "kernels/pdl.cuh"

namespace hcclb {

namespace {
using namespace tc05;

constexpr int kGemmThreads = 320, kEpiThreads = 256;
constexpr uint32_t kABytes = BM * BK * 2, kBBytes = BN * BK * 2;
constexpr uint32_t kTmemCols = 512;
template <bool kPair> constexpr uint32_t kStageBytes = kABytes + (kPair ? kBBytes / 2 : kBBytes);
template <bool kPair> constexpr int kStages = kPair ? 7 : 4;
constexpr int kMinShare = 8;  // k steps of 64 that a unit of a split tile has at least
constexpr int kMaxSplit = 4;

struct alignas(64) GemmParams {
    CUtensorMap tmA[kGemmShards], tmB[kGemmShards];
    __nv_bfloat16 *C[kGemmShards];
    int form, act;
    int um_tiles, n_tiles; // row units (128 rows, pair: 256) and 256-column tiles
    int shard_m, shard_n;  // rows of a row shard, columns of a column shard
    int k_seg, k_iters;    // k steps of one operand pair, of a whole tile
    int ldc, panel;        // panel: n tiles that are walked together
    int units;
    int wide;              // outputs are 32-byte aligned
    DevStatus *status;     // host-mapped, may be null
};

template <bool kPair> struct GemmShared {
    alignas(1024) uint8_t tiles[kStages<kPair> * kStageBytes<kPair>];
    alignas(8) uint64_t full_bar[kStages<kPair>];
    uint64_t empty_bar[kStages<kPair>];
    uint64_t tmem_full[2], tmem_empty[2];
    uint32_t tmem_base, fail;
};

// Panels of `panel` n tiles, m inside a panel, n fastest: the tiles that run together form a block of about panel x
// (units / panel) tiles, near-square in bytes, whose operands share L2.
__device__ __forceinline__ void tile_at(const GemmParams &P, int t, int &um, int &nt)
{
    const int per = P.um_tiles * P.panel, pn = t / per, n0 = pn * P.panel, w = min(P.panel, P.n_tiles - n0), r = t - pn * per;
    um = r / w;
    nt = n0 + r - um * w;
}

__device__ __forceinline__ void st_global_32B(void *p, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// 32 consecutive results of one row; 32-byte sectors where the output allows them
template <int ACT> __device__ __forceinline__ void store_row32(__nv_bfloat16 *dst, const float (&v)[32], bool wide)
{
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            o[i] = pack_bf16(__float_as_uint(activate<ACT>(v[16 * g + 2 * i])), __float_as_uint(activate<ACT>(v[16 * g + 2 * i + 1])));
        if (wide) st_global_32B(dst + 16 * g, o);
        else {
            ((uint4 *)(dst + 16 * g))[0] = make_uint4(o[0], o[1], o[2], o[3]);
            ((uint4 *)(dst + 16 * g))[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
    }
}
__device__ __forceinline__ void store_row32(__nv_bfloat16 *dst, const float (&v)[32], bool wide, int act)
{
    if (act == GEMM_ACT_SILU) store_row32<GEMM_ACT_SILU>(dst, v, wide);
    else if (act == GEMM_ACT_GELU) store_row32<GEMM_ACT_GELU>(dst, v, wide);
    else store_row32<GEMM_ACT_NONE>(dst, v, wide);
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// address of (row, column) of the tile space in its rank's output
__device__ __forceinline__ __nv_bfloat16 *out_row(const GemmParams &P, int row, int col)
{
    if (P.form == GEMM_GATHER) return P.C[col / P.shard_n] + (int64_t)row * P.ldc + col % P.shard_n;
    return P.C[row / P.shard_m] + (int64_t)(row % P.shard_m) * P.ldc + col;
}

template <bool kPair, int kSplit>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_local_kernel(const __grid_constant__ GemmParams P)
{
    extern __shared__ uint8_t smem_raw[];
    using Shared = GemmShared<kPair>;
    Shared &S = *(Shared *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int kSt = kStages<kPair>, kCtas = kPair ? 2 : 1;
    constexpr uint32_t kStB = kStageBytes<kPair>;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr bool kCluster = kPair || kSplit > 1;
    const uint32_t rank = kCluster ? cluster_ctarank() : 0u, cta_r = kPair ? rank & 1 : 0u, leader = rank - cta_r;
    const int unit = (int)blockIdx.x / (kCtas * kSplit), total = P.um_tiles * P.n_tiles;
    const int share = (int)rank / kCtas;  // of the tile's k steps
    const int k0 = P.k_iters * share / kSplit, k1 = P.k_iters * (share + 1) / kSplit;
    volatile uint32_t *fail = &S.fail;
    const int q4 = warp & 3, half = (warp - 2) >> 2, rl = q4 * 32 + lane;  // epilogue warps: TMEM lane quarter (a warp reaches its own only), column half, row
    float4 *sums = (float4 *)S.tiles;                                      // split tiles: [column / 4][row]
    static_assert(BM * BN * sizeof(float) <= sizeof(S.tiles), "the sums of a share fit the stages");

    pdl_trigger();
    if (threadIdx.x == 0) {
        S.fail = 0;
        for (int i = 0; i < kSt; ++i) { mbar_init(&S.full_bar[i], 1); mbar_init(&S.empty_bar[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&S.tmem_full[i], 1); mbar_init(&S.tmem_empty[i], kCtas * kEpiThreads / 32); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (kPair) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (kCluster) cluster_sync_all();  // the other CTA's barriers and TMEM are ready before anything of mine reaches them
    tc_fence_after();
    const uint32_t tmem_base = S.tmem_base;
    pdl_wait();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            uint32_t it = 0;
            for (int t = unit; t < total && !*fail; t += P.units) {
                int um, nt;
                tile_at(P, t, um, nt);
                int arow = (um * kCtas + (int)cta_r) * BM, brow = nt * BN + (kPair ? (int)cta_r * (BN / 2) : 0);
                const CUtensorMap *ma = &P.tmA[0], *mb = &P.tmB[0];
                if (P.form == GEMM_GATHER) {
                    const int sm = arow / P.shard_m, sn = brow / P.shard_n;
                    ma = &P.tmA[sm]; arow -= sm * P.shard_m;
                    mb = &P.tmB[sn]; brow -= sn * P.shard_n;
                }
                int kx = k0, seg = 0;
                if (P.form == GEMM_REDUCE) { seg = kx / P.k_seg; kx -= seg * P.k_seg; ma = &P.tmA[seg]; mb = &P.tmB[seg]; }
                for (int k = k0; k < k1; ++k, ++it, ++kx) {
                    if (kx == P.k_seg) { kx = 0; ++seg; ma = &P.tmA[seg]; mb = &P.tmB[seg]; }
                    const uint32_t s = it % kSt, ph = (it / kSt) & 1;
                    if (!mbar_wait_t<kPair>(&S.empty_bar[s], ph ^ 1, fail)) break;
                    uint8_t *sa = S.tiles + (size_t)s * kStB, *sb = sa + kABytes;
                    if (kPair) {  // the bytes of both CTAs' loads are counted on the leader's barrier
                        if (cta_r == 0) mbar_expect_tx(&S.full_bar[s], 2 * kStB);
                        const uint32_t full = mapa_u32(smem_u32(&S.full_bar[s]), leader);
                        tma_load_2d_pair(sa, ma, full, kx * BK, arow);
                        tma_load_2d_pair(sb, mb, full, kx * BK, brow);
                    } else {
                        mbar_expect_tx(&S.full_bar[s], kStB);
                        tma_load_2d(sa, ma, &S.full_bar[s], kx * BK, arow);
                        tma_load_2d(sb, mb, &S.full_bar[s], kx * BK, brow);
                    }
                }
            }
        }
        if (*fail)  // loads in flight land before the CTA lets go of its shared memory
            for (int i = 0; i < 200; ++i) __nanosleep(1000);
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (pair: the leader, for both CTAs)
        if (cta_r == 0 && elect_one()) {
            uint32_t it = 0, n = 0;
            const uint16_t both = (uint16_t)(3u << leader);
            for (int t = unit; t < total && !*fail; t += P.units, ++n) {
                const uint32_t buf = n & 1, use = n >> 1, d = tmem_base + buf * BN;
                if (!mbar_wait_t<kPair>(&S.tmem_empty[buf], (use & 1) ^ 1, fail)) break;
                tc_fence_after();
                for (int k = k0; k < k1; ++k, ++it) {
                    const uint32_t s = it % kSt, ph = (it / kSt) & 1;
                    if (!mbar_wait_t<kPair>(&S.full_bar[s], ph, fail)) break;
                    tc_fence_after();
                    const uint64_t da = make_smem_desc(S.tiles + (size_t)s * kStB), db = make_smem_desc(S.tiles + (size_t)s * kStB + kABytes);
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk) {  // 16 bf16 = 32 bytes along K inside the swizzle atom
                        if (kPair) umma_pair(d, da + (uint64_t)(2 * kk), db + (uint64_t)(2 * kk), k != k0 || kk != 0);
                        else umma(d, da + (uint64_t)(2 * kk), db + (uint64_t)(2 * kk), k != k0 || kk != 0);
                    }
                    if (kPair) umma_commit_pair(&S.empty_bar[s], both); else umma_commit(&S.empty_bar[s]);
                }
                if (kPair) umma_commit_pair(&S.tmem_full[buf], both); else umma_commit(&S.tmem_full[buf]);
            }
        }
    } else if (kSplit == 1) {
        // ------------------------------------------------------------------ epilogue
        uint32_t n = 0;
        for (int t = unit; t < total && !*fail; t += P.units, ++n) {
            int um, nt;
            tile_at(P, t, um, nt);
            __nv_bfloat16 *dst = out_row(P, (um * kCtas + (int)cta_r) * BM + rl, nt * BN + half * 128);
            const uint32_t buf = n & 1, use = n >> 1, taddr = tmem_base + buf * BN + half * 128 + ((uint32_t)(q4 * 32) << 16);
            if (!mbar_wait_t<kPair>(&S.tmem_full[buf], use & 1, fail)) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 128; c += 32) {
                uint32_t r[32];
                tmem_ld32(taddr + c, r);
                tmem_ld_wait();
                float v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
                store_row32(dst + c, v, P.wide, P.act);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (kPair) mbar_arrive_cluster(mapa_u32(smem_u32(&S.tmem_empty[buf]), leader)); else mbar_arrive(&S.tmem_empty[buf]);
            }
        }
    } else {
        // ------------------------------------------------------------------ one tile per cluster: this share's sums to shared memory
        // (every MMA and load of the share is over: the stages are free)
        if (mbar_wait_t<kPair>(&S.tmem_full[0], 0, fail)) {
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 128; c += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_base + half * 128 + c + ((uint32_t)(q4 * 32) << 16), r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    sums[(half * 32 + c / 4 + i) * BM + rl] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
            }
        }
    }
    if (kSplit > 1) {
        __syncwarp();
        cluster_sync_all();
        if (warp >= 2) {
            int um, nt;
            tile_at(P, unit, um, nt);
            constexpr int kCols = BN / kSplit / 2;  // per thread: half of this unit's columns
            const int col = share * (BN / kSplit) + half * kCols;
            __nv_bfloat16 *dst = out_row(P, (um * kCtas + (int)cta_r) * BM + rl, nt * BN + col);
#pragma unroll
            for (int c = 0; c < kCols; c += 32) {
                float4 x[kSplit][8];
#pragma unroll
                for (int q = 0; q < kSplit; ++q) {
                    const uint32_t base = mapa_u32(smem_u32(sums + ((col + c) / 4) * BM + rl), (uint32_t)(q * kCtas) + cta_r);
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[q][i] = ld_cluster_f4(base + (uint32_t)(i * BM * sizeof(float4)));
                }
                float v[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float4 t = x[0][i];
#pragma unroll
                    for (int q = 1; q < kSplit; ++q) { t.x += x[q][i].x; t.y += x[q][i].y; t.z += x[q][i].z; t.w += x[q][i].w; }
                    v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
                }
                store_row32(dst + c, v, P.wide, P.act);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (kCluster) cluster_sync_all();  // the leader's MMAs use both CTAs' stages and TMEM, its commits arrive on both; peers read `sums`
    if (warp == 1) {
        tc_fence_after();
        if (kPair) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
    if (threadIdx.x == 0 && *fail && P.status) {  // a bounded wait ran out: the result is not to be used
        P.status->step = 0; P.status->peer = -1; P.status->chan = blockIdx.x;
        __threadfence_system();
        *(volatile uint32_t *)&P.status->code = *fail;
    }
}

HcclResult encode_2d(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint32_t box_rows)
{
    const DriverApi &d = driver_api();
    if (!d.ok || !d.TensorMapEncodeTiled) return HCCL_E_DRV;
    cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, box_rows}, estr[2] = {1, 1};
    CUresult r = d.TensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { HLOG_ERROR("cuTensorMapEncodeTiled failed: %s", cu_err(r)); return HCCL_E_DRV; }
    return HCCL_SUCCESS;
}

template <bool kPair> size_t smem_bytes() { return sizeof(GemmShared<kPair>) + 1024; }

const void *kernel_of(bool pair, int split)
{
    if (pair) return split == 4 ? (const void *)gemm_local_kernel<true, 4> : split == 2 ? (const void *)gemm_local_kernel<true, 2> : (const void *)gemm_local_kernel<true, 1>;
    return split == 4 ? (const void *)gemm_local_kernel<false, 4> : split == 2 ? (const void *)gemm_local_kernel<false, 2> : (const void *)gemm_local_kernel<false, 1>;
}

// units[pair][split]: tiles that can be worked on at once (clusters of pair x split CTAs, each inside one GPC); 0: not known yet
struct DeviceShape { int units[2][kMaxSplit + 1] = {}; };

void set_cluster(cudaLaunchAttribute *a, int ctas)
{
    a->id = cudaLaunchAttributeClusterDimension;
    a->val.clusterDim.x = (unsigned)ctas; a->val.clusterDim.y = 1; a->val.clusterDim.z = 1;
}

// Asked once per device; sets the kernels' shared-memory limits on the way.
HcclResult device_shape(DeviceShape *out)
{
    static std::mutex mu;
    static DeviceShape known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return HCCL_E_RUNTIME;
    std::lock_guard<std::mutex> lk(mu);
    DeviceShape &d = known[dev];
    if (!d.units[0][1]) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        for (int pair = 0; pair < 2; ++pair)
            for (int split = kMaxSplit; split >= 1; split /= 2) {
                const void *fn = kernel_of(pair, split);
                const int ctas = (pair ? 2 : 1) * split;
                const size_t smem = pair ? smem_bytes<true>() : smem_bytes<false>();
                cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                int n = sms;
                if (e == cudaSuccess && ctas > 1) {
                    cudaLaunchConfig_t q;
                    memset(&q, 0, sizeof(q));
                    q.gridDim = dim3((unsigned)(sms / ctas * ctas)); q.blockDim = dim3(kGemmThreads); q.dynamicSmemBytes = smem;
                    cudaLaunchAttribute a[1];
                    set_cluster(a, ctas);
                    q.attrs = a; q.numAttrs = 1;
                    e = cudaOccupancyMaxActiveClusters(&n, fn, &q);
                }
                if (e != cudaSuccess || (split == 1 && n < 1)) { HLOG_ERROR("GEMM set-up failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
                if (!(pair == 0 && split == 1)) d.units[pair][split] = std::min(n, sms / ctas);
            }
        CHK_RET(tp_gemm_load());  // modules load on first use, which allocates: the allocation-free entry point finds its own loaded
        d.units[0][1] = sms;
    }
    *out = d;
    return HCCL_SUCCESS;
}

bool shape_ok(const GemmCall &c)
{
    const int shards = c.form == GEMM_PLAIN ? 1 : c.p;
    return c.p >= 1 && c.p <= kGemmShards && c.M > 0 && c.N > 0 && c.K > 0 && c.M % (BM * shards) == 0 && c.N % BN == 0 && c.K % BK == 0;
}

std::atomic<uint64_t> g_counts[2];

}  // namespace

void gemm_local_launch_counts(uint64_t *single, uint64_t *pair)
{
    *single = g_counts[0].load();
    *pair = g_counts[1].load();
}

HcclResult launch_gemm_local(const GemmCall &c, DevStatus *status, void *stream)
{
    if (!shape_ok(c)) {
        HLOG_ERROR("GEMM needs M %% %d == 0 per shard, N %% %d == 0, K %% %d == 0 (got %d x %d x %d, %d shards)", BM, BN, BK, c.M, c.N, c.K, c.p);
        return HCCL_E_PARA;
    }
    DeviceShape d;
    CHK_RET(device_shape(&d));
    const int na = c.form == GEMM_PLAIN ? 1 : c.p, rows = c.form == GEMM_PLAIN ? c.M : c.M / c.p;
    const bool pair = env_config().tp_gemm_pair && rows % (2 * BM) == 0;
    GemmParams P;
    memset(&P, 0, sizeof(P));
    P.um_tiles = c.M / (pair ? 2 * BM : BM);
    P.n_tiles = c.N / BN * (c.form == GEMM_GATHER ? c.p : 1);
    P.k_seg = c.K / BK;
    P.k_iters = P.k_seg * (c.form == GEMM_REDUCE ? c.p : 1);
    const int64_t tiles = (int64_t)P.um_tiles * P.n_tiles;
    // split along K while all tiles still fit the GPU at once and a unit keeps enough steps to be worth the meeting at the end
    int split = 1;
    while (split < kMaxSplit && tiles <= d.units[pair][2 * split] && P.k_iters / (2 * split) >= kMinShare) split *= 2;
    uintptr_t bits = 0;
    for (int i = 0; i < na; ++i) {
        if ((((uintptr_t)c.A[i]) | ((uintptr_t)c.B[i]) | ((uintptr_t)c.C[i])) & 15) return HCCL_E_PARA;
        CHK_RET(encode_2d(&P.tmA[i], c.A[i], (uint64_t)(c.form == GEMM_GATHER ? rows : c.M), (uint64_t)c.K, BM));
        CHK_RET(encode_2d(&P.tmB[i], c.B[i], (uint64_t)c.N, (uint64_t)c.K, pair ? BN / 2 : BN));
        P.C[i] = (__nv_bfloat16 *)c.C[i];
        bits |= (uintptr_t)c.C[i];
    }
    P.wide = (bits & 31) == 0;
    P.status = status;
    P.form = c.form; P.act = c.act;
    P.shard_m = rows;
    P.shard_n = c.N;
    P.ldc = c.N;
    // weights of a panel stay in L2 (40 MB of it) while the rows stream past, but a panel is never narrower than the square
    // block of tiles that run together: with K = 28672 two tiles would fill the 40 MB and every row of A crossed HBM 16 times
    P.panel = (int)std::min<int64_t>(P.n_tiles, std::max<int64_t>(8, (40ll << 20) / ((int64_t)BN * P.k_iters * BK * 2)));
    P.units = d.units[pair][split];
    const int ctas = (pair ? 2 : 1) * split;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(std::min<int64_t>(P.units, tiles) * ctas)); cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = pair ? smem_bytes<true>() : smem_bytes<false>();
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    set_cluster(&at[1], ctas);
    cfg.attrs = at; cfg.numAttrs = ctas > 1 ? 2 : 1;
    void *args[] = {&P};
    cudaError_t e = cudaLaunchKernelExC(&cfg, kernel_of(pair, split), args);
    if (e != cudaSuccess) { HLOG_ERROR("GEMM launch failed (clusters of %d): %s", ctas, cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    g_counts[pair ? 1 : 0]++;
    return HCCL_SUCCESS;
}

}  // namespace hcclb
