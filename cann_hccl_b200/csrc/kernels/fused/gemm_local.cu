// tcgen05 GEMM without communication (see gemm_local.h): bf16 operands, fp32 accumulation in TMEM, bf16 results, optional
// activation on the fp32 sums.  One persistent CTA per SM:
//   warp 0     TMA producer: 128-byte-swizzled stages of A and B (cp.async.bulk.tensor, never multicast);
//   warp 1     one thread issues tcgen05.mma into one of two accumulators of up to 256 columns;
//   warps 2-9  drain the other accumulator: two warps per TMEM lane quarter, half of the columns each, full 32-byte sectors per store.
// Pair form: a cluster of two CTAs shares a tile of 256 rows (cta_group::2), each CTA loading its 128 rows of A and half of the
// tile's B rows; single form: one CTA per 128 rows.  The two row blocks of a pair may belong to different ranks, and with an odd
// number of them the last pair computes one block of zeros.  A tile has 64 to 256 columns: the width, the form and the split
// follow from the shape (tiling_ns), so that the tiles fill whole waves of the GPU.
//
// Few tiles (a decode batch: one row block, deep K): a cluster of S units shares a tile along K (kSplit).  Each unit leaves
// its fp32 sums in its shared memory, the cluster meets, and the units take groups of 16 columns in turn, adding the S copies
// through distributed shared memory, in K order.  No scratch, no atomics, the same bits every time.
//
// Bound: tensor cores at the clock that the power cap leaves (prefill), HBM (decode: the weights are read once).
// Tried and left out: cutting the last wave along K over all units with fp32 shares in global memory (512 x 8192 x 28672:
// 210 -> 268 us; units at different k share nothing in L2, and under the power cap an idle last wave costs little).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include "common/env.h"
#include "common/log.h"
#include "kernels/fused/gemm_local.h"
#include "kernels/fused/tc05.cuh"
#include "kernels/fused/tensor_map.h"
#include "kernels/fused/tp_gemm.h"
#include "kernels/pdl.cuh"

namespace hcclb {

namespace {
using namespace tc05;

constexpr int kGemmThreads = 320, kEpiThreads = 256;
constexpr uint32_t kABytes = BM * BK * 2, kStageSpace = 7 * 32768;  // seven stages of the widest pair tile
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxStages = 8;
constexpr int kMinShare = 4;                       // k steps of 64 that a unit of a split tile has at least
constexpr int kMaxCluster = 8;                     // CTAs that share a tile at most
constexpr int kMinCols = 64, kMaxCols = BN;

struct alignas(64) GemmParams {
    CUtensorMap tmA[kGemmShards], tmB[kGemmShards];
    __nv_bfloat16 *C[kGemmShards];
    int form, act;
    int cols;                        // columns of a tile: multiple of 16, pair: of 32
    int um_tiles, n_tiles, shard_tiles;  // row units (128 rows, pair: 256), column tiles, column tiles of one shard (the last may be narrower)
    int rows, shards;                // rows of the tile space (pair: the last unit may be half outside), shards of A (gather)
    int shard_m, shard_n;            // rows of a row shard, columns of a column shard
    int k_seg, k_iters;              // k steps of one operand pair, of a whole tile
    int ldc, panel;                  // panel: n tiles that are walked together
    int units, split;                // split: units that share a tile along K
    int stages;
    uint32_t stage_bytes, idesc;
    int wide;                        // outputs are 32-byte aligned
    DevStatus *status;               // host-mapped, may be null
};

struct GemmShared {
    alignas(1024) uint8_t tiles[kStageSpace];
    alignas(8) uint64_t full_bar[kMaxStages];
    uint64_t empty_bar[kMaxStages];
    uint64_t tmem_full[2], tmem_empty[2];
    uint32_t tmem_base, fail;
};

// Panels of `panel` n tiles, m inside a panel, n fastest: the tiles that run together form a block of about panel x
// (units / panel) tiles, near-square in bytes, whose operands share L2.
struct Tile { int um, sn, col; };  // row unit, column shard, first column in it
__device__ __forceinline__ Tile tile_at(const GemmParams &P, int t)
{
    const int per = P.um_tiles * P.panel, pn = t / per, n0 = pn * P.panel, w = min(P.panel, P.n_tiles - n0), r = t - pn * per;
    const int um = r / w, nt = n0 + r - um * w, sn = nt / P.shard_tiles;
    return {um, sn, (nt - sn * P.shard_tiles) * P.cols};
}

__device__ __forceinline__ void st_global_32B(void *p, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// 16 consecutive results of one row; one 32-byte sector where the output allows it
template <int ACT> __device__ __forceinline__ void store_row16(__nv_bfloat16 *dst, const float *v, bool wide)
{
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = pack_bf16(__float_as_uint(activate<ACT>(v[2 * i])), __float_as_uint(activate<ACT>(v[2 * i + 1])));
    if (wide) st_global_32B(dst, o);
    else {
        ((uint4 *)dst)[0] = make_uint4(o[0], o[1], o[2], o[3]);
        ((uint4 *)dst)[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}
template <int COLS> __device__ __forceinline__ void store_row(__nv_bfloat16 *dst, const float (&v)[COLS], bool wide, int act)
{
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
        if (act == GEMM_ACT_SILU) store_row16<GEMM_ACT_SILU>(dst + c, v + c, wide);
        else if (act == GEMM_ACT_GELU) store_row16<GEMM_ACT_GELU>(dst + c, v + c, wide);
        else store_row16<GEMM_ACT_NONE>(dst + c, v + c, wide);
    }
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// address of (row, column of shard sn) in its rank's output; row lies inside the tile space
__device__ __forceinline__ __nv_bfloat16 *out_row(const GemmParams &P, int row, int sn, int col)
{
    if (P.form == GEMM_GATHER) return P.C[sn] + (int64_t)row * P.ldc + col;
    return P.C[row / P.shard_m] + (int64_t)(row % P.shard_m) * P.ldc + col;
}

template <bool kPair, bool kSplit>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_local_kernel(const __grid_constant__ GemmParams P)
{
    extern __shared__ uint8_t smem_raw[];
    GemmShared &S = *(GemmShared *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int kCtas = kPair ? 2 : 1;
    const uint32_t stages = (uint32_t)P.stages, stage_bytes = P.stage_bytes;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr bool kCluster = kPair || kSplit;
    const uint32_t rank = kCluster ? cluster_ctarank() : 0u, cta_r = kPair ? rank & 1 : 0u, leader = rank - cta_r;
    const int split = kSplit ? P.split : 1, unit = (int)blockIdx.x / (kCtas * split), total = P.um_tiles * P.n_tiles;
    const int share = (int)rank / kCtas;  // of the tile's k steps
    const int k0 = kSplit ? P.k_iters * share / split : 0, k1 = kSplit ? P.k_iters * (share + 1) / split : P.k_iters;
    volatile uint32_t *fail = &S.fail;
    // epilogue warps: TMEM lane quarter (a warp reaches its own only), column half, row
    const int q4 = warp & 3, half = (warp - 2) >> 2, rl = q4 * 32 + lane;
    const int mid = (P.cols / 16 + 1) / 2 * 16, c_lo = half ? mid : 0, c_hi = half ? P.cols : mid;
    float4 *sums = (float4 *)S.tiles;  // split tiles: [column / 4][row]
    static_assert(BM * kMaxCols * sizeof(float) <= sizeof(S.tiles), "the sums of a share fit the stages");

    pdl_trigger();
    if (threadIdx.x == 0) {
        S.fail = 0;
        for (int i = 0; i < kMaxStages; ++i) { mbar_init(&S.full_bar[i], 1); mbar_init(&S.empty_bar[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&S.tmem_full[i], 1); mbar_init(&S.tmem_empty[i], kCtas * kEpiThreads / 32); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_tensormap(&P.tmA[0]);
        prefetch_tensormap(&P.tmB[0]);
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
            uint32_t s = 0, ph = 0;
            for (int t = unit; t < total && !*fail; t += P.units) {
                const Tile w = tile_at(P, t);
                int arow = (w.um * kCtas + (int)cta_r) * BM;
                const int brow = w.col + (kPair ? (int)cta_r * (P.cols / 2) : 0);
                const CUtensorMap *ma = &P.tmA[0], *mb = &P.tmB[0];
                if (P.form == GEMM_GATHER) {
                    const int sm = min(arow / P.shard_m, P.shards - 1);  // past the last row: zeros
                    ma = &P.tmA[sm]; arow -= sm * P.shard_m;
                    mb = &P.tmB[w.sn];
                }
                int kx = k0, seg = 0;
                if (P.form == GEMM_REDUCE) { seg = kx / P.k_seg; kx -= seg * P.k_seg; ma = &P.tmA[seg]; mb = &P.tmB[seg]; }
                for (int k = k0; k < k1; ++k, ++kx) {
                    if (kx == P.k_seg) { kx = 0; ++seg; ma = &P.tmA[seg]; mb = &P.tmB[seg]; }
                    if (!mbar_wait_t<kPair>(&S.empty_bar[s], ph ^ 1, fail)) break;
                    uint8_t *sa = S.tiles + (size_t)s * stage_bytes, *sb = sa + kABytes;
                    if (kPair) {  // the bytes of both CTAs' loads are counted on the leader's barrier
                        if (cta_r == 0) mbar_expect_tx(&S.full_bar[s], 2 * stage_bytes);
                        const uint32_t full = mapa_u32(smem_u32(&S.full_bar[s]), leader);
                        tma_load_2d_pair(sa, ma, full, kx * BK, arow);
                        tma_load_2d_pair(sb, mb, full, kx * BK, brow);
                    } else {
                        mbar_expect_tx(&S.full_bar[s], stage_bytes);
                        tma_load_2d(sa, ma, &S.full_bar[s], kx * BK, arow);
                        tma_load_2d(sb, mb, &S.full_bar[s], kx * BK, brow);
                    }
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
            }
        }
        if (*fail)  // loads in flight land before the CTA lets go of its shared memory
            for (int i = 0; i < 200; ++i) __nanosleep(1000);
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (pair: the leader, for both CTAs)
        if (cta_r == 0 && elect_one()) {
            uint32_t s = 0, ph = 0, n = 0;
            const uint16_t both = (uint16_t)(3u << leader);
            for (int t = unit; t < total && !*fail; t += P.units, ++n) {
                const uint32_t buf = n & 1, use = n >> 1, d = tmem_base + buf * kMaxCols;
                if (!mbar_wait_t<kPair>(&S.tmem_empty[buf], (use & 1) ^ 1, fail)) break;
                tc_fence_after();
                for (int k = k0; k < k1; ++k) {
                    if (!mbar_wait_t<kPair>(&S.full_bar[s], ph, fail)) break;
                    tc_fence_after();
                    const uint64_t da = make_smem_desc(S.tiles + (size_t)s * stage_bytes), db = make_smem_desc(S.tiles + (size_t)s * stage_bytes + kABytes);
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk) {  // 16 bf16 = 32 bytes along K inside the swizzle atom
                        if (kPair) umma_pair(d, da + (uint64_t)(2 * kk), db + (uint64_t)(2 * kk), k != k0 || kk != 0, P.idesc);
                        else umma(d, da + (uint64_t)(2 * kk), db + (uint64_t)(2 * kk), k != k0 || kk != 0, P.idesc);
                    }
                    if (kPair) umma_commit_pair(&S.empty_bar[s], both); else umma_commit(&S.empty_bar[s]);
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
                if (kPair) umma_commit_pair(&S.tmem_full[buf], both); else umma_commit(&S.tmem_full[buf]);
            }
        }
    } else if (!kSplit) {
        // ------------------------------------------------------------------ epilogue
        uint32_t n = 0;
        for (int t = unit; t < total && !*fail; t += P.units, ++n) {
            const Tile w = tile_at(P, t);
            const int row0 = (w.um * kCtas + (int)cta_r) * BM;
            const int c_end = row0 < P.rows ? min(c_hi, P.shard_n - w.col) : 0;  // a shard's last tile may be narrower
            __nv_bfloat16 *dst = row0 < P.rows ? out_row(P, row0 + rl, w.sn, w.col) : nullptr;
            const uint32_t buf = n & 1, use = n >> 1, taddr = tmem_base + buf * kMaxCols + ((uint32_t)(q4 * 32) << 16);
            if (!mbar_wait_t<kPair>(&S.tmem_full[buf], use & 1, fail)) break;
            tc_fence_after();
            int c = c_lo;
#pragma unroll 1
            for (; c + 32 <= c_end; c += 32) {
                uint32_t r[32];
                tmem_ld32(taddr + c, r);
                tmem_ld_wait();
                float v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
                store_row(dst + c, v, P.wide, P.act);
            }
            if (c < c_end) {
                uint32_t r[16];
                tmem_ld16(taddr + c, r);
                tmem_ld_wait();
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
                store_row(dst + c, v, P.wide, P.act);
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
            for (int c = c_lo; c < c_hi; c += 16) {
                uint32_t r[16];
                tmem_ld16(tmem_base + c + ((uint32_t)(q4 * 32) << 16), r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    sums[(c / 4 + i) * BM + rl] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
            }
        }
    }
    if (kSplit) {
        __syncwarp();
        cluster_sync_all();
        if (warp >= 2) {  // groups of 16 columns in turn over the units and their column halves
            const Tile w = tile_at(P, unit);
            const int row0 = (w.um * kCtas + (int)cta_r) * BM;
            const int c_end = row0 < P.rows ? min(P.cols, P.shard_n - w.col) : 0;
            __nv_bfloat16 *dst = row0 < P.rows ? out_row(P, row0 + rl, w.sn, w.col) : nullptr;
#pragma unroll 1
            for (int c = 16 * (2 * share + half); c < c_end; c += 32 * split) {
                const uint32_t own = smem_u32(sums + (c / 4) * BM + rl);
                float v[16];
#pragma unroll 1
                for (int q0 = 0; q0 < split; q0 += 4) {
                    float4 x[4][4];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (q0 + q < split) {
                            const uint32_t base = mapa_u32(own, (uint32_t)((q0 + q) * kCtas) + cta_r);
#pragma unroll
                            for (int i = 0; i < 4; ++i) x[q][i] = ld_cluster_f4(base + (uint32_t)(i * BM * sizeof(float4)));
                        }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (q0 + q < split) {
                            const bool first = q0 + q == 0;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                v[4 * i] = first ? x[q][i].x : v[4 * i] + x[q][i].x;
                                v[4 * i + 1] = first ? x[q][i].y : v[4 * i + 1] + x[q][i].y;
                                v[4 * i + 2] = first ? x[q][i].z : v[4 * i + 2] + x[q][i].z;
                                v[4 * i + 3] = first ? x[q][i].w : v[4 * i + 3] + x[q][i].w;
                            }
                        }
                }
                store_row(dst + c, v, P.wide, P.act);
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

constexpr size_t kSmemBytes = sizeof(GemmShared) + 1024;

const void *kernel_of(bool pair, bool split)
{
    if (pair) return split ? (const void *)gemm_local_kernel<true, true> : (const void *)gemm_local_kernel<true, false>;
    return split ? (const void *)gemm_local_kernel<false, true> : (const void *)gemm_local_kernel<false, false>;
}

// units[pair][split]: tiles that can be worked on at once (clusters of pair x split CTAs, each inside one GPC)
struct DeviceShape { int units[2][kMaxCluster + 1] = {}; };

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
            for (int split = kMaxCluster / (pair ? 2 : 1); split >= 1; --split) {
                const void *fn = kernel_of(pair, split > 1);
                const int ctas = (pair ? 2 : 1) * split;
                cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
                int n = sms;
                if (e == cudaSuccess && ctas > 1) {
                    cudaLaunchConfig_t q;
                    memset(&q, 0, sizeof(q));
                    q.gridDim = dim3((unsigned)(sms / ctas * ctas)); q.blockDim = dim3(kGemmThreads); q.dynamicSmemBytes = kSmemBytes;
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

struct Tiling { bool pair; int cols, split; };

bool shape_ok(const GemmCall &c)
{
    const int shards = c.form == GEMM_PLAIN ? 1 : c.p;
    return c.p >= 1 && c.p <= kGemmShards && c.M > 0 && c.N > 0 && c.K > 0 && c.M % (BM * shards) == 0 && c.N % BN == 0 && c.K % BK == 0;
}

// Row units and column tiles of a call under a tiling.
int row_units(const GemmCall &c, bool pair) { return pair ? (c.M + 2 * BM - 1) / (2 * BM) : c.M / BM; }
int shard_tiles(const GemmCall &c, int cols) { return (c.N + cols - 1) / cols; }

// Estimated time (ns) of a tiling: the slowest unit (its rows of A and B per k step, which L2 delivers at 128 bytes per 0.8 to
// 1 ns, and the epilogues), against what the power cap leaves the tensor cores (a narrower tile reads more shared memory per
// product; of a wave that is partly idle about a quarter shows, the clock takes back the rest) and what HBM delivers.  The
// constants are a fit to measured (shape, tiling) pairs, 128 to 2048 rows, 1024 to 28672 columns and depth; over 21 such shapes the
// chosen tiling is within 5 % of the best one measured (20 of them within 3 %).  256 columns everywhere lose up to a factor of
// three: 128 x 4096 x 1024 10.7 us, with 64 columns 7.1; 640 x 4096 x 11008 71 us, with 144 columns 48; 128 x 28672 x 8192 83 us,
// with 208 columns 79; 2048 x 8192 x 28672 656 us, with 224 columns (four whole waves) 619; 128 x 2560 x 8192 51 us, with 80 columns
// split in four 15.
double tiling_ns(const GemmCall &c, const Tiling &t, int units)
{
    const int k_iters = c.K / BK * (c.form == GEMM_REDUCE ? c.p : 1);
    const double n = (double)c.N * (c.form == GEMM_GATHER ? c.p : 1), k = (double)k_iters * BK;
    const int64_t tiles = (int64_t)row_units(c, t.pair) * shard_tiles(c, t.cols) * (c.form == GEMM_GATHER ? c.p : 1);
    const double waves = t.split > 1 ? 1. : (double)((tiles + units - 1) / units), share = (k_iters + t.split - 1) / t.split;
    const double step = t.pair ? 0.99 * (BM + t.cols / 2) : 0.80 * (BM + t.cols), epi = 2.7 * t.cols;
    const double unit = waves * std::max(share * step, epi) + epi + (t.split > 1 ? 300. + 15. * t.cols : 0.);
    const double power = 2. * c.M * n * k / 1.30e6 * (1. + 0.12 * (BN - t.cols) / BN);
    const double hbm = 2. * (c.M * k + n * k + c.M * n) / 5.8e3;
    return std::max(std::max(unit, 0.75 * power + 0.25 * unit), hbm) + 0.06 * unit;
}

Tiling pick_tiling(const GemmCall &c, const DeviceShape &d, bool pair_ok)
{
    const int k_iters = c.K / BK * (c.form == GEMM_REDUCE ? c.p : 1);
    Tiling best{false, BN, 1};
    double least = 1e30;
    for (int pair = pair_ok; pair >= 0; --pair)
        for (int cols = kMaxCols; cols >= kMinCols; cols -= pair ? 32 : 16) {
            const int64_t tiles = (int64_t)row_units(c, pair) * shard_tiles(c, cols) * (c.form == GEMM_GATHER ? c.p : 1);
            for (int split = 1; split <= kMaxCluster / (pair ? 2 : 1); ++split) {
                // shares only while all tiles fit the GPU at once and a unit keeps a few steps
                if (split > 1 && (tiles > d.units[pair][split] || k_iters / split < kMinShare)) break;
                const Tiling t{pair != 0, cols, split};
                const double ns = tiling_ns(c, t, d.units[pair][split]);
                if (ns < least) { least = ns; best = t; }
            }
        }
    return best;
}

// The tilings of the last shapes, by device: a choice costs about as much as a small launch.
struct TilingMemo {
    int dev = -1, form = 0, p = 0, M = 0, N = 0, K = 0, pair_ok = 0;
    Tiling t{false, BN, 1};
};

Tiling tiling_for(const GemmCall &c, const DeviceShape &d, bool pair_ok)
{
    static std::mutex mu;
    static TilingMemo memo[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const uint32_t h = ((uint32_t)c.M * 2654435761u) ^ ((uint32_t)c.N * 2246822519u) ^ ((uint32_t)c.K * 3266489917u) ^ (uint32_t)(c.form * 4 + c.p);
    std::lock_guard<std::mutex> lk(mu);
    TilingMemo &m = memo[(h >> 16) % 64];
    if (m.dev != dev || m.form != c.form || m.p != c.p || m.M != c.M || m.N != c.N || m.K != c.K || m.pair_ok != (int)pair_ok) {
        m.t = pick_tiling(c, d, pair_ok);
        m.dev = dev; m.form = c.form; m.p = c.p; m.M = c.M; m.N = c.N; m.K = c.K; m.pair_ok = pair_ok;
    }
    return m.t;
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
    // an odd number of row blocks leaves a block of zeros in the last pair: worth it from eight row units on (7040 x 4352 x 5632
    // 252 -> 234 us, 2176 x 20992 x 6400 425 -> 392), not below (1152 x 2560 x 4864 22.5 -> 23.9, 640 x 11008 x 4096 46.5 -> 56.4)
    const Tiling til = tiling_for(c, d, env_config().tp_gemm_pair && (c.M / BM % 2 == 0 || c.M > 15 * BM));
    const bool pair = til.pair;
    GemmParams P;
    memset(&P, 0, sizeof(P));
    P.cols = til.cols; P.split = til.split;
    P.um_tiles = row_units(c, pair);
    P.shard_tiles = shard_tiles(c, til.cols);
    P.n_tiles = P.shard_tiles * (c.form == GEMM_GATHER ? c.p : 1);
    P.k_seg = c.K / BK;
    P.k_iters = P.k_seg * (c.form == GEMM_REDUCE ? c.p : 1);
    P.stage_bytes = kABytes + (uint32_t)(til.cols / (pair ? 2 : 1)) * BK * 2;
    P.stages = (int)std::min<uint32_t>(kMaxStages, kStageSpace / P.stage_bytes);
    P.idesc = instr_desc(pair ? 2 * BM : BM, (uint32_t)til.cols);
    const int64_t tiles = (int64_t)P.um_tiles * P.n_tiles;
    uintptr_t bits = 0;
    for (int i = 0; i < na; ++i) {
        if ((((uintptr_t)c.A[i]) | ((uintptr_t)c.B[i]) | ((uintptr_t)c.C[i])) & 15) return HCCL_E_PARA;
        CHK_RET(encode_2d(&P.tmA[i], c.A[i], (uint64_t)(c.form == GEMM_GATHER ? rows : c.M), (uint64_t)c.K, BM));
        CHK_RET(encode_2d(&P.tmB[i], c.B[i], (uint64_t)c.N, (uint64_t)c.K, (uint32_t)(pair ? til.cols / 2 : til.cols)));
        P.C[i] = (__nv_bfloat16 *)c.C[i];
        bits |= (uintptr_t)c.C[i];
    }
    P.wide = (bits & 31) == 0;
    P.status = status;
    P.form = c.form; P.act = c.act;
    P.rows = c.M; P.shards = na;
    P.shard_m = rows;
    P.shard_n = c.N;
    P.ldc = c.N;
    // weights of a panel stay in L2 (40 MB of it) while the rows stream past, but a panel is never narrower than the square
    // block of tiles that run together: with K = 28672 two tiles would fill the 40 MB and every row of A crossed HBM 16 times
    P.panel = (int)std::min<int64_t>(P.n_tiles, std::max<int64_t>(8, (40ll << 20) / ((int64_t)til.cols * P.k_iters * BK * 2)));
    P.units = d.units[pair][til.split];
    const int ctas = (pair ? 2 : 1) * til.split;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(std::min<int64_t>(P.units, tiles) * ctas)); cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    set_cluster(&at[1], ctas);
    cfg.attrs = at; cfg.numAttrs = ctas > 1 ? 2 : 1;
    void *args[] = {&P};
    cudaError_t e = cudaLaunchKernelExC(&cfg, kernel_of(pair, til.split > 1), args);
    if (e != cudaSuccess) { HLOG_ERROR("GEMM launch failed (clusters of %d): %s", ctas, cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    g_counts[pair ? 1 : 0]++;
    return HCCL_SUCCESS;
}

}  // namespace hcclb
