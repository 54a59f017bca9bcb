// MoE exchange where every rank is in this process on one GPU (a single rank included): three launches for a dispatch and a
// combine of all ranks, ordered by their stream (no barrier, no all-gather of counts), each a programmatic dependent launch.
//
//   count     every CTA numbers the (token, k) pairs of its chunk inside their experts with shared-memory counters; the CTA
//             that finishes last turns all histograms into row bases, so nothing waits and no counter needs clearing first;
//   dispatch  a CTA takes one token's row (or a part of it when tokens are few), reads it ONCE and stores it to its top-k
//             receive rows: tokens x (1 + k) rows of traffic, the least the exchange can do;
//   combine   the same split over the output rows, several tokens per CTA where top-k is small: eight expert rows in flight
//             per thread, fp32 sum in k order, one rounding.
//
// Up to 65536 pairs over all ranks, the rows come from ONE cluster that counts in shared memory and registers.
//
// Bound: HBM for prefill batches (8192 tokens x 7168, top 8, one rank: dispatch 165 us at 6.4 TB/s, combine 156 us at 6.8 TB/s,
// whole exchange 338 us, 468 us with a row read per expert, a launch per rank and step, and barriers), launches and L2 for
// decode batches (128 tokens on each of four ranks: 25.9 us, 294 us before; 25.4 us with activations and experts loaded ahead of
// the dispatch's own wait, which is not sound).  Dispatch with 16-byte instead of 32-byte vectors: 171 us.  Whole exchange,
// rows of 7224 pairs (903 tokens x 1280): 1 CTA 15.1 us, four CTAs 13.6 us, through global memory 16.1 us; of 26064 pairs (6516
// tokens x 3840, top 4) by the cluster 91.9 us, through global memory 94.0 us; of 65536 pairs 338 and 337 us.  Combine of 6516 tokens x 3840, top 4, with one token per CTA: 51 us, with
// two 45 us; 32-byte instead of 16-byte loads cost occupancy (8192 x 7168, top 8: 159 -> 171 us).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include "common/log.h"
#include "kernels/moe_a2a.h"
#include "kernels/pdl.cuh"

namespace hcclb {

namespace {

constexpr int kCountThreads = 1024, kScanRegs = 16, kRowsRegs = 8, kRowsCluster = 8, kDispatchThreads = 128, kRowThreads = 256, kRowBatch = 8;

struct alignas(32) Row32 { uint32_t w[8]; };
__device__ __forceinline__ uint4 ld_row(const uint4 *p) { return *p; }
__device__ __forceinline__ void st_row(uint4 *p, const uint4 &v) { *p = v; }
__device__ __forceinline__ Row32 ld_row(const Row32 *p)
{
    Row32 v;
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_row(Row32 *p, const Row32 &v)
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7]) : "memory");
}

// Exclusive prefix of t over the CTA's kCountThreads threads; *all becomes the sum.  Two barriers.
__device__ __forceinline__ int cta_prefix(int t, int *s_warp, int *all)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto inclusive = [&](int v) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += w;
        }
        return v;
    };
    const int v = inclusive(t);
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    const int sum = s_warp[lane], w = inclusive(sum);
    static_assert(kCountThreads == 1024, "one lane per warp of the CTA");
    const int before = __shfl_sync(0xffffffffu, w - sum, warp);
    *all = __shfl_sync(0xffffffffu, w, 31);
    __syncthreads();
    return before + v - t;
}

// The totals that the cluster's CTAs leave for each other.
__device__ __forceinline__ void moe_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ int ld_cluster_s32(const int32_t *own, int cta)
{
    uint32_t at;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(own)), "r"(cta));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}

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
    extern __shared__ int32_t sh[];  // [experts + 1], then [parts][experts]
    __shared__ int s_last;
    const int E = a.n_experts, r = blockIdx.y;
    const int64_t npairs = a.tokens * a.topk, i0 = (int64_t)blockIdx.x * a.chunk, i1 = min(i0 + a.chunk, npairs);
    for (int e = threadIdx.x; e < E; e += kCountThreads) sh[e] = 0;
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    for (int64_t i = i0 + threadIdx.x; i < i1; i += kCountThreads) {
        const int e = a.idx[r][i];
        a.pos[r][i] = e >= 0 && e < E ? atomicAdd(&sh[e], 1) : -1;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += kCountThreads) a.hist[((int64_t)r * a.nchunk + blockIdx.x) * E + e] = sh[e];
    __syncthreads();
    if (threadIdx.x == 0) {  // the barrier puts the CTA's histogram before this thread's fence
        __threadfence();
        s_last = atomicAdd(a.arrived, 1u) == gridDim.x * gridDim.y - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    // Rows of an owner are grouped [local expert][source rank][chunk].  `parts` threads share an expert's groups, so that their
    // loads are one round trip (a few registers each) where the experts leave threads over.
    const int groups = a.p * a.nchunk, El = E / a.p, parts = max(1, kCountThreads / E), per = (groups + parts - 1) / parts;
    int32_t *sub = sh + E + 1;  // [part][expert]: pairs of the part, then its first row within the expert
    __shared__ int s_warp[kCountThreads / 32];
    const bool once = parts * E <= kCountThreads && per <= kScanRegs;  // a thread's groups stay in its registers
    int n[kScanRegs];
    for (int i = threadIdx.x; i < parts * E; i += kCountThreads) {
        const int part = i / E, e = i - part * E, g0 = part * per, g1 = min(groups, g0 + per);
        int t = 0;
        for (int gb = g0; gb < g1; gb += kScanRegs) {
#pragma unroll
            for (int k = 0; k < kScanRegs; ++k) n[k] = gb + k < g1 ? __ldcg(a.hist + (int64_t)(gb + k) * E + e) : 0;
#pragma unroll
            for (int k = 0; k < kScanRegs; ++k) t += n[k];
        }
        sub[i] = t;
    }
    __syncthreads();
    // exclusive prefix over all experts, kCountThreads of them at a time
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += kCountThreads) {
        const int e = e0 + threadIdx.x;
        int t = 0;
        if (e < E)
            for (int q = 0; q < parts; ++q) { const int v = sub[q * E + e]; sub[q * E + e] = t; t += v; }
        int all;
        const int before = cta_prefix(t, s_warp, &all);
        if (e < E) sh[e] = carry + before;
        carry += all;
    }
    if (threadIdx.x == 0) { sh[E] = carry; *a.arrived = 0; }
    __syncthreads();
    for (int i = threadIdx.x; i < parts * E; i += kCountThreads) {
        const int part = i / E, e = i - part * E, q = e / El, first = sh[q * El], g0 = part * per, g1 = min(groups, g0 + per);
        int row = sh[e] - first + sub[i];
        for (int gb = g0; gb < g1; gb += kScanRegs) {
            if (!once)
#pragma unroll
                for (int k = 0; k < kScanRegs; ++k) n[k] = gb + k < g1 ? __ldcg(a.hist + (int64_t)(gb + k) * E + e) : 0;
#pragma unroll
            for (int k = 0; k < kScanRegs; ++k)
                if (gb + k < g1) {
                    a.hist[(int64_t)(gb + k) * E + e] = row;
                    row += n[k];
                }
        }
        if (part == 0) {
            a.expert_offsets[q][e - q * El] = sh[e] - first;
            if (e == q * El + El - 1) {
                const int total = sh[e + 1] - first;
                a.expert_offsets[q][El] = total;
                *a.recv_rows[q] = total;
                if (total > a.capacity) *a.overflow[q] = 1;
            }
        }
    }
}

// Up to 65536 pairs: one cluster numbers the pairs of all ranks and knows their rows without a trip through global memory (no
// histogram, no fence, no arrival).  CTA c takes a stretch of the pairs in rank order, a thread keeps its pairs in registers,
// and the CTAs read each other's totals per expert through distributed shared memory.  Dynamic shared memory: [rank][expert]
// counters, then first rows; [experts + 1] first row of an expert over all owners; [experts] pairs of this CTA.
__global__ void __launch_bounds__(kCountThreads) moe_local_rows_kernel(const __grid_constant__ MoeTables a)
{
    extern __shared__ int32_t sh[];
    __shared__ int s_warp[kCountThreads / 32];
    const int E = a.n_experts, El = E / a.p, npairs = (int)a.tokens * a.topk, total = npairs * a.p;
    const int ctas = (int)gridDim.x, c = (int)blockIdx.x, per = (total + ctas - 1) / ctas, i0 = c * per, i1 = min(total, i0 + per);
    int32_t *first = sh + a.p * E, *mine = first + E + 1;
    for (int i = threadIdx.x; i < a.p * E; i += kCountThreads) sh[i] = 0;
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    int ex[kRowsRegs], ps[kRowsRegs], rk[kRowsRegs];
#pragma unroll
    for (int k = 0; k < kRowsRegs; ++k) {
        const int i = i0 + k * kCountThreads + (int)threadIdx.x;
        rk[k] = 0;
        ex[k] = -1;
        if (i < i1) {
            rk[k] = i / npairs;
            ex[k] = a.idx[rk[k]][i - rk[k] * npairs];
        }
    }
#pragma unroll
    for (int k = 0; k < kRowsRegs; ++k) ps[k] = ex[k] >= 0 && ex[k] < E ? atomicAdd(&sh[rk[k] * E + ex[k]], 1) : -1;
    __syncthreads();
    if (ctas > 1) {
        for (int e = threadIdx.x; e < E; e += kCountThreads) {
            int t = 0;
            for (int r = 0; r < a.p; ++r) t += sh[r * E + e];
            mine[e] = t;
        }
        moe_cluster_sync();
    }
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += kCountThreads) {  // first row of every expert, counting over all owners
        const int e = e0 + threadIdx.x;
        int t = 0, earlier = 0;  // pairs of the expert, of them those of earlier CTAs
        if (e < E) {
            if (ctas > 1) {
                int n[kRowsCluster];
#pragma unroll
                for (int q = 0; q < kRowsCluster; ++q) n[q] = q < ctas ? ld_cluster_s32(mine + e, q) : 0;
#pragma unroll
                for (int q = 0; q < kRowsCluster; ++q) { t += n[q]; earlier += q < c ? n[q] : 0; }
            } else
                for (int r = 0; r < a.p; ++r) t += sh[r * E + e];
        }
        int all;
        const int before = cta_prefix(t, s_warp, &all);
        if (e < E) {
            first[e] = carry + before;
            int row = earlier;  // counted from the expert's first row
            for (int r = 0; r < a.p; ++r) { const int k = sh[r * E + e]; sh[r * E + e] = row; row += k; }
        }
        carry += all;
    }
    if (threadIdx.x == 0) first[E] = carry;
    __syncthreads();
    if (c == 0)
        for (int e = threadIdx.x; e < E; e += kCountThreads) {
            const int q = e / El, f = first[q * El];
            a.expert_offsets[q][e - q * El] = first[e] - f;
            if (e == q * El + El - 1) {
                const int rows = first[e + 1] - f;
                a.expert_offsets[q][El] = rows;
                *a.recv_rows[q] = rows;
                if (rows > a.capacity) *a.overflow[q] = 1;
            }
        }
#pragma unroll
    for (int k = 0; k < kRowsRegs; ++k)
        if (ps[k] >= 0) {
            const int e = ex[k];
            a.dst_row[rk[k]][i0 + k * kCountThreads + (int)threadIdx.x - rk[k] * npairs] = first[e] - first[e / El * El] + sh[rk[k] * E + e] + ps[k];
        }
    if (ctas > 1) moe_cluster_sync();  // the others may still read this CTA's totals
}

// grid (tokens x segments, ranks); kRows: the rows are in dst_row already; V: vectors of 32 bytes where the rows allow them, else of 16
template <class V, bool kRows>
__global__ void __launch_bounds__(kDispatchThreads) moe_local_dispatch_kernel(const __grid_constant__ MoeTables a)
{
    constexpr int kPer = 128 / sizeof(V);  // 128 bytes of a row per thread and round
    __shared__ V *s_dst[kRowBatch];
    pdl_trigger();
    const int r = blockIdx.y, k = a.topk, nvec = a.nvec / (int)(sizeof(V) / 16), nt = (int)blockDim.x;
    const int64_t t = a.nseg == 1 ? blockIdx.x : blockIdx.x / a.nseg;
    const int seg = (int)(blockIdx.x - t * a.nseg), per = (nvec + a.nseg - 1) / a.nseg, v1 = min(nvec, (seg + 1) * per);
    const V *src = (const V *)a.x[r] + t * nvec;
    const int v0 = seg * per + threadIdx.x;
    // Nothing is read before this grid's own wait: only that makes what earlier kernels wrote (activations and experts among it)
    // visible here, however early the kernel before this one triggered.
    pdl_wait();
    V x[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u)
        if (v0 + u * nt < v1) x[u] = ld_row(src + v0 + u * nt);
    for (int k0 = 0; k0 < k; k0 += kRowBatch) {
        if (k0) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < kPer; ++u)
                if (v0 + u * nt < v1) x[u] = ld_row(src + v0 + u * nt);
        }
        if (threadIdx.x < kRowBatch) {
            V *d = nullptr;
            if (k0 + (int)threadIdx.x < k) {
                const int64_t i = t * k + k0 + threadIdx.x;
                const int known = kRows ? a.dst_row[r][i] : a.pos[r][i], e = a.idx[r][i];
                if (e >= 0 && e < a.n_experts) {
                    const int64_t row = kRows ? known : a.hist[((int64_t)r * a.nchunk + (uint32_t)i / (uint32_t)a.chunk) * a.n_experts + e] + known;
                    if (!kRows && seg == 0) a.dst_row[r][i] = (int32_t)row;
                    if (row < a.capacity) d = (V *)a.rows[e / (a.n_experts / a.p)] + row * nvec;
                }
            }
            s_dst[threadIdx.x] = d;
        }
        __syncthreads();
        for (int vb = v0;;) {
#pragma unroll
            for (int j = 0; j < kRowBatch; ++j) {
                V *d = s_dst[j];
                if (!d) continue;
#pragma unroll
                for (int u = 0; u < kPer; ++u)
                    if (vb + u * nt < v1) st_row(d + vb + u * nt, x[u]);
            }
            vb += kPer * nt;
            if (vb >= v1) break;
#pragma unroll
            for (int u = 0; u < kPer; ++u)
                if (vb + u * nt < v1) x[u] = ld_row(src + vb + u * nt);
        }
    }
}

// grid (groups of G tokens x segments, ranks).  A thread has eight expert rows in flight: B = 8 / G of each token of the group, so
// that a small top-k does not leave it with two or four (the addresses of a group's rows are one round trip as well).
template <int G>
__global__ void __launch_bounds__(kRowThreads) moe_local_combine_kernel(const __grid_constant__ MoeTables a)
{
    constexpr int B = kRowBatch / G;
    __shared__ const uint4 *s_src[kRowBatch];
    __shared__ float s_gate[kRowBatch];
    pdl_trigger();
    const int r = blockIdx.y, k = a.topk, nt = (int)blockDim.x;
    const int64_t t0 = (int64_t)(blockIdx.x / a.nseg) * G;
    const int seg = (int)(blockIdx.x % a.nseg), per = (a.nvec + a.nseg - 1) / a.nseg, v1 = min(a.nvec, (seg + 1) * per);
    uint4 *out = (uint4 *)a.out[r] + t0 * a.nvec;
    pdl_wait();
    const bool one = k <= B;
    auto batch = [&](int k0) {
        if (threadIdx.x < kRowBatch) {
            const uint4 *s = nullptr;
            float g = 0.f;
            const int64_t t = t0 + threadIdx.x / B;
            const int kk = k0 + threadIdx.x % B;
            if (kk < k && t < a.tokens) {
                const int64_t i = t * k + kk;
                const int e = a.idx[r][i];
                const int64_t row = a.dst_row[r][i];
                const float gate = a.gates[r][i];
                if (e >= 0 && e < a.n_experts && row >= 0 && row < a.capacity) {
                    s = (const uint4 *)a.rows[e / (a.n_experts / a.p)] + row * a.nvec;
                    g = gate;
                }
            }
            s_src[threadIdx.x] = s;
            s_gate[threadIdx.x] = g;
        }
        __syncthreads();
    };
    if (one) batch(0);
    for (int vb = seg * per; vb < v1; vb += nt) {  // uniform trip count: the batches synchronise
        const int v = vb + (int)threadIdx.x;
        float acc[G][8];
#pragma unroll
        for (int u = 0; u < G; ++u)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[u][i] = 0.f;
        for (int k0 = 0; k0 < k; k0 += B) {
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
                        acc[j / B][2 * i] += g * f.x;
                        acc[j / B][2 * i + 1] += g * f.y;
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < G; ++u)
            if (v < v1 && t0 + u < a.tokens) {
                uint4 o;
                __nv_bfloat162 *h = (__nv_bfloat162 *)&o;
#pragma unroll
                for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(acc[u][2 * i], acc[u][2 * i + 1]);
                out[(int64_t)u * a.nvec + v] = o;
            }
    }
}

// Parts of a row per CTA row: whole rows once there is a CTA for every SM several times over.
int segments(int64_t units, int nvec, int threads)
{
    int s = 1;
    while (s < 4 && units * s < 4 * 148 && nvec / (2 * s) >= threads) s *= 2;
    return s;
}

// Threads of a CTA that goes through n vectors in the same number of rounds as `most` threads would, none of them half empty
// (a row of 2816 bf16, 352 vectors: two rounds of 192 threads instead of 256 and 96).
unsigned row_threads(int n, int most)
{
    const int rounds = std::max(1, (n + most - 1) / most);
    return (unsigned)std::max(32, ((n + rounds - 1) / rounds + 31) / 32 * 32);
}

void fill(MoeTables &t, const MoeLocalLayer &l)
{
    t.p = l.p; t.topk = l.topk; t.nvec = l.hidden / 8; t.n_experts = l.n_experts; t.tokens = l.tokens; t.capacity = l.capacity;
    moe_local_chunks(l.tokens * l.topk, &t.chunk, &t.nchunk);
    t.hist = l.scratch + 4;
    t.arrived = (uint32_t *)l.scratch;
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
    // one cluster for all ranks' pairs while a thread can keep its own in registers and the counters fit shared memory: a CTA
    // for every 2048 pairs (up to eight), one alone up to 4096, where meeting the others costs what it saves
    const size_t rows_smem = sizeof(int32_t) * ((size_t)l.p * l.n_experts + 2 * l.n_experts + 1);
    const int64_t total = l.tokens * l.topk * l.p;
    const bool rows = total <= kRowsCluster * kRowsRegs * kCountThreads && rows_smem <= 48 * 1024 - 256;
    const int ctas = rows && total > 4096 ? (int)std::min<int64_t>(kRowsCluster, (total + 2047) / 2048) : 1;
    HcclResult rc = rows ? launch_pdl((const void *)moe_local_rows_kernel, dim3((unsigned)ctas), kCountThreads, rows_smem, &t, stream, "moe rows", ctas)
                         : launch_pdl((const void *)moe_local_count_kernel, dim3((unsigned)t.nchunk, (unsigned)l.p), kCountThreads,
                                      sizeof(int32_t) * (l.n_experts + 1 + std::max(1, kCountThreads / l.n_experts) * l.n_experts), &t, stream, "moe count");
    if (rc != HCCL_SUCCESS) return rc;
    uintptr_t bits = (uintptr_t)(l.hidden * 2);
    for (int q = 0; q < l.p; ++q) bits |= (uintptr_t)x[q] | (uintptr_t)recv[q];
    const bool wide = (bits & 31) == 0;
    t.nseg = segments(l.tokens * l.p, wide ? t.nvec / 2 : t.nvec, kDispatchThreads);
    const void *fn = wide ? (rows ? (const void *)moe_local_dispatch_kernel<Row32, true> : (const void *)moe_local_dispatch_kernel<Row32, false>)
                          : (rows ? (const void *)moe_local_dispatch_kernel<uint4, true> : (const void *)moe_local_dispatch_kernel<uint4, false>);
    const int nv = wide ? t.nvec / 2 : t.nvec;
    return launch_pdl(fn, dim3((unsigned)(l.tokens * t.nseg), (unsigned)l.p), row_threads((nv + t.nseg - 1) / t.nseg, kDispatchThreads), 0, &t, stream, "moe dispatch");
}

HcclResult moe_local_combine(const MoeLocalLayer &l, void *const *rows, const int32_t *const *idx, const float *const *gates, void *const *out, void *stream)
{
    if (bad(l)) return HCCL_E_PARA;
    if (l.tokens == 0) return HCCL_SUCCESS;
    MoeTables t;
    fill(t, l);
    for (int q = 0; q < l.p; ++q) { t.idx[q] = idx[q]; t.rows[q] = (__nv_bfloat16 *)rows[q]; t.gates[q] = gates[q]; t.out[q] = (__nv_bfloat16 *)out[q]; }
    // tokens of a CTA: as many as eight rows in flight serve, while every SM keeps several CTAs
    int group = kRowBatch / 2;
    while (group > 1 && (group * l.topk > kRowBatch || l.tokens / group * l.p < 4 * 148)) group /= 2;
    const int64_t groups = (l.tokens + group - 1) / group;
    const void *fn = group == 4 ? (const void *)moe_local_combine_kernel<4> : group == 2 ? (const void *)moe_local_combine_kernel<2> : (const void *)moe_local_combine_kernel<1>;
    t.nseg = segments(groups * l.p, t.nvec, kRowThreads);
    return launch_pdl(fn, dim3((unsigned)(groups * t.nseg), (unsigned)l.p), row_threads((t.nvec + t.nseg - 1) / t.nseg, kRowThreads), 0, &t, stream, "moe combine");
}

}  // namespace hcclb
