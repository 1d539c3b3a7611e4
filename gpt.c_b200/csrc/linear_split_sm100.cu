// Linear products whose result has fewer tiles than the GPU has SMs (generation with a short prompt, small batches,
// narrow layers over few rows): y = x W^T + b and dx = dy W with the contraction shared out over a thread-block
// cluster.
//
// What bounds such a product is how fast the weights arrive: at 37 x 768 x 3072 the general kernel
// (linear_sm100.cu) keeps 6 SMs busy, each walking 96 contraction blocks one after the other with a 128-row tile of
// which 37 rows are real (24.4 us, 0.4 TB/s of weights).  Here
//   - the product is computed transposed: 128 columns of the result (rows or columns of W) are the tensor core's
//     128-row operand and the activations the other one, of just as many rows (rounded up to 16) as there are, so
//     a stage of the pipeline carries 16 KB of weights and little else, and the result leaves tensor memory with
//     consecutive columns in consecutive lanes: plain coalesced stores at any alignment;
//   - a cluster of `split` CTAs cuts the contraction of one tile; each leaves its partial tile in its own shared
//     memory and adds up a share of the rows over all of them through distributed shared memory, always in the
//     same order: no atomics, no zero-filled output, bias and bf16 planes come from the finished sum;
//   - the first weights are requested into L2 before the previous kernel of the stream has completed.
#include "linear_tf32.cuh"

#include "../../include/linear_sm100.h"

namespace lin {
namespace {

using namespace tc05;

constexpr int kMaxStages = 12;
constexpr int kMaxSplit = 8;  // CTAs on one tile: the portable cluster size
constexpr int kMostTmemCols = 128;  // an accumulator of at most 128 columns
// Epilogue warps (the first ones), one or two per tensor-memory lane quarter, then a TMA producer warp and a warp that
// issues the MMAs.  Several CTAs share an SM when tiles are not split: four warps each are enough there.
template <bool kSplit>
struct Roles {
    static constexpr int kEpiWarps = kSplit ? 8 : 4, kWarpTma = kEpiWarps, kWarpMma = kEpiWarps + 1;
    static constexpr int kThreads = 32 * (kEpiWarps + 2);
    static constexpr int kPerSm = kSplit ? 2 : 3;  // CTAs an SM's registers hold
    // The CTAs of a cluster wait for each other while they hold tensor memory: were an SM's columns fewer than its CTAs
    // want, two clusters could each hold what the other waits for.
    static_assert(kPerSm * kMostTmemCols <= 512, "tensor memory for every CTA of an SM");
};

struct Params {
    int M, cols;       // result
    int bm;            // activation rows per tile (multiple of 16, at most 128)
    int tiles_m, split, kb_total, kb_per_split;
    int stages, tmem_cols;
    int w_one;         // MN-major weight tile fetched with one 3-D copy per stage
    size_t plane_elems;
};

struct __align__(16) Control {
    uint64_t full[kMaxStages], empty[kMaxStages], acc_full;
    uint32_t tmem_base;
    int abort_flag;
};

enum Site : int { SITE_EMPTY = 231, SITE_FULL, SITE_ACC_FULL };

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

// kSplit: a cluster of CTAs per tile (else one CTA, several to an SM)
template <bool kWMN, bool kSplit>
__global__ void __launch_bounds__(Roles<kSplit>::kThreads, Roles<kSplit>::kPerSm) linear_split_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                const __grid_constant__ CUtensorMap map_act,
                                                                const float *__restrict__ bias, float *__restrict__ out,
                                                                __nv_bfloat16 *__restrict__ planes, Params p, int *status) {
    constexpr int kEpiWarps = Roles<kSplit>::kEpiWarps, kWarpTma = Roles<kSplit>::kWarpTma, kWarpMma = Roles<kSplit>::kWarpMma;
    extern __shared__ __align__(1024) uint8_t smem[];  // stages of {weights 16 KB, activations bm x 128 B}; then partials
    __shared__ Control ct;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = kSplit ? (int)cluster_rank() : 0;
    const int unit = kSplit ? (int)blockIdx.x / p.split : (int)blockIdx.x;
    const int n0 = unit / p.tiles_m * kBM, m0 = unit % p.tiles_m * p.bm;
    const int kb0 = rank * p.kb_per_split, kb1 = min(p.kb_total, kb0 + p.kb_per_split);
    const uint32_t stage_bytes = kATileBytes + p.bm * 128;
    WaitCtx ctx{&ct.abort_flag, status};

    if (threadIdx.x == 0) {
        ct.abort_flag = 0;
        for (int i = 0; i < p.stages; i++) {
            mbar_init(&ct.full[i], 1);
            mbar_init(&ct.empty[i], 1);
        }
        mbar_init(&ct.acc_full, 1);
        fence_barrier_init();
    }
    if (warp == kWarpMma) {
        tmem_alloc_then_launch_dependents(&ct.tmem_base, p.tmem_cols);
    }
    if (warp == kWarpTma && lane == 0) {
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_act);
        if (!kWMN || p.w_one) {
            // a prefetch into L2 has no result, so it need not wait for whatever wrote the weights last
            for (int kb = kb0; kb < min(kb1, kb0 + p.stages); kb++)
                asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(&map_w),
                             "r"(kWMN ? 0 : kb * kBK), "r"(kWMN ? kb * kBK : n0), "r"(kWMN ? n0 / 32 : 0), "r"(0)
                             : "memory");
        }
    }
    pdl_wait();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = ct.tmem_base;

    if (warp == kWarpTma) {
        if (lane == 0) {
            for (int kb = kb0, it = 0; kb < kb1; kb++, it++) {
                const int st = it % p.stages;
                if (it >= p.stages && !mbar_wait(&ct.empty[st], ((it / p.stages) - 1) & 1, ctx, SITE_EMPTY)) break;
                uint8_t *w = smem + st * stage_bytes, *a = w + kATileBytes;
                mbar_expect_tx(&ct.full[st], stage_bytes);
                if (!kWMN) {
                    tma_load_4d(w, &map_w, &ct.full[st], kb * kBK, n0, 0, 0);
                } else if (p.w_one) {
                    tma_load_4d(w, &map_w, &ct.full[st], 0, kb * kBK, n0 / 32, 0);
                } else {
                    for (int i = 0; i < 4; i++) tma_load_4d(w + i * 4096, &map_w, &ct.full[st], n0 + 32 * i, kb * kBK, 0, 0);
                }
                tma_load_4d(a, &map_act, &ct.full[st], kb * kBK, m0, 0, 0);
            }
        }
    } else if (warp == kWarpMma) {
        const uint32_t idesc = idesc_tf32(kBM, p.bm, kWMN ? 1 : 0, 0);
        const uint32_t leader = elect_leader();
        bool ok = true;
        for (int kb = kb0, it = 0; kb < kb1; kb++, it++) {
            const int st = it % p.stages;
            if (!mbar_wait_warp(&ct.full[st], (it / p.stages) & 1, ctx, SITE_FULL)) {
                ok = false;
                break;
            }
            tc_fence_after_sync();
            const uint32_t at = smem_u32(smem) + st * stage_bytes;
            const uint64_t ad = kWMN ? smem_desc_sw128_base32(at, 4096, 512) : smem_desc_sw128(at, 16, 1024);
            const uint64_t bd = smem_desc_sw128(at + kATileBytes, 16, 1024);
#pragma unroll
            for (int k = 0; k < kBK / 8; k++)
                mma_tf32_lead(leader, tmem, desc_advance(ad, k * (kWMN ? 1024 : 32)), desc_advance(bd, k * 32), idesc,
                              kb > kb0 || k > 0 ? 1u : 0u);
            tc_commit_lead(leader, &ct.empty[st]);
        }
        if (ok) tc_commit_lead(leader, &ct.acc_full);
    } else {
        // lane = column of the result, tensor-memory column = row; the two warps of a quarter take turns at 16 rows
        const int quarter = warp & 3, n = 32 * quarter + lane, col = n0 + n;
        const uint32_t src = tmem + ((uint32_t)(32 * quarter) << 16);
        const int rows = min(p.bm, p.M - m0);
        const float b = bias != nullptr && col < p.cols ? __ldg(bias + col) : 0.f;
        float *part = reinterpret_cast<float *>(smem) + n;
        if (mbar_wait_warp(&ct.acc_full, 0, ctx, SITE_ACC_FULL)) {
            tc_fence_after_sync();
#pragma unroll 1
            for (int c = 16 * (warp >> 2); c < rows; c += 4 * kEpiWarps) {
                uint32_t r[16];
                tmem_ld16(src + c, r);
                tmem_wait_ld();
                if (kSplit) {
#pragma unroll
                    for (int e = 0; e < 16; e++) part[(c + e) * kBM] = __uint_as_float(r[e]);
                    continue;
                }
                if (col >= p.cols) continue;
                const size_t at = (size_t)(m0 + c) * p.cols + col;
                float *o = out + at;
#pragma unroll
                for (int e = 0; e < 16; e++, o += p.cols)
                    if (c + e < rows) *o = __uint_as_float(r[e]) + b;
                if (planes == nullptr) continue;
                __nv_bfloat16 *h = planes + at;
#pragma unroll
                for (int e = 0; e < 16; e++, h += p.cols) {
                    const float v = __uint_as_float(r[e]) + b;
                    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
                    if (c + e < rows) h[0] = hi, h[p.plane_elems] = __float2bfloat16_rn(v - __bfloat162float(hi));
                }
            }
            tc_fence_before_sync();
        }
    }

    if (kSplit) {
        __syncwarp();
        cluster_sync_all();  // every partial tile is in place
        if (warp < kEpiWarps) {
            // rows rank, rank + split, ... of the tile: a row per warp at a time, four columns per lane
            const int rows = min(p.bm, p.M - m0), col = n0 + 4 * lane;
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (bias != nullptr) {
                if (col < p.cols) b.x = __ldg(bias + col);
                if (col + 1 < p.cols) b.y = __ldg(bias + col + 1);
                if (col + 2 < p.cols) b.z = __ldg(bias + col + 2);
                if (col + 3 < p.cols) b.w = __ldg(bias + col + 3);
            }
            const bool words = (p.cols & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
            const uint32_t mine = smem_u32(smem) + 16 * lane;
            uint32_t base[kMaxSplit];
#pragma unroll
            for (int s = 0; s < kMaxSplit; s++) base[s] = mapa(mine, s < p.split ? s : 0);
#pragma unroll 2
            for (int m = rank + p.split * warp; m < rows; m += kEpiWarps * p.split) {
                float4 u[kMaxSplit];  // all on their way before the first is added
#pragma unroll
                for (int s = 0; s < kMaxSplit; s++)
                    if (s < p.split) u[s] = ld_cluster_v4(base[s] + m * (kBM * 4));
                float4 v = u[0];
#pragma unroll
                for (int s = 1; s < kMaxSplit; s++)
                    if (s < p.split) v.x += u[s].x, v.y += u[s].y, v.z += u[s].z, v.w += u[s].w;
                v.x += b.x, v.y += b.y, v.z += b.z, v.w += b.w;
                const size_t at = (size_t)(m0 + m) * p.cols + col;
                if (words) {
                    if (col < p.cols) *reinterpret_cast<float4 *>(out + at) = v;
                } else {
                    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (col + e < p.cols) out[at + e] = f[e];
                }
                if (planes != nullptr && col < p.cols) {  // cols is a multiple of 8
                    uint32_t h0, l0, h1, l1;
                    split_bf16x2(v.x, v.y, h0, l0);
                    split_bf16x2(v.z, v.w, h1, l1);
                    *reinterpret_cast<uint2 *>(planes + at) = make_uint2(h0, h1);
                    *reinterpret_cast<uint2 *>(planes + p.plane_elems + at) = make_uint2(l0, l1);
                }
            }
        }
    }

    // ------------------------------ tear-down ------------------------------
    if (ct.abort_flag) __nanosleep(50000);
    __syncthreads();
    if (warp == kWarpMma) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, p.tmem_cols);
    }
    if (kSplit) cluster_sync_all();  // this CTA's partial tile stays until the others have read it
}

// CTAs of clusters of `split` that find an SM each at the same time; beyond it a second wave, or sharing, sets in.  A
// cluster stays inside a GPC, so larger ones leave SMs over: the table is what a GPU of 148 SMs had room for (clusters of
// seven leave too many), on one with fewer SMs it is taken in proportion.
int alone(int split, int sms) {
    constexpr int kOn148[kMaxSplit + 1] = {0, 148, 148, 117, 128, 120, 108, 0, 104};
    return kOn148[split] * sms / 148;
}

int rows_per_tile(int M) {
    const int tiles = (M + 127) / 128;
    return ((M + tiles - 1) / tiles + 15) / 16 * 16;
}

}  // namespace

// Time of the product in nanoseconds as measured on shapes of 16 to 1500 rows and 512 to 6400 columns (within 10 %): a
// CTA takes about 300 ns per contraction block, whatever the rows, because that is how fast one SM's loads of 128
// separate rows arrive; sharing an SM makes it 390 to 600 ns; cluster barriers and the exchange cost 1.3 us.
int plan_split(int M, int cols, int kc, int sms, int *split) {
    const int bm = rows_per_tile(M), units = (cols + kBM - 1) / kBM * ((M + bm - 1) / bm), kb = (kc + kBK - 1) / kBK;
    long long best = 0;
    for (int s = 1; s <= kMaxSplit; s++) {
        if (alone(s, sms) == 0 || s > kb || (s > 1 && units * s > 2 * alone(s, sms))) continue;
        const int per = (kb + s - 1) / s;
        const long long t = s == 1 ? 1650 + 16 * bm + (units <= sms ? 295ll * per : (400ll * per + 1000) * units / sms)
                             : 2900 + 16 * bm + (long long)per * (units * s <= alone(s, sms) ? 310 : 300 + 2 * bm);
        if (best == 0 || t < best) best = t, *split = s;
    }
    return best < 0x7fffffff ? (int)best : 0x7fffffff;
}

int launch_split(const float *act, const float *w, bool w_mn_major, int w_rows, const float *bias, float *out, void *planes, int M,
                 int cols, int kc, int split, int sms, int *status, cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    constexpr int kMostBytes = 224 * 1024;
    static bool ready[64] = {};
    using Kernel = decltype(&linear_split_kernel<false, false>);
    static const Kernel kernels[2][2] = {{linear_split_kernel<false, false>, linear_split_kernel<false, true>},
                                         {linear_split_kernel<true, false>, linear_split_kernel<true, true>}};
    if (dev >= 0 && dev < 64 && !ready[dev]) {
        for (int i = 0; i < 4; i++) {
            e = cudaFuncSetAttribute(kernels[i >> 1][i & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, kMostBytes);
            if (e != cudaSuccess) return (int)e;
        }
        ready[dev] = true;
    }
    Params p;
    p.M = M, p.cols = cols;
    p.bm = rows_per_tile(M);
    p.tiles_m = (M + p.bm - 1) / p.bm;
    p.kb_total = (kc + kBK - 1) / kBK;
    p.kb_per_split = (p.kb_total + split - 1) / split;
    p.split = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;  // every CTA has a share
    p.tmem_cols = p.bm <= 32 ? 32 : (p.bm <= 64 ? 64 : kMostTmemCols);
    p.plane_elems = attn::plane_bytes((size_t)M * cols) / sizeof(__nv_bfloat16);
    const int grid = (cols + kBM - 1) / kBM * p.tiles_m * p.split;
    const int stage = kATileBytes + p.bm * 128;
    // more CTAs than fit one to an SM: two or three share one, and its shared memory
    const int room = alone(p.split, sms), sharing = grid > 2 * room ? 3 : (grid > room ? 2 : 1);
    p.stages = kMostBytes / sharing / stage;
    if (p.stages > kMaxStages) p.stages = kMaxStages;
    if (p.stages > p.kb_per_split) p.stages = p.kb_per_split;
    const int partial = p.split > 1 ? p.bm * kBM * 4 : 0;
    const int bytes = p.stages * stage > partial ? p.stages * stage : partial;

    CUtensorMap mw, ma;
    int rc;
    p.w_one = 0;
    if (!w_mn_major) {
        // A tile fetches 128 bytes of each of its rows at a time: L2 asks HBM for the next 128 with them (37 x 50257 x 768 30.9 ->
        // 28.0 us, 37 x 50257 x 1600 58.9 -> 52.3; the tiles of linear_sm100.cu, which more rows share, gain nothing).
        if ((rc = map_k_major(&mw, w, cols, kc, kBM, 0, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) != 0) return rc;
    } else {
        p.w_one = map_mn_major_blocks(&mw, w, w_rows, cols, 4) == 0;
        if (!p.w_one && (rc = map_mn_major(&mw, w, w_rows, cols)) != 0) return rc;
    }
    if ((rc = map_k_major(&ma, act, M, kc, p.bm)) != 0) return rc;
    return (int)attn::launch_clusters_after_previous(kernels[w_mn_major ? 1 : 0][p.split > 1 ? 1 : 0], dim3(grid),
                                                     dim3(p.split > 1 ? Roles<true>::kThreads : Roles<false>::kThreads),
                                                     bytes, p.split, s, mw, ma, bias, out, static_cast<__nv_bfloat16 *>(planes), p, status);
}

}  // namespace lin
