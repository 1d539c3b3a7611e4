// Linear layer (y = x W^T + b) and its backward for sm_100a: one persistent tcgen05 GEMM kernel
// with TF32 inputs read straight from the fp32 tensors and fp32 accumulation in tensor memory.
//
// Replaces linear_forward_cuda_kernel / linear_backward_cuda_kernel of gpt.c
// (kernels/src/cuda/Linear.cu:37-92: one cuBLAS SGEMM in TF32 tensor-op math plus a separate
// bias kernel forward; two SGEMMs plus an atomic bias reduction backward) for the two Linear
// layers either side of the attention layer (src/self_attention.c:59-61, 78-80).  The forward
// epilogue adds the bias and can also emit the result as the two bf16 planes (hi, lo) the
// attention kernels consume, which removes the attention path's own split pass.
//
//     forward  y [M,N]  = x [M,K] . W[N,K]^T        A: x, K-major          B: W,  K-major
//     dx       dx[M,K]  = dy[M,N] . W[N,K]          A: dy, K-major (over N) B: W,  MN-major
// dx is made here where it is wanted alone or has few rows; dW, db and elsewhere dx are linear_backward_sm100.cu's.
// (K-major: the contraction index is the contiguous one.)  Contraction blocks are 32 fp32 values (one 128-byte
// swizzled row).  A tile is 128 rows by 128, 192 or 256 columns, or 256 rows by 192 or 256, with as many pipeline stages as shared memory holds;
// plan_tiles picks the width.
//
// What bounds the kernel: shared memory takes a contraction block's operands in and hands them to the tensor cores, 128 bytes a
// cycle in all, 2 R + n + R n / 128 cycles for R rows by n columns against R n / 64 in the tensor cores (128 x 192 60 %, 128 x 256
// 67, 256 x 192 71, 256 x 256 80 % of their rate; ncu: 48 % busy in the forward with bf16 planes, 82 % at 8192 x 768 x 3072).
// The result is written straight from registers, 64 bytes of a row per pair of lanes: staging it for the copy engine costs shared
// memory that the pipeline wants, bandwidth, and hand-overs between warps (QKV forward with bf16 planes 72 -> 67 us at 192 columns).
//
// Warp roles (384 threads, one CTA per SM, grid = number of SMs, tiles handed out round robin):
//   warp 0      TMA producer
//   warp 1      MMA issuer (kind::tf32, one elected lane)
//   warp 2      tensor-memory allocation (2 accumulators: the epilogue of one tile overlaps the main loop of the next)
//   warps 4-11  epilogue: 32 rows and half of the columns each, (+ bias, bf16 split) -> global memory, or through a
//               staging buffer of the warp's own to a bulk tensor reduction (dx in pieces) or unaligned rows (vocabulary)
// The waits on barriers are bounded (tc05.cuh).  Two others end for the reasons given there and need no limit: the
// allocation of tensor memory, and the wait for the previous kernel of the stream.
#include "linear_tf32.cuh"

#include "../../include/linear_sm100.h"
#include "../../include/tensor_sm100.h"

namespace lin {
namespace {

using namespace tc05;

constexpr int kThreads = 384;
constexpr int kEpiWarps = 8;

// Tile width kBN (128, 192 or 256 columns) and pipeline depth are chosen per problem: wide tiles halve the
// shared-memory and L2 traffic per flop, narrow ones fill the SMs better when there are few tiles.
template <int kRows, int kBN, int kStages, bool kStage>
struct __align__(1024) SmemT {
    uint8_t a[kStages][kRows * kATileBytes];
    uint8_t b[kStages][kBN * kBK * 4];
    uint8_t out[kStage ? kEpiWarps : 1][kStage ? 4096 : 16];  // output staging of the epilogue warps: 32 rows x 128 bytes
    uint64_t full[kStages], empty[kStages];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

struct Problem {
    int M, N, K;  // C is [M, N]; K is the contraction length
    int rows, bn;  // tile height in blocks of 128 rows, width
    int b_one;    // MN-major B fetched with one 3-D copy per stage (else one copy per 32-row block)
    int tiles_m, tiles_n, splits, kb_total, kb_per_split, total;
    int wide, wide_planes;  // rows of C / of the planes start on 32-byte boundaries
    size_t plane_words;     // distance from the hi to the lo plane
    size_t ldc;             // floats from one row of C to the next
    int m_fast;  // consecutive work items walk down the rows of C (else along its columns)
};

enum Site : int {
    SITE_EMPTY = 201, SITE_FULL, SITE_ACC_EMPTY, SITE_ACC_FULL, SITE_SMEM_ALIGN
};

struct Maps {
    CUtensorMap a, b, c;
};

struct Work {
    int m0, n0, kb0, kb1;  // first row of this CTA's 128, first column of the tile, contraction blocks
};
__device__ __forceinline__ Work decode(const Problem &p, int w) {
    const int split = w % p.splits;
    const int t = w / p.splits;
    // The operand whose tile index changes slowest is read from HBM once; the other one is streamed again for
    // every step of the slow index and has to live in L2.  The host picks the order by operand size.
    const int tn = p.m_fast ? t / p.tiles_m : t % p.tiles_n;
    const int tm = p.m_fast ? t % p.tiles_m : t / p.tiles_n;
    Work r;
    r.m0 = tm * p.rows * kBM;
    r.n0 = tn * p.bn;
    r.kb0 = split * p.kb_per_split;
    r.kb1 = min(p.kb_total, r.kb0 + p.kb_per_split);
    return r;
}

// kEpi 0: C = acc (+ bias), optional bf16 planes; kEpi 1: C += acc (bulk reduction)
// kDirect: the result goes out with plain coalesced 4-byte stores, for outputs whose row pitch is not a multiple of 16
// bytes (the 50257-wide vocabulary projection).
template <bool kBMN, int kEpi, int kRows, int kBN, int kStages, bool kPlanes, bool kDirect>
__global__ void __launch_bounds__(kThreads, 1)
linear_gemm_kernel(const __grid_constant__ Maps maps, const float *__restrict__ bias, float *__restrict__ c_direct,
                   uint32_t *__restrict__ planes, Problem p, int *status) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    using Smem = SmemT<kRows, kBN, kStages, kEpi == 1 || kDirect>;
    constexpr int kAccs = 2 / kRows;  // accumulators of 128 rows, one read out while the other is filled; or one of 256
    constexpr uint32_t kTmemCols = 2 * kBN <= 256 ? 256 : 512;  // a power of two that holds two accumulators
    constexpr int kBTileBytes = kBN * kBK * 4;
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0 && status) atomicCAS(status, 0, ST_TIMEOUT_BASE + SITE_SMEM_ALIGN);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WaitCtx ctx{&sm.abort_flag, status};
    const int first = (int)blockIdx.x, step = (int)gridDim.x;  // work items of this CTA

    if (threadIdx.x == 0) {
        sm.abort_flag = 0;
        for (int i = 0; i < kStages; i++) {
            mbar_init(&sm.full[i], 1);
            mbar_init(&sm.empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.acc_full[i], 1);
            mbar_init(&sm.acc_empty[i], kEpiWarps);  // one arrival per epilogue warp
        }
        fence_barrier_init();
    }
    if (warp == 2) {
        tmem_alloc_then_launch_dependents(&sm.tmem_base, kTmemCols);
    }
    if (warp == 3 && lane == 0) {
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    pdl_wait();  // every thread, before its first access to global memory
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int w = first; ok && w < p.total; w += step) {
                const Work wk = decode(p, w);
                for (int kb = wk.kb0; kb < wk.kb1; kb++, it++) {
                    const int st = it % kStages;
                    if (it >= kStages && !mbar_wait(&sm.empty[st], ((it / kStages) - 1) & 1, ctx, SITE_EMPTY)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&sm.full[st], kRows * kATileBytes + kBTileBytes);
                    auto load = [&](void *dst, const CUtensorMap *map, int c0, int c1, int c2) {
                        tma_load_4d(dst, map, &sm.full[st], c0, c1, c2, 0);
                    };
                    const int b0 = wk.n0;
                    // K-major: map {contraction, rows}, one box {32, 128}.  MN-major: map {rows, contraction},
                    // boxes {32, 32}: blocks of 32 rows, each [32 contraction steps x 128 bytes].
#pragma unroll
                    for (int h = 0; h < kRows; h++) load(sm.a[st] + h * kATileBytes, &maps.a, kb * kBK, wk.m0 + h * kBM, 0);
                    if (kBMN) {
                        if (p.b_one) {
                            load(sm.b[st], &maps.b, 0, kb * kBK, b0 / 32);
                        } else {
#pragma unroll
                            for (int i = 0; i < kBN / 32; i++)
                                load(sm.b[st] + i * 4096, &maps.b, b0 + 32 * i, kb * kBK, 0);
                        }
                    } else {
                        load(sm.b[st], &maps.b, kb * kBK, b0, 0);  // the B map's box is kBN rows
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        constexpr uint32_t idesc = idesc_tf32(kBM, kBN, 0, kBMN ? 1 : 0);
        const uint32_t leader = elect_leader();
        int it = 0, j = 0;
        bool ok = true;
        for (int w = first; ok && w < p.total; w += step, j++) {
            const Work wk = decode(p, w);
            const int acc = j % kAccs;
            if (j >= kAccs && !mbar_wait_warp(&sm.acc_empty[acc], (j / kAccs - 1) & 1, ctx, SITE_ACC_EMPTY)) break;
            tc_fence_after_sync();
            const uint32_t d = tmem + (uint32_t)acc * kBN;
            for (int kb = wk.kb0; kb < wk.kb1; kb++, it++) {
                const int st = it % kStages;
                if (!mbar_wait_warp(&sm.full[st], (it / kStages) & 1, ctx, SITE_FULL)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                // MN-major tiles: 32-row blocks 4096 bytes apart, groups of 4 contraction steps 512 bytes apart
                const uint64_t ad = smem_desc_sw128(smem_u32(sm.a[st]), 16, 1024);
                const uint64_t bd = kBMN ? smem_desc_sw128_base32(smem_u32(sm.b[st]), 4096, 512)
                                         : smem_desc_sw128(smem_u32(sm.b[st]), 16, 1024);
#pragma unroll
                for (int k = 0; k < kBK / 8; k++) {
                    const uint64_t ak = desc_advance(ad, k * 32), bk = desc_advance(bd, k * (kBMN ? 1024 : 32));
                    const uint32_t add = (kb > wk.kb0 || k > 0) ? 1u : 0u;
#pragma unroll
                    for (int h = 0; h < kRows; h++) mma_tf32_lead(leader, d + h * kBN, desc_advance(ak, h * kATileBytes), bk, idesc, add);
                }
                tc_commit_lead(leader, &sm.empty[st]);
            }
            if (!ok) break;
            tc_commit_lead(leader, &sm.acc_full[acc]);
        }
    } else if (warp >= 4) {
        // ------------------------------ epilogue ------------------------------
        // Every warp takes 32 rows (its tensor-memory lane quarter) and half of the columns, 32 at a time: accumulator
        // -> registers (+ bias) -> global memory; what is added into the result, and rows that are not 16-byte aligned,
        // by way of a staging buffer of the warp's own.  No warp waits for another one.
        const int quarter = warp & 3;
        const int half = (warp - 4) >> 2;
        uint8_t *buf = sm.out[kEpi == 1 || kDirect ? warp - 4 : 0];
        const uint32_t lane_addr = (uint32_t)(quarter << 5) << 16;
        constexpr int kChunks = kBN / 64;
        int j = 0;
        for (int w = first; w < p.total; w += step, j++) {
            const Work wk = decode(p, w);
            const int acc = j % kAccs;
            float bv[kChunks];  // bias of the columns col0 + lane, fetched while the tile is still being computed
#pragma unroll
            for (int c = 0; c < kChunks; c++) {
                const int col = wk.n0 + half * (kBN / 2) + 32 * c + lane;
                bv[c] = kEpi == 0 && bias != nullptr && col < p.N ? __ldg(bias + col) : 0.f;
            }
            if (!mbar_wait_warp(&sm.acc_full[acc], (j / kAccs) & 1, ctx, SITE_ACC_FULL)) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (int i = 0; i < kRows * kChunks; i++) {
                const int h = i / kChunks, c = i % kChunks;
                const int row0 = wk.m0 + h * kBM + 32 * quarter;
                const int off = half * (kBN / 2) + 32 * c, col0 = wk.n0 + off;
                uint32_t r[32];
                tmem_ld32(tmem + lane_addr + (uint32_t)(acc + h) * kBN + off, r);
                tmem_wait_ld();
                if (i == kRows * kChunks - 1) {  // the accumulator has been read out: the tensor cores may reuse it
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.acc_empty[acc]);
                }
                const float mine = c == 0 ? bv[0] : c == 1 ? bv[1] : c == 2 ? bv[2 % kChunks] : bv[3 % kChunks];
                if (kEpi == 0 && !kDirect) {
                    const int odd = lane & 1, col = col0 + 16 * odd;
                    exchange_halves(odd, r);
                    if (bias != nullptr) {
#pragma unroll
                        for (int e = 0; e < 16; e++) {
                            const float add = __shfl_sync(0xffffffffu, mine, 16 * odd + e);
                            r[e] = __float_as_uint(__uint_as_float(r[e]) + add);
                            r[16 + e] = __float_as_uint(__uint_as_float(r[16 + e]) + add);
                        }
                    }
#pragma unroll
                    for (int o = 0; o < 2; o++) {
                        const int row = row0 + lane - odd + o;
                        if (row >= p.M) continue;
                        store_words<4>(c_direct + (size_t)row * p.ldc + col, p.N - col, p.wide, r + 16 * o);
                        if (kPlanes) {
                            uint32_t hp[8], lp[8];
#pragma unroll
                            for (int e = 0; e < 8; e++)
                                split_bf16x2(__uint_as_float(r[16 * o + 2 * e]), __uint_as_float(r[16 * o + 2 * e + 1]), hp[e], lp[e]);
                            uint32_t *hi = planes + ((size_t)row * p.N + col) / 2;
                            store_words<2>(hi, (p.N - col) / 2, p.wide_planes, hp);
                            store_words<2>(hi + p.plane_words, (p.N - col) / 2, p.wide_planes, lp);
                        }
                    }
                    continue;
                }
                if (kDirect && bias != nullptr) {
#pragma unroll
                    for (int e = 0; e < 32; e++)
                        r[e] = __float_as_uint(__uint_as_float(r[e]) + __shfl_sync(0xffffffffu, mine, e));
                }
                if (!kDirect && lane == 0) bulk_wait_read_all();  // the copy engine has read the buffer out
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; q++)  // one row of 128 bytes per lane, 16-byte words swizzled
                    *reinterpret_cast<uint4 *>(buf + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                        make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                if (kDirect) {
                    // every row leaves as 32 consecutive floats in one warp instruction
                    __syncwarp();
#pragma unroll 8
                    for (int rr = 0; rr < 32; rr++) {
                        const float v = *reinterpret_cast<const float *>(buf + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) +
                                                                         ((lane & 3) << 2));
                        if (row0 + rr < p.M && col0 + lane < p.N) c_direct[(size_t)(row0 + rr) * p.N + col0 + lane] = v;
                    }
                    continue;
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_reduce_add_3d(buf, &maps.c, col0, row0, 0);
                    bulk_commit();
                }
            }
        }
        if (kEpi == 1 && lane == 0) bulk_wait_read_all();  // shared memory stays until it has been read
    }

    // ------------------------------ tear-down ------------------------------
    if (sm.abort_flag) __nanosleep(50000);
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// db[n] += sum_m dy[m, n].  A block covers 128 columns, four per lane, and every 8th row of its share of the rows; the
// loads of four rows are in flight per thread.  kWords: a lane's columns are one float4 (the pitch is a multiple of 4),
// else they are 32 apart and read one by one.
template <bool kWords>
__global__ void __launch_bounds__(256) bias_grad_kernel(const float *__restrict__ dy, float *__restrict__ db, int M, int N,
                                                        int pitch) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    __shared__ float4 part[8][32];
    const int lane = threadIdx.x & 31, rl = threadIdx.x >> 5;
    constexpr int kApart = kWords ? 1 : 32;
    const int col = blockIdx.x * 128 + (kWords ? 4 * lane : lane);
    auto load = [&](int m) -> float4 {
        const float *at = dy + (size_t)m * pitch + col;
        if (kWords) return __ldcs(reinterpret_cast<const float4 *>(at));
        return make_float4(__ldcs(at), col + 32 < N ? __ldcs(at + 32) : 0.f, col + 64 < N ? __ldcs(at + 64) : 0.f,
                           col + 96 < N ? __ldcs(at + 96) : 0.f);
    };
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (col < N) {
        const int step = gridDim.y * 8;
        int m = blockIdx.y * 8 + rl;
        for (; m + 3 * step < M; m += 4 * step) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = load(m + u * step);
#pragma unroll
            for (int u = 0; u < 4; u++) acc.x += v[u].x, acc.y += v[u].y, acc.z += v[u].z, acc.w += v[u].w;
        }
        for (; m < M; m += step) {
            const float4 v = load(m);
            acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
        }
    }
    part[rl][lane] = acc;
    __syncthreads();
    if (rl == 0 && col < N) {
        float4 t = part[0][lane];
#pragma unroll
        for (int i = 1; i < 8; i++) t.x += part[i][lane].x, t.y += part[i][lane].y, t.z += part[i][lane].z, t.w += part[i][lane].w;
        if (kWords && col + 3 < N && (reinterpret_cast<uintptr_t>(db + col) & 15u) == 0) {
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(db + col), "f"(t.x), "f"(t.y), "f"(t.z), "f"(t.w)
                         : "memory");
            return;
        }
        atomicAdd(db + col, t.x);
        if (col + kApart < N) atomicAdd(db + col + kApart, t.y);
        if (col + 2 * kApart < N) atomicAdd(db + col + 2 * kApart, t.z);
        if (col + 3 * kApart < N) atomicAdd(db + col + 3 * kApart, t.w);
    }
}

// A matrix as the sum of its pieces, `words` 16-byte words each, in their order: they come from L2, four at a time.
__global__ void __launch_bounds__(256) sum_pieces_kernel(float4 *__restrict__ out, const float4 *__restrict__ parts, size_t words, int pieces) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < words; i += (size_t)gridDim.x * 256) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p0 = 0; p0 < pieces; p0 += 4) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = p0 + u < pieces ? __ldcs(parts + (p0 + u) * words + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; u++) sum = make_float4(sum.x + v[u].x, sum.y + v[u].y, sum.z + v[u].z, sum.w + v[u].w);
        }
        out[i] = sum;
    }
}

// dst[M, Np] = src[M, N] with zero columns N..Np-1: a copy of dy whose rows start on 16-byte boundaries, for
// outputs of layers whose feature count is not a multiple of 4 (the vocabulary projection).
__global__ void __launch_bounds__(256) pad_rows_kernel(float *__restrict__ dst, const float *__restrict__ src, int M, int N,
                                                       int Np) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    // One block per row at a time.  The source row starts `o` floats past a 16-byte boundary (src itself is
    // 16-byte aligned): every thread loads the two aligned 16-byte words around its four values and picks them
    // out, so that loads and stores are all 16 bytes wide (the neighbour thread's copy of a word comes from L1).
    // Four such pairs are in flight per thread.  Words that reach past the end of src are read value by value.
    const size_t total = (size_t)M * N;
    const int nv = Np >> 2;
    auto load_word = [&](size_t at) -> float4 {
        if (at + 3 < total) return __ldg(reinterpret_cast<const float4 *>(src + at));
        float4 t;
        t.x = at < total ? src[at] : 0.f;
        t.y = at + 1 < total ? src[at + 1] : 0.f;
        t.z = at + 2 < total ? src[at + 2] : 0.f;
        t.w = at + 3 < total ? src[at + 3] : 0.f;
        return t;
    };
    constexpr int kU = 4;
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        const size_t start = (size_t)m * N;
        const int o = (int)(start & 3);
        const size_t base = start - o;  // multiple of 4
        float4 *out = reinterpret_cast<float4 *>(dst + (size_t)m * Np);
        for (int j0 = threadIdx.x; j0 < nv; j0 += 256 * kU) {
            float4 a[kU], b[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const int j4 = j0 + 256 * u;
                a[u] = b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j4 < nv) {
                    a[u] = load_word(base + 4 * (size_t)j4);
                    if (o != 0) b[u] = load_word(base + 4 * (size_t)(j4 + 1));
                }
            }
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const int j4 = j0 + 256 * u;
                if (j4 >= nv) continue;
                const float v[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
                float r[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float pick = o == 0 ? v[e] : (o == 1 ? v[e + 1] : (o == 2 ? v[e + 2] : v[e + 3]));
                    r[e] = 4 * j4 + e < N ? pick : 0.f;
                }
                __stcs(out + j4, make_float4(r[0], r[1], r[2], r[3]));
            }
        }
    }
}

// ---- host side ----

Problem make_problem(int M, int N, int K, int rows, int bn, int splits) {
    Problem p;
    p.M = M, p.N = N, p.K = K, p.rows = rows, p.bn = bn;
    p.b_one = 0;
    p.m_fast = 0;
    p.ldc = (size_t)N;
    p.tiles_m = (M + rows * kBM - 1) / (rows * kBM);
    p.tiles_n = (N + bn - 1) / bn;
    p.kb_total = (K + kBK - 1) / kBK;
    if (splits < 1) splits = 1;
    if (splits > p.kb_total) splits = p.kb_total;
    p.kb_per_split = (p.kb_total + splits - 1) / splits;
    p.splits = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;  // every split is non-empty
    p.total = p.tiles_m * p.tiles_n * p.splits;
    return p;
}

// Tile shape and number of pieces of the contraction for a [M, N] result of kb contraction blocks, chosen by expected
// time: a fixed part, and for every round over the SMs a charge and kb blocks at the slower of what one CTA takes when
// it is alone (`block`) and what L2 needs to feed all CTAs of the round.  The constants of 128 rows were fitted to the kernel's times
// on 224 shapes of 100 to 8192 rows and 512 to 6400 columns (mean error 5 %) before results left in pieces of 64 bytes of a row, which
// made the rounds of short contractions shorter; those of 256 rows come from the shapes below.  Wide tiles read the least per flop and
// win when there are many, narrow ones leave a smaller last round.
struct Plan {
    int rows, bn, splits;
    int ns;
};
struct Cost {
    int rows, bn, fixed, round, block;  // nanoseconds
};
// Tiles of 256 rows take a third less from L2 and shared memory per product (a block of 256 x 192 in 0.52 us where two of 128 x 192
// take 0.67), but have one accumulator: nothing is computed while a tile leaves.  They win where the contraction is long or they
// end in fewer rounds (us, 128 rows -> 256: 8192 x 768 x 3072 66 -> 59, 8192 x 2304 x 768 with planes 60 -> 57.5, 1500 x 4800 x
// 1600 with planes 54 -> 49; 8192 x 3072 x 768 67.7 -> 68.2, 1500 x 1600 x 6400 61 -> 99).
constexpr Cost kCosts[5] = {{1, 256, 4470, 2030, 283}, {1, 192, 4450, 900, 232}, {1, 128, 3920, 400, 226}, {2, 256, 5000, 5600, 620}, {2, 192, 4500, 4000, 520}};
constexpr int kL2BytesPerNs = 18190;

// Time of `tiles` tiles of kb contraction blocks each, without the fixed part.
long long rounds_ns(const Cost &c, long long tiles, int kb, int sms) {
    const long long bytes = c.rows * kATileBytes + (long long)c.bn * kBK * 4;  // a CTA's operands of one block
    auto round = [&](long long busy) {
        const long long fed = bytes * busy / kL2BytesPerNs;
        return c.round + kb * (fed > c.block ? fed : c.block);
    };
    const long long rest = tiles % sms;
    return tiles / sms * round(sms) + (rest ? round(rest) : 0);
}

int at_most_int(long long v) { return v < 0x7fffffff ? (int)v : 0x7fffffff; }

// What does not fit in L2 arrives from HBM at 5.0 TB/s, after a start of 6 us.
Plan plan_tiles(int M, int N, int kb, int sms) {
    Plan best{1, 128, 1, 0};
    const long long bytes = 4ll * ((long long)M * N + (long long)kb * kBK * (M + N));
    const long long least = bytes > (100ll << 20) ? 6000 + bytes / 5000 : 0;
    for (const Cost &c : kCosts) {
        if (c.bn > 128 && N < c.bn) continue;
        const long long tiles = (long long)((M + c.rows * kBM - 1) / (c.rows * kBM)) * ((N + c.bn - 1) / c.bn);
        long long t = c.fixed + rounds_ns(c, tiles, kb, sms);
        if (t < least) t = least;
        if (best.ns == 0 || t < best.ns) best = Plan{c.rows, c.bn, 1, at_most_int(t)};
    }
    return best;
}

// The same with the contraction cut into up to 32 pieces that add into the result with bulk reductions (dx when
// its contraction is very long); those cost 80 ns per megabyte and make a block 15 % slower.
Plan plan_pieces(int M, int N, int kb, int sms, int least_blocks, int most = 32) {
    Plan best{1, 128, 1, 0};
    for (const Cost &c : kCosts) {
        if (c.rows > 1 || (c.bn > 128 && N < c.bn)) continue;
        const long long tiles = (long long)((M + kBM - 1) / kBM) * ((N + c.bn - 1) / c.bn);
        const long long tile_bytes = (long long)kBM * c.bn * 4;
        for (int s = 1; s <= most && s <= kb; s++) {
            const int per = (kb + s - 1) / s;
            if (s > 1 && per < least_blocks) break;
            const long long t = c.fixed + rounds_ns(c, tiles * s, per, sms) * 115 / 100 +
                                tiles * s * tile_bytes / 1000 * 80 / 1000;
            if (best.ns == 0 || t < best.ns) best = Plan{1, c.bn, s, at_most_int(t)};
        }
    }
    return best;
}

template <bool kBMN, int kEpi, int kRows, int kBN, int kStages, bool kPlanes, bool kDirect>
int launch_one(const Maps &maps, const float *bias, float *c, void *planes, Problem p, int *status, cudaStream_t s) {
    using Smem = SmemT<kRows, kBN, kStages, kEpi == 1 || kDirect>;
    static_assert(sizeof(Smem) <= 227 * 1024, "shared memory of the Linear kernel");
    static bool attr_done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    auto kernel = linear_gemm_kernel<kBMN, kEpi, kRows, kBN, kStages, kPlanes, kDirect>;
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
        if (e != cudaSuccess) return (int)e;
        attr_done[dev] = true;
    }
    p.wide = p.ldc % 8 == 0 && p.N % 8 == 0 && (reinterpret_cast<uintptr_t>(c) & 31u) == 0;
    p.wide_planes = p.N % 16 == 0 && (reinterpret_cast<uintptr_t>(planes) & 31u) == 0;
    p.plane_words = attn::plane_bytes((size_t)p.M * p.N) / 4;
    const int most = attn::sm_count();
    const int grid = p.total < most ? p.total : most;
    return (int)attn::launch_after_previous(kernel, dim3(grid), dim3(kThreads), sizeof(Smem), s, maps, bias, c,
                                                     static_cast<uint32_t *>(planes), p, status);
}

// Pipeline depth by what fits in 227 KiB next to the output staging tile.
template <bool kBMN, int kEpi>
int launch(const Maps &maps, const float *bias, float *c, void *planes, const Problem &p, int *status, cudaStream_t s) {
#define GO(rows, bn, stages, with_planes) \
    return launch_one<kBMN, kEpi, rows, bn, stages, with_planes, false>(maps, bias, c, planes, p, status, s)
    constexpr bool kCanPlanes = !kBMN && kEpi == 0;  // only the forward product writes planes
    if constexpr (kCanPlanes) {
        if (planes && p.rows == 2 && p.bn == 256) GO(2, 256, 3, true);
        if (planes && p.rows == 2) GO(2, 192, 4, true);
        if (planes && p.bn == 256) GO(1, 256, 4, true);
        if (planes && p.bn == 192) GO(1, 192, 5, true);
        if (planes) GO(1, 128, 6, true);
    }
    if constexpr (kEpi == 0) {
        if (p.rows == 2 && p.bn == 256) GO(2, 256, 3, false);
        if (p.rows == 2) GO(2, 192, 4, false);
    }
    if (p.bn == 256) GO(1, 256, 4, false);
    if (p.bn == 192) GO(1, 192, kEpi == 1 ? 4 : 5, false);
    GO(1, 128, 6, false);
#undef GO
}

// C[M, N] = A[M, K] . B[N, K]^T: true when B (the weight) is too large to stay in L2 while every tile row of
// C passes over it and A is the smaller operand; the work items then run down the rows of C, so that B is read
// from HBM once and A (small) is what stays in L2.  (The vocabulary projection: B is 154 MB, A 25 MB.)
int stream_rows_of_c(int M, int N, int K) {
    const size_t a_bytes = (size_t)M * K * 4, b_bytes = (size_t)N * K * 4;
    return b_bytes > ((size_t)48 << 20) && b_bytes > a_bytes ? 1 : 0;
}

bool aligned16(const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; }

// Whether a caller has to bring room for the copy: wherever it may be made.
bool wants_scratch(int M, int N) { return N % 32 != 0 && (N % 4 == 0 || M < 4096 || (long long)M * N < (32 << 20)); }

// dx[M,K] = g[M,np] . w[N,K]: contraction over N (rows of w past N read as zeros)
struct InputGradient {
    Plan tiles;
    int split;  // > 0: the kernel for results of few tiles, with that many CTAs per tile
    int ns;
};
InputGradient plan_input_gradient(int M, int np, int K, int sms) {
    const int kb = np / kBK;
    InputGradient r;
    r.tiles = plan_tiles(M, K, kb, sms);
    // Pieces of the contraction may fill the SMs better, although dx has to be zeroed first.  Any number where it is very long
    // (the vocabulary projection), else two, whose sum does not depend on their order, and if they are expected to save more
    // than the estimate's error (M, N, K: 900, 5120, 1280 41 -> 26 us, 3000, 12032, 512 92 -> 78; without a margin 6000, 9999,
    // 768 214 -> 220).
    const bool very_long = kb >= 512;
    Plan cut = plan_pieces(M, K, kb, sms, 32, very_long ? 32 : 2);
    cut.ns += 2500 + (int)((long long)M * K * 4 / 5500);
    if (cut.splits > 1 && (very_long ? cut.ns : at_most_int(cut.ns * 21ll / 20)) < r.tiles.ns) r.tiles = cut;
    int split = 1;
    const int split_ns = plan_split(M, K, np, sms, &split);
    r.split = split_ns < r.tiles.ns ? split : 0;
    r.ns = r.split ? split_ns : r.tiles.ns;
    return r;
}
// Whether dx as a product of its own, below 4096 rows over a copy of dy, else over every fourth row, would be whole tiles or two pieces.
bool few_pieces(int M, int N, int K, int sms) {
    if (M < 4096) {
        const InputGradient how = plan_input_gradient(M, (N + 31) / 32 * 32, K, sms);
        return how.split || how.tiles.splits <= 2;
    }
    const int kb = (N + 3 + kBK - 1) / kBK;
    const Plan cut = plan_pieces((M + 3) / 4, K, kb, sms, 32);
    return cut.splits <= 2 || cut.ns + (2500 + (int)((long long)M * K * 4 / 5500)) / 4 >= plan_tiles((M + 3) / 4, K, kb, sms).ns;
}
// Whether the gradients of a [M, N] result come from views of every fourth row of dy, whose rows are not 16-byte aligned,
// and not from a copy with padded rows.  The copy is cheap as long as it stays in L2 (128 MB); the views add each tile of dW to
// memory four times, which costs more than the copy where K is large.  From 4096 rows on it is the views in any case.  Copy -> views,
// dx and dW | dx alone, in us (M, N, K):
//     1024, 50257, 768: 409 -> 402 | 251 -> 157       3000, 50257, 384: 712 -> 577 | 447 -> 269     1500, 30001, 768: 356 -> 338 | 222 -> 140
//     2300, 50257, 768: 857 -> 795 | 530 -> 351       3500, 50257, 384: 863 -> 662 | 546 -> 328     3100, 50257, 1024: 1482 -> 1401 | 892 -> 740
//     1800, 30001, 896: 497 -> 528 | 292 -> 250       1500, 22441, 960: 325 -> 340                  2700, 50257, 1024: 1192 -> 1291 | 755 -> 579
//     2400, 50257, 1600: 1644 -> 1807 | 840 -> 827    4090, 50257, 1600: 2481 -> 2986 | 1521 -> 1489
bool by_row_class(int M, int N, int K) {
    if (N % 4 == 0 || (long long)M * N < (32 << 20)) return false;
    return M >= 4096 || (N >= 16384 && M >= 1000 && 3ll * M >= 4ll * K && K <= (M < 2800 ? 768 : 1024));
}

// dx, dW and db (not all of them need be wanted) straight from a dy whose rows are not 16-byte aligned.  The contraction of dx is cut
// into pieces: long sums on the tensor cores, which truncate, lose precision (dx of N = 50257 is 3.9e-5 off from sums of 524 blocks
// of 32, 1.3e-5 from sums of 171).  They add into zeros, three or more of them in no fixed order.  But dx has the same bits in every
// call, with and without dW, where tiles of whole sums would keep the SMs as busy: below 4096 rows the pieces are kept apart, where
// the padded copy would be, and added up behind the launch (2300 x 50257 x 768 774 -> 795 us, elsewhere more: 1500 x 30001 x 768 338 ->
// 361); above, where there is no such room, a CTA takes a tile's pieces in turn (16384 x 50257 x 768 4609 -> 4583, dx alone 2118 -> 2374).
// In no order and without dW, whose ranges make up for it, their number decides how even the last round of tiles is (8192 x 50257 x 768:
// 1009 us from 3 pieces, 1111 from 4).
BackwardPlan plan_by_row_class(int M, int N, int K, bool want_dx, bool want_dw, int sms) {
    const int kb = (N + 3 + kBK - 1) / kBK;
    const int least = (kb + 523) / 524, by_tiles = plan_pieces((M + 3) / 4, K, kb, sms, 32).splits;
    int pieces = least > by_tiles ? least : by_tiles;
    const DxPieces how = pieces <= 2 || !few_pieces(M, N, K, sms) ? kDxAdded : M < 4096 ? kDxApart : kDxInTurn;
    if (how == kDxApart && pieces > (N + 31) / 32 * 32 / K) pieces = (N + 31) / 32 * 32 / K;  // as many as there is room for
    BackwardPlan plan = plan_backward(M, N, K, want_dx, want_dw, sms, 4, pieces, how);
    for (int more = 1; want_dx && !want_dw && pieces > 2 && how == kDxAdded && more <= 2; more++) {
        const BackwardPlan other = plan_backward(M, N, K, true, false, sms, 4, pieces + more);
        if (other.ns < plan.ns) plan = other;
    }
    return plan;
}
int gradients_by_row_class(const BackwardPlan &plan, const float *dy, const float *x, const float *w, float *dx, float *dw, float *db,
                           void *scratch, int M, int N, int K, int sms, int *status, cudaStream_t s) {
    const bool apart = dx && plan.dx_how == kDxApart;
    float *parts = static_cast<float *>(scratch);
    if (dx && plan.dx_how == kDxAdded && plan.dx_pieces > 1) {
        const int rc = tensor_sm100_fill(dx, (size_t)M * K, 0.f, s);
        if (rc != 0) return rc;
    }
    const int rc = launch_backward_by_row_class(plan, dy, x, w, apart ? parts : dx, dw, db, M, N, K, status, s);
    if (rc != 0 || !apart) return rc;
    return (int)attn::launch_after_previous(sum_pieces_kernel, dim3(sms * 8), dim3(256), 0, s, reinterpret_cast<float4 *>(dx),
                                            reinterpret_cast<const float4 *>(parts), (size_t)M * K / 4, plan.dx_pieces);
}

int input_gradient(const InputGradient &how, const float *g, const float *w, float *dx, int M, int N, int np, int K, int sms, int *status,
                   cudaStream_t s) {
    if (how.split) return launch_split(g, w, true, N, nullptr, dx, nullptr, M, K, np, how.split, sms, status, s);
    const Plan &plan = how.tiles;
    int rc;
    Maps maps = {};
    Problem p = make_problem(M, K, np, plan.rows, plan.bn, plan.splits);
    if ((rc = map_k_major(&maps.a, g, M, np, 128)) != 0) return rc;
    p.b_one = map_mn_major_blocks(&maps.b, w, N, K, p.bn / 32) == 0;
    if (!p.b_one && (rc = map_mn_major(&maps.b, w, N, K)) != 0) return rc;
    if (p.splits == 1) return launch<true, 0>(maps, nullptr, dx, nullptr, p, status, s);
    // the pieces of the contraction add into dx with bulk reductions: start from zeros
    if ((rc = map_out_f32(&maps.c, dx, M, K)) != 0) return rc;
    if ((rc = tensor_sm100_fill(dx, (size_t)M * K, 0.f, s)) != 0) return rc;
    return launch<true, 1>(maps, nullptr, dx, nullptr, p, status, s);
}

// Contraction blocks of dW that one accumulator sums up at most; it loses precision with them, since the tensor cores truncate.  As many
// as where every CTA had one piece of the same size, or 160: ranges of 158 blocks in two sums cost 8192 x 3072 x 768 139 -> 142 us, and
// one sum adds 1.2e-5 to the 7.7e-4 of the operands.  A longer range takes several sums, which add up in memory (18917 x
// 6368 x 544: four of 148 blocks, 1.0e-5 and 332 us, where one of 592 gives 3.2e-5 and 320).
int longest_dw_sum(int N, int K, int kb, int sms) {
    const int pieces = plan_pieces(N, K, kb, sms, 1).splits, even = (kb + pieces - 1) / pieces;
    return even > 160 ? even : 160;
}

// How the backward makes dx and dW; np: columns of a padded dy.  `in_parts`: one product after the other.
struct Gradients {
    bool classes, together;  // views of dy; dx and dW in one launch
    InputGradient alone;     // dx in a launch of its own, not from views
    BackwardPlan dx, dw;     // dx in a launch of its own, from views; the launch that makes dW, and dx if together
};
Gradients plan_gradients(int M, int N, int K, int np, bool want_dx, bool want_dw, bool in_parts, int sms) {
    Gradients g = {};
    g.classes = by_row_class(M, N, K);
    if (g.classes) {
        g.together = want_dx && want_dw && !in_parts;
        if (want_dx && !g.together) g.dx = plan_by_row_class(M, N, K, true, false, sms);
        if (want_dw) g.dw = plan_by_row_class(M, N, K, g.together, true, sms);
        return g;
    }
    if (want_dx) g.alone = plan_input_gradient(M, np, K, sms);
    if (!want_dw) return g;
    g.dw = plan_backward(M, N, K, false, true, sms);
    const int most = longest_dw_sum(N, K, g.dw.dw_kb, sms);
    g.dw.dw_most = most;
    // dx has the same bits with and without dW: one launch only where dx alone would be whole tiles too
    if (!want_dx || in_parts || g.alone.split || g.alone.tiles.splits > 1) return g;
    const BackwardPlan both = plan_backward(M, N, K, true, true, sms);
    g.together = both.ns < g.alone.ns + g.dw.ns;
    if (g.together) g.dw = both, g.dw.dw_most = most;
    return g;
}

// Whether a result lies over something that another product of the same call reads or writes: then the products have to
// follow each other, dx first and db last.
bool overlapping(const float *dy, const float *x, const float *w, const float *dx, const float *dw, const float *db, int M, int N, int K) {
    struct Range {
        const float *at;
        size_t n;
    };
    const Range r[6] = {{dx, (size_t)M * K}, {dw, (size_t)N * K}, {db, (size_t)N},
                        {dy, (size_t)M * N}, {x, (size_t)M * K},  {w, (size_t)N * K}};
    for (int i = 0; i < 3; i++)
        for (int j = i + 1; j < 6; j++)
            if (r[i].at && r[j].at && r[i].at < r[j].at + r[j].n && r[j].at < r[i].at + r[i].n) return true;
    return false;
}

}  // namespace
}  // namespace lin

extern "C" {

int linear_sm100_forward(const float *x, const float *w, const float *bias, float *y, void *planes, int M, int N, int K,
                         void *stream) {
    using namespace lin;
    if (!x || !w || !y) return ATTN_ERR_NULL;
    if (M <= 0 || N <= 0 || K <= 0 || (long long)M * N > 0x7fffffffLL || (long long)M * K > 0x7fffffffLL) return ATTN_ERR_SHAPE;
    const bool direct = N % 4 != 0;  // y's rows are not 16-byte aligned: no copy engine for the output
    if (K % 4 != 0 || (planes && N % 8 != 0)) return ATTN_ERR_UNSUPPORTED;
    if (!aligned16(x) || !aligned16(w) || (!direct && (!aligned16(y) || (bias && !aligned16(bias)))) ||
        (planes && !aligned16(planes)))
        return ATTN_ERR_ALIGN;
    int *status = nullptr;
    int rc = attn::device_status_word(&status);
    if (rc != ATTN_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int sms = attn::sm_count();
    const Plan plan = plan_tiles(M, N, (K + kBK - 1) / kBK, sms);
    int split = 1;
    if (plan_split(M, N, K, sms, &split) < plan.ns)
        return launch_split(x, w, false, 0, bias, y, planes, M, N, K, split, sms, status, s);
    Maps maps = {};
    // with plain stores (N not a multiple of 4) only the widest tiles are built
    Problem p = make_problem(M, N, K, direct ? 1 : plan.rows, direct ? 256 : plan.bn, 1);
    p.m_fast = stream_rows_of_c(M, N, K);
    if ((rc = map_k_major(&maps.a, x, M, K, 128)) != 0) return rc;
    if ((rc = map_k_major(&maps.b, w, N, K, p.bn)) != 0) return rc;
    if (direct) return launch_one<false, 0, 1, 256, 4, false, true>(maps, bias, y, nullptr, p, status, s);
    return launch<false, 0>(maps, bias, y, planes, p, status, s);
}

size_t linear_sm100_backward_scratch_bytes(int M, int N, int K) {
    (void)K;
    if (M <= 0 || N <= 0 || !lin::wants_scratch(M, N)) return 0;
    const size_t np = ((size_t)N + 31) / 32 * 32;
    return (size_t)M * np * sizeof(float);
}

int linear_sm100_backward(const float *dy, const float *x, const float *w, float *dx, float *dw, float *db, void *scratch,
                          int M, int N, int K, void *stream) {
    using namespace lin;
    if (!dy || !w || (!dx && !dw) || (dw && !x)) return ATTN_ERR_NULL;
    if (M <= 0 || N <= 0 || K <= 0 || (long long)M * N > 0x7fffffffLL || (long long)M * K > 0x7fffffffLL) return ATTN_ERR_SHAPE;
    if (K % 32 != 0) return ATTN_ERR_UNSUPPORTED;
    const int np = (N + 31) / 32 * 32;
    if ((long long)M * np > 0x7fffffffLL) return ATTN_ERR_SHAPE;
    if (wants_scratch(M, N) && !scratch) return ATTN_ERR_NULL;
    // dy itself must start on a 16-byte boundary in both cases: the padding kernel reads it in 16-byte words
    if (!aligned16(dy) || !aligned16(x) || !aligned16(w) || !aligned16(dx) || !aligned16(dw) ||
        (N % 32 == 0 && !aligned16(db)) || !aligned16(scratch))
        return ATTN_ERR_ALIGN;
    int *status = nullptr;
    int rc = attn::device_status_word(&status);
    if (rc != ATTN_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int sms = attn::sm_count();
    const bool in_parts = dw && overlapping(dy, x, w, dx, dw, db, M, N, K);
    const Gradients how = plan_gradients(M, N, K, np, dx != nullptr, dw != nullptr, in_parts, sms);
    float *dx_too = how.together ? dx : nullptr, *db_too = in_parts ? nullptr : db;
    const bool classes = how.classes;
    const float *g = dy;  // without row classes [M, np] from here on
    if (N % 32 != 0 && !classes) {  // dy's rows cannot be tiles of the copy engine: work on a padded copy
        rc = (int)attn::launch_after_previous(pad_rows_kernel, dim3(sms * 16), dim3(256), 0, s, static_cast<float *>(scratch), dy, M,
                                              N, np);
        if (rc != 0) return rc;
        g = static_cast<const float *>(scratch);
    }
    if (dx && !how.together) {
        rc = classes ? gradients_by_row_class(how.dx, dy, x, w, dx, nullptr, nullptr, scratch, M, N, K, sms, status, s)
                     : input_gradient(how.alone, g, w, dx, M, N, np, K, sms, status, s);
        if (rc != 0) return rc;
    }
    if (dw) {
        rc = classes ? gradients_by_row_class(how.dw, dy, x, w, dx_too, dw, db_too, scratch, M, N, K, sms, status, s)
                     : launch_backward(how.dw, g, x, w, N, dx_too, dw, db_too, M, N, np, K, status, s);
        if (rc != 0 || !in_parts) return rc;
    }
    if (db) {
        // eight blocks per SM, so that enough loads are on their way (six columns of 32 blocks took 9.2 us at
        // 8192 x 768), but at least four rows for each of a block's eight row lanes
        const int across = (N + 127) / 128, fill = 8 * sms / across, by = (M + 31) / 32 < fill ? (M + 31) / 32 : (fill > 1 ? fill : 1);
        dim3 grid((unsigned)((N + 127) / 128), (unsigned)by);
        rc = (int)attn::launch_after_previous(classes ? bias_grad_kernel<false> : bias_grad_kernel<true>, grid, dim3(256), 0, s, g,
                                              db, M, N, classes ? N : np);
    }
    return rc;
}

int linear_sm100_backward_plan(int M, int N, int K, int want_dx, int want_dw, int sms, int *plan) {
    using namespace lin;
    if (!plan) return ATTN_ERR_NULL;
    if (M <= 0 || N <= 0 || K <= 0 || sms <= 0 || (!want_dx && !want_dw) || (long long)M * N > 0x7fffffffLL || (long long)M * K > 0x7fffffffLL)
        return ATTN_ERR_SHAPE;
    if (K % 32 != 0) return ATTN_ERR_UNSUPPORTED;
    const Gradients how = plan_gradients(M, N, K, (N + 31) / 32 * 32, want_dx, want_dw, false, sms);
    const BackwardPlan &one = want_dw ? how.dw : how.dx;  // nothing in it for dx alone, not from views
    const int pieces = !want_dx ? 0 : how.classes ? one.dx_pieces : how.alone.split ? 1 : how.alone.tiles.splits;
    const DwLoad load = dw_load(one, M, N, K);
    const int out[9] = {how.together, how.classes ? 4 : 1, one.teams * one.team, one.team, one.down, pieces,
                        pieces <= 2 || (how.classes && one.dx_how != kDxAdded), load.cta, load.sum};
    for (int i = 0; i < 9; i++) plan[i] = out[i];
    return ATTN_OK;
}

}  // extern "C"
