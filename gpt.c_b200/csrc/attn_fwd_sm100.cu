// Fused causal attention forward for sm_100a, head size 64.
//
// Replaces attention_forward_cuda_kernel of gpt.c (kernels/src/cuda/Attention.cu:170-232): the
// permute kernel, the QK^T batched SGEMM, the mask and softmax kernels, the PV batched SGEMM and
// the unpermute kernel become one kernel that never writes the T x T matrix.
//
// A work item is one (batch, head) and one tile of 128 query rows; it walks the keys up to the
// diagonal in steps of 64.  Inputs are the bf16 hi/lo planes of the fused QKV tensor; Q/K/V tiles are
// addressed straight inside [B, T, 3C] by a 4-D tensor map (column, row, batch, plane).
//
// The grid has one CTA per item, heaviest first.  The first Q and K tiles are requested while the CTA is still being set
// up, the finished tile leaves by the copy engine from where Q was, or straight from registers where that is sooner.
// A sequence of at most 64 tokens takes one key step.
//
// A CTA is deliberately small (about 100 KiB of shared memory, 256 columns of tensor memory,
// 384 threads) so that TWO CTAs share an SM.  Inside a CTA two score buffers alternate, so the
// tensor cores compute S of the next key step while the softmax warps work on the current one.
// In the steady state a step takes about 1000 cycles of an SM, 800 of which its 24 MMAs execute.
//
// Warp roles (384 threads):
//   warp 0       TMA producer for Q and K (two-stage ring)
//   warp 1       tensor-memory allocation / release
//   warp 2       MMA issuer (not on the scheduler of the TMA warps: 2 % faster): S = Q K^T (Q from tensor memory, K K-major from shared memory) and O += P V (P from tensor memory,
//                V MN-major from shared memory), each as hi*hi + hi*lo + lo*hi; the whole warp
//                runs the loop, one elected lane issues
//   warp 3       TMA producer for V (two-stage ring)
//   warps 4-11   softmax: two threads per query row.  The warp quarter (warp % 4) selects the 32
//                rows the warp may touch in tensor memory, the warp half selects 32 of the 64
//                score columns of a step and 32 of the 64 output columns; the halves exchange
//                their row maximum through shared memory.
//
// Tensor memory (256 columns): S0 [0,64), S1 [64,128), O [128,192), Q hi/lo [192,256) (the A operand
// of S = Q K^T, copied once from shared memory).  P overwrites S in place: each run of 16
// score columns becomes 8 columns of packed bf16 hi parts followed by 8 columns of packed lo
// parts.  O accumulates in tensor memory across key tiles (the PV MMAs accumulate); the running
// reference maximum only moves when a row maximum exceeds it by more than 2^8, and only then is
// the accumulator rescaled in place.
#include "attn24.cuh"
#include "attn_internal.h"
#include "tc05.cuh"

namespace attn {
namespace {

using namespace tc05;

constexpr int kTile = 128;  // query rows per CTA
constexpr int kStep = 64;   // keys per step
constexpr int kD = 64;
constexpr int kPlaneTile = kTile * kD * 2;  // bytes of one bf16 plane of the Q tile (16 KiB)
constexpr int kPlaneStep = kStep * kD * 2;  // bytes of one bf16 plane of a K / V step (8 KiB)
constexpr int kThreads = 384;
constexpr int kSoftmaxWarps = 8;
constexpr uint32_t kTmemCols = 256;
static_assert(2 * kTmemCols <= 512, "the two CTAs of an SM have their columns at the same time");
constexpr uint32_t kColS = 0, kColO = 128, kColQ = 192;  // Q: hi plane [192,224), lo plane [224,256)

struct __align__(1024) FwdSmem {
    uint8_t q[2][kPlaneTile];  // [plane]
    uint8_t k[2][2][kPlaneStep];  // [stage][plane]
    uint8_t v[2][2][kPlaneStep];
    uint64_t q_full, q_tmem, k_full[2], k_empty[2], v_full[2], v_empty[2];
    uint64_t s_full[2], p_full[2], o_full;
    uint64_t pair_bar[4];       // [quarter]: the two halves of a row block meet here once per step
    uint64_t o_done;            // the last PV product of an item has completed
    uint64_t staged[2];         // [half]: 32 columns of the output are where Q was
    float xmax[2][2][kTile];    // [step parity][half][row]: row maxima exchanged between halves
    float lpart[2][kTile];      // [half][row]: partial row sums for the epilogue
    uint32_t tmem_base;
    int abort_flag;
};

enum Site : int {
    SITE_K_EMPTY = 1, SITE_V_EMPTY, SITE_Q_FULL, SITE_K_FULL, SITE_V_FULL, SITE_P_FULL, SITE_S_FULL, SITE_O_FULL,
    SITE_O_FULL_LAST, SITE_Q_TMEM, SITE_PAIR, SITE_SMEM_ALIGN, SITE_STAGED
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Rescale threshold of the running reference maximum, in log2 units: the reference only moves
// when a tile's row maximum exceeds it by more than this, so P stays below 2^8 and the O
// accumulator in tensor memory rarely needs rescaling after the first tile.
constexpr float kRescaleThreshold = 8.0f;

// Max pass of one key step.  kDiag: a step that touches the diagonal needs the causal mask; key0
// is the index of the step's first key relative to the first query row of the tile.  On return
// `alpha` is the factor by which the O accumulator must be rescaled before the PV product of
// this tile (1 when the reference maximum did not move).
// Returns false when the bounded wait on the partner half ran out.
template <bool kDiag>
__device__ __forceinline__ bool max_pass(FwdSmem &sm, const WaitCtx &ctx, uint32_t t_s, int row, int half, int par, int key0,
                                         uint64_t *pair_bar, uint32_t pair_parity, float scale_log2, float &m, float &alpha) {
    uint32_t r0[32];
    tmem_ld32(t_s + 32 * half, r0);
    tmem_wait_ld();
    float mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        float a0 = __uint_as_float(r0[e]), a1 = __uint_as_float(r0[e + 1]);
        if (kDiag) {
            if (key0 + 32 * half + e > row) a0 = -INFINITY;
            if (key0 + 32 * half + e + 1 > row) a1 = -INFINITY;
        }
        mx = max3(mx, a0, a1);
    }
    sm.xmax[par][half][row] = mx;
    mbar_arrive(pair_bar);
    if (!mbar_wait_warp(pair_bar, pair_parity, ctx, SITE_PAIR)) return false;
    mx = fmaxf(mx, sm.xmax[par][half ^ 1][row]) * scale_log2;
    const bool move = mx > m + kRescaleThreshold;  // always true on the first tile (m = -inf)
    alpha = move ? ex2(m - mx) : 1.0f;
    m = move ? mx : m;
    return true;
}

// exp pass: P = exp2(s * c - m), written over S in place as packed bf16 hi / lo.  The loads of
// the next 16 columns are in flight while the current 16 are processed.
// Returns this thread's partial row sum.
template <bool kDiag>
__device__ __forceinline__ float exp_pass(uint32_t t_s, int row, int half, int key0, float scale_log2, float m) {
    float2 lsum = make_float2(0.f, 0.f);
    const float2 sc2 = make_float2(scale_log2, scale_log2), mneg2 = make_float2(-m, -m);
    uint32_t r[2][16];
    tmem_ld16(t_s + 32 * half, r[0]);
#pragma unroll
    for (int c = 0; c < 2; c++) {
        tmem_wait_ld();
        if (c < 1) tmem_ld16(t_s + 32 * half + 16, r[1]);
        const uint32_t col = 32 * half + 16 * c;
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const float2 x = fma2(make_float2(__uint_as_float(r[c][2 * e]), __uint_as_float(r[c][2 * e + 1])), sc2, mneg2);
            float2 p = make_float2(ex2(x.x), ex2(x.y));
            if (kDiag) {
                if (key0 + (int)col + 2 * e > row) p.x = 0.f;
                if (key0 + (int)col + 2 * e + 1 > row) p.y = 0.f;
            }
            lsum = add2(lsum, p);
            split_bf16x2_packed(p, hi[e], lo[e]);
        }
        tmem_st8(t_s + col, hi);
        tmem_st8(t_s + col + 8, lo);
    }
    return lsum.x + lsum.y;
}

struct Item {
    int qt, b, h, nsteps;
};
// Items are numbered from the longest query tiles down, all (b, h) of one tile index together.
__device__ __forceinline__ Item decode(int item, int B, int T, int H) {
    const int BH = B * H, nqt = (T + kTile - 1) / kTile;
    Item r;
    r.qt = nqt - 1 - item / BH;
    const int bh = item % BH;
    r.b = bh / H;
    r.h = bh % H;
    r.nsteps = min(2 * (r.qt + 1), (T + kStep - 1) / kStep);  // key steps of 64 up to the diagonal or the end
    return r;
}

__device__ __forceinline__ void load_q(FwdSmem &sm, const CUtensorMap &map_x, const Item &w) {
    mbar_expect_tx(&sm.q_full, 2 * kPlaneTile);
    for (int hf = 0; hf < 2; hf++) {  // the tensor map's box is 64 rows
        tma_load_4d(sm.q[0] + hf * kPlaneStep, &map_x, &sm.q_full, w.h * kD, w.qt * kTile + hf * kStep, w.b, 0);
        tma_load_4d(sm.q[1] + hf * kPlaneStep, &map_x, &sm.q_full, w.h * kD, w.qt * kTile + hf * kStep, w.b, 1);
    }
}
__device__ __forceinline__ void load_k(FwdSmem &sm, const CUtensorMap &map_x, const Item &w, int C, int j, int st) {
    mbar_expect_tx(&sm.k_full[st], 2 * kPlaneStep);
    tma_load_4d(sm.k[st][0], &map_x, &sm.k_full[st], C + w.h * kD, j * kStep, w.b, 0);
    tma_load_4d(sm.k[st][1], &map_x, &sm.k_full[st], C + w.h * kD, j * kStep, w.b, 1);
}

// 32 columns of one row, scaled: 32 bytes per store when the pointer allows it.
__device__ __forceinline__ void store_row(float *dst, const uint32_t (&r)[32], float by) {
    if (aligned32(dst)) {
#pragma unroll
        for (int c = 0; c < 32; c += 8)
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + c), "f"(__uint_as_float(r[c]) * by),
                         "f"(__uint_as_float(r[c + 1]) * by), "f"(__uint_as_float(r[c + 2]) * by), "f"(__uint_as_float(r[c + 3]) * by),
                         "f"(__uint_as_float(r[c + 4]) * by), "f"(__uint_as_float(r[c + 5]) * by), "f"(__uint_as_float(r[c + 6]) * by),
                         "f"(__uint_as_float(r[c + 7]) * by)
                         : "memory");
    } else {
#pragma unroll
        for (int c = 0; c < 32; c += 4)
            *reinterpret_cast<float4 *>(dst + c) = make_float4(__uint_as_float(r[c]) * by, __uint_as_float(r[c + 1]) * by,
                                                               __uint_as_float(r[c + 2]) * by, __uint_as_float(r[c + 3]) * by);
    }
}

// Sequences of at most 64 tokens: the (only) item's Q, K and V come from the fp32 tensor, every thread splits its share
// into the two bf16 planes, in shared memory where the tensor cores read them; two warps with nothing else to do store
// them from there in `saved` for the backward.
// That takes the split kernel, its launch and a second trip through memory out of a pass that is all latency.
__device__ __forceinline__ size_t piece_at(int part, int row, int col, int b, int h, int T, int C) {
    return ((size_t)b * T + row) * 3 * C + part * C + h * kD + 8 * col;
}
__device__ __forceinline__ uint8_t *plane_of(FwdSmem &sm, int part, int lo) {
    return part == 0 ? sm.q[lo] : (part == 1 ? sm.k[0][lo] : sm.v[0][lo]);
}
__device__ __forceinline__ void take_fp32(FwdSmem &sm, const float *__restrict__ qkv, int b, int h, int T, int C) {
    constexpr int kEach = 3 * 8 * kStep / kThreads;  // 32-byte pieces of the 3 x 64 rows for a thread
    static_assert(kEach * kThreads == 3 * 8 * kStep, "every thread has the same number");
    float4 a[kEach][2];  // all on their way before the first is used
    const bool wide = aligned32(qkv);
#pragma unroll
    for (int u = 0; u < kEach; u++) {
        const int i = (int)threadIdx.x + u * kThreads, part = i >> 9, row = (i >> 3) & 63, c = i & 7;
        a[u][0] = a[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < T) load_f32x8(a[u][0], a[u][1], qkv + piece_at(part, row, c, b, h, T, C), wide);
    }
#pragma unroll
    for (int u = 0; u < kEach; u++) {
        const int i = (int)threadIdx.x + u * kThreads, part = i >> 9, row = (i >> 3) & 63, c = i & 7;
        uint4 vh, vl;
        split_bf16x2(a[u][0].x, a[u][0].y, vh.x, vl.x);
        split_bf16x2(a[u][0].z, a[u][0].w, vh.y, vl.y);
        split_bf16x2(a[u][1].x, a[u][1].y, vh.z, vl.z);
        split_bf16x2(a[u][1].z, a[u][1].w, vh.w, vl.w);
        const int at = row * 128 + ((c ^ (row & 7)) << 4);
        *reinterpret_cast<uint4 *>(plane_of(sm, part, 0) + at) = vh;
        *reinterpret_cast<uint4 *>(plane_of(sm, part, 1) + at) = vl;
    }
    fence_proxy_async_smem();
}
// i: 0..63, one of the threads of the two warps.  Stored by every thread, the planes held up the warps that the first product
// waits for (11 sequences of 50 tokens, 6 heads: 6.07 us, 5.28 this way).
__device__ __forceinline__ void save_planes(FwdSmem &sm, int i, __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo, int b,
                                            int h, int T, int C) {
    const int c = i & 7;
#pragma unroll 2
    for (int row = i >> 3; row < T; row += 8) {
        const int from = row * 128 + ((c ^ (row & 7)) << 4);
#pragma unroll
        for (int part = 0; part < 3; part++) {
            const size_t at = piece_at(part, row, c, b, h, T, C);
            *reinterpret_cast<uint4 *>(hi + at) = *reinterpret_cast<const uint4 *>(plane_of(sm, part, 0) + from);
            *reinterpret_cast<uint4 *>(lo + at) = *reinterpret_cast<const uint4 *>(plane_of(sm, part, 1) + from);
        }
    }
}

// Where an item comes from and goes.  kLong: the result leaves by the copy engine.  kRows: from registers, which is the
// shorter way for a CTA that stores part of a tile, once, and has its SM to itself (rows_from_registers).  kFp32: the same,
// and the item comes from the fp32 tensor (sequences of at most 64 tokens).
enum Form : int { kLong, kRows, kFp32 };
template <int kForm>
struct Maps {  // no tensor map that the form does not use: a launch carries them all
    CUtensorMap x, o, copy;
};
template <>
struct Maps<kRows> {
    CUtensorMap x;
};
template <>
struct Maps<kFp32> {};

template <int kForm>
__global__ void __launch_bounds__(kThreads, 2)
attn_fwd_kernel(const __grid_constant__ Maps<kForm> maps, const float *__restrict__ qkv, __nv_bfloat16 *__restrict__ hi,
                __nv_bfloat16 *__restrict__ lo, float *__restrict__ out, float *__restrict__ out_copy, float *__restrict__ lse, int B,
                int T, int H, float scale_log2, int *status) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    FwdSmem &sm = *reinterpret_cast<FwdSmem *>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0 && status) atomicCAS(status, 0, ST_TIMEOUT_BASE + SITE_SMEM_ALIGN);
        return;
    }
    // broadcast, so that the compiler knows the role branches and what they compute to be warp-uniform
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int C = H * kD;
    WaitCtx ctx{&sm.abort_flag, status};

    if constexpr (kForm == kLong) {
        if (threadIdx.x == 96) {
            tma_prefetch_desc(&maps.x);
            tma_prefetch_desc(&maps.o);
            if (out_copy) tma_prefetch_desc(&maps.copy);
        }
    }
    if (threadIdx.x == 0) {
        sm.abort_flag = 0;
        mbar_init(&sm.q_full, 1);
        mbar_init(&sm.q_tmem, kSoftmaxWarps);
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.k_full[i], 1);
            mbar_init(&sm.k_empty[i], 1);
            mbar_init(&sm.v_full[i], 1);
            mbar_init(&sm.v_empty[i], 1);
            mbar_init(&sm.s_full[i], 1);
            mbar_init(&sm.p_full[i], 32 * kSoftmaxWarps);
        }
        for (int i = 0; i < 4; i++) mbar_init(&sm.pair_bar[i], 64);
        mbar_init(&sm.o_full, 1);
        mbar_init(&sm.o_done, 1);
        for (int i = 0; i < 2; i++) mbar_init(&sm.staged[i], kSoftmaxWarps / 2);
        fence_barrier_init();
        // This thread is also the Q/K producer: the first Q and K tiles are requested right away, while the other
        // warps are still setting up (but not before the kernel that wrote them has completed).
        if constexpr (kForm != kFp32) {
            pdl_wait();
            fence_proxy_async_smem();
            if constexpr (kForm == kRows) tma_prefetch_desc(&maps.x);
            const Item w = decode((int)blockIdx.x, B, T, H);
            load_q(sm, maps.x, w);
            for (int j = 0; j < min(2, w.nsteps); j++) load_k(sm, maps.x, w, C, j, j);
        }
    }
    if (warp == 1) {
        tmem_alloc_then_launch_dependents(&sm.tmem_base, kTmemCols);
    }
    pdl_wait();  // every thread, before its first access to global memory
    if (kForm == kFp32) {
        const Item w = decode((int)blockIdx.x, B, T, H);
        take_fp32(sm, qkv, w.b, w.h, T, C);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);

    const Item w = decode((int)blockIdx.x, B, T, H);
    if (kForm == kFp32 && threadIdx.x == 0) {  // what the copy engine signals otherwise
        mbar_arrive(&sm.q_full);
        mbar_arrive(&sm.k_full[0]);
        mbar_arrive(&sm.v_full[0]);
    }

    if (kForm == kFp32 && (warp == 0 || warp == 3)) {
        // no loads to request; these two leave the planes for the backward
        save_planes(sm, (warp == 0 ? 0 : 32) + lane, hi, lo, w.b, w.h, T, C);
    } else if (warp == 0) {
        // ------------------------------ TMA producer: K ------------------------------
        if constexpr (kForm != kFp32) {
            if (lane == 0) {
                for (int n = 2; n < w.nsteps; n++) {  // Q and the first two steps were requested during set-up
                    if (!mbar_wait(&sm.k_empty[n & 1], ((n >> 1) - 1) & 1, ctx, SITE_K_EMPTY)) break;
                    load_k(sm, maps.x, w, C, n, n & 1);
                }
            }
        }
    } else if (warp == 3) {
        // ------------------------------ TMA producer: V ------------------------------
        if constexpr (kForm != kFp32) {
            if (lane == 0) {
                const int xv = 2 * C + w.h * kD;
                for (int n = 0; n < w.nsteps; n++) {
                    const int st = n & 1;
                    if (n >= 2 && !mbar_wait(&sm.v_empty[st], ((n >> 1) - 1) & 1, ctx, SITE_V_EMPTY)) break;
                    mbar_expect_tx(&sm.v_full[st], 2 * kPlaneStep);
                    tma_load_4d(sm.v[st][0], &maps.x, &sm.v_full[st], xv, n * kStep, w.b, 0);
                    tma_load_4d(sm.v[st][1], &maps.x, &sm.v_full[st], xv, n * kStep, w.b, 1);
                }
            }
        }
    } else if (warp == 2) {
        // ------------------------------ MMA issuer ------------------------------
        constexpr uint32_t idesc_s = idesc_bf16_f32(kTile, kStep, 0, 0);
        constexpr uint32_t idesc_o = idesc_bf16_f32(kTile, kD, 0, 1);
        const uint32_t leader = elect_leader();  // the one lane that issues every MMA and commit
        // S of step n+1 is issued before the wait for P of step n: the two score buffers alternate,
        // so the tensor cores work on the next scores while the softmax warps are busy.  S_{n+1}
        // overwrites P_{n-1}; the tensor pipe runs in issue order, so PV_{n-1} has read it by then.
        auto issue_qk = [&](int n) -> bool {
            const int st = n & 1;
            if (!mbar_wait_warp(&sm.k_full[st], (n >> 1) & 1, ctx, SITE_K_FULL)) return false;
            tc_fence_after_sync();
            const uint64_t kd[2] = {smem_desc_sw128(smem_u32(sm.k[st][0]), 16, 1024),
                                    smem_desc_sw128(smem_u32(sm.k[st][1]), 16, 1024)};
            uint32_t acc = 0;
#pragma unroll
            for (int term = 0; term < 3; term++) {
                const int qa = term == 2 ? 1 : 0, kb = term == 1 ? 1 : 0;  // hh, hl, lh
#pragma unroll
                for (int kk = 0; kk < kD / 16; kk++) {
                    mma_ts_lead(leader, tmem + kColS + st * kStep, tmem + kColQ + 32 * qa + 8 * kk, desc_advance(kd[kb], kk * 32),
                                 idesc_s, acc);
                    acc = 1;
                }
            }
            tc_commit_lead(leader, &sm.s_full[st]);
            tc_commit_lead(leader, &sm.k_empty[st]);
            return true;
        };
        bool ok = mbar_wait_warp(&sm.q_tmem, 0, ctx, SITE_Q_TMEM) && issue_qk(0);
        for (int n = 0; ok && n < w.nsteps; n++) {
            const int st = n & 1;
            ok = (n + 1 == w.nsteps || issue_qk(n + 1)) &&
                 // O += P_n V_n
                 mbar_wait_warp(&sm.v_full[st], (n >> 1) & 1, ctx, SITE_V_FULL) &&
                 mbar_wait_warp(&sm.p_full[st], (n >> 1) & 1, ctx, SITE_P_FULL);
            if (!ok) break;
            tc_fence_after_sync();
            const uint64_t vd[2] = {smem_desc_sw128(smem_u32(sm.v[st][0]), 1024, 1024),
                                    smem_desc_sw128(smem_u32(sm.v[st][1]), 1024, 1024)};
            uint32_t acc = n >= 1 ? 1u : 0u;
#pragma unroll
            for (int term = 0; term < 3; term++) {
                const int pa = term == 2 ? 1 : 0, vb = term == 1 ? 1 : 0;  // hh, hl, lh
#pragma unroll
                for (int kk = 0; kk < kStep / 16; kk++) {
                    mma_ts_lead(leader, tmem + kColO, tmem + kColS + st * kStep + 16 * kk + 8 * pa,
                                 desc_advance(vd[vb], kk * 2048), idesc_o, acc);
                    acc = 1;
                }
            }
            tc_commit_lead(leader, &sm.o_full);
            tc_commit_lead(leader, &sm.v_empty[st]);
            if (n == w.nsteps - 1) tc_commit_lead(leader, &sm.o_done);
        }
    } else if (warp >= 4) {
        // ------------------------------ softmax ------------------------------
        const int half = (warp - 4) >> 2;       // which 32 score columns / 32 output columns
        const int quarter = warp & 3;           // TMEM lane quarter this warp may access
        const int row = (quarter << 5) | lane;  // query row inside the tile == TMEM lane
        uint64_t *pair_bar = &sm.pair_bar[quarter];  // one phase per step and one at the end
        const uint32_t lane_addr = (uint32_t)(quarter << 5) << 16;
        const uint32_t t_o = tmem + lane_addr + kColO + 32 * half;

        // Copies this thread's Q row (half 0: hi plane, half 1: lo plane) from the swizzled shared
        // memory tile into tensor memory: 64 bf16 = 32 packed columns, lane = row.
        auto take_q = [&]() -> bool {
            if (!mbar_wait_warp(&sm.q_full, 0, ctx, SITE_Q_FULL)) return false;
            const uint8_t *qrow = sm.q[half] + row * 128;
            uint32_t r[32];
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const uint4 v = *reinterpret_cast<const uint4 *>(qrow + ((c ^ (row & 7)) << 4));
                r[4 * c] = v.x;
                r[4 * c + 1] = v.y;
                r[4 * c + 2] = v.z;
                r[4 * c + 3] = v.w;
            }
            tmem_st32(tmem + lane_addr + kColQ + 32 * half, r);
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.q_tmem);
            return true;
        };

        bool ok = take_q();
        float m = -INFINITY, l = 0.f;
        for (int n = 0; ok && n < w.nsteps; n++) {
            const int st = n & 1;
            const uint32_t t_s = tmem + lane_addr + kColS + st * kStep;
            const int key0 = n * kStep - w.qt * kTile;  // first key of the step relative to the tile's first row
            const bool diag = key0 + kStep - 1 > 0;     // some (row, key) pair of this step is above the diagonal
            if (!mbar_wait_warp(&sm.s_full[st], (n >> 1) & 1, ctx, SITE_S_FULL)) { ok = false; break; }
            tc_fence_after_sync();
            float alpha;
            const bool step_ok = diag
                ? max_pass<true>(sm, ctx, t_s, row, half, st, key0, pair_bar, n & 1, scale_log2, m, alpha)
                : max_pass<false>(sm, ctx, t_s, row, half, st, key0, pair_bar, n & 1, scale_log2, m, alpha);
            if (!step_ok) { ok = false; break; }
            // When the reference maximum of some row of this warp moved, rescale the warp's 32 rows x
            // 32 columns of O in place: after the previous PV product has finished, before P_j is
            // published.  (The barrier completes once per step, and not for this one before P_j is there.)
            if (n >= 1 && __any_sync(0xffffffffu, alpha != 1.0f)) {
                if (!mbar_wait_warp(&sm.o_full, (n - 1) & 1, ctx, SITE_O_FULL)) { ok = false; break; }
                tc_fence_after_sync();
                uint32_t r[32];
                tmem_ld32(t_o, r);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; e++) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
                tmem_st32(t_o, r);
            }
            l = l * alpha + (diag ? exp_pass<true>(t_s, row, half, key0, scale_log2, m)
                                  : exp_pass<false>(t_s, row, half, key0, scale_log2, m));
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(&sm.p_full[st]);
        }
        // O / l for this thread's 32 columns, log-sum-exp by the first half
        sm.lpart[half][row] = l;
        mbar_arrive(pair_bar);
        ok = ok && mbar_wait_warp(pair_bar, w.nsteps & 1, ctx, SITE_PAIR);
        const float l_all = sm.lpart[0][row] + sm.lpart[1][row];
        const float inv = 1.0f / l_all;
        // The last product of an item has a barrier of its own: o_full completes once per key step and this
        // thread has not followed its phases, so a parity wait on it could not tell the last product from the
        // one before.
        if (ok && mbar_wait_warp(&sm.o_done, 0, ctx, SITE_O_FULL_LAST)) {
            tc_fence_after_sync();
            uint32_t r[32];
            tmem_ld32(t_o, r);
            tmem_wait_ld();
            tc_fence_before_sync();
            const int tok = w.qt * kTile + row;
            if (half == 0 && tok < T) lse[((size_t)w.b * H + w.h) * T + tok] = (m + __log2f(l_all)) * 0.6931471805599453f;
            if constexpr (kForm != kLong) {
                if (tok < T) {
                    const size_t at = ((size_t)w.b * T + tok) * C + (size_t)w.h * kD + 32 * half;
                    store_row(out + at, r, inv);
                    if (out_copy) store_row(out_copy + at, r, inv);
                }
            } else {
                // This thread's own row and plane of Q, long in tensor memory, take its 32 columns, and the copy engine takes
                // them from there (rows past the end are dropped).  Rows written from registers, a row per lane in 32-byte
                // pieces, took 1640 cycles at the end of every CTA (B=8 T=128 H=12).
                uint8_t *at = sm.q[half] + row * 128;
#pragma unroll
                for (int c = 0; c < 8; c++)
                    *reinterpret_cast<float4 *>(at + ((c ^ (row & 7)) << 4)) =
                        make_float4(__uint_as_float(r[4 * c]) * inv, __uint_as_float(r[4 * c + 1]) * inv, __uint_as_float(r[4 * c + 2]) * inv,
                                    __uint_as_float(r[4 * c + 3]) * inv);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sm.staged[half]);
                    if (quarter == 0 && mbar_wait(&sm.staged[half], 0, ctx, SITE_STAGED)) {
                        tma_store_3d(sm.q[half], &maps.o, w.h * kD + 32 * half, w.qt * kTile, w.b);
                        if (out_copy) tma_store_3d(sm.q[half], &maps.copy, w.h * kD + 32 * half, w.qt * kTile, w.b);
                        bulk_commit();
                        bulk_wait_read_all();  // shared memory stays alive until then
                    }
                }
            }
        }
    }

    // ------------------------------ tear-down ------------------------------
    if (sm.abort_flag) __nanosleep(50000);  // let copies that are still in flight land
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// ---------------------------------------------------------------------------------------
// General forward: any head size up to 128, fp32 operands as three bf16 terms (attn24.cuh).
//
// One CTA per (b, h, 128 queries), heaviest first; it walks the keys in steps of 64.  S = Q K^T with Q from tensor memory
// and K from shared memory, P back to tensor memory as three terms, O_step = P V added to the running output in registers.
// The 16 worker warps convert K of the next step and start its scores before they turn to the softmax of this one, and
// convert V behind the softmax, so the tensor cores have the next scores and this step's P V ahead of them.
//
// The CTA of a query tile also leaves the bf16 planes of that tile's rows for the backward: Q at the start, K and V when it
// gets to the diagonal.
//
// What bounds it: the chain inside a step, conversion of K and V, softmax, sums in registers, beside 12 bf16 passes over both
// products: a step takes 3900 cycles at D = 128, of which the tensor cores need 3200 (active 51 % of the whole kernel, the
// start and end of its CTAs included).
// ---------------------------------------------------------------------------------------
namespace general {

using namespace attn24;

template <int kK>  // head columns in groups of 16
struct __align__(1024) Fwd24Smem {
    static constexpr int kBlocks = (kK + 3) / 4, kPlane = kBlocks * kStep * 128;  // bytes of one term of a K or V tile
    uint8_t k[3][kPlane], v[3][kPlane];  // before the first step: the three terms of Q, 128 rows each
    float raw[2][kStep * 16 * kK];       // K, V of the next step as they come; first the halves of Q
    uint64_t raw_full[2], raw_free[2];
    uint64_t go_s, go_pv, done_s, done_pv;
    float part[2][4][kTile];  // [step parity][column quarter][row]: row maxima, at the end row sums
    uint32_t odd[4][4];       // [column quarter][row / 32]: a bit per row of a result that is not finite
    uint32_t tmem_base;
    int abort_flag;
};

// The rows of this CTA's tile that are marked in `odd`, over again in fp32 arithmetic, a warp per row: a term of an infinite
// operand, or of a finite one that rounds up to infinity, is not a number, and so is the product of its infinite term with a
// zero term of the other operand.  A row that stays NaN ends at the first score that decides it: NaN in every input costs 15 to
// 30 us, a NaN in v of one of B=4 T=1024 H=6 D=128, where eight CTAs do 1021 rows again, 2.4 ms (one load after the other 6.3).
// A function of its own, behind the last barrier: inlined, or called from the workers' branch, it made the
// loop over the keys up to 10 % slower.
__device__ __noinline__ void exact_rows(const uint32_t (&odd)[4][4], const float *__restrict__ qkv, float *__restrict__ out,
                                        float *__restrict__ out_copy, float *__restrict__ lse, int T, int H, int D, float scale) {
    constexpr int kE = attn::kAttn24MaxD / 32, kAhead = 4;  // columns of a lane, keys whose loads are on their way together
    if (threadIdx.x == 0) bulk_wait_all();  // the copy engine has written the tile
    __syncthreads();
    const int nq = (T + kTile - 1) / kTile, nbh = (int)gridDim.x / nq;
    const int q0 = (nq - 1 - (int)blockIdx.x / nbh) * kTile, bh = (int)blockIdx.x % nbh, b = bh / H, h = bh % H, C = H * D;
    const size_t C3 = 3 * (size_t)C;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float *head = qkv + (size_t)b * T * C3 + (size_t)h * D, *k_rows = head + C, *v_rows = head + 2 * C;
#pragma unroll 1
    for (int r = warp; r < kTile; r += attn24::kThreads / 32) {
        if (!((odd[0][r >> 5] | odd[1][r >> 5] | odd[2][r >> 5] | odd[3][r >> 5]) >> (r & 31) & 1u)) continue;
        const int t = q0 + r;
        float q[kE], acc[kE];
#pragma unroll
        for (int e = 0; e < kE; e++) {
            q[e] = lane + 32 * e < D ? __ldg(head + (size_t)t * C3 + lane + 32 * e) : 0.f;
            acc[e] = 0.f;
        }
        // rows of keys j0 on, all on their way before the first is used; zeros past the diagonal
        auto fetch = [&](const float *rows, int j0, float (&x)[kAhead][kE]) {
#pragma unroll
            for (int u = 0; u < kAhead; u++)
#pragma unroll
                for (int e = 0; e < kE; e++)
                    x[u][e] = j0 + u <= t && lane + 32 * e < D ? __ldg(rows + (size_t)(j0 + u) * C3 + lane + 32 * e) : 0.f;
        };
        auto scores = [&](const float (&k)[kAhead][kE], int j0, float (&s)[kAhead]) {  // -inf past the diagonal
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                s[u] = 0.f;
#pragma unroll
                for (int e = 0; e < kE; e++) s[u] = fmaf(q[e], k[u][e], s[u]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < kAhead; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
            for (int u = 0; u < kAhead; u++) s[u] = j0 + u <= t ? s[u] * scale : -INFINITY;
        };
        float m = -INFINITY, l = 0.f, s[kAhead], k[kAhead][kE], v[kAhead][kE];
        bool is_nan = false;
#pragma unroll 1
        for (int j = 0; j <= t && !is_nan; j += kAhead) {
            fetch(k_rows, j, k);
            scores(k, j, s);
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                is_nan = is_nan || !(s[u] < INFINITY);  // an infinite maximum is subtracted from itself
                m = fmaxf(m, s[u]);
            }
        }
        const float minus = m == -INFINITY ? 0.f : m;
#pragma unroll 1
        for (int j = 0; j <= t && !is_nan; j += kAhead) {
            fetch(k_rows, j, k);
            fetch(v_rows, j, v);
            scores(k, j, s);
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                const float p = expf(s[u] - minus);  // 0 past the diagonal, where v is 0, too
                l += p;
#pragma unroll
                for (int e = 0; e < kE; e++) acc[e] = fmaf(p, v[u][e], acc[e]);
            }
        }
        const float by = is_nan ? NAN : 1.0f / l;
        const size_t at = ((size_t)b * T + t) * C + (size_t)h * D;
#pragma unroll
        for (int e = 0; e < kE; e++) {
            if (lane + 32 * e >= D) break;
            out[at + lane + 32 * e] = acc[e] * by;
            if (out_copy) out_copy[at + lane + 32 * e] = acc[e] * by;
        }
        if (lane == 0) lse[(size_t)bh * T + t] = is_nan ? NAN : m + logf(l);
    }
}

enum Site24 : int { SITE24_GO_S = 301, SITE24_GO_PV, SITE24_S, SITE24_PV, SITE24_RAW_FREE, SITE24_RAW_FULL, SITE24_SMEM_ALIGN };

// kTma: D is a multiple of 4, and the copy engine fetches and stores the rows, 16 kK columns of a head of which those past
// the D-th read as zeros and are not written; else the workers read them when they need them.
template <int kK, bool kTma>
__global__ void __launch_bounds__(attn24::kThreads, 1)
attn24_fwd_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_o,
                  const __grid_constant__ CUtensorMap map_copy, const float *__restrict__ qkv, __nv_bfloat16 *__restrict__ xhi,
                  __nv_bfloat16 *__restrict__ xlo, float *__restrict__ out, float *__restrict__ out_copy, float *__restrict__ lse,
                  int T, int H, int D, float scale, Scale scale_log2, int *status) {
    using Smem = Fwd24Smem<kK>;
    constexpr int kPlane = Smem::kPlane, kBlocks = Smem::kBlocks;
    constexpr uint32_t kColS = 0, kColO = 192, kColQ = 192 + 16 * kK;  // S (96 columns) twice; P takes its place
    constexpr uint32_t kCols = 192 + 40 * kK <= 256 ? 256 : 512;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0 && status) atomicCAS(status, 0, ST_TIMEOUT_BASE + SITE24_SMEM_ALIGN);
        return;
    }
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    constexpr bool vec = kTma;
    WaitCtx ctx{&sm.abort_flag, status};
    if (tid == 0) {
        sm.abort_flag = 0;
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.raw_full[i], 1);
            mbar_init(&sm.raw_free[i], kWorkWarps);
        }
        mbar_init(&sm.go_s, kWorkWarps);
        mbar_init(&sm.go_pv, kWorkWarps);
        mbar_init(&sm.done_s, 1);
        mbar_init(&sm.done_pv, 1);
        fence_barrier_init();
    }
    if (warp == kWorkWarps) {
        tmem_alloc_then_launch_dependents(&sm.tmem_base, kCols);
    }
    if (kTma && warp == kWorkWarps + 1 && lane == 0) {
        tma_prefetch_desc(&map_x);
        tma_prefetch_desc(&map_o);
    }
    pdl_wait();
    const int nq = (T + kTile - 1) / kTile, nbh = (int)gridDim.x / nq;
    const int q0 = (nq - 1 - (int)blockIdx.x / nbh) * kTile;  // longest rows first
    const int bh = (int)blockIdx.x % nbh, b = bh / H, h = bh % H;
    const int C = H * D, nsteps = (min(q0 + kTile, T) + kStep - 1) / kStep;
    const size_t C3 = 3 * (size_t)C;
    const float *head = qkv + (size_t)b * T * C3 + (size_t)h * D;
    int odd = 0;  // whether this thread has a value of the result that is not finite
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);

    if (warp > kWorkWarps) {
        // ------------------------------ producers: K, V (before the first step the halves of Q) ------------------------------
        const int kv = warp - kWorkWarps - 1;
        if (kTma && kv < 2 && lane == 0) {
            for (int n = 0; n <= nsteps; n++) {
                if (n > 0 && !await_thread(&sm.raw_free[kv], (n - 1) & 1, ctx, SITE24_RAW_FREE)) break;
                mbar_expect_tx(&sm.raw_full[kv], kStep * 16 * kK * 4);
                tma_load_4d(sm.raw[kv], &map_x, &sm.raw_full[kv], 0, (n > 0 ? (kv + 1) * H : 0) + h,
                            n > 0 ? (n - 1) * kStep : q0 + kv * kStep, b);
            }
        }
    } else if (warp == kWorkWarps) {
        // ------------------------------ MMA issuer ------------------------------
        constexpr uint32_t idesc_s = idesc_bf16_f32(kTile, kStep, 0, 0), idesc_o = idesc_bf16_f32(kTile, 16 * kK, 0, 1);
        constexpr int kTermA[6] = {2, 1, 0, 1, 0, 0}, kTermB[6] = {0, 1, 2, 0, 1, 0};  // smallest first
        const uint32_t leader = elect_leader();
        const uint64_t kd = smem_desc_sw128(smem_u32(sm.k[0]), 16, 1024);
        const uint64_t vd = smem_desc_sw128(smem_u32(sm.v[0]), kStep * 128, 1024);
        auto issue_s = [&](int n) {
            await(&sm.go_s, n & 1, ctx, SITE24_GO_S);
#pragma unroll
            for (int term = 0; term < 6; term++)
#pragma unroll
                for (int kk = 0; kk < kK; kk++)
                    mma_ts_lead(leader, tmem + kColS + (n & 1) * 96, tmem + kColQ + 8 * kK * kTermA[term] + 8 * kk,
                                desc_advance(kd, kTermB[term] * kPlane + (kk >> 2) * (kStep * 128) + (kk & 3) * 32), idesc_s,
                                term > 0 || kk > 0 ? 1u : 0u);
            tc_commit_lead(leader, &sm.done_s);
        };
        issue_s(0);
        for (int n = 0; n < nsteps; n++) {
            // S_n+1 goes where P_n-1 was, which P V of step n-1, earlier in the pipe, has read by then
            if (n + 1 < nsteps) issue_s(n + 1);
            await(&sm.go_pv, n & 1, ctx, SITE24_GO_PV);
#pragma unroll
            for (int term = 0; term < 6; term++)
#pragma unroll
                for (int kk = 0; kk < kStep / 16; kk++)
                    mma_ts_lead(leader, tmem + kColO, tmem + kColS + (n & 1) * 96 + term_column(kTermA[term], kk),
                                desc_advance(vd, kTermB[term] * kPlane + kk * 2048), idesc_o, term > 0 || kk > 0 ? 1u : 0u);
            tc_commit_lead(leader, &sm.done_pv);
        }
    } else {
        // ------------------------------ workers ------------------------------
        const int quarter = warp & 3, cq = warp >> 2, row = 32 * quarter + lane;
        const uint32_t lane_addr = (uint32_t)(quarter << 5) << 16;
        const uint32_t t_o = tmem + lane_addr + kColO + 4 * kK * cq;
        const Chunk mine(tid);
        // This thread's values of a 64-row tile (rows from t0 on, the columns of one head at src) as three terms into the
        // planes at `tile`; phase: how often the buffer has been filled before.
        auto put = [&](float (&f)[kBlocks][8], uint8_t *tile, int plane, int block, int kv, const float *src, int t0, int phase) {
            if (kTma) {
                await(&sm.raw_full[kv], phase & 1, ctx, SITE24_RAW_FULL);
#pragma unroll
                for (int i = 0; i < kBlocks; i++)
                    if (mine.has<kK>(i)) lds8(f[i], sm.raw[kv] + mine.r * (16 * kK) + mine.col(i), mine.c);
                warp_arrive(&sm.raw_free[kv], lane);  // its fence holds the copy engine back until these values are in registers
            } else {
                const float *from = src + (size_t)(t0 + mine.r) * C3;
#pragma unroll
                for (int i = 0; i < kBlocks; i++)
                    if (mine.has<kK>(i)) load8(f[i], from, mine.col(i), D, t0 + mine.r < T, vec);
            }
#pragma unroll
            for (int i = 0; i < kBlocks; i++)
                if (mine.has<kK>(i)) store_split3(tile, plane, mine.at + i * block, f[i]);
        };
        // The same values for the backward, behind the arrival that others wait for (its fence would wait for the stores).
        // part: 0, 1, 2 for Q, K, V
        auto save = [&](const float (&f)[kBlocks][8], int part, int t0) {
            const int t = t0 + mine.r;
            if (xhi == nullptr || t0 < q0 || t >= T) return;
            const size_t at = (size_t)b * T * C3 + (size_t)t * C3 + (size_t)part * C + (size_t)h * D;
#pragma unroll
            for (int i = 0; i < kBlocks; i++)
                if (mine.has<kK>(i)) save8(xhi + at, xlo + at, mine.col(i), D, f[i], vec);
        };
        // Q: split like K and V, 128 rows where those will be, and from there into tensor memory
        float f[kBlocks][8], q[2][kBlocks][8];
#pragma unroll
        for (int half = 0; half < 2; half++)
            put(q[half], sm.k[0] + half * (kStep * 128), 2 * kPlane, kTile * 128, half, head, q0 + half * kStep, 0);
        named_sync(5, kWorkers);
#pragma unroll
        for (int i = 0; i < kK; i++) {
            const int col = 4 * kK * cq + 4 * i;
            const uint8_t *from = sm.k[0] + (col >> 6) * (kTile * 128) + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4) + (col & 4) * 2;
            const uint32_t t_q = tmem + lane_addr + kColQ + 2 * kK * cq + 2 * i;
#pragma unroll
            for (int term = 0; term < 3; term++) {
                const uint2 w = *reinterpret_cast<const uint2 *>(from + term * 2 * kPlane);
                tmem_st2(t_q + term * 8 * kK, w.x, w.y);
            }
        }
        tmem_wait_st();
        named_sync(5, kWorkers);
        put(f, sm.k[0], kPlane, kStep * 128, 0, head + C, 0, 1);
        warp_arrive(&sm.go_s, lane);
        save(q[0], 0, q0);
        save(q[1], 0, q0 + kStep);
        save(f, 1, 0);

        float o[4 * kK], m = -INFINITY, l = 0.f, alpha_before = 1.f;
#pragma unroll
        for (int i = 0; i < 4 * kK; i++) o[i] = 0.f;
        for (int n = 0; n < nsteps; n++) {
            await(&sm.done_s, n & 1, ctx, SITE24_S);
            if (n + 1 < nsteps) {
                put(f, sm.k[0], kPlane, kStep * 128, 0, head + C, (n + 1) * kStep, n + 2);
                warp_arrive(&sm.go_s, lane);
                save(f, 1, (n + 1) * kStep);
            }
            const uint32_t t_s = tmem + lane_addr + kColS + (n & 1) * 96;
            uint32_t s[16];
            tmem_ld16(t_s + 16 * cq, s);
            tmem_wait_ld();
            float mx = -INFINITY;
            const int key0 = n * kStep + 16 * cq - q0;  // of this thread's columns, relative to the first query row
            if (key0 + 15 > 32 * quarter) {
#pragma unroll
                for (int e = 0; e < 16; e++)
                    if (key0 + e > row) s[e] = 0xff800000u;  // -inf
            }
#pragma unroll
            for (int e = 0; e < 16; e += 2) mx = max3(mx, __uint_as_float(s[e]), __uint_as_float(s[e + 1]));
            sm.part[n & 1][cq][row] = mx;
            named_sync(1 + quarter, 128);  // the four warps of these rows
            mx = fmaxf(fmaxf(sm.part[n & 1][0][row], sm.part[n & 1][1][row]), fmaxf(sm.part[n & 1][2][row], sm.part[n & 1][3][row]));
            mx = fmaxf(m, mx * scale_log2.hi);
            const bool none = mx == -INFINITY;  // nothing but -inf so far
            const float alpha = none ? 1.f : ex2f(m - mx);
            m = mx;
            const float2 by = make_float2(scale_log2.hi, scale_log2.hi), rest = make_float2(scale_log2.lo, scale_log2.lo);
            const float2 minus = make_float2(none ? 0.f : -mx, none ? 0.f : -mx);
            float2 sum = make_float2(0.f, 0.f);
            uint32_t hi[8], mid[8], lo[8];
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const float2 v = make_float2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1]));
                const float2 x = fma2(v, rest, fma2(v, by, minus));
                const float2 p = make_float2(ex2f(x.x), ex2f(x.y));
                sum = add2(sum, p);
                split3(p, hi[e], mid[e], lo[e]);
            }
            l = l * alpha + (sum.x + sum.y);
            tmem_st8(t_s + term_column(0, cq), hi);
            tmem_st8(t_s + term_column(1, cq), mid);
            tmem_st8(t_s + term_column(2, cq), lo);
            tmem_wait_st();
            if (n > 0) {
                await(&sm.done_pv, (n - 1) & 1, ctx, SITE24_PV);
                add_columns<kK>(o, t_o, alpha_before);
            }
            alpha_before = alpha;
            put(f, sm.v[0], kPlane, kStep * 128, 1, head + 2 * C, n * kStep, n + 1);
            warp_arrive(&sm.go_pv, lane);
            save(f, 2, n * kStep);
        }
        sm.part[nsteps & 1][cq][row] = l;
        named_sync(1 + quarter, 128);
        l = (sm.part[nsteps & 1][0][row] + sm.part[nsteps & 1][1][row]) + (sm.part[nsteps & 1][2][row] + sm.part[nsteps & 1][3][row]);
        await(&sm.done_pv, (nsteps - 1) & 1, ctx, SITE24_PV);
        add_columns<kK>(o, t_o, alpha_before);
        const int t = q0 + row;
        const float inv = 1.0f / l;
        {
            float zero[4] = {m * 0.f, 0.f, 0.f, 0.f};  // what is finite times zero is zero
#pragma unroll
            for (int i = 0; i < 4 * kK; i++) zero[i & 3] = fmaf(o[i] * inv, 0.f, zero[i & 3]);
            odd = t < T && !((zero[0] + zero[1]) + (zero[2] + zero[3]) == 0.f);
            const uint32_t rows = __ballot_sync(0xffffffffu, odd);
            if (lane == 0) sm.odd[cq][quarter] = rows;
        }
        if (kTma) {
            // by the copy engine, from the place of the raw K and V: groups of 16 columns, 128 rows of 64 bytes, swizzled
            uint8_t *stage = reinterpret_cast<uint8_t *>(sm.raw[0]);
#pragma unroll
            for (int i = 0; i < kK; i++) {
                const int col = 4 * kK * cq + 4 * i;
                *reinterpret_cast<float4 *>(stage + (col >> 4) * (kTile * 64) + row * 64 + ((((col >> 2) & 3) ^ ((row >> 1) & 3)) << 4)) =
                    make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
            }
            fence_proxy_async_smem();
            named_sync(5, kWorkers);
            if (tid == 0) {
                for (int g = 0; g < kK; g++) {
                    if (16 * g >= D) break;
                    tma_store_4d(stage + g * (kTile * 64), &map_o, 16 * g, h, q0, b);
                    if (out_copy) tma_store_4d(stage + g * (kTile * 64), &map_copy, 16 * g, h, q0, b);
                }
                bulk_commit();
                bulk_wait_read_all();  // shared memory stays alive until then
            }
        }
        if (t < T) {
            const size_t at = ((size_t)b * T + t) * C + (size_t)h * D;
            if (!kTma) {
                store_columns<kK>(out + at, 4 * kK * cq, D, o, inv, vec);
                if (out_copy) store_columns<kK>(out_copy + at, 4 * kK * cq, D, o, inv, vec);
            }
            // m ln 2 + ln l, ln 2 in two parts
            if (cq == 0) lse[(size_t)bh * T + t] = fmaf(m, 0.693147182464599609375f, fmaf(m, -1.904654299957768e-9f, logf(l)));
        }
    }
    if (sm.abort_flag) __nanosleep(50000);  // let copies and products that are still in flight end
    tc_fence_before_sync();
    const int again = __syncthreads_or(odd);
    if (warp == kWorkWarps) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kCols);
    }
    if (again) exact_rows(sm.odd, qkv, out, out_copy, lse, T, H, D, scale);
}

}  // namespace general

}  // namespace

cudaError_t fast_fwd_set_attributes() {
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel<kLong>, a, (int)sizeof(FwdSmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_fwd_kernel<kRows>, a, (int)sizeof(FwdSmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_fwd_kernel<kFp32>, a, (int)sizeof(FwdSmem));
    return e;
}

static const float kScaleLog2 = 0.125f * 1.4426950408889634f;  // 1/sqrt(64) * log2(e)

// Whether the result leaves from registers.  The last to end are the CTAs of the last query tile; where that tile has at most
// 96 rows, they are stored once and no second CTA on the SM covers the way through shared memory, barrier and copy engine, the
// rows are sooner out of registers.  Up to 64 tokens they are in any case.  Forward in us, copy engine / registers, without a
// copy of the result:
//     B=1 H=4:  T=65 6.7 / 6.3, 96 6.55 / 6.2, 120 7.1 / 6.9, 130 7.1 / 6.65, 192 7.2 / 6.8, 256 8.4 / 8.25, 448 10.5 / 10.2
//     B=1 H=12: T=700 15.1 / 14.8, 832 16.9 / 16.6, 960 18.8 / 18.4, 1088 20.7 / 20.3
//     B=6 H=12: T=96 9.45 / 9.4, 127 8.4 / 8.4, 192 9.5 / 9.3, 256 11.3 / 11.4
// with two CTAs on an SM (T, H=12): B=16 96 11.0 / 11.25, 127 12.2 / 12.7, B=8 130 10.6 / 10.65, 256 13.5 / 13.7; with a copy,
// core alone: B=3 T=100 H=8 6.6 / 6.7, B=6 T=192 H=12 8.15 / 8.2, B=8 T=128 H=12 7.5 / 8.6.
static bool rows_from_registers(int T, long long items, bool copied) {
    return T <= kTile / 2 || (!copied && T % kTile > 0 && T % kTile <= 96 && items <= sm_count());
}

cudaError_t launch_fast_forward(const CUtensorMap &map_x, const CUtensorMap &map_o, const CUtensorMap &map_copy, float *out,
                                float *out_copy, float *lse, int B, int T, int H, int *status, cudaStream_t s) {
    const long long items = (long long)((T + kTile - 1) / kTile) * B * H;
    const dim3 grid((unsigned)items);
    if (rows_from_registers(T, items, out_copy != nullptr))
        return launch_after_previous(attn_fwd_kernel<kRows>, grid, dim3(kThreads), sizeof(FwdSmem), s, Maps<kRows>{map_x}, nullptr, nullptr,
                                     nullptr, out, out_copy, lse, B, T, H, kScaleLog2, status);
    return launch_after_previous(attn_fwd_kernel<kLong>, grid, dim3(kThreads), sizeof(FwdSmem), s, Maps<kLong>{map_x, map_o, map_copy},
                                 nullptr, nullptr, nullptr, out, out_copy, lse, B, T, H, kScaleLog2, status);
}

cudaError_t launch_fast_forward_fp32(const float *qkv, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *out, float *out_copy, float *lse,
                                     int B, int T, int H, int *status, cudaStream_t s) {
    return launch_after_previous(attn_fwd_kernel<kFp32>, dim3((unsigned)(B * H)), dim3(kThreads), sizeof(FwdSmem), s,
                                 Maps<kFp32>{}, qkv, hi, lo, out, out_copy, lse, B, T, H, kScaleLog2, status);
}

cudaError_t attn24_fwd_set_attributes() {
    for (int n = 1; n <= kAttn24MaxD / 16; n++) {
        const cudaError_t e = attn24::with_groups(n, [](auto k) {
            constexpr int kK = decltype(k)::value, kBytes = (int)sizeof(general::Fwd24Smem<kK>);
            static_assert(kBytes <= 227 * 1024, "shared memory");
            const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
            const cudaError_t e = cudaFuncSetAttribute(general::attn24_fwd_kernel<kK, true>, a, kBytes);
            return e != cudaSuccess ? e : cudaFuncSetAttribute(general::attn24_fwd_kernel<kK, false>, a, kBytes);
        });
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_attn24_forward(const float *qkv, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *out, float *out_copy, float *lse, int B,
                                  int T, int H, int D, int *status, cudaStream_t s) {
    CUtensorMap map_x = {}, map_o = {}, map_copy = {};
    const bool tma = D % 4 == 0;
    if (tma) {
        int rc = attn24_heads_map(&map_x, qkv, B, T, 3 * H, D, (D + 15) / 16 * 16, attn24::kStep, CU_TENSOR_MAP_SWIZZLE_NONE);
        if (rc == 0) rc = attn24_heads_map(&map_o, out, B, T, H, D, 16, kTile, CU_TENSOR_MAP_SWIZZLE_64B);
        if (rc == 0 && out_copy) rc = attn24_heads_map(&map_copy, out_copy, B, T, H, D, 16, kTile, CU_TENSOR_MAP_SWIZZLE_64B);
        if (rc != 0) return (cudaError_t)rc;
    }
    return attn24::with_groups((D + 15) / 16, [&](auto k) {
        constexpr int kK = decltype(k)::value;
        const dim3 grid((unsigned)((size_t)B * H * ((T + kTile - 1) / kTile)));
        return launch_after_previous(tma ? general::attn24_fwd_kernel<kK, true> : general::attn24_fwd_kernel<kK, false>, grid,
                                     dim3(attn24::kThreads), sizeof(general::Fwd24Smem<kK>), s, map_x, map_o, map_copy, qkv, hi, lo,
                                     out, out_copy, lse, T, H, D, 1.0f / sqrtf((float)D), attn24::log2_scale(D), status);
    });
}

}  // namespace attn
