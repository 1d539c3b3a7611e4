// Backward of the Linear layer for sm_100a: dx = dy . W, dW += dy^T . x and db += column sums of dy in ONE launch.
//
// Replaces the two SGEMMs and the atomic bias reduction of linear_backward_cuda_kernel of gpt.c
// (kernels/src/cuda/Linear.cu:64-92).  The products run on the tensor cores with TF32 operands read straight from the
// fp32 tensors (linear_sm100.cu has the forward and says more about operands and pipeline).
//
// Why one launch: each product alone leaves SMs idle.  Tiles of dx = 8192 x 768 are 192 for 148 SMs, and every launch
// starts with empty pipelines and ends with a last tile's way out (about 4.5 us).  dW is added into what is there, so its
// contraction may be cut anywhere: every CTA first takes its tiles of dx, then as much of dW as makes all CTAs end together.
// dy is read from shared memory a second time for db, in fp32, by two warps that have nothing else to do.  Before, three
// launches, now (M, N, K in us, with db): 8192, 3072, 768 138 -> 124; 8192, 2304, 768 115 -> 95; 8192, 768, 768 51 -> 39;
// 1500, 6400, 1600 128 -> 106; 1500, 1600, 1600 45 -> 34; 1705, 129, 4288 32 -> 25.
// What bounds it: shared memory, which takes a block's 48 KB in and hands them to the tensor cores once (768 cycles at 128
// bytes each, 512 of products), and the power cap: 8192 x 3072 x 768 runs at 630 TFLOP/s.
//
//     dx[M,K]  = dy[M,N] . W[N,K]      A: dy, K-major (over N)   B: W, MN-major
//     dW[N,K] += dy[M,N]^T . x[M,K]    A: dy, MN-major           B: x, MN-major   (contraction over M, cut into ranges)
//
// Both results have K columns; a tile is 128 rows by up to 256 columns, and the columns are dealt out evenly in blocks of
// 32 (K = 1600: six tiles of 224 and one of 256 columns).
//
// Warp roles (384 threads, one CTA per SM):
//   warp 0      TMA producer
//   warp 1      MMA issuer
//   warp 2      tensor-memory allocation, db
//   warp 3      db
//   warps 4-11  epilogue: dx from registers, dW through a staging buffer to a bulk tensor reduction
// All waits on barriers are bounded (tc05.cuh).
#include <math.h>

#include <type_traits>

#include "linear_tf32.cuh"

namespace lin {
namespace {

using namespace tc05;

constexpr int kThreads = 384, kEpiWarps = 8;
constexpr int kBN = 256;                             // columns of an accumulator
constexpr int kMostStages = 6, kRingBytes = 192 * 1024;  // pipeline: as many stages as fit, of 16 KB of A and up to 32 KB of B

enum Site : int { SITE_EMPTY = 261, SITE_FULL, SITE_ACC_EMPTY, SITE_ACC_FULL, SITE_DB, SITE_SMEM_ALIGN };

struct __align__(1024) Smem {
    uint8_t ring[kRingBytes];
    uint8_t out[kEpiWarps][4096];  // output staging of the epilogue warps: 32 rows x 128 bytes
    uint64_t full[kMostStages], empty[kMostStages];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

// Rows of dy whose pitch is not a multiple of 16 bytes (the vocabulary projection: 50257 floats) cannot be tiled by the
// copy engine as they are, but every fourth row can: the rows m = 4 i + j form a matrix with a pitch of 4 N floats, whose
// base is moved down to a 16-byte boundary, by a_shift = (j N) mod 4 floats.  The view's column c is then column
// c - a_shift of dy.  In dx that is the contraction index, and W is fetched at rows c - a_shift (rows before the first
// and past the last read as zeros); one product per class, which leaves every fourth row of dx.  What the first a_shift
// columns hold is the end of the row of dy before: the MMA warp puts zeros there in shared memory (clear_leading), since
// the zeros of W alone would turn a value that is not finite into NaN.  In dW the view's column is the row of the
// result: each class is a piece of the contraction, added into dW a_shift rows higher up.  What this replaces is a
// copy of dy with padded rows, 536 us for the 1.65 GB of 8192 x 50257.
struct RowClass {
    const float *dy;  // base of the view
    int rows, shift;
};
RowClass row_class(const float *dy, int M, int N, int j) {
    const int shift = (int)(((long long)j * N) & 3);
    return RowClass{dy + (size_t)j * N - shift, (M - j + 3) / 4, shift};
}

// kClasses: the four views of dy (RowClass), and what goes with them.
template <bool kClasses>
struct Maps {
    static constexpr int kViews = kClasses ? 4 : 1;
    CUtensorMap dy_k[kViews], dy_mn[kViews];  // A of dx and of dW
    CUtensorMap x[kViews][2], w[2];           // B of dW and of dx, for tiles of p.cols and of p.cols + 1 blocks of 32 columns
    CUtensorMap dw;
    CUtensorMap dx[kViews];        // where dx is added up from pieces
    CUtensorMap dy_whole[kViews];  // dy_mn takes a copy per 32 columns and has the ones after the whole blocks too; this takes one per tile
};

// dW's tiles are cut across the contraction, and their ranges dealt out to teams of CTAs.  The members of a team work on the same
// range of neighbouring tiles at the same time, one tile each, so that what these tiles share comes from HBM once.
struct Problem {
    int M, N, K;
    int tiles_n, cols, wider;  // column tiles; blocks of 32 columns in each; the first `wider` have one more
    int dx_tiles, dx_kb;       // tiles of dx, handed out round robin; contraction blocks of one
    int classes;               // 4: views of every fourth row of dy
    int dx_pieces, piece_tiles, piece_kb;  // dx from so many pieces of the contraction; tiles and contraction blocks of a piece
    int dx_sums;               // or from so many in turn, added up by the CTA whose tile it is
    size_t dx_apart;           // from one piece of dx to the next, which are not added up here (0: they are)
    int whole[4], shift[4];    // columns of the views in whole blocks; before the first column of dy
    int dw_kb, dw_most;        // contraction blocks of a tile of dW; the most that go through one accumulator
    int team, down;            // CTAs of a team; their tiles are below (1) or beside each other (0)
    int rounds, strips;        // groups of `team` tiles: whole ones dealt out round robin; the ones after them, which are cut
    int teams, fewer;          // the first `fewer` teams (those with a tile of dx more) take share_fewer of dW, the others share
    uint32_t share_fewer, share;  // in units of 2^-32
    int snap;
    int uncut;                 // dW alone, whole tiles round robin
    int stages, stage_bytes;
    int wide;                  // rows of dx start on 32-byte boundaries
};

// Counted through all strips, team c takes the contraction blocks from range_start(c) to range_start(c + 1).  A range does not
// begin or end within `snap` blocks of a tile's edge.
__host__ __device__ __forceinline__ int range_start(const Problem &p, int c) {
    const int total = p.strips * p.dw_kb;
    if (c >= p.teams) return total;
    const uint32_t part = c < p.fewer ? c * p.share_fewer : p.fewer * p.share_fewer + (c - p.fewer) * p.share;
    const int u = (int)(((unsigned long long)(uint32_t)total * part) >> 32);
    const int in = u % p.dw_kb;
    return in < p.snap ? u - in : p.dw_kb - in < p.snap ? u + p.dw_kb - in : u;
}

// A tile of dx or of dW with a range of its contraction: what goes through one accumulator.
struct Item {
    bool dw;
    int cls, m0, tn, n0, cols, kb0, kb1;
};
struct Items {
    int cta, ctas;
    int i, whole;  // tiles of dx and whole tiles of dW taken so far
    int at, end;   // the team's range
    int team, member;
    int from, to, sums;  // what is left of the tile's range, and the accumulators it goes through
    __host__ __device__ __forceinline__ Items(const Problem &p, int cta, int ctas) : cta(cta), ctas(ctas), i(0), whole(0), sums(0) {
        team = cta / p.team;
        member = cta - team * p.team;
        at = range_start(p, team), end = range_start(p, team + 1);
    }
    // `t` is the item before, which the next one may continue.
    __host__ __device__ __forceinline__ bool next(const Problem &p, Item &t) {
        if (sums == 0 && !next_tile(p, t)) return false;
        t.kb0 = from;
        from = sums == 1 ? to : from + (to - from + sums - 1) / sums;
        t.kb1 = from;
        sums--;
        return true;
    }
    __host__ __device__ __forceinline__ bool next_tile(const Problem &p, Item &t) {
        int w = cta + i * ctas;
        int tm;
        sums = 1;
        if (p.uncut) {
            if (w >= p.strips) return false;
            t.dw = true;
            tm = w / p.tiles_n, t.tn = w - tm * p.tiles_n;
            from = 0, to = p.dw_kb;
            i++;
        } else if (w < p.dx_tiles) {
            t.dw = false;
            const int piece = p.dx_pieces > 1 ? w / p.piece_tiles : 0;
            w -= piece * p.piece_tiles;
            tm = w / p.tiles_n, t.tn = w - tm * p.tiles_n;
            from = piece * p.piece_kb, to = p.dx_kb - from < p.piece_kb ? p.dx_kb : from + p.piece_kb;
            sums = p.dx_sums;
            i++;
        } else {
            t.dw = true;
            int strip;
            if (whole < p.rounds) {
                strip = team + whole++ * p.teams;
                from = 0, to = p.dw_kb;
            } else {
                if (at >= end) return false;
                strip = at / p.dw_kb;
                from = at - strip * p.dw_kb;
                const int take = p.dw_kb - from < end - at ? p.dw_kb - from : end - at;
                to = from + take;
                at += take;
                strip += p.rounds * p.teams;
            }
            if (p.down) {
                t.tn = strip, tm = member;
            } else {
                const int tile = strip * p.team + member;
                tm = tile / p.tiles_n, t.tn = tile - tm * p.tiles_n;
            }
            if (to - from > p.dw_most) sums = (to - from + p.dw_most - 1) / p.dw_most;
        }
        t.cls = 0;
        if (p.classes > 1) {  // dW: the classes of a tile follow each other, so that what they add to stays in L2
            const int rows = p.piece_tiles / p.tiles_n / 4;
            t.cls = t.dw ? tm & 3 : tm / rows;
            tm = t.dw ? tm >> 2 : tm - t.cls * rows;
        }
        t.m0 = tm * kBM;
        t.cols = p.cols + (t.tn < p.wider ? 1 : 0);
        t.n0 = 32 * (t.tn * p.cols + (t.tn < p.wider ? t.tn : p.wider));
        return true;
    }
};

// A role's place in the ring of pipeline stages.
struct Place {
    int st = 0;
    uint32_t round = 0;
    __device__ __forceinline__ void next(int stages) {
        if (++st == stages) st = 0, round++;
    }
};

// Zeros for the first `columns` (at most 3) of a K-major A tile's 128 rows: they are in the first 16 bytes of a row, which
// the 128-byte swizzle puts at 16 * (row mod 8).  By a whole warp, one lane of which issues the tensor-core instructions
// that read the tile.
__device__ __forceinline__ void clear_leading(uint8_t *tile, int columns, int lane) {
    for (int r = lane; r < kBM; r += 32) {
        float *row = reinterpret_cast<float *>(tile + r * 128 + ((r & 7) << 4));
        row[0] = 0.f;
        if (columns > 1) row[1] = 0.f;
        if (columns > 2) row[2] = 0.f;
    }
    fence_proxy_async_smem();
    __syncwarp();
}

// r += what is at src, 4 * kQuads floats as far as `left` go (a multiple of 4).
template <int kQuads>
__device__ __forceinline__ void add_words(const float *src, int left, uint32_t *r) {
#pragma unroll
    for (int q = 0; q < kQuads; q++) {
        if (4 * q >= left) continue;
        float4 v;
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(src + 4 * q) : "memory");
        r[4 * q] = __float_as_uint(v.x + __uint_as_float(r[4 * q]));
        r[4 * q + 1] = __float_as_uint(v.y + __uint_as_float(r[4 * q + 1]));
        r[4 * q + 2] = __float_as_uint(v.z + __uint_as_float(r[4 * q + 2]));
        r[4 * q + 3] = __float_as_uint(v.w + __uint_as_float(r[4 * q + 3]));
    }
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    const float2 lo = add2(make_float2(a.x, a.y), make_float2(b.x, b.y)), hi = add2(make_float2(a.z, a.w), make_float2(b.z, b.w));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}

template <bool kClasses>
__global__ void __launch_bounds__(kThreads, 1)
linear_backward_kernel(const __grid_constant__ Maps<kClasses> maps, float *__restrict__ dx, float *__restrict__ dw, float *__restrict__ db, Problem p, int *status) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0 && status) atomicCAS(status, 0, ST_TIMEOUT_BASE + SITE_SMEM_ALIGN);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WaitCtx ctx{&sm.abort_flag, status};

    if (threadIdx.x == 0) {
        sm.abort_flag = 0;
        for (int i = 0; i < kMostStages; i++) {
            mbar_init(&sm.full[i], 1);
            mbar_init(&sm.empty[i], db != nullptr ? 3 : 1);  // the products, and the warps that sum up db
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.acc_full[i], 1);
            mbar_init(&sm.acc_empty[i], kEpiWarps);
        }
        fence_barrier_init();
    }
    if (warp == 2) tmem_alloc_then_launch_dependents(&sm.tmem_base, 2 * kBN);
    if (warp == 3 && lane == 0) {
        if (p.dx_tiles > 0) {
            tma_prefetch_desc(&maps.dy_k[0]);
            tma_prefetch_desc(&maps.w[0]);
        }
        if (dw != nullptr) {
            tma_prefetch_desc(&maps.dy_mn[0]);
            tma_prefetch_desc(&maps.x[0][0]);
            tma_prefetch_desc(&maps.dw);
        }
    }
    Items items(p, (int)blockIdx.x, (int)gridDim.x);  // the first item, before the wait for the previous kernel
    Item t;
    bool more = items.next(p, t);
    pdl_wait();  // every thread, before its first access to global memory
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            Place at;
            bool ok = true;
            for (; ok && more; more = items.next(p, t)) {
                const int wide = t.cols - p.cols;
                const int view = kClasses ? t.cls : 0;
                const CUtensorMap *map_b = t.dw ? &maps.x[view][wide] : &maps.w[wide];
                const int behind = kClasses && !t.dw ? p.shift[view] : 0;  // W's rows run this far behind the view's columns
                for (int kb = t.kb0; kb < t.kb1; kb++, at.next(p.stages)) {
                    const int st = at.st;
                    if (at.round > 0 && !mbar_wait(&sm.empty[st], (at.round - 1) & 1, ctx, SITE_EMPTY)) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = sm.ring + st * p.stage_bytes;
                    mbar_expect_tx(&sm.full[st], kATileBytes + t.cols * 4096);
                    // K-major: map {contraction, rows}, box {32, 128}.  MN-major: blocks of 32 rows, each
                    // [32 contraction steps x 128 bytes].
                    if (!t.dw) {
                        tma_load_4d(a, &maps.dy_k[view], &sm.full[st], kb * kBK, t.m0, 0, 0);
                    } else if (!kClasses) {
                        tma_load_4d(a, &maps.dy_mn[0], &sm.full[st], 0, kb * kBK, t.m0 / 32, 0);
                    } else if (t.m0 + kBM <= p.whole[view]) {
                        tma_load_4d(a, &maps.dy_whole[view], &sm.full[st], 0, kb * kBK, t.m0 / 32, 0);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            tma_load_4d(a + i * 4096, &maps.dy_mn[view], &sm.full[st], t.m0 + 32 * i, kb * kBK, 0, 0);
                    }
                    tma_load_4d(a + kATileBytes, map_b, &sm.full[st], 0, kb * kBK - behind, t.n0 / 32, 0);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        const uint32_t leader = elect_leader();
        Place at;
        int j = 0;
        bool ok = true;
        for (; ok && more; more = items.next(p, t)) {
            const int acc = j & 1;
            if (j >= 2 && !mbar_wait_warp(&sm.acc_empty[acc], ((j >> 1) - 1) & 1, ctx, SITE_ACC_EMPTY)) break;
            tc_fence_after_sync();
            const uint32_t d = tmem + (uint32_t)acc * kBN;
            // one loop per product, so that its operands' layouts are constants: what this warp issues per cycle is what the
            // tensor cores live on
            auto products = [&](auto dw) {
                constexpr bool kDW = decltype(dw)::value;
                const uint32_t idesc = idesc_tf32(kBM, 0, kDW ? 1 : 0, 1) | (uint32_t)(t.cols * 4) << 17;
                for (int kb = t.kb0; kb < t.kb1; kb++, at.next(p.stages)) {
                    const int st = at.st;
                    if (!mbar_wait_warp(&sm.full[st], at.round & 1, ctx, SITE_FULL)) return false;
                    tc_fence_after_sync();
                    const uint32_t a = smem_u32(sm.ring) + st * p.stage_bytes;
                    if (kClasses && !kDW && kb == 0 && p.shift[t.cls] > 0) clear_leading(sm.ring + st * p.stage_bytes, p.shift[t.cls], lane);
                    // MN-major tiles: 32-row blocks 4096 bytes apart, groups of 4 contraction steps 512 bytes apart
                    const uint64_t ad = kDW ? smem_desc_sw128_base32(a, 4096, 512)
                                            : smem_desc_sw128(a, 16, 1024);
                    const uint64_t bd = smem_desc_sw128_base32(a + kATileBytes, 4096, 512);
#pragma unroll
                    for (int k = 0; k < kBK / 8; k++)
                        mma_tf32_lead(leader, d, desc_advance(ad, k * (kDW ? 1024 : 32)), desc_advance(bd, k * 1024), idesc,
                                      (kb > t.kb0 || k > 0) ? 1u : 0u);
                    tc_commit_lead(leader, &sm.empty[st]);
                }
                return true;
            };
            ok = t.dw ? products(std::true_type()) : products(std::false_type());
            if (!ok) break;
            tc_commit_lead(leader, &sm.acc_full[acc]);
            j++;
        }
    } else if (warp < 4) {
        // ------------------------------ db ------------------------------
        // Column sums of dy, from the A tiles of dW.  The column tiles of the same 128 columns of dy share them out in blocks of
        // 32, since it slows a tile down to have its A read twice (all four blocks by the first column tile: 8192 x 3072 x 768
        // 134 us, shared out 131, among two warps 124, without db 122).  A lane reads 16 bytes of a row (of one value of M):
        // rows lane / 8 + 4 i, the 16-byte word lane % 8, which the swizzle makes the columns from `col` on.  Eight rows are
        // added up first, eight such sums next, so that long sums don't lose more than short ones.
        if (db != nullptr) {
            const int col = ((((lane & 7) >> 1) ^ (lane >> 3)) << 3) + ((lane & 1) << 2);
            Place at;
            bool ok = true;
            for (; ok && more; more = items.next(p, t)) {
                uint32_t mine = 0;
#pragma unroll
                for (int b = 0; b < 4; b++) mine |= t.dw && (b & 1) == (warp & 1) && b * (p.tiles_n < 4 ? p.tiles_n : 4) / 4 == t.tn ? 1u << b : 0u;
                float4 all[4] = {}, some[4] = {};
                for (int kb = t.kb0; kb < t.kb1; kb++, at.next(p.stages)) {
                    const int st = at.st;
                    if (!mbar_wait_warp(&sm.full[st], at.round & 1, ctx, SITE_DB)) {
                        ok = false;
                        break;
                    }
                    if (mine != 0) {
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            if (!(mine >> b & 1)) continue;
                            const float4 *rows = reinterpret_cast<const float4 *>(sm.ring + st * p.stage_bytes + b * 4096) + lane;
                            float4 v[8];
#pragma unroll
                            for (int i = 0; i < 8; i++) v[i] = rows[32 * i];
                            some[b] = add4(some[b], add4(add4(add4(v[0], v[1]), add4(v[2], v[3])), add4(add4(v[4], v[5]), add4(v[6], v[7]))));
                        }
                        if ((kb & 7) == 7 || kb + 1 == t.kb1) {
#pragma unroll
                            for (int b = 0; b < 4; b++) all[b] = add4(all[b], some[b]), some[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                    }
                    if (lane == 0) mbar_arrive(&sm.empty[st]);
                }
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    if (!(mine >> b & 1)) continue;
                    float *s = reinterpret_cast<float *>(&all[b]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {  // the lanes with the same columns
                        s[e] += __shfl_xor_sync(0xffffffffu, s[e], 10);
                        s[e] += __shfl_xor_sync(0xffffffffu, s[e], 20);
                    }
                    const int n = t.m0 + 32 * b + col - (kClasses ? p.shift[t.cls] : 0);
                    if (lane < 8) {
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (n + e >= 0 && n + e < p.N) atomicAdd(db + n + e, s[e]);
                    }
                }
            }
        }
    } else if (warp >= 4) {
        // ------------------------------ epilogue ------------------------------
        // Every warp takes 32 rows (its tensor-memory lane quarter) and half of the blocks of columns.  No warp waits for
        // another one.
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        uint8_t *buf = sm.out[warp - 4];
        const uint32_t lane_addr = (uint32_t)(quarter << 5) << 16;
        int j = 0;
        for (; more; more = items.next(p, t)) {
            const int acc = j & 1;
            if (!mbar_wait_warp(&sm.acc_full[acc], (j >> 1) & 1, ctx, SITE_ACC_FULL)) break;
            tc_fence_after_sync();
            const int row0 = t.m0 + 32 * quarter;
            const int c0 = half ? (t.cols + 1) / 2 : 0, c1 = half ? t.cols : (t.cols + 1) / 2;
            auto read_out = [&] {  // the tensor cores may reuse the accumulator
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.acc_empty[acc]);
            };
            if (c0 == c1) read_out();
#pragma unroll 1
            for (int c = c0; c < c1; c++) {
                const int col0 = t.n0 + 32 * c;
                uint32_t r[32];
                tmem_ld32(tmem + lane_addr + (uint32_t)acc * kBN + 32 * c, r);
                tmem_wait_ld();
                if (c + 1 == c1) read_out();
                if (!t.dw && (!kClasses || p.dx_pieces == 1 || p.dx_apart)) {
                    const int odd = lane & 1, col = col0 + 16 * odd;
                    float *piece = kClasses ? dx + t.kb0 / p.piece_kb * p.dx_apart : dx;
                    exchange_halves(odd, r);
#pragma unroll
                    for (int o = 0; o < 2; o++) {
                        const int row = row0 + lane - odd + o;
                        if (row * p.classes + t.cls >= p.M) continue;
                        float *to = piece + ((size_t)row * p.classes + t.cls) * p.K + col;
                        if (kClasses && p.dx_sums > 1 && t.kb0 > 0) add_words<4>(to, p.K - col, r + 16 * o);  // what this thread wrote for the range before
                        store_words<4>(to, p.K - col, p.wide, r + 16 * o);
                    }
                    continue;
                }
                const int up = kClasses && t.dw ? p.shift[t.cls] : 0;
                if (kClasses && row0 < up) {
                    // The first 32 rows of the result: up to three of them do not exist, and a copy must not start at a
                    // negative coordinate.
                    const int row = row0 + lane - up;
                    if (row >= 0 && row < p.N) {
                        float *dst = dw + (size_t)row * p.K + col0;
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4 * q),
                                         "f"(__uint_as_float(r[4 * q])), "f"(__uint_as_float(r[4 * q + 1])),
                                         "f"(__uint_as_float(r[4 * q + 2])), "f"(__uint_as_float(r[4 * q + 3]))
                                         : "memory");
                    }
                    continue;
                }
                if (lane == 0) bulk_wait_read_all();  // the copy engine has read the buffer out
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; q++)  // one row of 128 bytes per lane, 16-byte words swizzled
                    *reinterpret_cast<uint4 *>(buf + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                        make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_reduce_add_3d(buf, kClasses && !t.dw ? &maps.dx[t.cls] : &maps.dw, col0, row0 - up, 0);
                    bulk_commit();
                }
            }
            j++;
        }
        if (lane == 0) bulk_wait_read_all();  // shared memory stays until it has been read
    }

    // ------------------------------ tear-down ------------------------------
    if (sm.abort_flag) __nanosleep(50000);
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, 2 * kBN);
    }
}

// ---- host side ----

// Nanoseconds of a contraction block of a tile `cols` blocks of 32 columns wide while `busy` SMs of `sms` work on such tiles,
// of what a tile takes besides, and of adding pieces of dW to memory.  Fitted to dW alone at nine shapes, 5 widths, 1 to 11
// pieces (2795 x 3200 x 640: cut anywhere, 7 blocks wide 24.8 us, one whole piece of 5 or 4 blocks per CTA 30.8 and 28.6;
// 8192 x 768 x 768: 8 pieces of 18 tiles 20.3, cut anywhere 23.8).
double block_ns(int cols, int busy, int sms) {
    const double alone = 186 + 19 * cols, fed = (190.0 + 26 * cols) * busy / sms;
    return fed > alone ? fed : alone;
}
double tile_ns(int cols) { return cols > 6 ? 2000 : cols > 4 ? 900 : 400; }
double adding_ns(double pieces, int cols) { return pieces * cols * 16384 * 150e-6; }

Problem make_problem(const BackwardPlan &plan, int M, int N, int K) {
    Problem p = {};
    p.M = M, p.N = N, p.K = K;
    p.classes = plan.classes;
    p.dx_pieces = plan.dx_how == kDxInTurn ? 1 : plan.dx_pieces, p.dx_sums = plan.dx_how == kDxInTurn ? plan.dx_pieces : 1;
    p.dx_apart = plan.dx_how == kDxApart ? (size_t)M * K : 0;
    p.piece_tiles = plan.dx_tiles / p.dx_pieces, p.piece_kb = (plan.dx_kb + p.dx_pieces - 1) / p.dx_pieces;
    p.tiles_n = plan.tiles_n, p.cols = K / 32 / plan.tiles_n, p.wider = K / 32 % plan.tiles_n;
    p.dx_tiles = plan.dx_tiles, p.dx_kb = plan.dx_kb, p.dw_kb = plan.dw_kb, p.dw_most = plan.dw_most;
    p.team = plan.team, p.down = plan.down, p.rounds = plan.rounds, p.strips = plan.strips, p.teams = plan.teams, p.fewer = plan.fewer;
    const double all = plan.fewer * plan.share_fewer + (plan.teams - plan.fewer) * plan.share;
    // rounded up, so that shares of whole tiles begin where tiles do
    p.share_fewer = (uint32_t)ceil(plan.share_fewer / all * 4294967296.0);
    p.share = (uint32_t)fmin(ceil(plan.share / all * 4294967296.0), 4294967295.0);
    // pieces of the same size stay as they are; a few tiles of few blocks are cut anywhere, many are not
    p.snap = plan.even && p.strips < p.teams ? 0 : p.dw_kb >= 16 ? 4 : p.strips >= p.teams ? (p.dw_kb < 8 ? p.dw_kb : 2) : 0;
    p.uncut = p.dx_tiles == 0 && p.classes == 1 && p.team == 1 && p.snap == p.dw_kb;
    p.stage_bytes = kATileBytes + (p.cols + (p.wider > 0)) * 4096;
    p.stages = kRingBytes / p.stage_bytes < kMostStages ? kRingBytes / p.stage_bytes : kMostStages;
    return p;
}

}  // namespace

// The split of the work and the time in nanoseconds it is expected to take: see linear_tf32.cuh.
BackwardPlan plan_backward(int M, int N, int K, bool want_dx, bool want_dw, int sms, int classes, int dx_pieces, DxPieces how) {
    BackwardPlan best = {};
    const int blocks = K / 32;
    for (int width = 8; width >= 4; width--) {
        const int tiles_n = (blocks + width - 1) / width;
        if (tiles_n == best.tiles_n) continue;
        BackwardPlan c = {};
        c.tiles_n = tiles_n;
        const int cols = (blocks + tiles_n - 1) / tiles_n;
        const double tb = block_ns(cols, sms, sms), te = tile_ns(cols);
        const int rows = (M + classes - 1) / classes;  // of a class
        const int rows_m = (rows + kBM - 1) / kBM, rows_n = (N + classes - 1 + kBM - 1) / kBM;
        c.dx_kb = (N + classes - 1 + kBK - 1) / kBK;
        c.dw_kb = c.dw_most = (rows + kBK - 1) / kBK;
        c.classes = classes;
        const int piece_kb = (c.dx_kb + dx_pieces - 1) / dx_pieces;
        c.dx_pieces = (c.dx_kb + piece_kb - 1) / piece_kb;
        c.dx_how = how;
        c.dx_tiles = want_dx ? classes * rows_m * tiles_n * (how == kDxInTurn ? 1 : c.dx_pieces) : 0;
        const int dw_tiles = want_dw ? classes * rows_n * tiles_n : 0;
        // Where dy and x don't stay in L2 together, a team shares the larger of them, if that keeps most SMs busy.
        c.down = classes == 1 && N < K, c.team = c.down ? rows_n : tiles_n;
        if (4.0 * M * ((double)N + K) < (64 << 20) || c.team > sms || sms / c.team * c.team < sms * 24 / 25) c.down = 0, c.team = 1;
        c.strips = dw_tiles / c.team;
        c.teams = sms / c.team;
        if (!want_dx && (long long)c.strips * c.dw_kb < c.teams) c.teams = c.strips * c.dw_kb;
        const int ctas = c.teams * c.team;
        const double dx_ns = (piece_kb * tb + te) * (how == kDxInTurn ? c.dx_pieces : 1);
        // every CTA has about one piece of a tile more than its share of whole ones
        const double even = (c.dx_tiles * dx_ns + dw_tiles * (c.dw_kb * tb + te)) / ctas + te;
        const int most = (c.dx_tiles + ctas - 1) / ctas;
        c.fewer = (c.dx_tiles % ctas + c.team - 1) / c.team;
        // what is left for dW, in blocks, in a CTA with `most` tiles of dx and in one with a tile less
        c.share_fewer = (even - most * dx_ns - te) / tb, c.share = c.share_fewer + (c.fewer ? dx_ns / tb : 0);
        if (classes > 1) {
            // Most strips whole and in turn, so that teams work on neighbouring columns of dy at the same time
            const double least = c.fewer ? c.share_fewer : c.share;
            c.rounds = least > 0 ? (int)(least / c.dw_kb) : 0;
            if (c.rounds > c.strips / c.teams) c.rounds = c.strips / c.teams;
            c.strips -= c.rounds * c.teams;
            c.share_fewer -= c.rounds * c.dw_kb, c.share -= c.rounds * c.dw_kb;
        }
        if (c.share_fewer < 3) c.share_fewer = 0;
        if (c.share < 1) c.share = 1;
        double time = (even > most * dx_ns && want_dw ? even : most * dx_ns) + adding_ns(dw_tiles + ctas, cols);
        const int most_pieces = want_dx ? 0 : sms / dw_tiles < c.dw_kb ? sms / dw_tiles : c.dw_kb;
        auto as_deep = [&](int pieces) {  // fewest pieces that are no longer
            const int depth = (c.dw_kb + pieces - 1) / pieces;
            return (c.dw_kb + depth - 1) / depth;
        };
        for (int tries = 0, pieces = most_pieces > 0 ? as_deep(most_pieces) : 0; tries < 4 && pieces > 0; tries++) {
            // whole pieces of the same size, as many as SMs or fewer: no CTA has parts of two tiles, all of them the same rows
            const int busy = pieces * dw_tiles;
            const double whole = (c.dw_kb + pieces - 1) / pieces * block_ns(cols, busy, sms) + te + adding_ns(busy, cols);
            if (whole <= time) {
                c.team = 1, c.down = 0, c.rounds = 0, c.strips = dw_tiles, c.teams = busy, c.share = 1, c.even = 1;
                time = whole;
            }
            pieces = pieces > 1 ? as_deep(pieces - 1) : 0;
        }
        const double ns = 4470 + time;
        c.ns = ns < 2e9 ? (int)ns : 2000000000;
        if (best.ns == 0 || c.ns < best.ns) best = c;
    }
    return best;
}

DwLoad dw_load(const BackwardPlan &plan, int M, int N, int K) {
    DwLoad most = {};
    const int ctas = plan.teams * plan.team;
    if (ctas == 0) return most;
    const Problem p = make_problem(plan, M, N, K);
    for (int cta = 0; cta < ctas; cta++) {
        Items items(p, cta, ctas);
        int blocks = 0;
        for (Item t; items.next(p, t);) {
            if (!t.dw) continue;
            blocks += t.kb1 - t.kb0;
            if (t.kb1 - t.kb0 > most.sum) most.sum = t.kb1 - t.kb0;
        }
        if (blocks > most.cta) most.cta = blocks;
    }
    return most;
}

template <bool kClasses>
static int launch(const Maps<kClasses> &maps, float *dx, float *dw, float *db, const Problem &p, int ctas, int *status, cudaStream_t s) {
    static bool attr_done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    static_assert(sizeof(Smem) <= 227 * 1024, "shared memory of the Linear backward kernel");
    auto kernel = linear_backward_kernel<kClasses>;
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    return (int)attn::launch_after_previous(kernel, dim3(ctas), dim3(kThreads), sizeof(Smem), s, maps, dx, dw, db, p, status);
}

int launch_backward(const BackwardPlan &plan, const float *dy, const float *x, const float *w, int w_rows, float *dx, float *dw, float *db,
                    int M, int N, int np, int K, int *status, cudaStream_t s) {
    Problem p = make_problem(plan, M, N, K);
    p.wide = (reinterpret_cast<uintptr_t>(dx) & 31u) == 0;
    Maps<false> maps = {};
    int rc;
    if ((rc = map_mn_major_blocks(&maps.dy_mn[0], dy, M, np, 4)) != 0) return rc;
    if ((rc = map_out_f32(&maps.dw, dw, N, K)) != 0) return rc;
    for (int i = 0; i <= (p.wider > 0); i++) {
        if ((rc = map_mn_major_blocks(&maps.x[0][i], x, M, K, p.cols + i)) != 0) return rc;
        if (dx && (rc = map_mn_major_blocks(&maps.w[i], w, w_rows, K, p.cols + i)) != 0) return rc;
    }
    if (dx && (rc = map_k_major(&maps.dy_k[0], dy, M, np, 128)) != 0) return rc;
    return launch<false>(maps, dx, dw, db, p, plan.teams * plan.team, status, s);
}

int launch_backward_by_row_class(const BackwardPlan &plan, const float *dy, const float *x, const float *w, float *dx, float *dw, float *db,
                                 int M, int N, int K, int *status, cudaStream_t s) {
    Problem p = make_problem(plan, M, N, K);
    p.wide = (reinterpret_cast<uintptr_t>(dx) & 31u) == 0;
    Maps<true> maps = {};  // those of products that are not wanted stay empty: x may be NULL without dw
    int rc;
    if (dw && (rc = map_out_f32(&maps.dw, dw, N, K)) != 0) return rc;
    for (int j = 0; j < 4; j++) {
        const RowClass c = row_class(dy, M, N, j);
        const size_t pitch = 4 * (size_t)N;
        p.shift[j] = c.shift, p.whole[j] = (N + c.shift) / 32 * 32;
        if (dw) {
            if (p.whole[j] > 0 && (rc = map_mn_major_blocks(&maps.dy_whole[j], c.dy, c.rows, p.whole[j], 4, pitch)) != 0) return rc;
            if ((rc = map_mn_major(&maps.dy_mn[j], c.dy, c.rows, N + c.shift, pitch)) != 0) return rc;
            for (int i = 0; i <= (p.wider > 0); i++)
                if ((rc = map_mn_major_blocks(&maps.x[j][i], x + (size_t)j * K, c.rows, K, p.cols + i, 4 * (size_t)K)) != 0) return rc;
        }
        if (!dx) continue;
        if ((rc = map_k_major(&maps.dy_k[j], c.dy, c.rows, N + c.shift, 128, pitch)) != 0) return rc;
        if (p.dx_pieces > 1 && !p.dx_apart && (rc = map_out_f32(&maps.dx[j], dx + (size_t)j * K, c.rows, K, 4 * (size_t)K)) != 0) return rc;
    }
    for (int i = 0; dx && i <= (p.wider > 0); i++)
        if ((rc = map_mn_major_blocks(&maps.w[i], w, N, K, p.cols + i)) != 0) return rc;
    return launch<true>(maps, dx, dw, db, p, plan.teams * plan.team, status, s);
}

}  // namespace lin
