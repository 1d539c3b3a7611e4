// Shared by the general attention kernels on the tensor cores (attn_fwd_sm100.cu, attn_bwd_sm100.cu): fp32 operands as
// sums of bf16 terms, tiles of them in shared memory, tensor-memory accesses of any multiple of four columns.
//
// An fp32 value is the sum of three bf16 values exactly (24 = 3 x 8 significant bits).  A product of two such sums is
// evaluated as the six term products that reach 2^-24 of it, the smallest first: every tcgen05.mma truncates its sum to
// fp32, which costs next to nothing while the sum is small.  Sums that run on over many tiles are kept in registers and
// added to with ordinary (rounded) additions, the tensor cores start every tile at zero.
#pragma once

#include <math.h>

#include <type_traits>

#include "tc05.cuh"

namespace attn24 {

using namespace tc05;

// Threads that compute: a thread owns one row of the 128-row tile (its tensor-memory lane) and a quarter of the columns.
constexpr int kWorkers = 512;
constexpr int kThreads = kWorkers + 128;  // and a group of which one warp issues the tensor-core instructions
constexpr int kWorkWarps = kWorkers / 32;
constexpr int kStep = 64;  // rows of the smaller tile operand

// log2(e) / sqrt(D) as the sum of two floats, both positive (a score of -inf times either is -inf), and a little more than
// that: the tensor cores truncate, so the last k = D / 16 products of a score, which are not small, leave it too small by
// (0.18 k + 0.5) * 2^-24 of it on average.  That is what scores of 2^3 and more showed at D = 16 ... 128 against 64 bits (0.36 k
// + 0.36 would follow from cutting off half a unit of the sum so far after each product, and is too much: the sums seem to
// have a bit more on the way).  Relative error of the log-sum-exp without it, with twice of it and with it, and in fp32
// arithmetic, 1e-8: D = 128, q and k of standard deviation one 3.6, 2.8, 2.8, 3.1, of two 11.0, 7.7, 4.2, 6.6; D = 64, of two
// 6.8, 4.6, 3.3, 4.9.  In the backward, which takes its scores from 16-bit operands, it is 1 % of the error (dq at D = 128, of
// two: 1.67e-5 without it, 1.65e-5 with it, 1.66e-5 in fp32 arithmetic).
struct Scale {
    float hi, lo;
};
inline Scale log2_scale(int D) {
    const double c = 1.4426950408889634 / sqrt((double)D) * (1.0 + (0.18 * ((D + 15) / 16) + 0.5) / 16777216.0);
    float hi = (float)c;
    if ((double)hi >= c) hi = nextafterf(hi, 0.f);
    return Scale{hi, (float)(c - (double)hi)};
}

__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// p = hi + mid + lo for both halves: hi rounded, mid the next eight bits cut off, lo what is left.  The rounding is an
// integer addition: conversions share the quarter-rate pipe with exp2.  What is not finite stays so in one of the terms, but
// not what it was: an infinity leaves inf and NaN (inf - inf), a finite value above 3.396e38 rounds up to inf, a NaN may leave
// hi, but not mid.  Products with them are NaN, and whoever uses this looks for that.  half: 0 to cut hi off, too.
__device__ __forceinline__ void split3(float2 p, uint32_t &hi, uint32_t &mid, uint32_t &lo, uint32_t half = 0x8000u) {
    const float2 minus = make_float2(-1.f, -1.f);
    const uint32_t a = __float_as_uint(p.x) + half, b = __float_as_uint(p.y) + half;
    hi = __byte_perm(a, b, 0x7632);
    const float2 r = fma2(make_float2(__uint_as_float(a & 0xFFFF0000u), __uint_as_float(b & 0xFFFF0000u)), minus, p);
    mid = __byte_perm(__float_as_uint(r.x), __float_as_uint(r.y), 0x7632);
    const float2 s = fma2(make_float2(__uint_as_float(__float_as_uint(r.x) & 0xFFFF0000u),
                                      __uint_as_float(__float_as_uint(r.y) & 0xFFFF0000u)),
                          minus, r);
    lo = __byte_perm(__float_as_uint(s.x), __float_as_uint(s.y), 0x7632);
}

// Eight consecutive values of a row of `width`, from column col on; zeros past the end and where the row is not `in`.
// vec: width is a multiple of 4, so rows and the groups of four in them are 16-byte aligned.
__device__ __forceinline__ void load8(float (&f)[8], const float *row, int col, int width, bool in, bool vec) {
    if (vec) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (in && col < width) a = __ldg(reinterpret_cast<const float4 *>(row + col));
        if (in && col + 4 < width) b = __ldg(reinterpret_cast<const float4 *>(row + col + 4));
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++) f[e] = in && col + e < width ? __ldg(row + col + e) : 0.f;
    }
}
// The same for bf16 values, into shared memory.
__device__ __forceinline__ void copy8(uint8_t *dst, const __nv_bfloat16 *row, int col, int width, bool in, bool vec) {
    uint32_t w[4];
    if (vec) {
        uint2 a = make_uint2(0, 0), b = a;
        if (in && col < width) a = __ldg(reinterpret_cast<const uint2 *>(row + col));
        if (in && col + 4 < width) b = __ldg(reinterpret_cast<const uint2 *>(row + col + 4));
        w[0] = a.x, w[1] = a.y, w[2] = b.x, w[3] = b.y;
    } else {
        const uint16_t *bits = reinterpret_cast<const uint16_t *>(row);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t x = in && col + 2 * e < width ? __ldg(bits + col + 2 * e) : 0u;
            const uint32_t y = in && col + 2 * e + 1 < width ? __ldg(bits + col + 2 * e + 1) : 0u;
            w[e] = x | y << 16;
        }
    }
    *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}
// Eight floats from shared memory, by threads whose column 8 c differs: half of them start with the second word, so that
// eight neighbours read 128 different bytes at a time.
__device__ __forceinline__ void lds8(float (&f)[8], const float *src, int c) {
    const int swap = c & 4;
    const float4 a = *reinterpret_cast<const float4 *>(src + swap), b = *reinterpret_cast<const float4 *>(src + (swap ^ 4));
    const float4 x = swap ? b : a, y = swap ? a : b;
    f[0] = x.x, f[1] = x.y, f[2] = x.z, f[3] = x.w, f[4] = y.x, f[5] = y.y, f[6] = y.z, f[7] = y.w;
}

// Eight values from column col of a row as the two bf16 planes the backward reads, rounded as launch_split rounds them.
__device__ __forceinline__ void save8(__nv_bfloat16 *hi, __nv_bfloat16 *lo, int col, int width, const float (&f)[8], bool vec) {
    if (col >= width) return;
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; e++) split_bf16x2(f[2 * e], f[2 * e + 1], h[e], l[e]);
    if (vec && width % 8 == 0) {
        *reinterpret_cast<uint4 *>(hi + col) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4 *>(lo + col) = make_uint4(l[0], l[1], l[2], l[3]);
    } else if (vec) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            if (col + 4 * i >= width) break;
            *reinterpret_cast<uint2 *>(hi + col + 4 * i) = make_uint2(h[2 * i], h[2 * i + 1]);
            *reinterpret_cast<uint2 *>(lo + col + 4 * i) = make_uint2(l[2 * i], l[2 * i + 1]);
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++) {
            if (col + e >= width) break;
            reinterpret_cast<uint16_t *>(hi)[col + e] = (uint16_t)(h[e >> 1] >> (16 * (e & 1)));
            reinterpret_cast<uint16_t *>(lo)[col + e] = (uint16_t)(l[e >> 1] >> (16 * (e & 1)));
        }
    }
}

// Tiles in shared memory: planes of 64-column blocks, in a block a row of 128 bytes per row, with the 128-byte swizzle.
// A worker moves eight values at a time: column 8 c of row r (of 64) and, from 64 columns on, the same in the next block.
struct Chunk {
    int r, c, at;  // at: bytes into a block
    __device__ __forceinline__ Chunk(int tid) : r(tid >> 3), c(tid & 7), at(r * 128 + ((c ^ (r & 7)) << 4)) {}
    template <int kK>
    __device__ __forceinline__ bool has(int i) const { return c + 8 * i < 2 * kK; }
    __device__ __forceinline__ int col(int i) const { return 8 * c + 64 * i; }
};

// Splits eight values into the three planes at `tile`, `plane` bytes apart.  kLarge: hi is cut off instead of rounded where one
// of the values would round up to infinity (three terms of eight bits all the same).
template <bool kLarge = false>
__device__ __forceinline__ void store_split3(uint8_t *tile, int plane, int at, const float (&f)[8]) {
    uint32_t half = 0x8000u;
    if (kLarge) {
        float top = fmaxf(fabsf(f[0]), fabsf(f[1]));
#pragma unroll
        for (int e = 2; e < 8; e += 2) top = max3(top, fabsf(f[e]), fabsf(f[e + 1]));
        half = top >= __uint_as_float(0x7f7f8000u) ? 0u : half;
    }
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; e++) split3(make_float2(f[2 * e], f[2 * e + 1]), h[e], m[e], l[e], half);
    *reinterpret_cast<uint4 *>(tile + at) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(tile + plane + at) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4 *>(tile + 2 * plane + at) = make_uint4(l[0], l[1], l[2], l[3]);
}

// ------------------------------------------------------------------------------------------
// Tensor memory: consecutive columns of this thread's lane
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st2(uint32_t taddr, uint32_t a, uint32_t b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}
template <int kN>  // 4 or 8
__device__ __forceinline__ void tmem_load(uint32_t taddr, uint32_t *r) {
    if (kN == 4) tmem_ld4(taddr, r);
    else tmem_ld8(taddr, r);
}
template <int kN>  // 2 or 4
__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t *r) {
    if (kN == 2) tmem_st2(taddr, r[0], r[1]);
    else tmem_st4(taddr, r);
}

// The 64 columns of a score tile become the three terms of P (or dS) in 96: each run of 16 score columns makes 8 of packed
// mid parts and 8 of packed lo parts in its place, the hi parts are in the 32 columns behind.  Where a term's columns for
// contraction step kk (16 scores) start:
__device__ __forceinline__ constexpr uint32_t term_column(int term, int kk) {
    return term == 0 ? 64 + 8 * kk : 16 * kk + 8 * (term - 1);
}

// acc = acc * by + the 4 kN columns at taddr, eight of them in registers at a time
template <int kN>
__device__ __forceinline__ void add_columns(float (&acc)[4 * kN], uint32_t taddr, float by) {
#pragma unroll
    for (int c = 0; c < kN; c += 2) {
        uint32_t r[8];
        if (c + 1 < kN) tmem_ld8(taddr + 4 * c, r);
        else tmem_ld4(taddr + 4 * c, r);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < (c + 1 < kN ? 8 : 4); e++) acc[4 * c + e] = fmaf(acc[4 * c + e], by, __uint_as_float(r[e]));
    }
}

// 4 kN consecutive values of a row of `width`, from column col on, scaled.
template <int kN>
__device__ __forceinline__ void store_columns(float *row, int col, int width, const float (&acc)[4 * kN], float by, bool vec) {
#pragma unroll
    for (int c = 0; c < kN; c++) {
        const int at = col + 4 * c;
        if (vec) {
            if (at < width)
                *reinterpret_cast<float4 *>(row + at) =
                    make_float4(acc[4 * c] * by, acc[4 * c + 1] * by, acc[4 * c + 2] * by, acc[4 * c + 3] * by);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (at + e < width) row[at + e] = acc[4 * c + e] * by;
        }
    }
}

// One arrival per warp, after what its lanes wrote to shared memory or did to tensor memory.
__device__ __forceinline__ void warp_arrive(uint64_t *bar, int lane) {
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// A bounded wait.  When one runs out, all others of the CTA return at once; threads that request copies stop then, every
// other role goes through the rest of its loop (of which it skips nothing that another thread waits for) to the common end.
// As a parity is all a waiter can name, no barrier may get two phases ahead of any of its waiters.
__device__ __forceinline__ bool await_thread(uint64_t *bar, uint32_t parity, const WaitCtx &ctx, int site) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    while (!*ctx.cta_abort) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_timer_ns() - t0 > TC05_WAIT_LIMIT_NS) {
            *ctx.cta_abort = 1;
            if (ctx.status) atomicCAS(ctx.status, 0, ST_TIMEOUT_BASE + site);
        }
    }
    return false;
}
__device__ __forceinline__ void await(uint64_t *bar, uint32_t parity, const WaitCtx &ctx, int site) {
    await_thread(bar, parity, ctx, site);
    __syncwarp();
    tc_fence_after_sync();
}

// Named barrier `id` (not 0): waits for, or only counts towards, `count` threads.
__device__ __forceinline__ void named_sync(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int count) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }

// f(std::integral_constant<int, n>{}) for n = 1 .. 8, the number of 16-column groups of the head size
template <class Fn>
inline cudaError_t with_groups(int n, Fn f) {
    switch (n) {
        case 1: return f(std::integral_constant<int, 1>{});
        case 2: return f(std::integral_constant<int, 2>{});
        case 3: return f(std::integral_constant<int, 3>{});
        case 4: return f(std::integral_constant<int, 4>{});
        case 5: return f(std::integral_constant<int, 5>{});
        case 6: return f(std::integral_constant<int, 6>{});
        case 7: return f(std::integral_constant<int, 7>{});
        default: return f(std::integral_constant<int, 8>{});
    }
}

}  // namespace attn24
