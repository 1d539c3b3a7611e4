// General-shape causal attention kernels (fp32 SIMT, tiled) and the elementwise
// preparation kernels shared with the tensor-core path.
//
// These kernels serve the head sizes the tcgen05 kernels do not take, 129 to 256, and any T <= 8192.  They replace
// the same reference code as those: kernels/src/cuda/Attention.cu:170-324 of gpt.c.
#include "attn_internal.h"
#include "tc05.cuh"

namespace attn {

namespace {

constexpr int kWarp = 32;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------------
// split: x -> hi, lo
// ---------------------------------------------------------------------------------------
// Small tensors, whose planes the next kernel reads from L2.
__global__ void __launch_bounds__(256) split_small_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ hi,
                                                     __nv_bfloat16 *__restrict__ lo, size_t n) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    const size_t n8 = n / 8;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n8; v += stride) {
        const float4 a = __ldcs(reinterpret_cast<const float4 *>(x) + 2 * v);
        const float4 b = __ldcs(reinterpret_cast<const float4 *>(x) + 2 * v + 1);
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
            const float r0 = f[2 * k] - __low2float(hh), r1 = f[2 * k + 1] - __high2float(hh);
            __nv_bfloat162 ll = __floats2bfloat162_rn(r0, r1);
            h[k] = *reinterpret_cast<uint32_t *>(&hh);
            l[k] = *reinterpret_cast<uint32_t *>(&ll);
        }
        reinterpret_cast<uint4 *>(hi)[v] = make_uint4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<uint4 *>(lo)[v] = make_uint4(l[0], l[1], l[2], l[3]);
    }
    // ragged tail (n not a multiple of 8)
    for (size_t i = n8 * 8 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float f = x[i];
        const __nv_bfloat16 hh = __float2bfloat16_rn(f);
        hi[i] = hh;
        lo[i] = __float2bfloat16_rn(f - __bfloat162float(hh));
    }
}

// Read once and written once: HBM bound.  32 bytes per load, two of them in flight per thread, every block one piece;
// results leave the cache first (the loop above, 16 bytes per load, took 133 us for 805 MB, this 121 us; 125 us at the
// copy rate).  On small tensors it is no slower itself, but a forward of B=8 T=128 H=12 went from 10.7 to 12.3 us.
__global__ void __launch_bounds__(256) split_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ hi,
                                                     __nv_bfloat16 *__restrict__ lo, size_t n) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    constexpr int kU = 2;
    const size_t n8 = n / 8, v0 = (size_t)blockIdx.x * (256 * kU) + threadIdx.x;
    const bool wide = (reinterpret_cast<uintptr_t>(x) & 31u) == 0;
    float f[kU][8];
#pragma unroll
    for (int u = 0; u < kU; u++) {
        const size_t v = v0 + 256 * u;
        if (v >= n8) break;
        if (wide) {
            asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=f"(f[u][0]), "=f"(f[u][1]), "=f"(f[u][2]), "=f"(f[u][3]), "=f"(f[u][4]), "=f"(f[u][5]), "=f"(f[u][6]),
                           "=f"(f[u][7])
                         : "l"(x + 8 * v));
        } else {
            const float4 a = __ldcs(reinterpret_cast<const float4 *>(x) + 2 * v), b = __ldcs(reinterpret_cast<const float4 *>(x) + 2 * v + 1);
            f[u][0] = a.x, f[u][1] = a.y, f[u][2] = a.z, f[u][3] = a.w, f[u][4] = b.x, f[u][5] = b.y, f[u][6] = b.z, f[u][7] = b.w;
        }
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
        const size_t v = v0 + 256 * u;
        if (v >= n8) break;
        uint4 h, l;
        tc05::split_bf16x2(f[u][0], f[u][1], h.x, l.x);
        tc05::split_bf16x2(f[u][2], f[u][3], h.y, l.y);
        tc05::split_bf16x2(f[u][4], f[u][5], h.z, l.z);
        tc05::split_bf16x2(f[u][6], f[u][7], h.w, l.w);
        __stcs(reinterpret_cast<uint4 *>(hi) + v, h);
        __stcs(reinterpret_cast<uint4 *>(lo) + v, l);
    }
    // ragged tail (n not a multiple of 8)
    if (blockIdx.x == 0 && n8 * 8 + threadIdx.x < n) {
        const size_t i = n8 * 8 + threadIdx.x;
        const float t = x[i];
        const __nv_bfloat16 hh = __float2bfloat16_rn(t);
        hi[i] = hh;
        lo[i] = __float2bfloat16_rn(t - __bfloat162float(hh));
    }
}

// ---------------------------------------------------------------------------------------
// backward preparation for the general kernels: delta[b,h,t] = sum_d dout*out, and zero-fill of the
// dq third of dqkv (the backward accumulates dq in memory), or of all of it.  One warp per (b, t, h): D elements.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) bwd_prepare_kernel(const float *__restrict__ dout, const float *__restrict__ out,
                                                           float *__restrict__ delta, float *__restrict__ dqkv, bool zero_all,
                                                           int B, int T, int H, int D) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    const int lane = threadIdx.x & 31;
    const size_t nrows = (size_t)B * T * H;
    const size_t wstride = (size_t)gridDim.x * (blockDim.x >> 5);
    const int C = H * D;
    for (size_t w = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < nrows; w += wstride) {
        const int h = (int)(w % H);
        const size_t bt = w / H;
        const int t = (int)(bt % T);
        const int b = (int)(bt / T);
        const size_t base = bt * C + (size_t)h * D;
        float acc = 0.f;
        for (int d = lane; d < D; d += kWarp) {
            const float g = dout[base + d];
            acc += g * out[base + d];
            float *zero = dqkv + bt * 3 * C + (size_t)h * D + d;
            zero[0] = 0.f;
            if (zero_all) zero[C] = zero[2 * C] = 0.f;
        }
        acc = warp_sum(acc);
        if (lane == 0) delta[((size_t)b * H + h) * T + t] = acc;
    }
}

// The same for up to 64 columns, a multiple of 4: 8 or 16 lanes per row, a 16-byte word each (B=32 T=1024 H=16 D=64 120 ->
// 70 ... 77 us, B=8 T=1024 H=4 D=48 7.5 -> 5.4; at D = 128 the kernel above is faster, 6.5 against 8.2 us for B=4 T=1024 H=6).
__global__ void __launch_bounds__(256) bwd_prepare_words_kernel(const float *__restrict__ dout, const float *__restrict__ out,
                                                                 float *__restrict__ delta, float *__restrict__ dqkv, bool zero_all,
                                                                 int lanes, int B, int T, int H, int D) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    const size_t w = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / lanes, nrows = (size_t)B * T * H, bt = w / H;
    const int d = 4 * (threadIdx.x % lanes), h = (int)(w % H), C = H * D;
    float acc = 0.f;
    if (w < nrows && d < D) {
        const float4 g = __ldcs(reinterpret_cast<const float4 *>(dout + w * D + d)), o = __ldcs(reinterpret_cast<const float4 *>(out + w * D + d));
        acc = g.x * o.x + g.y * o.y + g.z * o.z + g.w * o.w;
        for (int part = 0; part < (zero_all ? 3 : 1); part++)
            *reinterpret_cast<float4 *>(dqkv + (bt * 3 + part) * C + (size_t)h * D + d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int o = lanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (w < nrows && d == 0) delta[(bt / T * H + h) * T + bt % T] = acc;
}

// ---------------------------------------------------------------------------------------
// backward preparation for head size 64 (the tensor-core path): the same work as above with
// 8 consecutive elements per thread, so 8 lanes cover one (b, t, h) row of 64 values.  HBM bound: 32 bytes per access,
// one piece per block (1.68 GB: 283 us with 16-byte accesses in a grid-stride loop, 261 us now; 260 at the copy rate).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void load8_last_use(const float *p, float4 &a, float4 &b) {
    asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}
__global__ void __launch_bounds__(256) bwd_prepare64_kernel(const float *__restrict__ dout, const float *__restrict__ out,
                                                             float *__restrict__ delta, __nv_bfloat16 *__restrict__ dhi,
                                                             __nv_bfloat16 *__restrict__ dlo, float *__restrict__ dq_zero,
                                                             int *__restrict__ sched, int B, int T, int H) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    if (sched && blockIdx.x == 0 && threadIdx.x < 2) sched[threadIdx.x] = 0;  // item counter of the backward core
    const int C = H * 64;
    const size_t nvec = (size_t)B * T * C / 8;  // multiple of 8, so whole groups of 8 lanes stay together
    const int lane = threadIdx.x & 31;
    const bool wide = ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dq_zero)) & 31u) == 0;
    const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v - lane < nvec) {  // warp-uniform (shuffles below need every lane); memory accesses are guarded
        const bool active = v < nvec;
        const size_t bt = v / (C / 8);
        const int c8 = (int)(v % (C / 8));
        const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 g0 = zero4, g1 = zero4, o0 = zero4, o1 = zero4;
        if (active && wide) {
            load8_last_use(dout + 8 * v, g0, g1);
            load8_last_use(out + 8 * v, o0, o1);
        } else if (active) {
            g0 = __ldcs(reinterpret_cast<const float4 *>(dout) + 2 * v), g1 = __ldcs(reinterpret_cast<const float4 *>(dout) + 2 * v + 1);
            o0 = __ldcs(reinterpret_cast<const float4 *>(out) + 2 * v), o1 = __ldcs(reinterpret_cast<const float4 *>(out) + 2 * v + 1);
        }
        float acc = g0.x * o0.x + g0.y * o0.y + g0.z * o0.z + g0.w * o0.w + g1.x * o1.x + g1.y * o1.y + g1.z * o1.z +
                    g1.w * o1.w;
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        const float f[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        uint32_t hw[4], lw[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
            __nv_bfloat162 ll = __floats2bfloat162_rn(f[2 * k] - __low2float(hh), f[2 * k + 1] - __high2float(hh));
            hw[k] = *reinterpret_cast<uint32_t *>(&hh);
            lw[k] = *reinterpret_cast<uint32_t *>(&ll);
        }
        if (!active) return;
        reinterpret_cast<uint4 *>(dhi)[v] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        reinterpret_cast<uint4 *>(dlo)[v] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        float4 *z = reinterpret_cast<float4 *>(dq_zero + bt * 3 * C + (size_t)c8 * 8);
        if (wide) {
            asm volatile("st.global.v8.f32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"l"(z), "f"(0.f) : "memory");
        } else {
            z[0] = zero4;
            z[1] = zero4;
        }
        if ((c8 & 7) == 0) {
            const int h = c8 >> 3, t = (int)(bt % T), b = (int)(bt / T);
            delta[((size_t)b * H + h) * T + t] = acc;
        }
    }
}

// ---------------------------------------------------------------------------------------
// General kernels: causal attention in fp32 for head sizes above 128, tiled over queries and keys.
//
// What bounds them is the fp32 pipe, so they are built around register tiles: a thread owns kR rows and
// several columns of every product and reads its operands from shared memory in 16-byte words, 16 packed
// multiply-adds (fma.rn.f32x2) for each such word of a score tile and 6 for each word of an output tile.
// A warp covers 4 row groups x 8 column groups, which lets the 8 (or 4) lanes that want the same word get
// it in one access; rows are padded to an odd number of 16-byte words, so 8 rows in a column do not collide.
//   score products (contraction over the head size, contiguous in both operands): the two halves of a packed
//     accumulator hold the sums over even and odd head columns, added once at the end;
//   output products (contraction over keys or queries): they hold two neighbouring head columns, the other
//     operand is broadcast into both halves.
// kNI = head columns in blocks of 32 (the output tile's width), so D = 140 does 160 columns of output work; the
// score products run over exactly the 4-column words that hold data.
// ---------------------------------------------------------------------------------------
typedef unsigned long long f32x2;  // two floats of a packed instruction

__device__ __forceinline__ f32x2 fma_x2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul_x2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 both(float v) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ float2 halves(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ ulonglong2 lds_x4(const float *p) { return *reinterpret_cast<const ulonglong2 *>(p); }

// Row pitch of a tile in shared memory, in floats: wide enough for the output product's columns, an odd number
// of 16-byte words.
template <int kNI>
struct Pitch {
    static constexpr int value = 32 * kNI + 4;
};

// Rows r0 .. r0+kRows-1 of one head (D columns starting at src, rows `stride` apart) into a shared-memory tile, by
// asynchronous copies; rows at or past `rows` and the columns that fill the last 16-byte word become zeros.
template <int kRows, int kPitch, int kThreads, bool kVec>
__device__ __forceinline__ void load_rows_async(float *tile, const float *src, size_t stride, int r0, int rows, int D, int tid) {
    const int words = (D + 3) >> 2;
    for (int r = tid >> 3; r < kRows; r += kThreads / 8) {
        const bool in = r0 + r < rows;
        const float *row = src + (size_t)(in ? r0 + r : 0) * stride;
        const uint32_t dst = tc05::smem_u32(tile + r * kPitch);
        for (int w = tid & 7; w < words; w += 8) {
            if (kVec) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 16 * w), "l"(row + 4 * w),
                             "r"(in ? 16 : 0)
                             : "memory");
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int c = 4 * w + e;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * c),
                                 "l"(row + (c < D ? c : 0)), "r"(in && c < D ? 4 : 0)
                                 : "memory");
                }
            }
        }
    }
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// The same for rows held as two bf16 planes: the sum of the two is stored.
template <int kRows, int kPitch, int kThreads, bool kVec>
__device__ __forceinline__ void load_rows_split(float *tile, const __nv_bfloat16 *hi, const __nv_bfloat16 *lo, size_t stride,
                                                int r0, int rows, int D) {
    const int words = (D + 3) >> 2;
#pragma unroll 2
    for (int r = threadIdx.x >> 3; r < kRows; r += kThreads / 8) {
        const bool in = r0 + r < rows;
        const size_t at = (size_t)(in ? r0 + r : 0) * stride;
#pragma unroll 2
        for (int w = threadIdx.x & 7; w < words; w += 8) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in) {
                if (kVec) {
                    const uint2 h = __ldg(reinterpret_cast<const uint2 *>(hi + at) + w);
                    const uint2 l = __ldg(reinterpret_cast<const uint2 *>(lo + at) + w);
                    v.x = __uint_as_float(h.x << 16) + __uint_as_float(l.x << 16);
                    v.y = __uint_as_float(h.x & 0xffff0000u) + __uint_as_float(l.x & 0xffff0000u);
                    v.z = __uint_as_float(h.y << 16) + __uint_as_float(l.y << 16);
                    v.w = __uint_as_float(h.y & 0xffff0000u) + __uint_as_float(l.y & 0xffff0000u);
                } else {
                    float f[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int c = 4 * w + e;
                        f[e] = c < D ? __bfloat162float(hi[at + c]) + __bfloat162float(lo[at + c]) : 0.f;
                    }
                    v = make_float4(f[0], f[1], f[2], f[3]);
                }
            }
            *reinterpret_cast<float4 *>(tile + r * kPitch + 4 * w) = v;
        }
    }
}

// acc[r][c] += rows a0 + 4 r of A (pitch floats apart) times rows b0 + 8 c of B, over `words` 4-column words.
template <int kR, int kC, int kPitch>
__device__ __forceinline__ void score_product(f32x2 (&acc)[kR][kC], const float *a0, const float *b0, int words) {
#pragma unroll
    for (int r = 0; r < kR; r++)
#pragma unroll
        for (int c = 0; c < kC; c++) acc[r][c] = 0ull;
#pragma unroll 2
    for (int w = 0; w < words; w++) {
        ulonglong2 a[kR], b[kC];
#pragma unroll
        for (int r = 0; r < kR; r++) a[r] = lds_x4(a0 + 4 * r * kPitch + 4 * w);
#pragma unroll
        for (int c = 0; c < kC; c++) b[c] = lds_x4(b0 + 8 * c * kPitch + 4 * w);
#pragma unroll
        for (int r = 0; r < kR; r++)
#pragma unroll
            for (int c = 0; c < kC; c++) {
                acc[r][c] = fma_x2(a[r].x, b[c].x, acc[r][c]);
                acc[r][c] = fma_x2(a[r].y, b[c].y, acc[r][c]);
            }
    }
}
__device__ __forceinline__ float total(f32x2 v) {
    const float2 h = halves(v);
    return h.x + h.y;
}

template <bool kVec>
__device__ __forceinline__ void store_cols(float *row, int col, int D, float4 v) {
    if (kVec) {
        if (col < D) *reinterpret_cast<float4 *>(row + col) = v;  // D is a multiple of 4
    } else {
        if (col < D) row[col] = v.x;
        if (col + 1 < D) row[col + 1] = v.y;
        if (col + 2 < D) row[col + 2] = v.z;
        if (col + 3 < D) row[col + 3] = v.w;
    }
}

// ---------------------------------------------------------------------------------------
// forward: one block per (b, h, 64 queries), key tiles of 8 kC, online softmax.  Two groups of four warps take the
// key tiles in turns, each with its own K, V and P tiles, and the two partial results are merged at the end: a block
// then has its SM to itself and the longest-first order balances the SMs.  (With one group per block and two blocks per
// SM, the SMs were busy for 71 % of the launch on average, because the long blocks that start together share an SM.)
// ---------------------------------------------------------------------------------------
constexpr int kFwdGroup = 128, kFwdThreads = 2 * kFwdGroup, kFwdRows = 64;

template <int kNI, int kC>
struct FwdTile {
    static constexpr int kPitch = Pitch<kNI>::value, kKeys = 8 * kC, kPPitch = kKeys + 4;
    static constexpr int kQ = kFwdRows * kPitch;
    static constexpr int kKP = kKeys * kPitch > kFwdRows * kPPitch ? kKeys * kPitch : kFwdRows * kPPitch;  // K, then P
    static constexpr int kV = kKeys * kPitch;
    static constexpr size_t kBytes = (size_t)(kQ + 2 * (kKP + kV)) * sizeof(float);
};

// one group's barrier
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

template <int kNI, int kC, bool kVec>
__global__ void __launch_bounds__(kFwdThreads) generic_fwd_kernel(const float *__restrict__ qkv, float *__restrict__ out,
                                                                  float *__restrict__ out_copy, float *__restrict__ lse,
                                                                  int T, int H, int D, float scale) {
    using S = FwdTile<kNI, kC>;
    constexpr int kR = 4, kPitch = S::kPitch, kKeys = S::kKeys, kPPitch = S::kPPitch;
    extern __shared__ __align__(16) float sm[];
    const int group = threadIdx.x / kFwdGroup, tid = threadIdx.x % kFwdGroup;
    float *sq = sm, *sk = sm + S::kQ + group * (S::kKP + S::kV), *sp = sk, *sv = sk + S::kKP;
    const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
    const int row0 = 16 * (tid >> 5) + ty;  // this thread's rows: row0 + 4 r
    const int nq = (T + kFwdRows - 1) / kFwdRows;
    const int nbh = gridDim.x / nq;
    const int q0 = (nq - 1 - (int)blockIdx.x / nbh) * kFwdRows;  // longest rows first
    const int bh = (int)blockIdx.x % nbh, b = bh / H, h = bh % H;
    const int C = H * D;
    const size_t C3 = 3 * (size_t)C;
    const int words = (D + 3) >> 2;
    const float *head = qkv + (size_t)b * T * C3 + (size_t)h * D;

    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    load_rows_async<kFwdRows, kPitch, kFwdThreads, kVec>(sq, head, C3, q0, T, D, threadIdx.x);
    async_wait_all();
    __syncthreads();
    f32x2 o[kR][2 * kNI];
    float m[kR], l[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        m[r] = -INFINITY, l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 2 * kNI; i++) o[r][i] = 0ull;
    }
    const int last = min(q0 + kFwdRows, T) - 1;
    for (int j0 = group * kKeys; j0 <= last; j0 += 2 * kKeys) {
        load_rows_async<kKeys, kPitch, kFwdGroup, kVec>(sk, head + C, C3, j0, T, D, tid);
        async_commit();
        load_rows_async<kKeys, kPitch, kFwdGroup, kVec>(sv, head + 2 * C, C3, j0, T, D, tid);
        async_commit();
        async_wait<1>();
        group_sync(group);
        float p[kR][kC];
        {
            f32x2 acc[kR][kC];
            score_product<kR, kC, kPitch>(acc, sq + row0 * kPitch, sk + tx * kPitch, words);
#pragma unroll
            for (int r = 0; r < kR; r++)
#pragma unroll
                for (int c = 0; c < kC; c++) p[r][c] = total(acc[r][c]) * scale;
        }
        if (j0 + kKeys > q0) {  // the diagonal passes through this tile
#pragma unroll
            for (int r = 0; r < kR; r++)
#pragma unroll
                for (int c = 0; c < kC; c++)
                    if (j0 + tx + 8 * c > q0 + row0 + 4 * r) p[r][c] = -INFINITY;
        }
#pragma unroll
        for (int r = 0; r < kR; r++) {
            float mx = p[r][0];
#pragma unroll
            for (int c = 1; c < kC; c++) mx = fmaxf(mx, p[r][c]);
#pragma unroll
            for (int s = 1; s < 8; s <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
            mx = fmaxf(mx, m[r]);
            const float alpha = mx == -INFINITY ? 1.f : expf(m[r] - mx);
            m[r] = mx;
            if (mx == -INFINITY) mx = 0.f;  // group 1 may start with a tile that lies past all keys of a row
            l[r] *= alpha;
            const f32x2 a2 = both(alpha);
#pragma unroll
            for (int i = 0; i < 2 * kNI; i++) o[r][i] = mul_x2(o[r][i], a2);
#pragma unroll
            for (int c = 0; c < kC; c++) {
                p[r][c] = expf(p[r][c] - mx);
                l[r] += p[r][c];
            }
        }
        group_sync(group);  // K has been read by everybody: its place takes P
#pragma unroll
        for (int r = 0; r < kR; r++)
#pragma unroll
            for (int c = 0; c < kC; c++) sp[(row0 + 4 * r) * kPPitch + tx + 8 * c] = p[r][c];
        async_wait<0>();
        group_sync(group);
#pragma unroll 1
        for (int j = 0; j < kKeys; j += 4) {
            float4 pr[kR];
#pragma unroll
            for (int r = 0; r < kR; r++) pr[r] = *reinterpret_cast<const float4 *>(sp + (row0 + 4 * r) * kPPitch + j);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                ulonglong2 v[kNI];
#pragma unroll
                for (int i = 0; i < kNI; i++) v[i] = lds_x4(sv + (j + e) * kPitch + 4 * tx + 32 * i);
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    const f32x2 pe = both(e == 0 ? pr[r].x : e == 1 ? pr[r].y : e == 2 ? pr[r].z : pr[r].w);
#pragma unroll
                    for (int i = 0; i < kNI; i++) {
                        o[r][2 * i] = fma_x2(pe, v[i].x, o[r][2 * i]);
                        o[r][2 * i + 1] = fma_x2(pe, v[i].y, o[r][2 * i + 1]);
                    }
                }
            }
        }
        group_sync(group);  // P and V have been read: the next tile may overwrite them
    }
#pragma unroll
    for (int r = 0; r < kR; r++)
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], s);
    // group 1 leaves its output sums in its own tiles, maximum and sum of every row in the Q tile
    f32x2 *po = reinterpret_cast<f32x2 *>(sm + S::kQ + S::kKP + S::kV);
    float *ml = sm;
    __syncthreads();
    if (group == 1) {
#pragma unroll
        for (int r = 0; r < kR; r++) {
            ml[r * kFwdGroup + tid] = m[r];
            ml[(kR + r) * kFwdGroup + tid] = l[r];
#pragma unroll
            for (int i = 0; i < 2 * kNI; i++) po[(r * 2 * kNI + i) * kFwdGroup + tid] = o[r][i];
        }
    }
    __syncthreads();
    if (group == 1) return;
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int t = q0 + row0 + 4 * r;
        if (t >= T) continue;
        // the other group's thread of this number has the same rows and columns
        const float m1 = ml[r * kFwdGroup + tid], top = fmaxf(m[r], m1);
        const float by0 = expf(m[r] - top), by1 = expf(m1 - top);  // m1 is -inf when that group had no tile
        const float sum = l[r] * by0 + ml[(kR + r) * kFwdGroup + tid] * by1;
        const f32x2 w0 = both(by0), w1 = both(by1);
#pragma unroll
        for (int i = 0; i < 2 * kNI; i++) o[r][i] = fma_x2(o[r][i], w0, mul_x2(po[(r * 2 * kNI + i) * kFwdGroup + tid], w1));
        const float inv = 1.0f / sum;
        const size_t at = ((size_t)b * T + t) * C + (size_t)h * D;
#pragma unroll
        for (int i = 0; i < kNI; i++) {
            const float2 lo = halves(o[r][2 * i]), hi = halves(o[r][2 * i + 1]);
            const float4 v = make_float4(lo.x * inv, lo.y * inv, hi.x * inv, hi.y * inv);
            store_cols<kVec>(out + at, 4 * tx + 32 * i, D, v);
            if (out_copy) store_cols<kVec>(out_copy + at, 4 * tx + 32 * i, D, v);
        }
        if (tx == 0) lse[(size_t)bh * T + t] = top + logf(sum);
    }
}

// ---------------------------------------------------------------------------------------
// backward: one block per (b, h, key tile of 8 kC keys), query tiles from the diagonal on.  K, V, the query tile's Q
// and dO, P and dS sit in shared memory (one block of 8 warps per SM).  Two groups of four
// warps share the five products: one computes S and then dV, the other dP, dS and then dK; each keeps its gradient
// tile in registers over all query tiles; dQ of the query tile is shared out by blocks of 32 head columns and added
// to memory with fp32 atomics (a second kernel that owns the queries would do S and dP again, seven products
// instead of five).  dq has been zero-filled by the preparation kernel.
// ---------------------------------------------------------------------------------------
constexpr int kBwdThreads = 256;

template <int kNI, int kC>
struct BwdTile {
    static constexpr int kPitch = Pitch<kNI>::value, kRows = 8 * kC, kPPitch = kRows + 4;
    static constexpr int kX = kRows * kPitch, kP = kRows * kPPitch;
    static constexpr size_t kBytes = (size_t)(4 * kX + 2 * kP + 2 * kRows) * sizeof(float);
};

// g[k][..] += sum over the query tile of p[q][key k] * x[q][columns of this thread]
template <int kR, int kNI, int kRows, int kPPitch, int kPitch>
__device__ __forceinline__ void key_gradient(f32x2 (&g)[kR][2 * kNI], const float *p, const float *x) {
#pragma unroll 2
    for (int q = 0; q < kRows; q++) {
        float pk[kR];
        const float2 v = *reinterpret_cast<const float2 *>(p + q * kPPitch);
        pk[0] = v.x, pk[1] = v.y;
        ulonglong2 xv[kNI];
#pragma unroll
        for (int i = 0; i < kNI; i++) xv[i] = lds_x4(x + q * kPitch + 32 * i);
#pragma unroll
        for (int k = 0; k < kR; k++) {
            const f32x2 pe = both(pk[k]);
#pragma unroll
            for (int i = 0; i < kNI; i++) {
                g[k][2 * i] = fma_x2(pe, xv[i].x, g[k][2 * i]);
                g[k][2 * i + 1] = fma_x2(pe, xv[i].y, g[k][2 * i + 1]);
            }
        }
    }
}

template <int kNI, int kC, bool kVec>
__global__ void __launch_bounds__(kBwdThreads) generic_bwd_kernel(const __nv_bfloat16 *__restrict__ xhi,
                                                                  const __nv_bfloat16 *__restrict__ xlo,
                                                                  const float *__restrict__ lse,
                                                                  const float *__restrict__ delta,
                                                                  const float *__restrict__ dout,
                                                                  float *__restrict__ dqkv, int T, int H, int D,
                                                                  float scale) {
    using S = BwdTile<kNI, kC>;
    constexpr int kR = kC / 2;  // 16 row groups cover the tile
    constexpr int kPitch = S::kPitch, kRows = S::kRows, kPPitch = S::kPPitch;
    constexpr int kQI = (kNI + 1) / 2;  // column blocks of dQ per group
    extern __shared__ __align__(16) float sm[];
    float *sk = sm, *sv = sk + S::kX, *sq = sv + S::kX, *sg = sq + S::kX;
    float *sp = sg + S::kX, *sd = sp + S::kP, *s_lse = sd + S::kP, *s_delta = s_lse + kRows;
    const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
    const int group = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3;
    const int row0 = 4 * kR * warp + ty;  // score tiles: rows row0 + 4 r, columns tx + 8 c
    const int key0 = 4 * kR * warp + kR * ty;  // gradient tiles: keys key0 .. key0 + kR - 1, columns 4 tx + 32 i
    const int nt = (T + kRows - 1) / kRows;
    const int nbh = gridDim.x / nt;
    const int k0 = (int)blockIdx.x / nbh * kRows;  // the first keys are seen by the most queries
    const int bh = (int)blockIdx.x % nbh, b = bh / H, h = bh % H;
    const int C = H * D;
    const size_t C3 = 3 * (size_t)C;
    const int words = (D + 3) >> 2;
    const size_t head = (size_t)b * T * C3 + (size_t)h * D;
    const float *dhead = dout + (size_t)b * T * C + (size_t)h * D;

    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    load_rows_split<kRows, kPitch, kBwdThreads, kVec>(sk, xhi + head + C, xlo + head + C, C3, k0, T, D);
    load_rows_split<kRows, kPitch, kBwdThreads, kVec>(sv, xhi + head + 2 * C, xlo + head + 2 * C, C3, k0, T, D);
    f32x2 grad[kR][2 * kNI];  // dV in group 0, dK in group 1
#pragma unroll
    for (int r = 0; r < kR; r++)
#pragma unroll
        for (int i = 0; i < 2 * kNI; i++) grad[r][i] = 0ull;

    // A query tile is loaded while dQ of the one before it is computed, the last product, which reads neither: dO by
    // asynchronous copies, Q (split rows) and the row statistics through registers.
    constexpr int kRowsEach = kRows / (kBwdThreads / 8);
    uint2 qh[kRowsEach][kNI], ql[kRowsEach][kNI];
    float stat = 0.f;
    auto request = [&](int q0) {
        load_rows_async<kRows, kPitch, kBwdThreads, kVec>(sg, dhead, (size_t)C, q0, T, D, threadIdx.x);
        async_commit();
        if (kVec) {
#pragma unroll
            for (int i = 0; i < kRowsEach; i++) {
                const int r = q0 + ((int)threadIdx.x >> 3) + i * (kBwdThreads / 8);
                const size_t at = head + (size_t)(r < T ? r : 0) * C3;
#pragma unroll
                for (int u = 0; u < kNI; u++) {
                    const int w = (threadIdx.x & 7) + 8 * u;
                    const bool in = r < T && w < words;
                    qh[i][u] = in ? __ldg(reinterpret_cast<const uint2 *>(xhi + at) + w) : make_uint2(0, 0);
                    ql[i][u] = in ? __ldg(reinterpret_cast<const uint2 *>(xlo + at) + w) : make_uint2(0, 0);
                }
            }
        }
        if (threadIdx.x < 2 * kRows) {
            const int t = q0 + (int)threadIdx.x % kRows;
            const float *src = threadIdx.x < kRows ? lse : delta;
            stat = t < T ? src[(size_t)bh * T + t] : 0.f;
        }
    };
    auto place = [&](int q0) {  // what request() holds in registers; the tile is complete behind the next barrier
        if (kVec) {
#pragma unroll
            for (int i = 0; i < kRowsEach; i++) {
                float *row = sq + (((int)threadIdx.x >> 3) + i * (kBwdThreads / 8)) * kPitch;
#pragma unroll
                for (int u = 0; u < kNI; u++) {
                    const int w = (threadIdx.x & 7) + 8 * u;
                    const uint2 h = qh[i][u], l = ql[i][u];
                    if (w < words)
                        *reinterpret_cast<float4 *>(row + 4 * w) =
                            make_float4(__uint_as_float(h.x << 16) + __uint_as_float(l.x << 16),
                                        __uint_as_float(h.x & 0xffff0000u) + __uint_as_float(l.x & 0xffff0000u),
                                        __uint_as_float(h.y << 16) + __uint_as_float(l.y << 16),
                                        __uint_as_float(h.y & 0xffff0000u) + __uint_as_float(l.y & 0xffff0000u));
                }
            }
        } else {
            load_rows_split<kRows, kPitch, kBwdThreads, kVec>(sq, xhi + head, xlo + head, C3, q0, T, D);
        }
        if (threadIdx.x < 2 * kRows) s_lse[threadIdx.x] = stat;
        async_wait<0>();
    };
    request(k0);
    place(k0);
    __syncthreads();
    for (int q0 = k0; q0 < T; q0 += kRows) {
        {
            f32x2 acc[kR][kC];
            if (group == 0) {
                score_product<kR, kC, kPitch>(acc, sq + row0 * kPitch, sk + tx * kPitch, words);
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    const int q = q0 + row0 + 4 * r;
#pragma unroll
                    for (int c = 0; c < kC; c++) {
                        const float e = expf(total(acc[r][c]) * scale - s_lse[row0 + 4 * r]);
                        sp[(row0 + 4 * r) * kPPitch + tx + 8 * c] = q < T && k0 + tx + 8 * c <= q ? e : 0.f;
                    }
                }
            } else {
                score_product<kR, kC, kPitch>(acc, sg + row0 * kPitch, sv + tx * kPitch, words);
            }
            __syncthreads();  // P is complete
            if (group == 1) {
#pragma unroll
                for (int r = 0; r < kR; r++)
#pragma unroll
                    for (int c = 0; c < kC; c++) {
                        const int at = (row0 + 4 * r) * kPPitch + tx + 8 * c;
                        sd[at] = sp[at] * (total(acc[r][c]) - s_delta[row0 + 4 * r]);
                    }
                asm volatile("bar.sync 1, 128;" ::: "memory");  // dS is complete for the warps of this group
            }
        }
        if (group == 0) key_gradient<kR, kNI, kRows, kPPitch, kPitch>(grad, sp + key0, sg + 4 * tx);
        else key_gradient<kR, kNI, kRows, kPPitch, kPitch>(grad, sd + key0, sq + 4 * tx);
        __syncthreads();  // dS is complete for everybody; Q, dO, P and the statistics have been read
        const bool more = q0 + kRows < T;
        if (more) request(q0 + kRows);
        {
            f32x2 dq[kR][2 * kQI];
#pragma unroll
            for (int r = 0; r < kR; r++)
#pragma unroll
                for (int i = 0; i < 2 * kQI; i++) dq[r][i] = 0ull;
#pragma unroll 1
            for (int j = 0; j < kRows; j += 4) {
                float4 ds[kR];
#pragma unroll
                for (int r = 0; r < kR; r++) ds[r] = *reinterpret_cast<const float4 *>(sd + (row0 + 4 * r) * kPPitch + j);
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    ulonglong2 kv[kQI];
#pragma unroll
                    for (int i = 0; i < kQI; i++) {
                        const int block = min(group + 2 * i, kNI - 1);  // an odd last block is done by group 0
                        kv[i] = lds_x4(sk + (j + e) * kPitch + 4 * tx + 32 * block);
                    }
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const f32x2 de = both(e == 0 ? ds[r].x : e == 1 ? ds[r].y : e == 2 ? ds[r].z : ds[r].w);
#pragma unroll
                        for (int i = 0; i < kQI; i++) {
                            dq[r][2 * i] = fma_x2(de, kv[i].x, dq[r][2 * i]);
                            dq[r][2 * i + 1] = fma_x2(de, kv[i].y, dq[r][2 * i + 1]);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < kR; r++) {
                const int t = q0 + row0 + 4 * r;
                if (t >= T) continue;
                float *dst = dqkv + head + (size_t)t * C3;
#pragma unroll
                for (int i = 0; i < kQI; i++) {
                    const int col = 4 * tx + 32 * (group + 2 * i);
                    const float2 lo = halves(dq[r][2 * i]), hi = halves(dq[r][2 * i + 1]);
                    if (group + 2 * i >= kNI || col >= D) continue;
                    if (kVec) {
                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + col), "f"(lo.x * scale),
                                     "f"(lo.y * scale), "f"(hi.x * scale), "f"(hi.y * scale)
                                     : "memory");
                    } else {
                        const float v[4] = {lo.x * scale, lo.y * scale, hi.x * scale, hi.y * scale};
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (col + e < D) atomicAdd(dst + col + e, v[e]);
                    }
                }
            }
        }
        if (more) place(q0 + kRows);
        __syncthreads();  // the next tile is in place, dS may be overwritten
    }
    const float by = group == 0 ? 1.0f : scale;
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const int t = k0 + key0 + r;
        if (t >= T) continue;
        float *dst = dqkv + head + (size_t)t * C3 + (group == 0 ? 2 * C : C);
#pragma unroll
        for (int i = 0; i < kNI; i++) {
            const float2 lo = halves(grad[r][2 * i]), hi = halves(grad[r][2 * i + 1]);
            store_cols<kVec>(dst, 4 * tx + 32 * i, D, make_float4(lo.x * by, lo.y * by, hi.x * by, hi.y * by));
        }
    }
}

template <int kNI>
struct Generic {
    static constexpr int kC = 4;  // key tiles of 32: 64 would not fit with rows this wide
    using F = FwdTile<kNI, kC>;
    using G = BwdTile<kNI, kC>;

    static cudaError_t set_attributes() {
        cudaError_t e;
        const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if ((e = cudaFuncSetAttribute(generic_fwd_kernel<kNI, kC, true>, a, (int)F::kBytes)) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(generic_fwd_kernel<kNI, kC, false>, a, (int)F::kBytes)) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(generic_bwd_kernel<kNI, kC, true>, a, (int)G::kBytes)) != cudaSuccess) return e;
        return cudaFuncSetAttribute(generic_bwd_kernel<kNI, kC, false>, a, (int)G::kBytes);
    }
    static cudaError_t forward(const float *qkv, float *out, float *out_copy, float *lse, int B, int T, int H, int D,
                               cudaStream_t s) {
        const dim3 grid((unsigned)((size_t)B * H * ((T + kFwdRows - 1) / kFwdRows)));
        return launch_after_previous(D % 4 == 0 ? generic_fwd_kernel<kNI, kC, true> : generic_fwd_kernel<kNI, kC, false>, grid,
                                     dim3(kFwdThreads), F::kBytes, s, qkv, out, out_copy, lse, T, H, D,
                                     1.0f / sqrtf((float)D));
    }
    static cudaError_t backward(const __nv_bfloat16 *xhi, const __nv_bfloat16 *xlo, const float *lse, const float *delta,
                                const float *dout, float *dqkv, int B, int T, int H, int D, cudaStream_t s) {
        const dim3 grid((unsigned)((size_t)B * H * ((T + G::kRows - 1) / G::kRows)));
        return launch_after_previous(D % 4 == 0 ? generic_bwd_kernel<kNI, kC, true> : generic_bwd_kernel<kNI, kC, false>, grid,
                                     dim3(kBwdThreads), G::kBytes, s, xhi, xlo, lse, delta, dout, dqkv, T, H, D,
                                     1.0f / sqrtf((float)D));
    }
};

}  // namespace

// f(Generic<n>{}) for n = 5 .. 8, the number of 32-column blocks of the head size
template <class Fn>
static cudaError_t with_blocks(int n, Fn f) {
    switch (n) {
        case 5: return f(Generic<5>{});
        case 6: return f(Generic<6>{});
        case 7: return f(Generic<7>{});
        default: return f(Generic<8>{});
    }
}

cudaError_t generic_set_attributes() {
    for (int n = kAttn24MaxD / 32 + 1; n <= kGenericMaxD / 32; n++) {
        const cudaError_t e = with_blocks(n, [](auto g) { return decltype(g)::set_attributes(); });
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_split(const float *x, __nv_bfloat16 *hi, __nv_bfloat16 *lo, size_t n, cudaStream_t s) {
    const size_t pieces = (n / 8 + 255) / 256;
    if (pieces <= (size_t)sm_count() * 16)  // one trip of the loop
        return launch_after_previous(split_small_kernel, dim3((unsigned)(pieces ? pieces : 1)), dim3(256), 0, s, x, hi, lo, n);
    return launch_after_previous(split_kernel, dim3((unsigned)((pieces + 1) / 2)), dim3(256), 0, s, x, hi, lo, n);
}

cudaError_t launch_bwd_prepare(const float *dout, const float *out, float *delta, __nv_bfloat16 *dhi,
                               __nv_bfloat16 *dlo, float *dqkv, bool zero_all, int *sched, int B, int T, int H, int D, cudaStream_t s) {
    if (D == 64 && dhi && dlo) {
        const size_t nvec = (size_t)B * T * H * 8;
        const size_t blocks = (nvec + 255) / 256;
        return launch_after_previous(bwd_prepare64_kernel, dim3((unsigned)blocks), dim3(256), 0, s, dout, out, delta, dhi,
                                     dlo, dqkv, sched, B, T, H);
    }
    const size_t rows = (size_t)B * T * H;
    if (D % 4 == 0 && D <= 64) {
        const int lanes = D > 32 ? 16 : 8;
        return launch_after_previous(bwd_prepare_words_kernel, dim3((unsigned)((rows * lanes + 255) / 256)), dim3(256), 0, s, dout, out,
                                     delta, dqkv, zero_all, lanes, B, T, H, D);
    }
    const size_t most = (size_t)sm_count() * 16;
    const size_t blocks = (rows + 7) / 8 < most ? (rows + 7) / 8 : most;
    return launch_after_previous(bwd_prepare_kernel, dim3((unsigned)blocks), dim3(256), 0, s, dout, out, delta, dqkv, zero_all, B, T,
                                 H, D);
}

cudaError_t launch_generic_forward(const float *qkv, float *out, float *out_copy, float *lse, int B, int T, int H,
                                   int D, cudaStream_t s) {
    return with_blocks((D + 31) / 32,
                       [&](auto g) { return decltype(g)::forward(qkv, out, out_copy, lse, B, T, H, D, s); });
}

cudaError_t launch_generic_backward(const __nv_bfloat16 *xhi, const __nv_bfloat16 *xlo, const float *lse,
                                    const float *delta, const float *dout, float *dqkv, int B, int T, int H, int D,
                                    cudaStream_t s) {
    return with_blocks((D + 31) / 32, [&](auto g) {
        return decltype(g)::backward(xhi, xlo, lse, delta, dout, dqkv, B, T, H, D, s);
    });
}

}  // namespace attn
