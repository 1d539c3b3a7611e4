// Cross-entropy loss over the vocabulary for sm_100a: HBM-bound row kernels.
//
// Replaces cross_entropy_forward_cuda_kernel / cross_entropy_backward_cuda_kernel of gpt.c
// (kernels/src/cuda/CrossEntropyLoss.cu:136-178 and their kernels :8-79, :82-129: one warp per row of
// 50257 logits, three passes forward).  Same results and the same buffer semantics:
//   forward   logsm[r, :] = logits[r, :] - max - log(sum exp(logits - max));  loss += -logsm[r, target_r] / rows
//   backward  dout[r, target_r] = -g[r] / rows;  s = sum_j dout[r, j];  dout[r, j] -= exp(logsm[r, j]) * s
// (the backward works on whatever dout holds, like the reference, whose layer hands in zeros).
//
// One block of 1024 threads per row (the forward of long rows: below); the rows of a [rows, 50257] tensor start on 4-byte boundaries only,
// so loads and stores are 4 bytes wide but fully coalesced.  Forward: maximum and sum of exponentials in
// one online pass, then the write pass re-reads the row (200 KB): 8 bytes of HBM traffic per element when the
// re-read hits L2.  The forward loops keep eight loads per thread in flight: with one load per trip, which is
// what the dependent maximum / sum update compiles to, the pass was bound by memory latency, not bandwidth.
// What has had its last use, and what is written, is marked to leave the cache first: the row has to stay in L2
// between its two reads (8192 x 50257: 677 -> 640 us; the bytes alone take 510).
// Backward: 12 bytes per element (dout is read-modify-write; its second read hits L2 the same way), four pairs of loads
// in flight and the same marks in the write pass, eight loads in the pass before it (973 -> 870 us; 766 for the bytes).
#include "attn_internal.h"
#include "tc05.cuh"

#include "../../include/xent_sm100.h"

namespace xent {
namespace {

constexpr int kThreads = 1024;
constexpr int kBatch = 8;  // independent loads per thread and loop trip

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(kThreads) xent_forward_kernel(const float *__restrict__ logits,
                                                                const float *__restrict__ targets,
                                                                float *__restrict__ logsm, float *__restrict__ loss,
                                                                int rows, int C) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    __shared__ float s_m[kThreads / 32], s_s[kThreads / 32];
    __shared__ float s_shift;
    const int r = blockIdx.x;
    const float *x = logits + (size_t)r * C;
    float *y = logsm + (size_t)r * C;
    // online maximum / sum of exponentials
    float m = -INFINITY, s = 0.f;
    for (int j0 = threadIdx.x; j0 < C; j0 += kThreads * kBatch) {
        float v[kBatch];  // kBatch loads in flight per thread: the pass is bound by HBM latency otherwise
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int j = j0 + u * kThreads;
            v[u] = j < C ? __ldg(x + j) : -INFINITY;
        }
        float bm = v[0];
#pragma unroll
        for (int u = 1; u < kBatch; u++) bm = fmaxf(bm, v[u]);
        if (bm > m) {
            s *= __expf(m - bm);  // exp(-inf) = 0 on the first batch
            m = bm;
        }
        const float low = m == -INFINITY ? 0.f : m;  // a thread that has seen nothing but -inf so far adds nothing
#pragma unroll
        for (int u = 0; u < kBatch; u++) s += __expf(v[u] - low);  // exp(-inf) = 0 past the end of the row
    }
    // combine (m, s) pairs across the warp, then across the block
    const float wm = warp_max(m);
    s = warp_sum(m == -INFINITY ? s : s * __expf(m - wm));  // s is 0, or NaN, where there was nothing but -inf
    if ((threadIdx.x & 31) == 0) {
        s_m[threadIdx.x >> 5] = wm;
        s_s[threadIdx.x >> 5] = s;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const float pm = threadIdx.x < kThreads / 32 ? s_m[threadIdx.x] : -INFINITY;
        const float ps = threadIdx.x < kThreads / 32 ? s_s[threadIdx.x] : 0.f;
        const float bm = warp_max(pm);
        const float bs = warp_sum(pm == -INFINITY ? ps : ps * __expf(pm - bm));
        if (threadIdx.x == 0) s_shift = bm + logf(bs);
    }
    __syncthreads();
    const float shift = s_shift;
    for (int j0 = threadIdx.x; j0 < C; j0 += kThreads * kBatch) {
        float v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int j = j0 + u * kThreads;
            v[u] = j < C ? __ldcs(x + j) : 0.f;  // last use
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int j = j0 + u * kThreads;
            if (j < C) __stcs(y + j, v[u] - shift);
        }
    }
    if (threadIdx.x == 0) {
        const int t = (int)targets[r];
        atomicAdd(loss, -(x[t] - shift) / (float)rows);
    }
}

__global__ void __launch_bounds__(kThreads) xent_backward_kernel(const float *__restrict__ g,
                                                                 const float *__restrict__ targets,
                                                                 const float *__restrict__ logsm, float *__restrict__ dout,
                                                                 int rows, int C) {
    tc05::pdl_launch_dependents();
    tc05::pdl_wait();
    __shared__ float s_part[kThreads / 32];
    __shared__ float s_total;
    const int r = blockIdx.x;
    const float *c = logsm + (size_t)r * C;
    float *d = dout + (size_t)r * C;
    const int t = (int)targets[r];
    const float at_target = -g[r] / (float)rows;
    // sum of the row as it will be once the target entry is set
    float s = 0.f;
    for (int j0 = threadIdx.x; j0 < C; j0 += kThreads * kBatch) {
        float v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int j = j0 + u * kThreads;
            v[u] = j < C ? d[j] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) s += j0 + u * kThreads == t ? at_target : v[u];
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        float p = threadIdx.x < kThreads / 32 ? s_part[threadIdx.x] : 0.f;
        p = warp_sum(p);
        if (threadIdx.x == 0) s_total = p;
    }
    __syncthreads();
    const float total = s_total;
    constexpr int kPairs = 4;  // two loads each
    for (int j0 = threadIdx.x; j0 < C; j0 += kThreads * kPairs) {
        float v[kPairs], e[kPairs];
#pragma unroll
        for (int u = 0; u < kPairs; u++) {
            const int j = j0 + u * kThreads;
            v[u] = j < C ? __ldcs(d + j) : 0.f;
            e[u] = j < C ? __ldcs(c + j) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kPairs; u++) {
            const int j = j0 + u * kThreads;
            if (j < C) __stcs(d + j, (j == t ? at_target : v[u]) - __expf(e[u]) * total);
        }
    }
}

// ---- forward of rows that fit in shared memory ----
//
// One CTA per SM goes through rows of up to kSlots * kSlot values, which the copy engine brings in pieces of 16 KB: a row is
// read once, and while its results leave piece by piece the next rows follow into the places that become free, so that HBM
// always has up to 200 KB of reads from every SM ahead of it (8192 x 50257: 628 -> 544 us, 6.05 TB/s).  The backward the same
// way, its log-probabilities through registers, was no faster than its kernel above (883 and 880 us; rows of 16384 356, 270).
constexpr int kSlot = 4096, kSlots = 13;  // floats of a piece; pieces of the ring: 208 KB
constexpr int kWorkers = 512, kRowThreads = kWorkers + 32;
constexpr int kPerThread = kSlot / 4 / kWorkers;  // 16-byte words of a piece per thread

struct __align__(128) RowSmem {
    float ring[kSlots][kSlot];
    uint64_t full[kSlots], empty[kSlots];
    float m[2][kWorkers / 32], s[2][kWorkers / 32];  // per warp, of this row and of the one before
    int abort_flag, drain_flag;  // a wait has run out; so has the wait for copies on their way at the end
};
enum Site : int { SITE_EMPTY = 251, SITE_FULL, SITE_DRAIN };

// The words of a row that start on 16-byte boundaries, and the up to three values either side of them.
struct Row {
    int head, words;  // values before the first word, words
    __device__ __forceinline__ Row(const float *x, int C) {
        head = min(C, (int)((16 - (reinterpret_cast<uintptr_t>(x) & 15)) & 15) / 4);
        words = (C - head) / 4;
    }
    __device__ __forceinline__ int pieces() const { return (words * 4 + kSlot - 1) / kSlot; }
    // the loose values, one each for the first threads: -1 for the others
    __device__ __forceinline__ int loose(int thread, int C) const {
        const int j = thread < head ? thread : head + 4 * words + thread - head;
        return thread < head || (thread < 6 && j < C) ? j : -1;
    }
};

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(tc05::smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(tc05::smem_u32(bar))
                 : "memory");
}
// A barrier of the workers that tells each of them whether one has given up.  They leave together or not at all: the flag in
// shared memory may change while they look at it, and those that stayed would wait at the next barrier for ever.
__device__ __forceinline__ bool workers_any(bool gave_up) {
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"((uint32_t)gave_up), "n"(kWorkers)
        : "memory");
    return any != 0;
}

__device__ __forceinline__ void init_ring(RowSmem &sm) {
    if (threadIdx.x == 0) {
        sm.abort_flag = sm.drain_flag = 0;
        for (int i = 0; i < kSlots; i++) {
            tc05::mbar_init(&sm.full[i], 1);
            tc05::mbar_init(&sm.empty[i], kWorkers / 32);
        }
        tc05::fence_barrier_init();
    }
    __syncthreads();
}
// The place of a piece in the ring: pieces are counted through all rows of the CTA.
struct Place {
    int slot = 0;
    uint32_t round = 0;
    __device__ __forceinline__ void next() {
        if (++slot == kSlots) slot = 0, round++;
    }
};
// One thread: the pieces of every row of this CTA.  Returns the place behind the last one.
__device__ __forceinline__ Place load_rows(RowSmem &sm, const float *x, int rows, int C, const tc05::WaitCtx &ctx) {
    Place at;
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const float *from = x + (size_t)r * C;
        const Row row(from, C);
        for (int c = 0; c < row.pieces(); c++, at.next()) {
            if (at.round > 0 && !tc05::mbar_wait(&sm.empty[at.slot], (at.round - 1) & 1, ctx, SITE_EMPTY)) return at;
            const uint32_t bytes = min(kSlot, row.words * 4 - c * kSlot) * 4;
            tc05::mbar_expect_tx(&sm.full[at.slot], bytes);
            bulk_load(sm.ring[at.slot], from + row.head + c * kSlot, bytes, &sm.full[at.slot]);
        }
    }
    return at;
}
// The same thread, last: nothing is on its way into shared memory that the CTA gives back, also where the workers have left.
__device__ __forceinline__ void drain(RowSmem &sm, const Place &end, const tc05::WaitCtx &ctx) {
    const tc05::WaitCtx last{&sm.drain_flag, ctx.status, ctx.limit_ns};
    for (int i = 0; i < kSlots; i++) {
        const uint32_t pieces = end.round + (i < end.slot);  // that this place has been given
        if (pieces > 0) tc05::mbar_wait(&sm.full[i], (pieces - 1) & 1, last, SITE_DRAIN);
    }
}
// After a warp's last look at a piece: the copy engine may overwrite it.
__device__ __forceinline__ void release(RowSmem &sm, int c) {
    tc05::fence_proxy_async_smem();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) tc05::mbar_arrive(&sm.empty[c]);
}

__global__ void __launch_bounds__(kRowThreads, 1) xent_forward_rows_kernel(const float *__restrict__ logits, const float *__restrict__ targets,
                                                                         float *__restrict__ logsm, float *__restrict__ loss, int rows,
                                                                         int C, int loaded, uint64_t limit_ns, int *status) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    RowSmem &sm = *reinterpret_cast<RowSmem *>(smem_raw);
    tc05::pdl_launch_dependents();
    init_ring(sm);
    tc05::pdl_wait();
    tc05::WaitCtx ctx{&sm.abort_flag, status, limit_ns};
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid >= kWorkers) {
        if (tid == kWorkers) drain(sm, load_rows(sm, logits, loaded, C, ctx), ctx);
        return;
    }
    Place first;
    for (int r = blockIdx.x, n = 0; r < rows; r += gridDim.x, n++) {
        const float *x = logits + (size_t)r * C;
        float *y = logsm + (size_t)r * C;
        const Row row(x, C);
        const int loose = row.loose(tid, C), pieces = row.pieces();
        const float mine = loose >= 0 ? x[loose] : -INFINITY, at_target = tid == 0 ? x[(int)targets[r]] : 0.f;
        // maximum so far and four sums of exponentials; what is below the maximum of nothing (all -inf) adds nothing
        float m = mine, s0 = loose >= 0 && mine != -INFINITY ? __expf(mine - m) : 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        Place at = first;
        bool arrived = true;
        for (int c = 0; c < pieces; c++, at.next()) {
            arrived = tc05::mbar_wait_warp(&sm.full[at.slot], at.round & 1, ctx, SITE_FULL);
            if (!arrived) break;
            const int words = min(kSlot / 4, row.words - c * (kSlot / 4));
            const float4 *from = reinterpret_cast<const float4 *>(sm.ring[at.slot]);
            float4 v[kPerThread];
            float bm = -INFINITY;
#pragma unroll
            for (int u = 0; u < kPerThread; u++) {
                const int i = tid + u * kWorkers;
                v[u] = i < words ? from[i] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
                bm = fmaxf(fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)), bm);
            }
            if (bm > m) {
                const float f = __expf(m - bm);  // exp(-inf) = 0 on the first piece
                s0 *= f, s1 *= f, s2 *= f, s3 *= f;
                m = bm;
            }
            const float low = m == -INFINITY ? 0.f : m;
#pragma unroll
            for (int u = 0; u < kPerThread; u++)
                s0 += __expf(v[u].x - low), s1 += __expf(v[u].y - low), s2 += __expf(v[u].z - low), s3 += __expf(v[u].w - low);
        }
        float s = (s0 + s1) + (s2 + s3);
        const float wm = warp_max(m);
        s = warp_sum(m == -INFINITY ? s : s * __expf(m - wm));  // as in the kernel above
        if (lane == 0) sm.m[n & 1][warp] = wm, sm.s[n & 1][warp] = s;
        if (workers_any(!arrived)) return;
        const float pm = lane < kWorkers / 32 ? sm.m[n & 1][lane] : -INFINITY, ps = lane < kWorkers / 32 ? sm.s[n & 1][lane] : 0.f;
        const float top = warp_max(pm);
        const float shift = top + logf(warp_sum(pm == -INFINITY ? ps : ps * __expf(pm - top)));
        const bool whole = ((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(y)) & 15) == 0;
        at = first;
        for (int c = 0; c < pieces; c++, at.next()) {
            const int words = min(kSlot / 4, row.words - c * (kSlot / 4));
            const float4 *from = reinterpret_cast<const float4 *>(sm.ring[at.slot]);
            float *to = y + row.head + c * kSlot;
#pragma unroll
            for (int u = 0; u < kPerThread; u++) {
                const int i = tid + u * kWorkers;
                if (i >= words) continue;
                const float4 v = from[i];
                const float4 o = make_float4(v.x - shift, v.y - shift, v.z - shift, v.w - shift);
                if (whole) __stcs(reinterpret_cast<float4 *>(to) + i, o);
                else __stcs(to + 4 * i, o.x), __stcs(to + 4 * i + 1, o.y), __stcs(to + 4 * i + 2, o.z), __stcs(to + 4 * i + 3, o.w);
            }
            release(sm, at.slot);
        }
        first = at;
        if (loose >= 0) y[loose] = mine - shift;
        if (tid == 0) atomicAdd(loss, -(at_target - shift) / (float)rows);
    }
}

// Shorter rows gain nothing, several of whose blocks share an SM (8192 rows of 16384: 197 us there, 206 here, 24576: 271, 279,
// 32000: 367, 351, 50257: 628, 544; 1 row of 50257: 9.8, 9.9, 37 rows: 12.1, 10.5).
bool row_fits(int C) { return C >= 30000 && C <= kSlot * kSlots; }
// Nor do more rows than SMs, up to two for each, which the kernel above takes all at once and this one in two turns, unless their
// addresses modulo 16 differ (214 rows of 30000: 13.6 us there, 15.6 here, 34000: 16.1, 17.1, 36001: 18.3, 17.7, 50257: 25.1, 24.0).
bool in_two_turns(int rows, int C) { return C % 4 == 0 && rows > attn::sm_count() && rows <= 2 * attn::sm_count(); }

// `loaded` rows are fetched: all of them, or in the test of what happens when one never arrives fewer.
int launch_rows(const float *logits, const float *targets, float *logsm, float *loss, int rows, int C, cudaStream_t s, int loaded,
                uint64_t limit_ns = 0) {
    static bool ready[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64 || !ready[dev]) {
        e = cudaFuncSetAttribute(xent_forward_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RowSmem));
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) ready[dev] = true;
    }
    int *status = nullptr;
    const int rc = attn::device_status_word(&status);
    if (rc != ATTN_OK) return rc;
    const int sms = attn::sm_count();
    return (int)attn::launch_after_previous(xent_forward_rows_kernel, dim3(rows < sms ? rows : sms), dim3(kRowThreads), sizeof(RowSmem), s,
                                            logits, targets, logsm, loss, rows, C, loaded, limit_ns, status);
}

}  // namespace
}  // namespace xent

extern "C" {

int xent_sm100_forward(const float *logits, const float *targets, float *logsm, float *loss, int rows, int C, void *stream) {
    if (!logits || !targets || !logsm || !loss) return ATTN_ERR_NULL;
    if (rows <= 0 || C <= 0) return ATTN_ERR_SHAPE;
    if (xent::row_fits(C) && !xent::in_two_turns(rows, C))
        return xent::launch_rows(logits, targets, logsm, loss, rows, C, static_cast<cudaStream_t>(stream), rows);
    return (int)attn::launch_after_previous(xent::xent_forward_kernel, dim3(rows), dim3(xent::kThreads), 0,
                                            static_cast<cudaStream_t>(stream), logits, targets, logsm, loss, rows, C);
}

int xent_sm100_selftest_wait_limit(const float *logits, const float *targets, float *logsm, float *loss, int rows, int C, int loaded,
                                   unsigned limit_us, void *stream) {
    if (!logits || !targets || !logsm || !loss) return ATTN_ERR_NULL;
    if (rows <= 0 || !xent::row_fits(C) || loaded < 0 || loaded > rows || limit_us == 0 || limit_us > 100000u) return ATTN_ERR_SHAPE;
    return xent::launch_rows(logits, targets, logsm, loss, rows, C, static_cast<cudaStream_t>(stream), loaded, limit_us * 1000ull);
}

int xent_sm100_backward(const float *g, const float *targets, const float *logsm, float *dout, int rows, int C, void *stream) {
    if (!g || !targets || !logsm || !dout) return ATTN_ERR_NULL;
    if (rows <= 0 || C <= 0) return ATTN_ERR_SHAPE;
    return (int)attn::launch_after_previous(xent::xent_backward_kernel, dim3(rows), dim3(xent::kThreads), 0,
                                            static_cast<cudaStream_t>(stream), g, targets, logsm, dout, rows, C);
}

}  // extern "C"
