// Internal launch interface between the C-ABI shim (attn_api.cu) and the kernel files.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>

namespace attn {

// SMs of the current device (1 when that cannot be found out: the launch that follows reports why).
inline int sm_count() {
    static std::atomic<int> known[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    const bool slot = dev >= 0 && dev < 64;
    if (slot && (sms = known[dev].load(std::memory_order_relaxed)) > 0) return sms;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1;
    if (slot) known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

constexpr int kShortT = 128;  // one query and key tile: the kernels that read the fp32 tensors themselves
constexpr int kAttn24MaxD = 128;  // general kernels on the tensor cores; above, fp32 arithmetic
constexpr int kGenericMaxD = 256;
constexpr int kGenericMaxT = 8192;

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// One bf16 plane of n elements, padded so the next plane starts 256-byte aligned.
inline size_t plane_bytes(size_t n) { return align_up(n * sizeof(__nv_bfloat16), 256); }

// fp32 -> (hi, lo) bf16 planes, hi = bf16(x), lo = bf16(x - hi).
cudaError_t launch_split(const float *x, __nv_bfloat16 *hi, __nv_bfloat16 *lo, size_t n, cudaStream_t s);

// rowsum(dout * out) per (b, h, t) -> delta [B, H, T], and zero-fill of the dq third of dqkv ([B, T, 3C]), or of all of it;
// also splits dout into bf16 planes when dhi/dlo are given and zeroes the two ints at `sched` (the item counter
// of the tensor-core backward kernel) when that is given.
cudaError_t launch_bwd_prepare(const float *dout, const float *out, float *delta, __nv_bfloat16 *dhi,
                               __nv_bfloat16 *dlo, float *dqkv, bool zero_all, int *sched, int B, int T, int H, int D, cudaStream_t s);

// General-shape SIMT kernels (kAttn24MaxD < D <= kGenericMaxD, T <= kGenericMaxT).
cudaError_t generic_set_attributes();
cudaError_t launch_generic_forward(const float *qkv, float *out, float *out_copy, float *lse, int B, int T, int H,
                                   int D, cudaStream_t s);
cudaError_t launch_generic_backward(const __nv_bfloat16 *xhi, const __nv_bfloat16 *xlo, const float *lse,
                                    const float *delta, const float *dout, float *dqkv, int B, int T, int H, int D,
                                    cudaStream_t s);

// The general kernels on the tensor cores (D <= kAttn24MaxD, T <= kGenericMaxT), fp32 operands as three bf16 terms.
// fp32 [B, T, heads, D] (D a multiple of 4) as a 4-D map {D, heads, T, B} with boxes of `cols` columns of one head by `rows`
// tokens; columns past the D-th read as zeros and are not written.
int attn24_heads_map(CUtensorMap *map, const void *base, int B, int T, int heads, int D, int cols, int rows, CUtensorMapSwizzle swizzle);
// The bf16 planes at `saved` (D a multiple of 8) as a 5-D map {D, 3 H, T, B, plane}, boxes of 64 columns by 64 tokens.
int attn24_planes_map(CUtensorMap *map, const void *saved, int B, int T, int H, int D);
cudaError_t attn24_fwd_set_attributes();
cudaError_t attn24_bwd_set_attributes();
// hi, lo: receive the planes that launch_split would write (NULL: they are there already)
cudaError_t launch_attn24_forward(const float *qkv, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *out, float *out_copy, float *lse, int B,
                                  int T, int H, int D, int *status, cudaStream_t s);
// map_x: attn24_planes_map where D is a multiple of 8, else not looked at
cudaError_t launch_attn24_backward(const CUtensorMap &map_x, const __nv_bfloat16 *xhi, const __nv_bfloat16 *xlo, const float *lse, const float *delta,
                                   const float *dout, float *dqkv, int pieces, int B, int T, int H, int D, int *status, cudaStream_t s);
// Into how many pieces (1 or 2, D a multiple of 4 only) the queries of a key tile are best cut: with 2 dk and dv are added to
// memory, which has to be zero.
int attn24_backward_pieces(int B, int T, int H, int sms);

// Tensor-core (tcgen05) kernels, D == 64.  The tensor maps cover the bf16 hi/lo planes:
//   map_x : dims {3C, T, B, 2 planes}, box {64, 64, 1, 1}, 128-byte swizzle
//   map_do: dims { C, T, B, 2 planes}, same box
cudaError_t fast_fwd_set_attributes();
cudaError_t fast_bwd_set_attributes();
// map_o, map_copy (used only if out_copy is not null): out and out_copy, dims {C, T, B}, box {32, 128, 1}, 128-byte swizzle.
cudaError_t launch_fast_forward(const CUtensorMap &map_x, const CUtensorMap &map_o, const CUtensorMap &map_copy, float *out,
                                float *out_copy, float *lse, int B, int T, int H, int *status, cudaStream_t s);
// T <= kShortT / 2 only: splits qkv itself (hi, lo receive the planes), in place of launch_split and launch_fast_forward.
cudaError_t launch_fast_forward_fp32(const float *qkv, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *out, float *out_copy, float *lse,
                                     int B, int T, int H, int *status, cudaStream_t s);
// T <= kShortT and B * H <= num_sms only: prepares dout itself (everything launch_bwd_prepare leaves in the scratch
// buffer is written too), in place of launch_bwd_prepare and launch_fast_backward.
cudaError_t launch_fast_backward_fp32(const CUtensorMap &map_x, const CUtensorMap &map_dx, const float *dout, const float *out,
                                      const float *lse, float *delta, __nv_bfloat16 *dhi, __nv_bfloat16 *dlo, float *dqkv, int B,
                                      int T, int H, int *sched, int *status, cudaStream_t s);
cudaError_t launch_fast_backward(const CUtensorMap &map_x, const CUtensorMap &map_do, const CUtensorMap &map_dx,
                                 const float *lse, const float *delta, float *dqkv, int B, int T, int H, int num_sms,
                                 int *sched, int *status, cudaStream_t s);

// Launches `kernel` so that it may begin (up to its pdl_wait(), tc05.cuh) while the previous kernel of the
// stream is still running: its launch latency and set-up overlap that kernel's tail.
// cluster > 1: in clusters of that many CTAs along x.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_clusters_after_previous(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, unsigned cluster,
                                                  cudaStream_t s, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_after_previous(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                         Args &&...args) {
    return launch_clusters_after_previous(kernel, grid, block, smem, 1, s, static_cast<Args &&>(args)...);
}

// Helpers shared with the Linear kernels (linear_sm100.cu).
// cuTensorMapEncodeTiled with the given swizzle, no interleave, no L2 promotion, zero fill; the encoder
// is resolved by attn_sm100_init.  Returns 0 or a cudaError_t.
int encode_tiled(CUtensorMap *map, CUtensorMapDataType dtype, unsigned rank, const void *base, const cuuint64_t *dims,
                 const cuuint64_t *strides, const cuuint32_t *box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B,
                 CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_NONE);
// Status word of the current device (initialises the library on first use).  Returns ATTN_OK or an error.
int device_status_word(int **status);

}  // namespace attn
