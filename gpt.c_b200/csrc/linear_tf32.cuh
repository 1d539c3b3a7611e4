// What the two Linear kernels share: TF32 tensor-core instructions, operand descriptors and tensor maps.
#pragma once

#include "attn_internal.h"
#include "tc05.cuh"

namespace lin {

constexpr int kBM = 128, kBK = 32;
constexpr int kATileBytes = kBM * kBK * 4;  // A tile of one stage: 16 KiB

// Instruction descriptor for kind::tf32 (A and B formats = 2), fp32 accumulation.
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N, int a_mn_major, int b_mn_major) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32_lead(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                              uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t"
        "}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}

// Shared-memory descriptor for 32-bit operands read MN-major: layout type 1 (128-byte swizzle with
// 32-byte atoms); rows of 32 values along M/N, LBO = distance between 32-value blocks, SBO = distance
// between groups of 4 contraction steps.
__device__ __forceinline__ uint64_t smem_desc_sw128_base32(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)1 << 61;
    return d;
}

// Writes 4 * kQuads consecutive 32-bit words to dst, as far as `left` words go (a multiple of
// 4): 32 bytes per store where dst allows it, else 16.
template <int kQuads>
__device__ __forceinline__ void store_words(void *dst, int left, int wide, const uint32_t *r) {
    uint32_t *d = static_cast<uint32_t *>(dst);
    if (wide) {
#pragma unroll
        for (int q = 0; q < kQuads / 2; q++)
            if (8 * q < left)
                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(d + 8 * q), "r"(r[8 * q]),
                             "r"(r[8 * q + 1]), "r"(r[8 * q + 2]), "r"(r[8 * q + 3]), "r"(r[8 * q + 4]), "r"(r[8 * q + 5]),
                             "r"(r[8 * q + 6]), "r"(r[8 * q + 7])
                             : "memory");
    } else {
#pragma unroll
        for (int q = 0; q < kQuads; q++)
            if (4 * q < left) *reinterpret_cast<uint4 *>(d + 4 * q) = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
    }
}

// The 32 columns of a row that every lane holds leave from registers: a pair of lanes (odd: the second one) holds two rows and
// exchanges halves, so that both have 16 columns of either row, r[0..15] of the even lane's and r[16..31] of the odd one's,
// and a store instruction touches 16 rows instead of 32.  L2 takes 32-byte pieces of a line one by one at 4.0 TB/s, pieces of
// 64 bytes and more at 5.3 (forward of K = 32, 8192 x 3072: 28 -> 22 us).
__device__ __forceinline__ void exchange_halves(int odd, uint32_t (&r)[32]) {
#pragma unroll
    for (int e = 0; e < 16; e++) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? r[e] : r[16 + e], 1);
        r[e] = odd ? other : r[e];
        r[16 + e] = odd ? r[16 + e] : other;
    }
}

// ---- host side ----

// Operand read K-major: matrix [rows, kc] row-major (kc contiguous = contraction); boxes of 32 x box_rows.
// `pitch`: floats from one row to the next (0: kc).
inline int map_k_major(CUtensorMap *map, const float *base, int rows, int kc, int box_rows, size_t pitch = 0,
                       CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_NONE) {
    if (pitch == 0) pitch = (size_t)kc;
    const cuuint64_t dims[4] = {(cuuint64_t)kc, (cuuint64_t)rows, 1, 1};
    const cuuint64_t strides[3] = {(cuuint64_t)pitch * 4, (cuuint64_t)pitch * 4 * (cuuint64_t)rows, (cuuint64_t)pitch * 4 * (cuuint64_t)rows};
    const cuuint32_t box[4] = {32, (cuuint32_t)box_rows, 1, 1};
    return attn::encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, promotion);
}
// Operand read MN-major, whole tile in one copy: the matrix [kc, rows] seen as {32 values, kc, rows / 32 blocks}
// with the block index as the slowest box dimension, box {32, 32, nblocks}: shared memory receives
// [block][contraction step][32 values], the layout the descriptor expects.  rows % 32 == 0.
inline int map_mn_major_blocks(CUtensorMap *map, const float *base, int kc, int rows, int nblocks, size_t pitch = 0) {
    if (pitch == 0) pitch = (size_t)rows;
    const cuuint64_t dims[4] = {32, (cuuint64_t)kc, (cuuint64_t)(rows / 32), 1};
    const cuuint64_t strides[3] = {(cuuint64_t)pitch * 4, 128, (cuuint64_t)pitch * 4 * (cuuint64_t)kc};
    const cuuint32_t box[4] = {32, 32, (cuuint32_t)nblocks, 1};
    return attn::encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box,
                              CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B);
}
// Operand read MN-major: matrix [kc, rows] row-major (rows contiguous, kc = contraction), boxes of 32 x 32.
inline int map_mn_major(CUtensorMap *map, const float *base, int kc, int rows, size_t pitch = 0) {
    if (pitch == 0) pitch = (size_t)rows;
    const cuuint64_t dims[4] = {(cuuint64_t)rows, (cuuint64_t)kc, 1, 1};
    const cuuint64_t strides[3] = {(cuuint64_t)pitch * 4, (cuuint64_t)pitch * 4 * (cuuint64_t)kc, (cuuint64_t)pitch * 4 * (cuuint64_t)kc};
    const cuuint32_t box[4] = {32, 32, 1, 1};
    // 32-bit operands read MN-major need the 128-byte swizzle with 32-byte atoms (rows of 128 bytes, the
    // 32-byte quarter of a row XORed with the row index modulo 4)
    return attn::encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box,
                              CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B);
}
inline int map_out_f32(CUtensorMap *map, const float *base, int rows, int cols, size_t pitch = 0) {
    if (pitch == 0) pitch = (size_t)cols;
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 1};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * 4, (cuuint64_t)pitch * 4 * (cuuint64_t)rows};
    const cuuint32_t box[3] = {32, 32, 1};
    return attn::encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box);
}
// Pieces of the contraction of dx: added to zeros in memory, in no fixed order; added up by one CTA, which takes them in turn; left
// apart, one matrix behind the other.
enum DxPieces : int { kDxAdded, kDxInTurn, kDxApart };
// All of a backward in one launch (linear_backward_sm100.cu), or dW and db alone (dx NULL), or dx alone (dw and db NULL).  What is cut how, and the time in
// nanoseconds it is expected to take.
struct BackwardPlan {
    int tiles_n;                 // column tiles of both results
    int dx_tiles, dx_kb, dw_kb;  // tiles of dx (of all its pieces); contraction blocks of a tile of dx, of dW
    int classes, dx_pieces;      // views of dy; pieces of the contraction of dx,
    DxPieces dx_how;             // and what becomes of them
    int team, down;              // CTAs that work on neighbouring tiles of dW, below (1) or beside each other
    int rounds, strips;          // groups of such tiles that a team takes whole; groups that are cut
    int teams, fewer, even;      // even: whole pieces of the same size, one per team
    int dw_most;                 // contraction blocks of dW that go through one accumulator
    double share_fewer, share;   // how much of dW the first `fewer` teams take, and the others
    int ns;
};
BackwardPlan plan_backward(int M, int N, int K, bool want_dx, bool want_dw, int sms, int classes = 1, int dx_pieces = 1, DxPieces how = kDxAdded);
// Contraction blocks of dW: the most that one CTA takes, and the most that one accumulator sums up.
struct DwLoad {
    int cta, sum;
};
DwLoad dw_load(const BackwardPlan &plan, int M, int N, int K);
// dy [M, np] with zeros from column N on, w [w_rows, K].
int launch_backward(const BackwardPlan &plan, const float *dy, const float *x, const float *w, int w_rows, float *dx, float *dw, float *db,
                    int M, int N, int np, int K, int *status, cudaStream_t s);
// The same from views of every fourth row of dy [M, N] (plan.classes = 4).  With several pieces that are added dx has to be zero, with pieces
// apart it has room for them all.
int launch_backward_by_row_class(const BackwardPlan &plan, const float *dy, const float *x, const float *w, float *dx, float *dw, float *db,
                                 int M, int N, int K, int *status, cudaStream_t s);
// The kernel for results of few tiles (linear_split_sm100.cu): out[M, cols] = act[M, kc] . w^T + bias, with w [cols, kc],
// or with w_mn_major [w_rows, cols] (its rows past w_rows, up to kc, read as zeros); optionally the bf16 planes of out.
// `split` CTAs share the contraction of a tile.  Returns ATTN_OK or an error.
int launch_split(const float *act, const float *w, bool w_mn_major, int w_rows, const float *bias, float *out, void *planes, int M,
                 int cols, int kc, int split, int sms, int *status, cudaStream_t s);
// The best `split` and the time in nanoseconds it is expected to take.
int plan_split(int M, int cols, int kc, int sms, int *split);

}  // namespace lin
