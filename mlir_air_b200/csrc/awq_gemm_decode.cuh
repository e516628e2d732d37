// Pieces shared by the batched-decode GEMM kernels (awq_gemm_decode.cu: 16-bit operands; awq_gemm_decode_f8.cu: the
// packed nibbles and split token rows as fp8 operands): the stream-K walk over (tile, k-block) units, the slots the
// partial sums go through, and the second pass that adds them up.
#pragma once

#include <cudaTypedefs.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "awq_common.cuh"

namespace awq {

int encode_tensor_map_2d(CUtensorMap *map, int dtype, const void *base, uint64_t dim0, uint64_t dim1,
                         uint64_t stride1_bytes, uint32_t box0, uint32_t box1, int swizzle);
int encode_tensor_map_3d(CUtensorMap *map, int dtype, const void *base, uint64_t dim0, uint64_t dim1, uint64_t dim2,
                         uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t box0, uint32_t box1, uint32_t box2,
                         int swizzle);

constexpr int DG_BN = 256, DG_BK = 64, DG_GROUP = 128;
constexpr int DG_W_BYTES = DG_GROUP * (DG_BN / 8) * 4;  // 16 KB of packed words: a unit (128 k, one quantisation group)
constexpr int DG_S_BYTES = DG_BN * 2;
constexpr int DG_Z_BYTES = DG_BN / 8 * 4;
constexpr int DG_MAX_TILES = 4096;

// The walk over a CTA's units, the same for every warp role: unit u = tile * KB + kb (KB units of 128 k per tile),
// range [u0, u1).
struct UnitWalk {
    int KB, u, u1;
    __device__ __forceinline__ UnitWalk(int tiles, int kb_count) : KB(kb_count) {
        const long long U = (long long)tiles * kb_count, C = gridDim.x, c = blockIdx.x;
        u = (int)(c * U / C);
        u1 = (int)((c + 1) * U / C);
    }
    __device__ __forceinline__ bool valid() const { return u < u1; }
    __device__ __forceinline__ int tile() const { return u / KB; }
    __device__ __forceinline__ int kb() const { return u - tile() * KB; }
    // units of the current tile that this CTA still has, from u on
    __device__ __forceinline__ int left_in_tile() const {
        const int end = (tile() + 1) * KB;
        return (end < u1 ? end : u1) - u;
    }
};

// The first CTA whose range (UnitWalk) reaches into tile t.
__device__ __forceinline__ int dg_first_cta(int t, int KB, int tiles) {
    const long long U = (long long)tiles * KB, C = gridDim.x;
    return (int)((((long long)t * KB + 1) * C + U - 1) / U) - 1;
}
// Partial sums of a tile in the workspace: slot [contributor][token row m][column of the tile], so that the 32 lanes
// of a warp (columns) touch one 128-byte line.
template <int NB>
__device__ __forceinline__ float *dg_slot_word(float *slots, int slots_per_tile, int tile, int contributor, int m, int col) {
    return slots + (((size_t)tile * slots_per_tile + contributor) * NB + m) * DG_BN + col;
}

// ---- token rows split into two e4m3 pieces, with a power of two per (row, quantisation group) ----------------------
// x 2^p = hi + lo / 16, where 2^p brings the group's largest magnitude into [128, 256).  One block per group, as it is to lie in
// shared memory, so that one untiled copy brings it:
//   [2 rows][128] bytes: row m = hi pieces of token m, row rows + m = its lo pieces; k permuted inside 32-k steps, 128-byte swizzle
//   [2 rows] f32: sums over the group of hi + lo / 16, then the powers of two that undo the scaling
// `rows` is the batch rounded up to what the MMA sees; the rows past the batch are never written, and whatever they hold
// reaches only sums that nobody reads.
struct SplitRows {
    uint8_t *blocks;
    int rows;
};
__host__ __device__ __forceinline__ size_t split_block_bytes(int rows) { return (size_t)2 * rows * (DG_GROUP + 4); }
// Values k and k + 1 (k even) of group g of token row m; `mx` = bits of the group's largest magnitude.  Returns their part of
// the group sum.  Element k = 8 i + 2 t + b of a 32-k step goes to byte 8 t + 2 i + b: the order in which the kernel's regroup
// warps produce the weights.
__device__ __forceinline__ int split_exponent(uint32_t mx) { return max((int)(mx >> 23), 27); }  // (a group of tiny values: keep 2^p finite)
__device__ __forceinline__ float split_pair(const SplitRows &o, int m, int g, int k, float a, float b, uint32_t mx) {
    const float scale = __uint_as_float((uint32_t)(261 - split_exponent(mx)) << 23);
    a *= scale, b *= scale;
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    const float2 hf = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(hi, __NV_E4M3)));
    const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(16.f * (a - hf.x), 16.f * (b - hf.y)), __NV_SATFINITE, __NV_E4M3);
    const float2 lf = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(lo, __NV_E4M3)));
    const int at = (k & ~31) + 8 * ((k & 7) >> 1) + 2 * ((k & 31) >> 3);  // byte inside the row, before the swizzle
    uint8_t *row = o.blocks + (size_t)g * split_block_bytes(o.rows) + (size_t)m * DG_GROUP + (at ^ ((m & 7) << 4));
    *reinterpret_cast<__nv_fp8x2_storage_t *>(row) = hi;
    *reinterpret_cast<__nv_fp8x2_storage_t *>(row + (size_t)o.rows * DG_GROUP) = lo;  // (rows is a multiple of 8: the same swizzle)
    return (hf.x + 0.0625f * lf.x) + (hf.y + 0.0625f * lf.y);
}
__device__ __forceinline__ void split_finish(const SplitRows &o, int m, int g, float sum, uint32_t mx) {
    float *w = reinterpret_cast<float *>(o.blocks + (size_t)g * split_block_bytes(o.rows) + (size_t)2 * o.rows * DG_GROUP) + m;
    w[0] = sum;
    // an infinity or a NaN in the group shows in everything that it is multiplied into
    w[o.rows] = mx >= 0x7F800000u ? __uint_as_float(0x7F800000u) : __uint_as_float((uint32_t)(split_exponent(mx) - 7) << 23);
}

int dg_rows(int M);       // token rows the MMA sees: the batch rounded up to 16, 32 or 64
int dg_sm_count();
int dg_slots_per_tile(int tiles);
// The second pass over the slots of a main kernel of `main_ctas` CTAs: sums (* row_scale[m] if given), then the epilogue.
// `split` (SwiGLU only): the outputs are written as split rows instead of to C.
int launch_gemm_decode_fixup(int rows, uint16_t *C, const uint16_t *residual, int epilogue, int c_f16, const float *row_scale, int M,
                             int N, int KB, int tiles, int main_ctas, const float *slots, int slots_per_tile, cudaStream_t stream,
                             const SplitRows *split = nullptr);

}  // namespace awq
