// Shared pieces of the attention / memory kernels: tile geometry (128-token chunks, head_dim 64),
// the 128-byte-swizzled shared-memory tile layout that both TMA and tcgen05 descriptors use, and
// row-per-thread helpers (RoPE with interleaved pairs restarting every chunk, tanh).
#pragma once
#include "ws_ptx.cuh"
#include "ws_tma_host.h"

namespace ws {

constexpr int CHUNK = 128;
constexpr int HD = 64;
constexpr int TILE_BYTES = CHUNK * HD * 2;  // one [128 x 64] BF16 tile, 16 KiB

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}
__device__ __forceinline__ float sigmoid_f(float x) { return sigmoid_fast(x); }

// The arithmetic that two forms of a kernel must share bit for bit is written with explicitly rounded operations,
// so that the compiler's choice of which product to fuse into which addition cannot differ between them.
__device__ __forceinline__ float2 rope_rotate(float2 x, float2 cs) {  // (cos, sin) of the pair's angle
  return make_float2(__fmaf_rn(x.x, cs.x, -__fmul_rn(x.y, cs.y)), __fmaf_rn(x.y, cs.x, __fmul_rn(x.x, cs.y)));
}
// exp2((s - m) * k): the unnormalised softmax weight of a score
__device__ __forceinline__ float softmax_term(float s, float m, float k) { return exp2f(__fmul_rn(__fsub_rn(s, m), k)); }
// g * (o * inv_l) + (1 - g) * (mem / 8)
__device__ __forceinline__ float gate_blend(float g, float o, float inv_l, float mem) {
  return __fmaf_rn(g, __fmul_rn(o, inv_l), __fmul_rn(__fsub_rn(1.f, g), __fmul_rn(mem, 0.125f)));
}

// Address of the 16-byte chunk `j` (8 BF16 columns) of row `r` in a [rows x 64] swizzled tile.
__device__ __forceinline__ uint8_t* tile_chunk(uint8_t* tile, int r, int j) {
  return tile + r * 128 + ((j ^ (r & 7)) << 4);
}

// In place on row `r` of a tile: optional rotary embedding at in-chunk position r (pairs are
// adjacent elements; rope[p*128 + r] = (cos, sin) of pair p at position r -- pair-major, so that
// the 32 rows of a warp read 256 contiguous bytes instead of 32 cache lines), then optional tanh;
// of the row's eight 16-byte pieces only `count` from `first` on.
__device__ __forceinline__ void rope_tanh_row(uint8_t* tile, int r, const float2* __restrict__ rope,
                                              bool do_rope, bool do_tanh, int first = 0, int count = 8) {
#pragma unroll
  for (int i = 0; i < count; ++i) {
    const int j = first + i;
    uint4* p = reinterpret_cast<uint4*>(tile_chunk(tile, r, j));
    uint4 v = *p;
    uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w[t]));
      if (do_rope) x = rope_rotate(x, rope[(j * 4 + t) * CHUNK + r]);
      if (do_tanh) {
        x.x = tanh_fast(x.x);
        x.y = tanh_fast(x.y);
      }
      w[t] = pack_bf16x2(x.x, x.y);
    }
    *p = v;
  }
}

// Store 32 BF16 values (16 packed words) of row r, columns [c0, c0+32), into a [128 x 128]
// K-major operand made of two swizzled [128 x 64] tiles (columns 0-63 | 64-127).
__device__ __forceinline__ void store_row_chunk32(uint8_t* tiles, int r, int c0, const uint32_t (&pk)[16]) {
  uint8_t* tile = tiles + (c0 >> 6) * TILE_BYTES;
  const int j0 = (c0 & 63) >> 3;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<uint4*>(tile_chunk(tile, r, j0 + q)) = make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
}
__device__ __forceinline__ void load_row_chunk32(uint8_t* tiles, int r, int c0, uint32_t (&pk)[16]) {
  uint8_t* tile = tiles + (c0 >> 6) * TILE_BYTES;
  const int j0 = (c0 & 63) >> 3;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile_chunk(tile, r, j0 + q));
    pk[4 * q] = v.x; pk[4 * q + 1] = v.y; pk[4 * q + 2] = v.z; pk[4 * q + 3] = v.w;
  }
}

// Host: 2-D map over a row-major BF16 matrix for [box_rows x box_cols] swizzled tiles.
inline int make_tile_map(CUtensorMap* map, const void* base, uint64_t cols, uint64_t rows, uint64_t ld,
                         uint32_t box_cols, uint32_t box_rows) {
  return make_map_bf16(map, base, cols, rows, ld, box_cols, box_rows);
}

// Host: 3-D map (column, position, sequence) over a token-major BF16 matrix [sequences * length, cols], for swizzled
// tiles of one sequence: a box that reaches past the sequence's last position is filled with zeros on a load and
// clipped on a store, instead of running into the next sequence.
inline int make_sequence_map(CUtensorMap* map, const void* base, uint64_t cols, uint64_t length, uint64_t sequences,
                             uint32_t box_cols, uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return -10;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (cols * 2) % 16 != 0) return -11;
  cuuint64_t dims[3] = {cols, length, sequences};
  cuuint64_t strides[2] = {cols * 2, length * cols * 2};
  cuuint32_t box[3] = {box_cols, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -12;
}

// out[q][h] = sigmoid'(logit_q[h]) * sum over the head's B * 16 partials of the reverse scan: one warp, fixed order.
__device__ __forceinline__ void logit_grad(const float* partials, const float* fast_logit, const float* slow_logit, const float* mix_logit,
                                           int B, int H, int h, int q, float* out) {
  const int lane = threadIdx.x & 31;
  float v = 0.f;
  for (int i = lane; i < B * 16; i += 32)
    v += partials[((static_cast<size_t>(i >> 4) * H + h) * 16 + (i & 15)) * 3 + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) {
    const float* logit = q == 0 ? fast_logit : q == 1 ? slow_logit : mix_logit;
    const float s = 1.f / (1.f + expf(-logit[h]));
    out[q * H + h] = v * s * (1.f - s);
  }
}

}  // namespace ws
