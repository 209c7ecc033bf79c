// Bandwidth-bound row kernels: RMSNorm forward / backward (with the depth modulation of the
// residual stream folded in), casts, column sums and the embedding gather / scatter.
//
// One warp owns one row (few rows of a forward norm: a block owns one); a lane owns columns {lane*4 + 128*i}.  Row statistics
// are FP32 (the reference norm, warpstate/model.py:22-28; its Triton twin ops/activation_execution.py:96-158).
// Weight-gradient column sums are accumulated per lane in registers, reduced across the warps
// of a block in shared memory and written as one partial row per block; a second kernel adds the
// partial rows in a fixed order, so the result does not depend on scheduling.
#include "ws_ptx.cuh"
#include "ws_api.h"
#include "attention_common.cuh"
#include "ws_launch.h"

#include <utility>

namespace ws {

extern "C" void ws_count_launch(void);

constexpr int ROW_WARPS = 8;
constexpr int ROW_THREADS = ROW_WARPS * 32;
constexpr int MAX_CHUNKS = 16;  // d <= 2048 for the register-accumulating backward

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// A parameter vector, which no kernel that is launched as a dependent writes: through the read-only path, whose loads pass
// stores.  The statement is volatile, so that the compiler leaves it behind the wait all the same.
__device__ __forceinline__ float4 ld4_parameter(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(__nv_bfloat16* p, float4 v) {
  uint2 o;
  o.x = pack_bf16x2(v.x, v.y);
  o.y = pack_bf16x2(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = o;
}

// --------------------------------------------------------------------------- RMSNorm forward
// x_mod = x * (1 + col_scale) + col_bias (when given); z = bf16(x_mod * rstd * w).
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
rmsnorm_fwd_kernel(const T* x, const float* col_scale,
                   const float* col_bias, const float* w, float eps, int rows,
                   int d, T* __restrict__ xmod_out, __nv_bfloat16* __restrict__ z,
                   float* __restrict__ rstd_out) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int row = blockIdx.x * ROW_WARPS + warp; row < rows; row += gridDim.x * ROW_WARPS) {
    const T* xr = x + static_cast<size_t>(row) * d;
    float ss = 0.f;
    for (int c = lane * 4; c < d; c += 128) {
      float4 v = ld4(xr + c);
      if (col_scale != nullptr) {
        v = modulated(v, ld4(col_scale + c), ld4(col_bias + c));
        if (sizeof(T) == 2) { v.x = bf16_round(v.x); v.y = bf16_round(v.y); v.z = bf16_round(v.z); v.w = bf16_round(v.w); }
      }
      ss += square_sum(v);
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / static_cast<float>(d) + eps);
    if (lane == 0 && rstd_out != nullptr) rstd_out[row] = rstd;
    for (int c = lane * 4; c < d; c += 128) {
      float4 v = ld4(xr + c);
      if (col_scale != nullptr) {
        v = modulated(v, ld4(col_scale + c), ld4(col_bias + c));
        if (sizeof(T) == 2) { v.x = bf16_round(v.x); v.y = bf16_round(v.y); v.z = bf16_round(v.z); v.w = bf16_round(v.w); }
      }
      const float4 ww = ld4(w + c);
      if (xmod_out != nullptr) st4(xmod_out + static_cast<size_t>(row) * d + c, v);
      float4 o;
      if (sizeof(T) == 2) {  // BF16 stream: round x_hat and w first, as an eager BF16 norm does
        o.x = bf16_round(v.x * rstd) * bf16_round(ww.x); o.y = bf16_round(v.y * rstd) * bf16_round(ww.y);
        o.z = bf16_round(v.z * rstd) * bf16_round(ww.z); o.w = bf16_round(v.w * rstd) * bf16_round(ww.w);
      } else {
        o.x = v.x * rstd * ww.x; o.y = v.y * rstd * ww.y; o.z = v.z * rstd * ww.z; o.w = v.w * rstd * ww.w;
      }
      st4(z + static_cast<size_t>(row) * d + c, o);
    }
  }
}

// The same with the row held in registers between the two passes (d = 128 * CHUNKS known at compile time):
// x is read from memory once, and all CHUNKS loads of a lane are in flight together.  The weights go through `ld4_parameter`:
// as plain loads they do not pass the stores between them, and 300 x 2048 rows take 5.3 us instead of 3.1, 3456 rows 9.8
// instead of 6.9.
template <typename T, int CHUNKS>
__global__ void __launch_bounds__(ROW_THREADS)
rmsnorm_fwd_rows_kernel(const T* x, const float* col_scale,
                        const float* col_bias, const float* w, float eps, int rows,
                        T* __restrict__ xmod_out, __nv_bfloat16* __restrict__ z, float* __restrict__ rstd_out) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int d = 128 * CHUNKS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int row = blockIdx.x * ROW_WARPS + warp; row < rows; row += gridDim.x * ROW_WARPS) {
    const T* xr = x + static_cast<size_t>(row) * d;
    float4 v[CHUNKS];
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) v[i] = ld4(xr + i * 128 + lane * 4);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      if (col_scale != nullptr) {
        const int c = i * 128 + lane * 4;
        v[i] = modulated(v[i], ld4(col_scale + c), ld4(col_bias + c));
        if (sizeof(T) == 2) {
          v[i].x = bf16_round(v[i].x); v[i].y = bf16_round(v[i].y); v[i].z = bf16_round(v[i].z); v[i].w = bf16_round(v[i].w);
        }
      }
      ss += square_sum(v[i]);
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / static_cast<float>(d) + eps);
    if (lane == 0 && rstd_out != nullptr) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = i * 128 + lane * 4;
      if (xmod_out != nullptr) st4(xmod_out + static_cast<size_t>(row) * d + c, v[i]);
      const float4 ww = ld4_parameter(w + c);
      float4 o;
      if (sizeof(T) == 2) {  // BF16 stream: round x_hat and w first, as an eager BF16 norm does
        o.x = bf16_round(v[i].x * rstd) * bf16_round(ww.x); o.y = bf16_round(v[i].y * rstd) * bf16_round(ww.y);
        o.z = bf16_round(v[i].z * rstd) * bf16_round(ww.z); o.w = bf16_round(v[i].w * rstd) * bf16_round(ww.w);
      } else {
        o.x = v[i].x * rstd * ww.x; o.y = v[i].y * rstd * ww.y; o.z = v[i].z * rstd * ww.z; o.w = v[i].w * rstd * ww.w;
      }
      st4(z + static_cast<size_t>(row) * d + c, o);
    }
  }
}

// The same for few rows, a block per row: with a warp per row, 300 rows are 38 blocks whose lanes walk 16 loads, as many pairs
// of modulation values and 16 stores each.  A thread has two pieces of four columns; the squares are added in the order of
// the kernels above (lane l of a warp: columns 128 i + 4 l), so that they agree bit for bit.  d <= 2048.
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
rmsnorm_fwd_block_kernel(const T* x, const float* col_scale, const float* col_bias, const float* w, float eps, int d,
                         T* __restrict__ xmod_out, __nv_bfloat16* __restrict__ z, float* __restrict__ rstd_out) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float squares[512];
  __shared__ float factor;
  const size_t base = static_cast<size_t>(blockIdx.x) * d;
  float4 v[2], ww[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = (threadIdx.x + i * ROW_THREADS) * 4;
    if (c >= d) continue;
    v[i] = ld4(x + base + c);
    ww[i] = ld4_parameter(w + c);
    if (col_scale != nullptr) {
      v[i] = modulated(v[i], ld4(col_scale + c), ld4(col_bias + c));
      if (sizeof(T) == 2) {
        v[i].x = bf16_round(v[i].x); v[i].y = bf16_round(v[i].y); v[i].z = bf16_round(v[i].z); v[i].w = bf16_round(v[i].w);
      }
    }
    squares[c >> 2] = square_sum(v[i]);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < d / 4; i += 32) ss += squares[i];
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / static_cast<float>(d) + eps);
    if (threadIdx.x == 0) {
      factor = rstd;
      if (rstd_out != nullptr) rstd_out[blockIdx.x] = rstd;
    }
  }
  __syncthreads();
  const float rstd = factor;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = (threadIdx.x + i * ROW_THREADS) * 4;
    if (c >= d) continue;
    if (xmod_out != nullptr) st4(xmod_out + base + c, v[i]);
    float4 o;
    if (sizeof(T) == 2) {  // BF16 stream: round x_hat and w first, as an eager BF16 norm does
      o.x = bf16_round(v[i].x * rstd) * bf16_round(ww[i].x); o.y = bf16_round(v[i].y * rstd) * bf16_round(ww[i].y);
      o.z = bf16_round(v[i].z * rstd) * bf16_round(ww[i].z); o.w = bf16_round(v[i].w * rstd) * bf16_round(ww[i].w);
    } else {
      o.x = v[i].x * rstd * ww[i].x; o.y = v[i].y * rstd * ww[i].y; o.z = v[i].z * rstd * ww[i].z; o.w = v[i].w * rstd * ww[i].w;
    }
    st4(z + base + c, o);
  }
}

// --------------------------------------------------------------------------- RMSNorm backward
// dxn = rstd * (dz*w - x_hat * mean(dz*w*x_hat));  out = (dres + dxn) * (1 + out_scale)
// dw_partial[block] = sum over the block's rows of dz * x_hat.
//
// Column-owner layout: thread t owns columns 8t .. 8t+7 (256 threads cover d <= 2048) and the
// block walks over pairs of rows, so every operand is read from global memory exactly
// once, the per-row mean needs one block reduction per step of one or two rows
// (double-buffered, one __syncthreads), and the weight-gradient column sums stay in 8 registers.
//
// Bound by DRAM (14 bytes an element, 470 MB at 16384 x 2048: 72 us at the rate of a copy).  While a block has a step of rows in
// hand, the rows of its next steps are on their way into shared memory, past L1 and without registers; requested into registers
// in one step and used in the next, behind the barrier and the stores of the step before, they came at 4.7 TB/s.  16384 x 2048: 97 -> 82 us,
// MOD 100 -> 76; 8192 x 1280 45 -> 29 and 45 -> 31; BF16 stream 76 -> 59 (alone, in a chain of launches).  In a block's backward pass:
// 1792 x 1280 11.8 -> 8.8 us and 11.7 -> 9.3, 128 x 2048 4.6 -> 3.7 and 4.8 -> 4.6.
//
// MOD (FP32 stream, the norm behind a depth modulation xmod = x * (1 + scale) + bias): `x` is the modulation's input and
// xmod is formed again from it.  The gradients of scale and bias are column sums of dxmod * x and dxmod, and dxmod is in
// registers here; x is what it was, so nothing is lost where the bias is much larger than x * (1 + scale).  Summed in the
// same pass they cost 16 registers; as a pass of their own (colsum2_kernel, still used for the BF16 stream, whose xmod is
// rounded) 268 MB more per 16384 x 2048 rows.  A block's forward + backward at 1792 x 1280, where the launches count:
// 691 -> 604 us; at 16384 x 2048 within the noise of 6.5 ms.
constexpr int RB_ROWS = 2;

template <typename T>
__device__ __forceinline__ void ld8(const T* p, float (&v)[8]) {
  const float4 a = ld4(p), b = ld4(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <typename T>
__device__ __forceinline__ void st8(T* p, const float (&v)[8]) {
  st4(p, make_float4(v[0], v[1], v[2], v[3]));
  st4(p + 4, make_float4(v[4], v[5], v[6], v[7]));
}

// DEPTH steps of STEP rows of dz, x, dres and rstd in shared memory; a warp fetches its own 256 columns of each.
template <typename T, bool MOD, int STEP>
struct NormBackward {
  static constexpr int BF16_BYTES = ROW_THREADS * 16, T_BYTES = ROW_THREADS * 8 * (int)sizeof(T);
  static constexpr int SLOT = BF16_BYTES + 2 * T_BYTES + ROW_THREADS * 4;   // a row
  static constexpr int BLOCKS_PER_SM = STEP == 2 ? 2 : 3;
  static constexpr int DEPTH = STEP == 2 ? 2 : 3;
  static constexpr int SMEM = DEPTH * STEP * SLOT;
};

// Eight columns of a lane, and how its warp's 256 of them get there: 16 bytes a lane in the order of memory, so that a request covers
// whole sectors.  FP32: two rounds, and the pieces' low bit flipped in every other eight, so that lanes that read 32 bytes each do
// not meet in a bank.
__device__ __forceinline__ void fetch_columns(uint32_t warp_to, int lane, const float* warp_from, int columns, bool) {
#pragma unroll
  for (int p = lane; p < 64; p += 32)
    if (p * 4 < columns) cp_async_16(warp_to + ((p ^ ((p >> 3) & 1)) << 4), warp_from + p * 4);
}
__device__ __forceinline__ void fetch_columns(uint32_t warp_to, int lane, const __nv_bfloat16* warp_from, int columns, bool whole) {
  if (lane * 8 >= columns) return;
  const __nv_bfloat16* from = warp_from + lane * 8;
  if (whole) {
    cp_async_16(warp_to + lane * 16, from);
  } else {   // BF16 operands may begin at any 8 bytes
    cp_async_small<8>(warp_to + lane * 16, from);
    cp_async_small<8>(warp_to + lane * 16 + 8, from + 4);
  }
}
__device__ __forceinline__ void fetched_columns(uint32_t warp_at, int lane, float (&v)[8], float) {
  const uint32_t at = warp_at + lane * 32, flip = ((lane >> 2) & 1) << 4;
  float4 a, b;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w) : "r"(at ^ flip) : "memory");
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "r"((at ^ flip) ^ 16) : "memory");
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void fetched_columns(uint32_t warp_at, int lane, float (&v)[8], __nv_bfloat16) {
  uint32_t w[4];
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(warp_at + lane * 16) : "memory");
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]));
    v[2 * j] = a.x;
    v[2 * j + 1] = a.y;
  }
}

template <typename T, bool MOD, int STEP>
__global__ void __launch_bounds__(ROW_THREADS, (NormBackward<T, MOD, STEP>::BLOCKS_PER_SM))
rmsnorm_bwd_kernel(const __nv_bfloat16* dz, const T* x,
                   const float* rstd_in, const float* w,
                   const T* dres, const float* out_scale, int rows, int d,
                   T* __restrict__ dx_out, __nv_bfloat16* __restrict__ dx_bf16,
                   float* __restrict__ dw_partial, const float* mod_bias) {
  using Cfg = NormBackward<T, MOD, STEP>;
  extern __shared__ __align__(16) uint8_t ring[];
  __shared__ float red[2][STEP][ROW_WARPS];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = threadIdx.x * 8;
  const bool active = c < d;
  const float inv_d = 1.0f / static_cast<float>(d);
  const int columns = d - warp * 256;   // the warp's, at most 256 of them
  const uint32_t at_dz = smem_u32(ring) + warp * 512, at_x = smem_u32(ring) + Cfg::BF16_BYTES + warp * (256 * (int)sizeof(T));
  const uint32_t at_dres = at_x + Cfg::T_BYTES, at_rstd = smem_u32(ring) + Cfg::BF16_BYTES + 2 * Cfg::T_BYTES + threadIdx.x * 4;
  const bool whole = (reinterpret_cast<uintptr_t>(dz) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dres)) % 16 == 0;
  // this block's k-th row: pairs of neighbours, the blocks' pairs by turns
  auto row_of = [&](int k) { return (static_cast<int>(blockIdx.x) + (k / RB_ROWS) * static_cast<int>(gridDim.x)) * RB_ROWS + k % RB_ROWS; };
  auto request = [&](int k, int slot) {
#pragma unroll
    for (int r = 0; r < STEP; ++r) {
      const int row = row_of(k + r);
      if (row < rows && columns > 0) {
        const size_t base = static_cast<size_t>(row) * d + warp * 256;
        const uint32_t at = (slot * STEP + r) * Cfg::SLOT;
        fetch_columns(at_dz + at, lane, dz + base, columns, whole);
        fetch_columns(at_x + at, lane, x + base, columns, whole);
        if (dres != nullptr) fetch_columns(at_dres + at, lane, dres + base, columns, whole);
        cp_async_small<4>(at_rstd + at, rstd_in + row);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int n = 0; n < Cfg::DEPTH - 1; ++n) request(n * STEP, n);
  float wv[8], sv[8], acc[8];
  [[maybe_unused]] float bi[8], acc_bias[8], acc_scale[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { wv[j] = 0.f; sv[j] = 1.f; bi[j] = 0.f; acc[j] = 0.f; acc_bias[j] = 0.f; acc_scale[j] = 0.f; }
  if (active) {
    ld8(w + c, wv);
    if constexpr (MOD) ld8(mod_bias + c, bi);
    if (out_scale != nullptr) {
      ld8(out_scale + c, sv);
#pragma unroll
      for (int j = 0; j < 8; ++j) sv[j] += 1.f;
    }
  }
  int slot = 0, turn = 0;
  for (int k = 0; row_of(k) < rows; k += STEP, turn ^= 1) {
    __syncwarp();   // every lane has read the rows before these
    request(k + (Cfg::DEPTH - 1) * STEP, slot == 0 ? Cfg::DEPTH - 1 : slot - 1);   // into their place
    cp_async_wait<Cfg::DEPTH - 1>();
    __syncwarp();
    float g[STEP][8], xh[STEP][8], rs[STEP];
#pragma unroll
    for (int r = 0; r < STEP; ++r) {
      const uint32_t at = (slot * STEP + r) * Cfg::SLOT;
      float part = 0.f;
      rs[r] = 0.f;
      if (active && row_of(k + r) < rows) {
        fetched_columns(at_dz + at, lane, g[r], __nv_bfloat16());
        fetched_columns(at_x + at, lane, xh[r], T());
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(rs[r]) : "r"(at_rstd + at) : "memory");
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) { g[r][j] = 0.f; xh[r][j] = 0.f; }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if constexpr (MOD) xh[r][j] = xh[r][j] * sv[j] + bi[j];
        xh[r][j] *= rs[r];
        part += g[r][j] * wv[j] * xh[r][j];
      }
      part = warp_sum(part);
      if (lane == 0) red[turn][r][warp] = part;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < STEP; ++r) {
      const int row = row_of(k + r);
      if (row < rows && active) {
        const uint32_t at = (slot * STEP + r) * Cfg::SLOT;
        float dot = 0.f;
#pragma unroll
        for (int wi = 0; wi < ROW_WARPS; ++wi) dot += red[turn][r][wi];
        dot *= inv_d;  // mean(dz * w * x_hat)
        const size_t base = static_cast<size_t>(row) * d + c;
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[j] += g[r][j] * xh[r][j];
          o[j] = rs[r] * (g[r][j] * wv[j] - xh[r][j] * dot);
        }
        if (dres != nullptr) {
          float rr[8];
          fetched_columns(at_dres + at, lane, rr, T());
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += rr[j];
        }
        if constexpr (MOD) {
          float xv[8];
          fetched_columns(at_x + at, lane, xv, T());
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            acc_bias[j] += o[j];
            acc_scale[j] += o[j] * xv[j];
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] *= sv[j];
        st8(dx_out + base, o);
        if (dx_bf16 != nullptr) st8(dx_bf16 + base, o);
      }
    }
    slot = slot + 1 == Cfg::DEPTH ? 0 : slot + 1;
  }
  if (dw_partial != nullptr && active) st8(dw_partial + static_cast<size_t>(blockIdx.x) * d + c, acc);
  if constexpr (MOD) {
    if (active) {
      st8(dw_partial + (static_cast<size_t>(gridDim.x) + blockIdx.x) * d + c, acc_bias);
      st8(dw_partial + (2 * static_cast<size_t>(gridDim.x) + blockIdx.x) * d + c, acc_scale);
    }
  }
}

template <typename T, bool MOD, int STEP>
static int launch_rmsnorm_bwd_step(const void* dz, const void* x, const float* rstd, const float* w, const void* dres,
                                   const float* out_scale, int rows, int d, void* dx_out, void* dx_bf16, float* dw_partial,
                                   const float* mod_bias, int grid, cudaStream_t stream) {
  using Cfg = NormBackward<T, MOD, STEP>;
  if (!allow_shared_memory<rmsnorm_bwd_kernel<T, MOD, STEP>>(Cfg::SMEM)) return -20;
  launch_dependent(rmsnorm_bwd_kernel<T, MOD, STEP>, dim3(grid), dim3(ROW_THREADS), Cfg::SMEM, stream, static_cast<const __nv_bfloat16*>(dz),
                   static_cast<const T*>(x), rstd, w, static_cast<const T*>(dres), out_scale, rows, d, static_cast<T*>(dx_out),
                   static_cast<__nv_bfloat16*>(dx_bf16), dw_partial, mod_bias);
  ws_count_launch();
  return 0;
}

// Two rows to a step where all of the blocks are resident that way, two on an SM (up to 592 rows, and always with MOD, whose registers allow
// no third): half the barriers, and a block's only pair of rows is fetched at once (128 x 2048: 3.7 us against 4.1).  Past that three blocks on an
// SM with one row to a step: 82 us against 89 at 16384 x 2048.  MOD with one: 79.5 against 75.6 there, within 0.5 us below 2048 rows.
template <typename T, bool MOD>
static int launch_rmsnorm_bwd(const void* dz, const void* x, const float* rstd, const float* w, const void* dres, const float* out_scale,
                              int rows, int d, void* dx_out, void* dx_bf16, float* dw_partial, const float* mod_bias, int grid,
                              cudaStream_t stream) {
  if constexpr (!MOD) {
    if (grid > CHIP_SMS * 2)
      return launch_rmsnorm_bwd_step<T, MOD, 1>(dz, x, rstd, w, dres, out_scale, rows, d, dx_out, dx_bf16, dw_partial, mod_bias, grid, stream);
  }
  return launch_rmsnorm_bwd_step<T, MOD, 2>(dz, x, rstd, w, dres, out_scale, rows, d, dx_out, dx_bf16, dw_partial, mod_bias, grid, stream);
}

// --------------------------------------------------------------------------- column sums
// partial_a[block] = sum_rows a ; partial_ab[block] = sum_rows a*b  (a, b: [rows, d])
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
colsum2_kernel(const T* a, const T* b, int rows, int d,
               float* __restrict__ partial_a, float* __restrict__ partial_ab) {
  pdl_launch_dependents();
  pdl_wait();
  // thread t owns columns t*4 .. t*4+3 of a 1024-wide panel; rows strided over blocks
  for (int c0 = 0; c0 < d; c0 += ROW_THREADS * 4) {
    const int c = c0 + threadIdx.x * 4;
    if (c >= d) continue;
    float4 sa = make_float4(0.f, 0.f, 0.f, 0.f), sab = sa;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
      const float4 va = ld4(a + static_cast<size_t>(row) * d + c);
      sa.x += va.x; sa.y += va.y; sa.z += va.z; sa.w += va.w;
      if (b != nullptr) {
        const float4 vb = ld4(b + static_cast<size_t>(row) * d + c);
        sab.x += va.x * vb.x; sab.y += va.y * vb.y; sab.z += va.z * vb.z; sab.w += va.w * vb.w;
      }
    }
    st4(partial_a + static_cast<size_t>(blockIdx.x) * d + c, sa);
    if (b != nullptr) st4(partial_ab + static_cast<size_t>(blockIdx.x) * d + c, sab);
  }
}

// out[c] = beta*out[c] + scale(c) * sum_p partial[p][c];  scale(c) = 1/(1+inv_scale[c]) if given.  gridDim.y sums of
// that kind lie behind one another ([gridDim.y][parts][d] -> [gridDim.y][d]).
// One block per 32 columns; warp w sums parts w, w+32, ... (independent 128-byte loads in flight), then the warp sums are
// combined in a fixed order: the result is deterministic.  Its time is that of its rounds of loads one after another, so
// 32 warps with four loads each at once: the sums of 1792 x 1280 rows 6.1 us with eight warps, 3.8 so.
constexpr int FIN_COLS = 32, FIN_WARPS = 32;
__device__ __forceinline__ void column_sums(const float* partial, int parts, int d, const float* inv_scale, float beta, float* out) {
  __shared__ float red[FIN_WARPS][FIN_COLS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * FIN_COLS + lane;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  if (c < d) {
    for (int p = warp; p < parts; p += 4 * FIN_WARPS) {
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        v[q] = p + q * FIN_WARPS < parts ? partial[static_cast<size_t>(p + q * FIN_WARPS) * d + c] : 0.f;
      s0 += v[0]; s1 += v[1]; s2 += v[2]; s3 += v[3];
    }
  }
  red[warp][lane] = (s0 + s1) + (s2 + s3);
  __syncthreads();
  if (warp == 0 && c < d) {
    float s = 0.f;
#pragma unroll
    for (int wi = 0; wi < FIN_WARPS; ++wi) s += red[wi][lane];
    if (inv_scale != nullptr) {
      const float den = 1.f + inv_scale[c];
      s = den != 0.f ? s / den : 0.f;
    }
    out[c] = (beta != 0.f ? beta * out[c] : 0.f) + s;
  }
}

__global__ void __launch_bounds__(FIN_WARPS * 32)
colsum_finalize_kernel(const float* partial, int parts, int d,
                       const float* inv_scale, float beta, float* out) {
  pdl_launch_dependents();
  pdl_wait();
  column_sums(partial + static_cast<size_t>(blockIdx.y) * parts * d, parts, d, inv_scale, beta, out + static_cast<size_t>(blockIdx.y) * d);
}

// The small sums that a block's backward pass leaves, in one launch behind it: blockIdx.y 0 the second norm's weight gradient, 1 .. `first_sums` the
// first norm's, and one more the logits' (d = 64 H: two blocks for every head).  None of them is needed before.  A block's pass has
// two launches less for it, which no whole step shows beyond its spread (the smoke model's, four blocks: 1.74 ms; 2 x 896 tokens at width 1280: 0.44 ms).
struct BlockSums {
  const float *second, *first, *scan, *fast_logit, *slow_logit, *mix_logit;
  int second_parts, first_parts, first_sums, B, H, d;
  float *second_out, *first_out, *logits_out;
};
__global__ void __launch_bounds__(FIN_WARPS * 32)
block_sums_kernel(const BlockSums p) {
  pdl_launch_dependents();
  pdl_wait();
  const int y = blockIdx.y;
  if (y == 0) {
    column_sums(p.second, p.second_parts, p.d, nullptr, 0.f, p.second_out);
  } else if (y <= p.first_sums) {
    column_sums(p.first + static_cast<size_t>(y - 1) * p.first_parts * p.d, p.first_parts, p.d, nullptr, 0.f, p.first_out + static_cast<size_t>(y - 1) * p.d);
  } else if (static_cast<int>(blockIdx.x) < p.H && threadIdx.x < 96) {
    logit_grad(p.scan, p.fast_logit, p.slow_logit, p.mix_logit, p.B, p.H, blockIdx.x, threadIdx.x >> 5, p.logits_out);
  }
}

// --------------------------------------------------------------------------- casts
__global__ void cast_f32_bf16_kernel(const float* in, __nv_bfloat16* __restrict__ out,
                                     size_t n4) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    st4(out + i * 4, ld4(in + i * 4));
  }
}

// --------------------------------------------------------------------------- embedding
// out[row] = table[ids[row]] ; table FP32 (master) or BF16, out FP32 or BF16
template <typename TT, typename TO>
__global__ void __launch_bounds__(ROW_THREADS)
embed_fwd_kernel(const long long* __restrict__ ids, const TT* __restrict__ table, int rows, int d,
                 int vocab, TO* __restrict__ out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int row = blockIdx.x * ROW_WARPS + warp; row < rows; row += gridDim.x * ROW_WARPS) {
    long long id = ids[row];
    if (id < 0 || id >= vocab) id = 0;
    const TT* src = table + static_cast<size_t>(id) * d;
    for (int c = lane * 4; c < d; c += 128) st4(out + static_cast<size_t>(row) * d + c, ld4(src + c));
  }
}

// Deterministic embedding backward: rows were sorted by token id on the host side of the op
// (`order` = argsort of ids).  The unit of work is (position p of the sorted ids, 128-column chunk): a warp
// works only if a run of equal ids starts at p, and then adds that chunk of all gradient rows of the run, in
// order, into the FP32 gradient table - no atomics, run-to-run identical.  A run is therefore shared by d / 128
// warps, which keeps a run of thousands of equal ids (the padding of a fine-tuning batch) from being one
// warp's serial work.  The runs are found on the device, so the host needs no count of distinct tokens (which
// would cost a device-to-host read, and with it a drained launch queue, in every micro-batch).
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
embed_bwd_kernel(const T* __restrict__ dx, const long long* __restrict__ sorted_ids,
                 const long long* __restrict__ order, int rows, int d, int vocab, float* __restrict__ grad_table) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = d / 128;
  const long long units = static_cast<long long>(rows) * chunks;
  for (long long unit = blockIdx.x * ROW_WARPS + warp; unit < units; unit += static_cast<long long>(gridDim.x) * ROW_WARPS) {
    const int begin = static_cast<int>(unit / chunks);
    const int c = static_cast<int>(unit % chunks) * 128 + lane * 4;
    const long long id = sorted_ids[begin];
    if (begin > 0 && sorted_ids[begin - 1] == id) continue;  // not the head of a run
    if (id < 0 || id >= vocab) continue;
    // the end of the run, 32 positions per step
    int end = begin + 1;
    for (;;) {
      const int at = end + lane;
      const bool same = at < rows && sorted_ids[at] == id;
      const unsigned mask = __ballot_sync(0xffffffffu, same);
      if (mask == 0xffffffffu) {
        end += 32;
        continue;
      }
      end += __ffs(~mask) - 1;
      break;
    }
    float* dst = grad_table + static_cast<size_t>(id) * d + c;
    float4 s = ld4(dst);
    int j = begin;
    for (; j + 4 <= end; j += 4) {  // four independent loads in flight; the sum keeps the row order
      const float4 v0 = ld4(dx + static_cast<size_t>(order[j]) * d + c);
      const float4 v1 = ld4(dx + static_cast<size_t>(order[j + 1]) * d + c);
      const float4 v2 = ld4(dx + static_cast<size_t>(order[j + 2]) * d + c);
      const float4 v3 = ld4(dx + static_cast<size_t>(order[j + 3]) * d + c);
      s.x += v0.x; s.y += v0.y; s.z += v0.z; s.w += v0.w;
      s.x += v1.x; s.y += v1.y; s.z += v1.z; s.w += v1.w;
      s.x += v2.x; s.y += v2.y; s.z += v2.z; s.w += v2.w;
      s.x += v3.x; s.y += v3.y; s.z += v3.z; s.w += v3.w;
    }
    for (; j < end; ++j) {
      const float4 v = ld4(dx + static_cast<size_t>(order[j]) * d + c);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    st4(dst, s);
  }
}

constexpr int CHIP_BLOCKS = CHIP_SMS * 8;   // blocks of ROW_THREADS that the chip holds at once
static int row_grid(int rows) {
  int blocks = (rows + ROW_WARPS - 1) / ROW_WARPS;
  return blocks < CHIP_BLOCKS ? (blocks > 0 ? blocks : 1) : CHIP_BLOCKS;
}

template <typename T>
using RmsnormRows = void (*)(const T*, const float*, const float*, const float*, float, int, T*, __nv_bfloat16*, float*);
// The kernel that holds rows of 128 * chunks columns (1..MAX_CHUNKS) in registers.
template <typename T, int... I>
static RmsnormRows<T> rmsnorm_rows(int chunks, std::integer_sequence<int, I...>) {
  static constexpr RmsnormRows<T> kernels[] = {rmsnorm_fwd_rows_kernel<T, I + 1>...};
  return kernels[chunks - 1];
}

// Up to how many rows a block for each is faster than a warp.  Wide rows: one round of blocks over the chip.  Narrow ones leave
// most of a block idle, and past two blocks to an SM its start costs more than the warp's longer walk; the modulation's loads
// lengthen that walk.  Measured in a chain of launches (a warp -> a block per row, FP32, us): modulated 2048 columns 64 rows 3.9 ->
// 2.0, 300 3.9 -> 2.4, 1100 6.2 -> 4.3; 1280 columns 300 rows 3.4 -> 2.2, 1100 5.6 -> 3.4; 384 columns 592 rows 2.0 -> 1.8, 1100 2.9 ->
// 2.2; 256 columns 64 rows 1.6 -> 1.5, 1024 2.0 -> 2.0; 128 columns 64 rows 1.2 -> 1.4.  Plain 1280 columns 1100 rows 3.5 -> 2.5; 640 columns
// 64 rows 1.6 -> 1.4, 1100 2.3 -> 2.1; 512 columns 296 rows 1.5 -> 1.4, 400 1.5 -> 1.6; 256 columns 1000 rows 1.5 -> 2.0.
static int rmsnorm_block_rows(int d, bool modulated) {
  if (d > 128 * MAX_CHUNKS || d < 256) return 0;
  return d >= (modulated ? 384 : 640) ? CHIP_BLOCKS : CHIP_BLOCKS / 4;
}

template <typename T>
static void launch_rmsnorm_fwd(const T* x, const float* col_scale, const float* col_bias, const float* w, float eps, int rows, int d,
                               T* xmod_out, __nv_bfloat16* z, float* rstd, bool dependent, cudaStream_t stream) {
  if (rows <= rmsnorm_block_rows(d, col_scale != nullptr))
    launch_kernel(dependent, rmsnorm_fwd_block_kernel<T>, dim3(rows), dim3(ROW_THREADS), 0, stream, x, col_scale, col_bias, w, eps, d,
                     xmod_out, z, rstd);
  else if (d <= 128 * MAX_CHUNKS)   // the general kernel reads its rows twice: 4096 rows of 384, 1024, 1920 columns 5.1, 10.7, 19.7 us, 3.6, 6.5, 12.2 so
    launch_kernel(dependent, rmsnorm_rows<T>(d / 128, std::make_integer_sequence<int, MAX_CHUNKS>{}), dim3(row_grid(rows)),
                     dim3(ROW_THREADS), 0, stream, x, col_scale, col_bias, w, eps, rows, xmod_out, z, rstd);
  else
    launch_kernel(dependent, rmsnorm_fwd_kernel<T>, dim3(row_grid(rows)), dim3(ROW_THREADS), 0, stream, x, col_scale, col_bias, w, eps,
                     rows, d, xmod_out, z, rstd);
  ws_count_launch();
}

}  // namespace ws

using namespace ws;

extern "C" int ws_rmsnorm_fwd(const void* x, int x_bf16, const float* col_scale, const float* col_bias,
                              const float* w, float eps, int rows, int d, void* xmod_out, void* z,
                              float* rstd, int first, cudaStream_t stream) {
  if (d % 128 != 0 || rows <= 0) return -1;
  if (x_bf16)
    launch_rmsnorm_fwd(static_cast<const __nv_bfloat16*>(x), col_scale, col_bias, w, eps, rows, d,
                       static_cast<__nv_bfloat16*>(xmod_out), static_cast<__nv_bfloat16*>(z), rstd, first == 0, stream);
  else
    launch_rmsnorm_fwd(static_cast<const float*>(x), col_scale, col_bias, w, eps, rows, d, static_cast<float*>(xmod_out),
                       static_cast<__nv_bfloat16*>(z), rstd, first == 0, stream);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Number of partial rows ws_rmsnorm_bwd writes (the caller sizes dw_partial as parts*d floats).
constexpr int kRmsBwdMaxParts = CHIP_SMS * 3;  // three resident blocks per SM
extern "C" int ws_rmsnorm_bwd_parts(int rows) {
  int blocks = (rows + RB_ROWS - 1) / RB_ROWS;
  return blocks < kRmsBwdMaxParts ? (blocks > 0 ? blocks : 1) : kRmsBwdMaxParts;
}

extern "C" int ws_rmsnorm_bwd(const void* dz, const void* x, int x_bf16, const float* rstd, const float* w,
                              const void* dres, const float* out_scale, int rows, int d, void* dx_out,
                              void* dx_bf16, float* dw_partial, cudaStream_t stream) {
  if (d % 128 != 0 || d > ROW_THREADS * 8 || rows <= 0) return -1;
  const int grid = ws_rmsnorm_bwd_parts(rows);
  auto* run = x_bf16 ? &launch_rmsnorm_bwd<__nv_bfloat16, false> : &launch_rmsnorm_bwd<float, false>;
  const int rc = run(dz, x, rstd, w, dres, out_scale, rows, d, dx_out, dx_bf16, dw_partial, nullptr, grid, stream);
  return rc ? rc : cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Two resident blocks per SM: the modulation's column sums take the registers of the third.
extern "C" int ws_rmsnorm_bwd_mod_parts(int rows) {
  const int blocks = (rows + RB_ROWS - 1) / RB_ROWS;
  return blocks < CHIP_SMS * 2 ? (blocks > 0 ? blocks : 1) : CHIP_SMS * 2;
}

extern "C" int ws_rmsnorm_bwd_mod(const void* dz, const float* x, const float* rstd, const float* w, const float* dres,
                                  const float* scale, const float* bias, int rows, int d, float* dx_out,
                                  float* partial, float* grads, cudaStream_t stream) {
  if (d % 128 != 0 || d > ROW_THREADS * 8 || rows <= 0) return -1;
  const int parts = ws_rmsnorm_bwd_mod_parts(rows);
  const int rc = launch_rmsnorm_bwd<float, true>(dz, x, rstd, w, dres, scale, rows, d, dx_out, nullptr, partial, bias, parts, stream);
  if (rc || grads == nullptr) return rc ? rc : cudaGetLastError() == cudaSuccess ? 0 : -2;
  launch_dependent(colsum_finalize_kernel, dim3((d + FIN_COLS - 1) / FIN_COLS, 3), dim3(FIN_WARPS * 32), 0, stream, partial,
                   parts, d, nullptr, 0.f, grads);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_colsum_parts(int rows) { return rows < 296 ? (rows > 0 ? rows : 1) : 296; }

extern "C" int ws_colsum2(const void* a, const void* b, int is_bf16, int rows, int d, float* partial_a,
                          float* partial_ab, cudaStream_t stream) {
  if (d % 4 != 0 || rows <= 0) return -1;
  const int grid = ws_colsum_parts(rows);
  if (is_bf16)
    launch_dependent(colsum2_kernel<__nv_bfloat16>, dim3(grid), dim3(ROW_THREADS), 0, stream, (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, rows, d, partial_a, partial_ab);
  else
    launch_dependent(colsum2_kernel<float>, dim3(grid), dim3(ROW_THREADS), 0, stream, (const float*)a, (const float*)b, rows, d,
                                                            partial_a, partial_ab);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_colsum_finalize(const float* partial, int parts, int d, const float* inv_scale, float beta,
                                  float* out, cudaStream_t stream) {
  launch_dependent(colsum_finalize_kernel, dim3((d + FIN_COLS - 1) / FIN_COLS), dim3(FIN_WARPS * 32), 0, stream, partial, parts, d, inv_scale, beta, out);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_block_sums(const float* second, int second_parts, float* second_out, const float* first, int first_parts, int first_sums,
                             float* first_out, const float* scan, const float* fast_logit, const float* slow_logit, const float* mix_logit, int B,
                             int H, float* logits_out, int d, cudaStream_t stream) {
  if (d != 64 * H || first_sums < 1) return -1;
  const BlockSums p{second, first, scan, fast_logit, slow_logit, mix_logit, second_parts, first_parts, first_sums, B, H, d, second_out, first_out,
                    logits_out};
  launch_dependent(block_sums_kernel, dim3((d + FIN_COLS - 1) / FIN_COLS, first_sums + 2), dim3(FIN_WARPS * 32), 0, stream, p);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_cast_f32_bf16(const float* in, void* out, size_t n, cudaStream_t stream) {
  if (n % 4 != 0) return -1;
  if (n == 0) return 0;
  const size_t n4 = n / 4;
  size_t blocks = (n4 + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  launch_dependent(cast_f32_bf16_kernel, dim3((int)blocks), dim3(256), 0, stream, in, (__nv_bfloat16*)out, n4);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_embed_fwd(const long long* ids, const void* table, int table_bf16, int rows, int d,
                            int vocab, void* out, int out_bf16, cudaStream_t stream) {
  if (d % 4 != 0 || rows <= 0) return -1;
  const int grid = row_grid(rows);
  if (table_bf16 && out_bf16)
    embed_fwd_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, ROW_THREADS, 0, stream>>>(
        ids, (const __nv_bfloat16*)table, rows, d, vocab, (__nv_bfloat16*)out);
  else if (!table_bf16 && out_bf16)
    embed_fwd_kernel<float, __nv_bfloat16><<<grid, ROW_THREADS, 0, stream>>>(
        ids, (const float*)table, rows, d, vocab, (__nv_bfloat16*)out);
  else if (!table_bf16 && !out_bf16)
    embed_fwd_kernel<float, float><<<grid, ROW_THREADS, 0, stream>>>(ids, (const float*)table, rows, d,
                                                                     vocab, (float*)out);
  else if (table_bf16 && !out_bf16)  // BF16 table of a frozen model feeding an FP32 residual stream
    embed_fwd_kernel<__nv_bfloat16, float><<<grid, ROW_THREADS, 0, stream>>>(ids, (const __nv_bfloat16*)table, rows,
                                                                              d, vocab, (float*)out);
  else
    return -3;
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_embed_bwd(const void* dx, int dx_bf16, const long long* sorted_ids, const long long* order, int rows,
                            int d, int vocab, float* grad_table, cudaStream_t stream) {
  if (d % 128 != 0 || rows <= 0 || vocab <= 0) return -1;
  const int grid = 148 * 8;
  if (dx_bf16)
    embed_bwd_kernel<__nv_bfloat16><<<grid, ROW_THREADS, 0, stream>>>((const __nv_bfloat16*)dx, sorted_ids, order, rows,
                                                                      d, vocab, grad_table);
  else
    embed_bwd_kernel<float><<<grid, ROW_THREADS, 0, stream>>>((const float*)dx, sorted_ids, order, rows, d, vocab,
                                                              grad_table);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// =============================================================================== no-allocation entry
// RMSNorm backward whose partial-sum scratch is part of the library image (see
// ws_static_scratch.h for who needs this and for the sharing rules).
#include "ws_static_scratch.h"
#include <mutex>

// Lives in every GPU that loads this library until the process exits.  In host code this name is
// only a handle for cudaGetSymbolAddress, never a device address.
static __device__ __align__(256) float g_static_scratch[WS_STATIC_SCRATCH_FLOATS];
// The array is exactly what the largest accepted problem writes: the most partial rows the kernel ever
// uses times the widest row it accepts.
static_assert(WS_STATIC_SCRATCH_FLOATS == kRmsBwdMaxParts * 128 * MAX_CHUNKS,
              "WS_STATIC_SCRATCH_FLOATS must equal the maximum number of partial rows times the maximum width");

namespace {
constexpr int kMaxDevices = 64;
float* g_scratch_addr[kMaxDevices] = {};
std::mutex g_scratch_mutex;

// Device address of the scratch array on the current device, looked up once per device.
int static_scratch_for_current_device(float** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return WS_STATIC_ERR_SYMBOL;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_addr[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || ptr == nullptr) return WS_STATIC_ERR_SYMBOL;
    g_scratch_addr[dev] = static_cast<float*>(ptr);
  }
  *out = g_scratch_addr[dev];
  return 0;
}
}  // namespace

extern "C" const char* ws_static_scratch_strerror(int code) {
  switch (code) {
    case 0: return "success";
    case WS_STATIC_ERR_BAD_SHAPE: return "rows must be positive and d a multiple of 128 not above 2048";
    case WS_STATIC_ERR_LAUNCH: return "kernel launch failed";
    case WS_STATIC_ERR_TOO_LARGE: return "problem needs more partial sums than the built-in scratch array holds "
                                         "(cannot happen while d <= 2048 is enforced; kept as a guard)";
    case WS_STATIC_ERR_SYMBOL: return "could not resolve the device address of the built-in scratch array";
    default: return "unknown error";
  }
}

extern "C" int ws_rmsnorm_bwd_static(const void* dz, const void* x, int x_bf16, const float* rstd, const float* w,
                                     const void* dres, const float* out_scale, int rows, int d, void* dx_out,
                                     void* dx_bf16, float* dw_out, cudaStream_t stream) {
  if (d % 128 != 0 || d > 128 * MAX_CHUNKS || rows <= 0) return WS_STATIC_ERR_BAD_SHAPE;
  const int parts = ws_rmsnorm_bwd_parts(rows);
  if (static_cast<long long>(parts) * d > static_cast<long long>(WS_STATIC_SCRATCH_FLOATS)) return WS_STATIC_ERR_TOO_LARGE;
  float* scratch = nullptr;
  const int rc = static_scratch_for_current_device(&scratch);
  if (rc != 0) return rc;
  // Every partial row that the reduction reads below is written by the kernel first, so the
  // previous call's contents never leak into this result.
  auto* run = x_bf16 ? &launch_rmsnorm_bwd<__nv_bfloat16, false> : &launch_rmsnorm_bwd<float, false>;
  if (run(dz, x, rstd, w, dres, out_scale, rows, d, dx_out, dx_bf16, scratch, nullptr, parts, stream) != 0) return WS_STATIC_ERR_LAUNCH;
  launch_dependent(colsum_finalize_kernel, dim3((d + FIN_COLS - 1) / FIN_COLS), dim3(FIN_WARPS * 32), 0, stream, scratch, parts, d, nullptr, 0.f, dw_out);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : WS_STATIC_ERR_LAUNCH;
}
