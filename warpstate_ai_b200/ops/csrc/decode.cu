// Decode-step kernels: one new token for every sequence of a batch (batch <= 64; the projections also for the rows of a prompt of up
// to 128 tokens).
//
// A decode step is bound by streaming the weights once (4.0 GB for the 2.005 B model) and the
// current chunk's K/V cache, so the GEMMs here are weight-streaming kernels, not tile kernels:
//
//   decode_gemm_kernel     out[b, n] = sum_k x[b, k] W[n, k].  The roles of the MMA operands are
//                          swapped with respect to training: 128 weight rows are the M dimension of
//                          tcgen05.mma, the (padded) batch is its N dimension, so one CTA streams a
//                          128-row slab of W exactly once through an 8-stage TMA ring while the
//                          tiny activation block comes from L2.  Slabs x K-splits give >= 128 CTAs
//                          for every projection of the model; split partials are FP32.
//                          Epilogues: BF16, FP32 (logits), FP32 split-K partial, SwiGLU (64 up rows
//                          and their 64 gate rows share a slab).
//   decode_reduce_norm_kernel  x += sum of split partials (or x = embedding row), optional depth
//                          modulation of the next layer, RMSNorm -> BF16: everything between two
//                          GEMMs of the residual stream in one pass, one CTA per sequence.
//   decode_attn_kernel     one CTA per (sequence, head): RoPE of q/k at the in-chunk position,
//                          append k/v/u to the chunk cache, causal attention over the cache rows
//                          <= position, memory read q.M, gate blend.  decode_attn_warp_kernel: a warp for each, where there are many.
//
//   decode_norm_gemm_kernel    the residual + norm and the projection that reads it in one launch, for one sequence.
//
// The 140 to 200 launches of a step form one chain of programmatic dependent launches: every kernel lets
// its successor start at once, and a GEMM fills its whole TMA ring with weight tiles (which no
// kernel of the step writes) before it waits for its predecessor, so the weight stream of the
// next projection runs under the small kernels and the tail of the previous GEMM.
//
// Reference semantics: WarpStateCore.step (reference warpstate/model.py:222-274) in the
// training-consistent form of ops/posttrain_chat.py:94-142.  The reference runs these as
// ~40 eager PyTorch ops per layer at batch 1.
#include "ws_ptx.cuh"
#include "ws_api.h"
#include "ws_launch.h"
#include "ws_tma_host.h"

#include <cuda_bf16.h>

#include <cstdlib>

namespace ws {

extern "C" void ws_count_launch(void);

namespace dec {
constexpr int TM = 128;  // weight rows per slab
constexpr int BK = 64;
constexpr int THREADS = 192;  // warp 0 TMA, warp 1 MMA + TMEM, warps 2..5 epilogue
constexpr int W_BYTES = TM * BK * 2;
}  // namespace dec

struct DecodeGemmParams {
  int n;        // output features (SwiGLU: hidden size h; W has 2h rows)
  int k;
  int batch;
  int kb_per_split;
  int packed;   // W is stored tile by tile: [slab][k block][128 rows][64 columns], each tile contiguous
  void* out;    // BF16 [batch, ldo] | FP32 [batch, ldo] | FP32 partial [splits, batch, n]
  int ldo;
  int* error_flag;
};

// DEPTH = stages of the TMA ring.  8: one CTA per SM with 192 KiB of tiles in flight.  4: half the ring, so that
// two CTAs fit on an SM -- the successor of a launch in the dependent chain can then become resident, set up and
// request its first ring of weights while its predecessor still occupies every SM.  The SwiGLU exchange buffer
// overlays the first ring stages (the ring is idle once the last MMA has completed).
template <int BPAD, int DEPTH>
struct DecodeCfg {
  static constexpr int STAGES = DEPTH;
  static constexpr int X_BYTES = BPAD * dec::BK * 2;
  static constexpr int STAGE_BYTES = dec::W_BYTES + X_BYTES;
  static constexpr int EXCHANGE_BYTES = 64 * BPAD * 4;
  static_assert(EXCHANGE_BYTES <= STAGES * dec::W_BYTES, "the exchange buffer overlays the weight stages");
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = BPAD <= 32 ? 32 : BPAD <= 64 ? 64 : 128;   // a power of two
  static constexpr int CTAS_PER_SM = 2 * (SMEM + 1024) <= 233472 ? 2 : 1;
};

// EPI: 0 = BF16 out, 1 = FP32 split-K partial, 2 = SwiGLU (BF16 activation), 3 = FP32 out
// Epilogue of one slab (128 weight rows from n0, or 64 up rows and their gate rows) by the four warps whose TMEM quarters it is.
template <int BPAD, int EPI>
__device__ __forceinline__ void decode_epilogue(const DecodeGemmParams& p, uint32_t tmem, int warp, int lane, int n0, float* sG, bool ok) {
  const int quarter = warp & 3;  // TMEM lane quarter this warp may read
  const int row = quarter * 32 + lane;
  tc_fence_after_sync();
  const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
  if (EPI == 2) {
    // rows 0..63 = up, 64..127 = gate: the gate warps hand silu-ready values over through smem
    if (row >= 64 && ok) {
#pragma unroll
      for (int c0 = 0; c0 < BPAD; c0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(taddr + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float g = __uint_as_float(r[j]);
          sG[(c0 + j) * 64 + (row - 64)] = g * sigmoid_fast(g);
        }
      }
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (row < 64 && ok) {
      const int hcol = n0 + row;
      __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out);
#pragma unroll
      for (int c0 = 0; c0 < BPAD; c0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(taddr + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int b = c0 + j;
          if (b < p.batch && hcol < p.n)
            out[static_cast<size_t>(b) * p.ldo + hcol] = __float2bfloat16(__uint_as_float(r[j]) * sG[b * 64 + row]);
        }
      }
    }
  } else if (ok) {
    const int n = n0 + row;
#pragma unroll
    for (int c0 = 0; c0 < BPAD; c0 += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(taddr + c0, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int b = c0 + j;
        if (b >= p.batch || n >= p.n) continue;
        const float v = __uint_as_float(r[j]);
        if (EPI == 0) {
          static_cast<__nv_bfloat16*>(p.out)[static_cast<size_t>(b) * p.ldo + n] = __float2bfloat16(v);
        } else if (EPI == 3) {
          static_cast<float*>(p.out)[static_cast<size_t>(b) * p.ldo + n] = v;
        } else {
          static_cast<float*>(p.out)[(static_cast<size_t>(blockIdx.y) * p.batch + b) * p.n + n] = v;
        }
      }
    }
  }
}

template <int BPAD, int EPI, int DEPTH>
__global__ void __launch_bounds__(dec::THREADS, DecodeCfg<BPAD, DEPTH>::CTAS_PER_SM)
decode_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                   const DecodeGemmParams p) {
  using namespace dec;
  using Cfg = DecodeCfg<BPAD, DEPTH>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sW = smem;
  uint8_t* sX = smem + Cfg::STAGES * W_BYTES;
  float* sG = reinterpret_cast<float*>(sW);  // written only after the last MMA has read the ring
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + Cfg::STAGES;
  uint64_t* tfull = bars + 2 * Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * Cfg::STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();

  const int slab = blockIdx.x;
  const int total_kb = (p.k + BK - 1) / BK;
  const int kb0 = blockIdx.y * p.kb_per_split;
  const int kb1 = min(total_kb, kb0 + p.kb_per_split);
  const int rows_per_slab = EPI == 2 ? 64 : TM;
  const int n0 = slab * rows_per_slab;

  if (warp == 0) {
    if (lane == 0) {
      auto load_w = [&](int s, int kb) {
        mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
        if (p.packed) {  // one contiguous 16 KiB tile (SwiGLU: the up and gate rows are already paired)
          tma_load_2d(sW + s * W_BYTES, &tm_w, &full[s], 0, (slab * total_kb + kb) * TM);
          return;
        }
        tma_load_2d(sW + s * W_BYTES, &tm_w, &full[s], kb * BK, n0);
        if (EPI == 2)  // 64 up rows + the 64 matching gate rows
          tma_load_2d(sW + s * W_BYTES + 64 * 128, &tm_w, &full[s], kb * BK, p.n + n0);
      };
      // Every CTA walks its k blocks from a different starting block (wrapping around): all CTAs of a
      // launch read the same activation tiles, and in lock step they would queue on the few L2
      // slices that hold the current one.
      const int nkb = kb1 - kb0;
      const int rot = nkb > 0 ? static_cast<int>((blockIdx.x * 5u + blockIdx.y * 3u) % static_cast<unsigned>(nkb)) : 0;
      auto block_of = [&](int it) {
        const int r = it + rot;
        return kb0 + (r >= nkb ? r - nkb : r);
      };
      // The weights are constant during a step: the first ring of weight tiles is requested before
      // the wait for the previous kernel, whose output is this kernel's activation block.
      const int pre = min(nkb, Cfg::STAGES);
      for (int it = 0; it < pre; ++it) load_w(it, block_of(it));
      pdl_wait();
      for (int it = 0; it < pre; ++it) tma_load_2d(sX + it * Cfg::X_BYTES, &tm_x, &full[it], block_of(it) * BK, 0);
      for (int it = pre; it < nkb; ++it) {
        const int s = it % Cfg::STAGES;
        const uint32_t ph = (it / Cfg::STAGES) & 1;
        if (!mbar_wait(&empty[s], ph ^ 1, abort_flag)) break;
        const int kb = block_of(it);
        load_w(s, kb);
        tma_load_2d(sX + s * Cfg::X_BYTES, &tm_x, &full[s], kb * BK, 0);
      }
    }
  } else if (warp == 1) {
    // A slab of in_proj or up/gate is 128 products of 128 x BPAD x 16, 40-49 clocks of tensor core each: what bounded this
    // loop was their issue, 165 clocks a product (11 us a slab, longer than its bytes take).  One elected lane, descriptors
    // as 32-bit sums and a counter instead of a remainder: 28 layers at one sequence 1195 -> 1034 us a step, 8 layers at 64
    // 570 -> 522, 16 layers of width 1280 at one 534 -> 457.
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(TM, BPAD, false, false);
      bool ok = true;
      int s = 0;
      uint32_t ph = 0;
      const uint32_t a0 = desc_low_sw128(smem_u32(sW)), b0 = desc_low_sw128(smem_u32(sX));
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[s], ph, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t a = a0 + s * (W_BYTES / 16), b = b0 + s * (Cfg::X_BYTES / 16);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16_low(tmem, a + 2 * k, b + 2 * k, idesc, k != 0 || kb != kb0 ? 1u : 0u);
        umma_commit(&empty[s]);
        if (++s == Cfg::STAGES) {
          s = 0;
          ph ^= 1;
        }
      }
      if (ok) umma_commit(tfull);
    }
  } else {
    const bool ok = kb1 > kb0 && mbar_wait_warp(tfull, 0, abort_flag);
    decode_epilogue<BPAD, EPI>(p, tmem, warp, lane, n0, sG, ok);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 8);
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, Cfg::TMEM_COLS);
  }
}

// --------------------------------------------------------------------------- residual + norm
// One CTA per sequence.  x (FP32 residual stream, [batch, d]) is updated in place:
//   token != null : x = table[token[b]]           (embedding gather)
//   partial != null: x += sum_s partial[s][b]     (split-K partials of the previous projection)
//   scale != null : x = x * (1 + scale) + bias    (depth modulation of the layer that follows)
// then out = BF16(x * rsqrt(mean(x^2) + eps) * w).
// This form takes rows of more than 2048 columns; shorter ones, those of every configuration, take the one below.
__global__ void __launch_bounds__(256)
decode_reduce_norm_kernel(float* x, const float* partial, int splits,
                          const long long* token, const float* table, int vocab,
                          const float* scale, const float* bias, const float* w,
                          float eps, int d, int batch, __nv_bfloat16* __restrict__ out) {
  __shared__ float red[8];
  pdl_launch_dependents();
  const int b = blockIdx.x;
  // The first HELD * 1024 columns stay in registers between the two passes; what no kernel of the step writes (norm weight,
  // modulation) is requested before the wait for the previous kernel.
  constexpr int HELD = 2;
  float4 held[HELD], ww[HELD], sc[HELD], bi[HELD];
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c >= d) continue;
    if (out != nullptr) ww[i] = *reinterpret_cast<const float4*>(w + c);
    if (scale != nullptr) {
      sc[i] = *reinterpret_cast<const float4*>(scale + c);
      bi[i] = *reinterpret_cast<const float4*>(bias + c);
    }
  }
  pdl_wait();
  float* xr = x + static_cast<size_t>(b) * d;
  const float* src = xr;
  if (token != nullptr) {
    long long id = token[b];
    if (id < 0) id = 0;
    if (id >= vocab) id = vocab - 1;
    src = table + static_cast<size_t>(id) * d;
  }
  auto updated = [&](int c, const float4& m, const float4& a) {
    float4 v = *reinterpret_cast<const float4*>(src + c);
    for (int s = 0; s < splits; ++s) {
      const float4 q = *reinterpret_cast<const float4*>(partial + (static_cast<size_t>(s) * batch + b) * d + c);
      v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
    }
    if (scale != nullptr) v = modulated(v, m, a);
    *reinterpret_cast<float4*>(xr + c) = v;
    return v;
  };
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c >= d) continue;
    held[i] = updated(c, sc[i], bi[i]);
    ss = __fadd_rn(ss, square_sum(held[i]));
  }
  for (int c = (threadIdx.x + HELD * 256) * 4; c < d; c += 256 * 4) {
    float4 m = make_float4(0.f, 0.f, 0.f, 0.f), a = m;
    if (scale != nullptr) {
      m = *reinterpret_cast<const float4*>(scale + c);
      a = *reinterpret_cast<const float4*>(bias + c);
    }
    const float4 v = updated(c, m, a);
    ss = __fadd_rn(ss, square_sum(v));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float total = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) total += red[i];
  const float rstd = rsqrtf(total / static_cast<float>(d) + eps);
  if (out == nullptr) return;
  auto emit = [&](int c, const float4& v, const float4& g) {
    uint2 o;
    o.x = pack_bf16x2(v.x * rstd * g.x, v.y * rstd * g.y);
    o.y = pack_bf16x2(v.z * rstd * g.z, v.w * rstd * g.w);
    *reinterpret_cast<uint2*>(out + static_cast<size_t>(b) * d + c) = o;
  };
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    const int c = (threadIdx.x + i * 256) * 4;
    if (c < d) emit(c, held[i], ww[i]);
  }
  for (int c = (threadIdx.x + HELD * 256) * 4; c < d; c += 256 * 4)  // xr: this thread's own stores
    emit(c, *reinterpret_cast<const float4*>(xr + c), *reinterpret_cast<const float4*>(w + c));
}

// The same for rows of at most 2048 columns, four to a thread of 512: the partials of a thread are one or two rounds of loads
// instead of one for every few of them, and this kernel is nothing but the time of its loads, twice in every layer.  The
// squares are added as the kernel above adds them (its thread t owns the columns of threads t and t + 256 here).
// A step of 28 layers at one sequence 1042 -> 1013 us, of 8 layers at 16 365 -> 353, at 64 522 -> 507, of 16 layers of width 1280 459 -> 431.
__global__ void __launch_bounds__(512)
decode_reduce_norm_short_kernel(float* x, const float* partial, int splits, const long long* token, const float* table,
                                int vocab, const float* scale, const float* bias, const float* w, float eps, int d, int batch,
                                __nv_bfloat16* __restrict__ out) {
  __shared__ float upper[256], red[8];
  pdl_launch_dependents();
  const int b = blockIdx.x, c = threadIdx.x * 4;
  const bool mine = c < d;
  float4 ww = make_float4(0.f, 0.f, 0.f, 0.f), sc = ww, bi = ww, v = ww;
  if (mine) {
    if (out != nullptr) ww = *reinterpret_cast<const float4*>(w + c);
    if (scale != nullptr) {
      sc = *reinterpret_cast<const float4*>(scale + c);
      bi = *reinterpret_cast<const float4*>(bias + c);
    }
  }
  pdl_wait();
  float* xr = x + static_cast<size_t>(b) * d;
  if (mine) {
    const float* src = xr;
    if (token != nullptr) {
      long long id = token[b];
      if (id < 0) id = 0;
      if (id >= vocab) id = vocab - 1;
      src = table + static_cast<size_t>(id) * d;
    }
    v = *reinterpret_cast<const float4*>(src + c);
    for (int s0 = 0; s0 < splits; s0 += 8) {
      float4 q[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s0 + s < splits) q[s] = *reinterpret_cast<const float4*>(partial + (static_cast<size_t>(s0 + s) * batch + b) * d + c);
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s0 + s < splits) { v.x += q[s].x; v.y += q[s].y; v.z += q[s].z; v.w += q[s].w; }
    }
    if (scale != nullptr) v = modulated(v, sc, bi);
    *reinterpret_cast<float4*>(xr + c) = v;
  }
  if (out == nullptr) return;
  const float square = square_sum(v);
  if (threadIdx.x >= 256) upper[threadIdx.x - 256] = square;
  __syncthreads();
  if (threadIdx.x < 256) {
    float ss = __fadd_rn(square, upper[threadIdx.x]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  }
  __syncthreads();
  float total = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) total += red[i];
  const float rstd = rsqrtf(total / static_cast<float>(d) + eps);
  if (mine)
    *reinterpret_cast<uint2*>(out + static_cast<size_t>(b) * d + c) =
        make_uint2(pack_bf16x2(v.x * rstd * ww.x, v.y * rstd * ww.y), pack_bf16x2(v.z * rstd * ww.z, v.w * rstd * ww.w));
}

// --------------------------------------------------------------------------- residual + norm + projection
// One sequence: the two kernels above in front of the projection that reads their result, in its launch.  Every CTA adds the
// partials and forms the norm itself, as its MMAs' operand, and CTA 0 leaves the residual for the next such launch (in another
// buffer: the others may still be reading).  A boundary of the chain and a round trip through memory less, twice a layer,
// against reading (1 + splits) rows of x per CTA from L2.  Bit for bit what the two launches give: same order of partials, squares
// and k blocks.  d <= 2048.  A step of 28 layers of width 2048 1018 -> 940 us, of 16 of 1280 416 -> 375, of 8 of 256 122 -> 112.  With more sequences
// those reads take longer than the boundary did: two 1023 -> 1065 and 418 -> 442, eight 1056 -> 1654.  Rings of four to six stages, with
// which a CTA would fit beside its predecessor's: 1064-1153.
struct DecodeNormParams {
  const float* x;         // residual before, [d]; behind a token its embedding row instead
  float* x_out;           // and after
  const float* partial;   // [splits, d]
  int splits;
  const long long* token;
  const float* table;
  int vocab;
  const float *scale, *bias, *w;
  float eps;
};
constexpr int NORM_WORKERS = 512;                 // of four columns each
constexpr int NORM_THREADS = 64 + NORM_WORKERS;   // warp 0 TMA, warp 1 MMA + TMEM, warps 2..17 the norm, 2..5 of them the epilogue
constexpr int NORM_STAGES = 8;
constexpr int NORM_ROUND = 12;                    // partials of a thread requested at once

// The MMA's operand has 16 rows, of which the sequence is the first: eight rows of 128 bytes per k block, taken twice.
static int norm_gemm_smem(int d) { return NORM_STAGES * dec::W_BYTES + d / dec::BK * 1024 + 1024 + 256; }

template <int EPI>
__global__ void __launch_bounds__(NORM_THREADS, 1)
decode_norm_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const DecodeGemmParams p, const DecodeNormParams q) {
  using namespace dec;
  constexpr int BPAD = 16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ float upper[256], red[8];
  const int total_kb = p.k / BK;
  uint8_t* sW = smem;
  uint8_t* sX = smem + NORM_STAGES * W_BYTES;    // [k block][8 rows][64 columns]; the columns of D that rows 1.. give are not read
  float* sG = reinterpret_cast<float*>(sW);      // written only after the last MMA has read the ring
  uint64_t* bars = reinterpret_cast<uint64_t*>(sX + total_kb * 1024);
  uint64_t* full = bars;
  uint64_t* empty = bars + NORM_STAGES;
  uint64_t* tfull = bars + 2 * NORM_STAGES;
  uint64_t* ready = tfull + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NORM_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(ready, NORM_WORKERS / 32);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 32);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();

  const int slab = blockIdx.x, n0 = slab * (EPI == 2 ? 64 : TM);
  const int rot = static_cast<int>((blockIdx.x * 5u) % static_cast<unsigned>(total_kb));   // as decode_gemm_kernel walks them
  auto block_of = [&](int it) {
    const int r = it + rot;
    return r >= total_kb ? r - total_kb : r;
  };

  if (warp == 0) {
    if (lane == 0) {
      // Weights only, which no kernel of the step writes: as far ahead as the ring goes, whatever the predecessor does.
      for (int it = 0; it < total_kb; ++it) {
        const int s = it % NORM_STAGES, kb = block_of(it);
        if (!mbar_wait(&empty[s], ((it / NORM_STAGES) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(&full[s], W_BYTES);
        if (p.packed) {
          tma_load_2d(sW + s * W_BYTES, &tm_w, &full[s], 0, (slab * total_kb + kb) * TM);
        } else {
          tma_load_2d(sW + s * W_BYTES, &tm_w, &full[s], kb * BK, n0);
          if (EPI == 2) tma_load_2d(sW + s * W_BYTES + 64 * 128, &tm_w, &full[s], kb * BK, p.n + n0);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(TM, BPAD, false, false);
      const uint32_t a0 = desc_low_sw128(smem_u32(sW)), b0 = desc_low_sw128(smem_u32(sX));
      bool ok = mbar_wait(ready, 0, abort_flag);
      int s = 0;
      uint32_t ph = 0;
      for (int it = 0; it < total_kb && ok; ++it) {
        ok = mbar_wait(&full[s], ph, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t a = a0 + s * (W_BYTES / 16), b = b0 + block_of(it) * (1024 / 16);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16_low<0>(tmem, a + 2 * k, b + 2 * k, idesc, (it | k) != 0 ? 1u : 0u);
        umma_commit(&empty[s]);
        if (++s == NORM_STAGES) {
          s = 0;
          ph ^= 1;
        }
      }
      if (ok) umma_commit(tfull);
    }
  } else {
    const int worker = threadIdx.x - 64, c = worker * 4;
    float4 weight = make_float4(0.f, 0.f, 0.f, 0.f), scale = weight, bias = weight;
    if (c < p.k) {   // what no kernel of the step writes is requested before the wait
      weight = *reinterpret_cast<const float4*>(q.w + c);
      if (q.scale != nullptr) {
        scale = *reinterpret_cast<const float4*>(q.scale + c);
        bias = *reinterpret_cast<const float4*>(q.bias + c);
      }
    }
    pdl_wait();
    const bool mine = c < p.k;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mine) {
      const float* src = q.x;
      if (q.token != nullptr) {
        long long id = *q.token;
        if (id < 0) id = 0;
        if (id >= q.vocab) id = q.vocab - 1;
        src = q.table + static_cast<size_t>(id) * p.k;
      }
      v = *reinterpret_cast<const float4*>(src + c);
      for (int s0 = 0; s0 < q.splits; s0 += NORM_ROUND) {
        float4 part[NORM_ROUND];
#pragma unroll
        for (int s = 0; s < NORM_ROUND; ++s)
          if (s0 + s < q.splits) part[s] = *reinterpret_cast<const float4*>(q.partial + static_cast<size_t>(s0 + s) * p.k + c);
#pragma unroll
        for (int s = 0; s < NORM_ROUND; ++s)
          if (s0 + s < q.splits) { v.x += part[s].x; v.y += part[s].y; v.z += part[s].z; v.w += part[s].w; }
      }
      if (q.scale != nullptr) v = modulated(v, scale, bias);
      if (blockIdx.x == 0 && q.x_out != nullptr) *reinterpret_cast<float4*>(q.x_out + c) = v;
    }
    const float square = square_sum(v);   // added as decode_reduce_norm_short_kernel adds them
    if (worker >= 256) upper[worker - 256] = square;
    asm volatile("bar.sync 2, 512;" ::: "memory");
    if (worker < 256) {
      float ss = __fadd_rn(square, upper[worker]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) red[worker >> 5] = ss;
    }
    asm volatile("bar.sync 2, 512;" ::: "memory");
    if (mine) {
      float total = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) total += red[i];
      const float rstd = rsqrtf(total / static_cast<float>(p.k) + q.eps);
      *reinterpret_cast<uint2*>(sX + (c >> 6) * 1024 + (c & 63) * 2) =
          make_uint2(pack_bf16x2(v.x * rstd * weight.x, v.y * rstd * weight.y), pack_bf16x2(v.z * rstd * weight.z, v.w * rstd * weight.w));
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(ready);
    if (warp < 6) {
      const bool ok = mbar_wait_warp(tfull, 0, abort_flag);
      decode_epilogue<BPAD, EPI>(p, tmem, warp, lane, n0, sG, ok);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 8);
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 32);
  }
}

// --------------------------------------------------------------------------- attention step
// One CTA of 128 threads per (sequence, head); head_dim 64, chunk 128.
// qkvgu: [batch, 5*d] BF16 (q | k | v | gate | u); caches kc/vc/uc: [batch, H, 128, 64] BF16;
// mixed: [batch, H, 64, 64] BF16 (mix*fast + (1-mix)*slow); rope: [128, 32] (cos, sin);
// y: [batch, d] BF16.  `pos_ptr` is the in-chunk position (device scalar, so that one captured
// graph serves every position).
__global__ void __launch_bounds__(128)
decode_attn_kernel(const __nv_bfloat16* qkvgu, __nv_bfloat16* kc, __nv_bfloat16* vc,
                   __nv_bfloat16* uc,
                   const __nv_bfloat16* mixed, const float2* rope,
                   const long long* pos_ptr, int H, int d, __nv_bfloat16* __restrict__ y, bool early) {
  constexpr int HD = 64, C = 128;
  __shared__ float sq[HD], sk[HD], sp[C], sl[16][HD + 1], sm[16][HD + 1], sred[4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x % H, b = blockIdx.x / H;
  pdl_launch_dependents();
  if (!early) pdl_wait();
  int pos = static_cast<int>(*pos_ptr);
  pos = pos < 0 ? 0 : (pos >= C ? C - 1 : pos);
  const __nv_bfloat16* row = qkvgu + static_cast<size_t>(b) * 5 * d + h * HD;
  const size_t cache = (static_cast<size_t>(b) * H + h) * C * HD;
  // Thread (rg, jg) owns columns 8*jg .. 8*jg+7 of the rows rg, rg+16, ... of the K and V caches and of M: a warp
  // instruction reads four whole 128-byte rows.  Every load the step needs from the caches is issued here, before
  // the RoPE of the new token, so that the three dependent phases below (scores, softmax, P.V) wait for memory once.
  // `early`: they are issued before the wait for the previous kernel, too, and run under the tail of the projection.  Only
  // `row` is this step's; the position, the cache rows before it and M are what was there before the step, and a replay of
  // the graph that captured the step starts after everything before it.  A step launched kernel by kernel has no such
  // start: its first kernels may be resident while the kernel that writes the position still runs, and only the wait
  // makes that visible.  48 steps of 28 layers at batch 1, a prompt of 100 tokens included: 62.6 -> 61.2 ms; 40 of 8 layers
  // at batch 64: 29.9 -> 29.5.
  const int jg = tid & 7, rg = tid >> 3;
  uint4 kreg[C / 16], vreg[C / 16], mreg[HD / 16];
#pragma unroll
  for (int it = 0; it < C / 16; ++it) {
    const int c = rg + it * 16;
    if (c < pos) {
      kreg[it] = *reinterpret_cast<const uint4*>(kc + cache + static_cast<size_t>(c) * HD + jg * 8);
      vreg[it] = *reinterpret_cast<const uint4*>(vc + cache + static_cast<size_t>(c) * HD + jg * 8);
    }
  }
  const __nv_bfloat16* mbase = mixed + (static_cast<size_t>(b) * H + h) * HD * HD;
#pragma unroll
  for (int it = 0; it < HD / 16; ++it) mreg[it] = *reinterpret_cast<const uint4*>(mbase + (rg + it * 16) * HD + jg * 8);
  const float2 cs = rope[pos * 32 + lane];
  if (early) pdl_wait();
#pragma unroll
  for (int it = 0; it < C / 16; ++it)
    if (rg + it * 16 == pos) vreg[it] = *reinterpret_cast<const uint4*>(row + 2 * d + jg * 8);  // the new token's own value row
  // RoPE (adjacent pairs) of q and k; append k, v, u at `pos`
  if (tid < 32) {
    const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + 2 * tid));
    const float2 k = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + d + 2 * tid));
    // round through BF16 as the cached / batched path does
    const __nv_bfloat162 qr = __floats2bfloat162_rn(q.x * cs.x - q.y * cs.y, q.y * cs.x + q.x * cs.y);
    const __nv_bfloat162 kr = __floats2bfloat162_rn(k.x * cs.x - k.y * cs.y, k.y * cs.x + k.x * cs.y);
    const float2 qf = __bfloat1622float2(qr), kf = __bfloat1622float2(kr);
    sq[2 * tid] = qf.x; sq[2 * tid + 1] = qf.y;
    sk[2 * tid] = kf.x; sk[2 * tid + 1] = kf.y;
    *reinterpret_cast<__nv_bfloat162*>(kc + cache + static_cast<size_t>(pos) * HD + 2 * tid) = kr;
  } else if (tid < 64) {
    const int t = tid - 32;
    *reinterpret_cast<__nv_bfloat162*>(vc + cache + static_cast<size_t>(pos) * HD + 2 * t) =
        *reinterpret_cast<const __nv_bfloat162*>(row + 2 * d + 2 * t);
  } else if (tid < 96) {
    const int t = tid - 64;
    *reinterpret_cast<__nv_bfloat162*>(uc + cache + static_cast<size_t>(pos) * HD + 2 * t) =
        *reinterpret_cast<const __nv_bfloat162*>(row + 4 * d + 2 * t);
  }
  __syncthreads();
  // scores: the eight lanes of a row group each hold an eighth of q . k[c]; key `pos` is the new token's own
  {
    float qv[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) qv[t] = sq[jg * 8 + t];
#pragma unroll
    for (int it = 0; it < C / 16; ++it) {
      const int c = rg + it * 16;
      float acc = 0.f;
      if (c < pos) {
        const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&kreg[it]);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = __bfloat1622float2(pb[t]);
          acc += qv[2 * t] * f.x + qv[2 * t + 1] * f.y;
        }
      } else if (c == pos) {
#pragma unroll
        for (int t = 0; t < 8; ++t) acc += qv[t] * sk[jg * 8 + t];
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      if (jg == 0) sp[c] = acc * 0.125f;
    }
  }
  __syncthreads();
  const float score = tid <= pos ? sp[tid] : -INFINITY;
  float m = score;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) sred[warp] = m;
  __syncthreads();
  m = fmaxf(fmaxf(sred[0], sred[1]), fmaxf(sred[2], sred[3]));
  const float e = tid <= pos ? __expf(score - m) : 0.f;
  float s = e;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __syncthreads();
  if (lane == 0) sred[warp] = s;
  sp[tid] = e;
  __syncthreads();
  const float inv = 1.f / (sred[0] + sred[1] + sred[2] + sred[3]);
  // local = sum_c p[c] V[c] and memory = q . M from the rows already in registers; the 16 row groups are then
  // summed through shared memory.
  {
    float accl[8], accm[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) { accl[t] = 0.f; accm[t] = 0.f; }
#pragma unroll
    for (int it = 0; it < C / 16; ++it) {
      const int c = rg + it * 16;
      if (c <= pos) {
        const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&vreg[it]);
        const float pc = sp[c];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = __bfloat1622float2(pb[t]);
          accl[2 * t] += pc * f.x;
          accl[2 * t + 1] += pc * f.y;
        }
      }
    }
#pragma unroll
    for (int it = 0; it < HD / 16; ++it) {
      const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&mreg[it]);
      const float qi = sq[rg + it * 16];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = __bfloat1622float2(pb[t]);
        accm[2 * t] += qi * f.x;
        accm[2 * t + 1] += qi * f.y;
      }
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      sl[rg][jg * 8 + t] = accl[t];
      sm[rg][jg * 8 + t] = accm[t];
    }
  }
  __syncthreads();
  if (tid < HD) {
    float local = 0.f, mem = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      local += sl[r][tid];
      mem += sm[r][tid];
    }
    local *= inv;
    mem *= 0.125f;
    const float g = sigmoid_fast(__bfloat162float(row[3 * d + tid]));
    y[static_cast<size_t>(b) * d + h * HD + tid] = __float2bfloat16(g * local + (1.f - g) * mem);
  }
}

// --------------------------------------------------------------------------- attention step, row-per-thread scores
// The earlier form of decode_attn_kernel (WS_DECODE_ATTN=rows): thread c computes the score of key c from its own
// 128-byte cache row, and the value / memory rows are read after the softmax.  Fewer registers (more CTAs per SM),
// three dependent memory phases.  One CTA of 128 threads per (sequence, head); head_dim 64, chunk 128.
// qkvgu: [batch, 5*d] BF16 (q | k | v | gate | u); caches kc/vc/uc: [batch, H, 128, 64] BF16;
// mixed: [batch, H, 64, 64] BF16 (mix*fast + (1-mix)*slow); rope: [128, 32] (cos, sin);
// y: [batch, d] BF16.  `pos_ptr` is the in-chunk position (device scalar, so that one captured
// graph serves every position).
__global__ void __launch_bounds__(128)
decode_attn_rows_kernel(const __nv_bfloat16* qkvgu, __nv_bfloat16* kc, __nv_bfloat16* vc,
                   __nv_bfloat16* uc,
                   const __nv_bfloat16* mixed, const float2* rope,
                   const long long* pos_ptr, int H, int d, __nv_bfloat16* __restrict__ y, bool) {
  constexpr int HD = 64, C = 128;
  __shared__ float sq[HD], sk[HD], sp[C], sl[16][HD + 1], sm[16][HD + 1], sred[4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x % H, b = blockIdx.x / H;
  pdl_launch_dependents();
  pdl_wait();
  int pos = static_cast<int>(*pos_ptr);
  pos = pos < 0 ? 0 : (pos >= C ? C - 1 : pos);
  const __nv_bfloat16* row = qkvgu + static_cast<size_t>(b) * 5 * d + h * HD;
  const size_t cache = (static_cast<size_t>(b) * H + h) * C * HD;
  // RoPE (adjacent pairs) of q and k; append k, v, u at `pos`
  if (tid < 32) {
    const float2 cs = rope[pos * 32 + tid];
    const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + 2 * tid));
    const float2 k = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + d + 2 * tid));
    // round through BF16 as the cached / batched path does
    const __nv_bfloat162 qr = __floats2bfloat162_rn(q.x * cs.x - q.y * cs.y, q.y * cs.x + q.x * cs.y);
    const __nv_bfloat162 kr = __floats2bfloat162_rn(k.x * cs.x - k.y * cs.y, k.y * cs.x + k.x * cs.y);
    const float2 qf = __bfloat1622float2(qr), kf = __bfloat1622float2(kr);
    sq[2 * tid] = qf.x; sq[2 * tid + 1] = qf.y;
    sk[2 * tid] = kf.x; sk[2 * tid + 1] = kf.y;
    *reinterpret_cast<__nv_bfloat162*>(kc + cache + static_cast<size_t>(pos) * HD + 2 * tid) = kr;
  } else if (tid < 64) {
    const int t = tid - 32;
    *reinterpret_cast<__nv_bfloat162*>(vc + cache + static_cast<size_t>(pos) * HD + 2 * t) =
        *reinterpret_cast<const __nv_bfloat162*>(row + 2 * d + 2 * t);
  } else if (tid < 96) {
    const int t = tid - 64;
    *reinterpret_cast<__nv_bfloat162*>(uc + cache + static_cast<size_t>(pos) * HD + 2 * t) =
        *reinterpret_cast<const __nv_bfloat162*>(row + 4 * d + 2 * t);
  }
  __syncthreads();
  // scores: thread c owns key c
  float score = -INFINITY;
  if (tid <= pos) {
    float acc = 0.f;
    if (tid == pos) {
#pragma unroll
      for (int i = 0; i < HD; ++i) acc += sq[i] * sk[i];
    } else {
      const uint4* kr = reinterpret_cast<const uint4*>(kc + cache + static_cast<size_t>(tid) * HD);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint4 v = kr[j];
        const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = __bfloat1622float2(pb[t]);
          acc += sq[j * 8 + 2 * t] * f.x + sq[j * 8 + 2 * t + 1] * f.y;
        }
      }
    }
    score = acc * 0.125f;
  }
  float m = score;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) sred[warp] = m;
  __syncthreads();
  m = fmaxf(fmaxf(sred[0], sred[1]), fmaxf(sred[2], sred[3]));
  const float e = tid <= pos ? __expf(score - m) : 0.f;
  float s = e;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __syncthreads();
  if (lane == 0) sred[warp] = s;
  sp[tid] = e;
  __syncthreads();
  const float inv = 1.f / (sred[0] + sred[1] + sred[2] + sred[3]);
  // local = sum_c p[c] V[c] and memory = q . M in one pass of wide loads: thread (rg, jg) owns
  // columns 8*jg .. 8*jg+7 and the rows rg, rg+16, ... of V (keys) and of M; the 16 row groups
  // are then summed through shared memory.
  {
    const int jg = tid & 7, rg = tid >> 3;
    float accl[8], accm[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) { accl[t] = 0.f; accm[t] = 0.f; }
#pragma unroll
    for (int it = 0; it < C / 16; ++it) {
      const int c = rg + it * 16;
      if (c <= pos) {
        const uint4 v = (c == pos) ? *reinterpret_cast<const uint4*>(row + 2 * d + jg * 8)
                                   : *reinterpret_cast<const uint4*>(vc + cache + static_cast<size_t>(c) * HD + jg * 8);
        const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&v);
        const float pc = sp[c];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = __bfloat1622float2(pb[t]);
          accl[2 * t] += pc * f.x;
          accl[2 * t + 1] += pc * f.y;
        }
      }
    }
    const __nv_bfloat16* mbase = mixed + (static_cast<size_t>(b) * H + h) * HD * HD;
#pragma unroll
    for (int it = 0; it < HD / 16; ++it) {
      const int i = rg + it * 16;
      const uint4 v = *reinterpret_cast<const uint4*>(mbase + i * HD + jg * 8);
      const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&v);
      const float qi = sq[i];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = __bfloat1622float2(pb[t]);
        accm[2 * t] += qi * f.x;
        accm[2 * t + 1] += qi * f.y;
      }
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      sl[rg][jg * 8 + t] = accl[t];
      sm[rg][jg * 8 + t] = accm[t];
    }
  }
  __syncthreads();
  if (tid < HD) {
    float local = 0.f, mem = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      local += sl[r][tid];
      mem += sm[r][tid];
    }
    local *= inv;
    mem *= 0.125f;
    const float g = sigmoid_fast(__bfloat162float(row[3 * d + tid]));
    y[static_cast<size_t>(b) * d + h * HD + tid] = __float2bfloat16(g * local + (1.f - g) * mem);
  }
}

// --------------------------------------------------------------------------- attention step, a warp per head
// The same for many (sequence, head) pairs: one warp each, four to a CTA.  With a CTA of 128 threads to a pair, 64 sequences x 32 heads are
// 3.5 rounds of CTAs that meet at six barriers each; here they are one round of warps that meet at none.  Cache rows come 32 at a time,
// only as many as the position asks for, and the softmax is carried from one 32 to the next (running maximum and sum).  Lane (rg, jg) has
// the 16-byte piece jg of the rows rg, rg + 4, ...: eight lanes hold a score, all of them its weight, and the sums over rows meet at the end.
// The first 32 rows of K and V and half of M are requested ahead of the wait where that is allowed (`early`, as above).
// us a layer with a CTA per pair -> so, at positions 20, 70 and 120: 64 sequences x 32 heads 13.5 -> 7.2, 16.4 -> 12.4, 20.3 -> 15.8; 32 sequences
// 7.4 -> 5.4, 8.9 -> 9.7, 10.4 -> 11.9; one 2.6 -> 2.4, 2.6 -> 4.1, 2.6 -> 4.8.  So from more than two rounds of CTAs (four to an SM) on, where
// the third begins; at 20, 70, 100 and 127 there: 38 sequences x 32 heads 9.0 -> 6.1, 10.6 -> 10.6, 11.8 -> 12.7, 12.9 -> 13.0; 40 9.5 -> 6.2,
// 11.5 -> 10.8, 12.8 -> 12.7, 14.0 -> 13.0; 48 10.4 -> 6.5, 12.6 -> 11.0, 13.9 -> 13.2, 15.1 -> 13.7; 60 x 20 heads as 38 x 32.  Over the positions
// of a chunk that is a gain at every count; only at 38 and around position 100 is a step slower by 8 % of this kernel.
constexpr int ATTN_WARPS = 4;
constexpr int ATTN_ROUND = CHIP_SMS * 4;   // CTAs of decode_attn_kernel that the chip holds at once

__global__ void __launch_bounds__(32 * ATTN_WARPS, 4)
decode_attn_warp_kernel(const __nv_bfloat16* qkvgu, __nv_bfloat16* kc, __nv_bfloat16* vc, __nv_bfloat16* uc, const __nv_bfloat16* mixed,
                        const float2* rope, const long long* pos_ptr, int H, int d, int items, __nv_bfloat16* __restrict__ y, bool early) {
  constexpr int HD = 64, C = 128;
  __shared__ __align__(16) float query[ATTN_WARPS][HD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, jg = lane & 7, rg = lane >> 3;
  const int item = blockIdx.x * ATTN_WARPS + warp;
  pdl_launch_dependents();
  if (!early) pdl_wait();
  if (item >= items) return;
  const int h = item % H, b = item / H;
  int pos = static_cast<int>(*pos_ptr);
  pos = pos < 0 ? 0 : (pos >= C ? C - 1 : pos);
  const __nv_bfloat16* row = qkvgu + static_cast<size_t>(b) * 5 * d + h * HD;
  const size_t cache = static_cast<size_t>(item) * C * HD;
  const __nv_bfloat16* memory = mixed + static_cast<size_t>(item) * HD * HD;
  uint4 k[8], v[8], m[8];
  auto request = [&](uint4 (&to)[8], const __nv_bfloat16* from, int r0) {   // rows from `pos` on as zeros
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = r0 + rg + 4 * i;
      to[i] = make_uint4(0u, 0u, 0u, 0u);
      if (r < pos) to[i] = *reinterpret_cast<const uint4*>(from + cache + r * HD + jg * 8);
    }
  };
  auto request_memory = [&](int r0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) m[i] = *reinterpret_cast<const uint4*>(memory + (r0 + rg + 4 * i) * HD + jg * 8);
  };
  request(k, kc, 0);
  request(v, vc, 0);
  request_memory(0);
  const float2 cs = rope[pos * 32 + lane];
  if (early) pdl_wait();
  // RoPE (adjacent pairs) of q and k, rounded through BF16 as the cached / batched path does; k, v, u are appended at `pos`
  const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(row);
  const float2 q = __bfloat1622float2(pairs[lane]), kk = __bfloat1622float2(pairs[d / 2 + lane]);
  const __nv_bfloat162 v_new = pairs[d + lane], u_new = pairs[2 * d + lane];
  const uint4 own = *reinterpret_cast<const uint4*>(row + 2 * d + jg * 8), gate = *reinterpret_cast<const uint4*>(row + 3 * d + jg * 8);
  const __nv_bfloat162 qr = __floats2bfloat162_rn(q.x * cs.x - q.y * cs.y, q.y * cs.x + q.x * cs.y);
  const __nv_bfloat162 kr = __floats2bfloat162_rn(kk.x * cs.x - kk.y * cs.y, kk.y * cs.x + kk.x * cs.y);
  const float2 qf = __bfloat1622float2(qr), kf = __bfloat1622float2(kr);
  query[warp][2 * lane] = qf.x;
  query[warp][2 * lane + 1] = qf.y;
  *reinterpret_cast<__nv_bfloat162*>(kc + cache + pos * HD + 2 * lane) = kr;
  *reinterpret_cast<__nv_bfloat162*>(vc + cache + pos * HD + 2 * lane) = v_new;
  *reinterpret_cast<__nv_bfloat162*>(uc + cache + pos * HD + 2 * lane) = u_new;
  float top = qf.x * kf.x + qf.y * kf.y;   // the new token's own score, with which the softmax begins
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top += __shfl_xor_sync(0xffffffffu, top, o);
  top *= 0.125f;
  __syncwarp();
  float qv[8];
  *reinterpret_cast<float4*>(qv) = *reinterpret_cast<const float4*>(&query[warp][jg * 8]);
  *reinterpret_cast<float4*>(qv + 4) = *reinterpret_cast<const float4*>(&query[warp][jg * 8 + 4]);
  float sum = 1.f, local[8], mem[8];
  const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&own);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float2 f = __bfloat1622float2(ob[t]);
    local[2 * t] = rg == 0 ? f.x : 0.f;
    local[2 * t + 1] = rg == 0 ? f.y : 0.f;
    mem[2 * t] = mem[2 * t + 1] = 0.f;
  }
  auto add_memory = [&](int r0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&m[i]);
      const float qi = query[warp][r0 + rg + 4 * i];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = __bfloat1622float2(pb[t]);
        mem[2 * t] += qi * f.x;
        mem[2 * t + 1] += qi * f.y;
      }
    }
  };
  add_memory(0);
  request_memory(32);
  for (int r0 = 0; r0 < pos; r0 += 32) {
    float s[8], most = top;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&k[i]);
      float acc = 0.f;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = __bfloat1622float2(pb[t]);
        acc += qv[2 * t] * f.x + qv[2 * t + 1] * f.y;
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      s[i] = r0 + rg + 4 * i < pos ? acc * 0.125f : -INFINITY;
      most = fmaxf(most, s[i]);
    }
    request(k, kc, r0 + 32);   // under the sum over V, as V's next rows are under the scores
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 8));
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 16));
    const float keep = __expf(top - most);
    top = most;
    float here = 0.f;
#pragma unroll
    for (int t = 0; t < 8; ++t) local[t] *= keep;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float e = __expf(s[i] - most);
      here += e;
      const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = __bfloat1622float2(pb[t]);
        local[2 * t] += e * f.x;
        local[2 * t + 1] += e * f.y;
      }
    }
    request(v, vc, r0 + 32);
    here += __shfl_xor_sync(0xffffffffu, here, 8);
    here += __shfl_xor_sync(0xffffffffu, here, 16);
    sum = sum * keep + here;
  }
  add_memory(32);
#pragma unroll
  for (int t = 0; t < 8; ++t) {
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      local[t] += __shfl_xor_sync(0xffffffffu, local[t], o);
      mem[t] += __shfl_xor_sync(0xffffffffu, mem[t], o);
    }
  }
  if (rg == 0) {
    const float inv = 1.f / sum;
    const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gate);
    uint4 out;
    uint32_t* w = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 gf = __bfloat1622float2(gb[t]);
      const float g0 = sigmoid_fast(gf.x), g1 = sigmoid_fast(gf.y);
      w[t] = pack_bf16x2(g0 * (local[2 * t] * inv) + (1.f - g0) * (mem[2 * t] * 0.125f),
                         g1 * (local[2 * t + 1] * inv) + (1.f - g1) * (mem[2 * t + 1] * 0.125f));
    }
    *reinterpret_cast<uint4*>(y + static_cast<size_t>(b) * d + h * HD + jg * 8) = out;
  }
}

// --------------------------------------------------------------------------- end of a chunk
// The 128 positions of a finished chunk enter the memories: write = tanh(K)^T tanh(U) / 128, then
// fast <- df fast + (1 - df) write, slow alike, mixed <- BF16(mix fast + (1 - mix) slow).  One CTA per (sequence, head),
// a thread owns 4 x 4 of the 64 x 64 elements; K and U go through shared memory as FP32 tanh, everything is read and
// written once (217 MB per layer at 64 sequences x 32 heads, about as long as the 2.1 GFLOP take on the CUDA cores).
// 48 steps of 28 layers at batch 1 with one end of a chunk: 64.9 ms with a dozen framework operations per layer, 63.1 so.
constexpr int CHUNK_END_SMEM = 2 * 128 * 64 * 4;

__global__ void __launch_bounds__(256)
decode_chunk_end_kernel(const __nv_bfloat16* kc, const __nv_bfloat16* uc,
                        float* fast, float* slow, __nv_bfloat16* __restrict__ mixed,
                        const float* fast_keep, const float* slow_keep,
                        const float* mix_of, int H) {
  constexpr int HD = 64, C = 128;
  extern __shared__ float chunk_smem[];
  float* sK = chunk_smem;
  float* sU = chunk_smem + C * HD;
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, h = blockIdx.x % H;
  const size_t cache = static_cast<size_t>(blockIdx.x) * C * HD, state = static_cast<size_t>(blockIdx.x) * HD * HD;
#pragma unroll
  for (int i = 0; i < C * HD / 8 / 256; ++i) {
    const int at = (tid + i * 256) * 8;
    const uint4 kv = *reinterpret_cast<const uint4*>(kc + cache + at), uv = *reinterpret_cast<const uint4*>(uc + cache + at);
    const __nv_bfloat162* kb = reinterpret_cast<const __nv_bfloat162*>(&kv);
    const __nv_bfloat162* ub = reinterpret_cast<const __nv_bfloat162*>(&uv);
#pragma unroll
    for (int t = 0; t < 4; t += 2) {
      const float2 k0 = __bfloat1622float2(kb[t]), k1 = __bfloat1622float2(kb[t + 1]);
      const float2 u0 = __bfloat1622float2(ub[t]), u1 = __bfloat1622float2(ub[t + 1]);
      *reinterpret_cast<float4*>(sK + at + 2 * t) = make_float4(tanh_fast(k0.x), tanh_fast(k0.y), tanh_fast(k1.x), tanh_fast(k1.y));
      *reinterpret_cast<float4*>(sU + at + 2 * t) = make_float4(tanh_fast(u0.x), tanh_fast(u0.y), tanh_fast(u1.x), tanh_fast(u1.y));
    }
  }
  __syncthreads();
  const int x0 = (tid >> 4) * 4, y0 = (tid & 15) * 4;
  float acc[4][4] = {};
#pragma unroll 4
  for (int c = 0; c < C; ++c) {
    const float4 a = *reinterpret_cast<const float4*>(sK + c * HD + x0), b = *reinterpret_cast<const float4*>(sU + c * HD + y0);
    const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i][0] += av[i] * b.x;
      acc[i][1] += av[i] * b.y;
      acc[i][2] += av[i] * b.z;
      acc[i][3] += av[i] * b.w;
    }
  }
  const float df = fast_keep[h], ds = slow_keep[h], mix = mix_of[h];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t at = state + static_cast<size_t>(x0 + i) * HD + y0;
    float4 f = *reinterpret_cast<const float4*>(fast + at), s = *reinterpret_cast<const float4*>(slow + at);
    float* fv = reinterpret_cast<float*>(&f);
    float* sv = reinterpret_cast<float*>(&s);
    float m[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float w = acc[i][j] * (1.f / C);
      fv[j] = df * fv[j] + (1.f - df) * w;
      sv[j] = ds * sv[j] + (1.f - ds) * w;
      m[j] = mix * fv[j] + (1.f - mix) * sv[j];
    }
    *reinterpret_cast<float4*>(fast + at) = f;
    *reinterpret_cast<float4*>(slow + at) = s;
    *reinterpret_cast<uint2*>(mixed + at) = make_uint2(pack_bf16x2(m[0], m[1]), pack_bf16x2(m[2], m[3]));
  }
}

// --------------------------------------------------------------------------- greedy pick
// One CTA per sequence: token[b] = argmax of logits[b, :] (the lowest index among equal maxima, as torch.argmax
// picks), written where the next step's embedding gather reads it and into column `*cursor` of the history
// [batch, capacity]; CTA 0 then advances the in-chunk position and the cursor.  With this kernel as the last node of
// the step graph a greedy decode needs nothing from the host between steps.
__global__ void __launch_bounds__(256)
decode_pick_kernel(const float* logits, int vocab, long long* __restrict__ token,
                   long long* __restrict__ history, int capacity, long long* cursor, long long* pos) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float best_v[8];
  __shared__ int best_i[8];
  const int b = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* row = logits + static_cast<size_t>(b) * vocab;
  float v = -INFINITY;
  int at = 0x7fffffff;
  for (int c = threadIdx.x * 4; c < vocab; c += 256 * 4) {  // vocab % 4 == 0 (checked by the caller)
    const float4 q = *reinterpret_cast<const float4*>(row + c);
    const float e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (e[j] > v || (e[j] == v && c + j < at)) {
        v = e[j];
        at = c + j;
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, at, o);
    if (ov > v || (ov == v && oi < at)) {
      v = ov;
      at = oi;
    }
  }
  if (lane == 0) {
    best_v[warp] = v;
    best_i[warp] = at;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w)
      if (best_v[w] > v || (best_v[w] == v && best_i[w] < at)) {
        v = best_v[w];
        at = best_i[w];
      }
    if (at == 0x7fffffff) at = 0;  // a row of NaNs: any token, as long as it is a valid one
    const long long column = *cursor;
    token[b] = at;
    if (history != nullptr && column < capacity) history[static_cast<size_t>(b) * capacity + column] = at;
  }
  // every CTA has read the cursor before CTA 0 may advance it: CTA 0 waits for the others' arrival count
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned arrived = atomicAdd(reinterpret_cast<unsigned*>(cursor + 1), 1u) + 1u;
    if (arrived == gridDim.x) {
      *reinterpret_cast<unsigned*>(cursor + 1) = 0u;
      *cursor += 1;
      *pos += 1;
    }
  }
}

// Launch with the programmatic-stream-serialization attribute (WS_DECODE_PDL=0 launches normally).
template <typename... KArgs, typename... Args>
static cudaError_t launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  Args... args) {
  static const bool chained = [] {
    const char* e = std::getenv("WS_DECODE_PDL");
    return e == nullptr || e[0] != '0';
  }();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

template <int BPAD, int EPI, int DEPTH>
static int launch_decode_gemm_depth(const CUtensorMap& tw, const CUtensorMap& tx, const DecodeGemmParams& p, dim3 grid,
                                    cudaStream_t stream) {
  static bool configured = false;
  auto kern = decode_gemm_kernel<BPAD, EPI, DEPTH>;
  using Cfg = DecodeCfg<BPAD, DEPTH>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM) != cudaSuccess) return -20;
    configured = true;
  }
  const cudaError_t err = launch_chained(kern, grid, dim3(dec::THREADS), Cfg::SMEM, stream, tw, tx, p);
  ws_count_launch();
  return err == cudaSuccess ? 0 : -21;
}

// WS_DECODE_STAGES=9 is the deepest ring that fits (217 KiB at batch 64).  WS_DECODE_STAGES=4 selects the shallow ring (two CTAs per SM); the default is 8
// (one CTA per SM): measured at batch 64, 2.14 ms per token with 8 stages against 2.42 with 4 (2.21 with twice the K splits) -- the bytes a
// CTA keeps in flight matter more than letting the next launch become resident early.  The switch is for batches that are padded to 16
// and 64 rows; those padded to 32 and 48 have 8 stages, prompts past 64 tokens what fits.
static int decode_ring_depth() {
  static const int depth = [] {
    const char* e = std::getenv("WS_DECODE_STAGES");
    return e != nullptr && e[0] == '4' ? 4 : e != nullptr && e[0] == '9' ? 9 : 8;
  }();
  return depth;
}

template <int EPI>
static int launch_norm_gemm(const CUtensorMap& tw, const DecodeGemmParams& p, const DecodeNormParams& q, int slabs, cudaStream_t stream) {
  static bool configured = false;
  auto kern = decode_norm_gemm_kernel<EPI>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, norm_gemm_smem(2048)) != cudaSuccess) return -20;
    configured = true;
  }
  const cudaError_t err = launch_chained(kern, dim3(slabs), dim3(NORM_THREADS), norm_gemm_smem(p.k), stream, tw, p, q);
  ws_count_launch();
  return err == cudaSuccess ? 0 : -21;
}

template <int BPAD, int EPI>
static int launch_decode_gemm(const CUtensorMap& tw, const CUtensorMap& tx, const DecodeGemmParams& p, dim3 grid,
                              cudaStream_t stream) {
  // up to 16 KiB of X go to a stage, and the ring is what fits
  if constexpr (BPAD > 64) return launch_decode_gemm_depth<BPAD, EPI, BPAD <= 96 ? 7 : 6>(tw, tx, p, grid, stream);
  else if constexpr (BPAD != 16 && BPAD != 64) return launch_decode_gemm_depth<BPAD, EPI, 8>(tw, tx, p, grid, stream);
  else switch (decode_ring_depth()) {
    case 4: return launch_decode_gemm_depth<BPAD, EPI, 4>(tw, tx, p, grid, stream);
    case 9: return launch_decode_gemm_depth<BPAD, EPI, 9>(tw, tx, p, grid, stream);
    default: return launch_decode_gemm_depth<BPAD, EPI, 8>(tw, tx, p, grid, stream);
  }
}

template <int BPAD>
static int launch_decode_epilogue(int epilogue, const CUtensorMap& tw, const CUtensorMap& tx, const DecodeGemmParams& p, dim3 grid,
                                  cudaStream_t stream) {
  switch (epilogue) {
    case 0: return launch_decode_gemm<BPAD, 0>(tw, tx, p, grid, stream);
    case 1: return launch_decode_gemm<BPAD, 1>(tw, tx, p, grid, stream);
    case 2: return launch_decode_gemm<BPAD, 2>(tw, tx, p, grid, stream);
    default: return launch_decode_gemm<BPAD, 3>(tw, tx, p, grid, stream);
  }
}

}  // namespace ws

using namespace ws;

// Number of K splits ws_decode_gemm uses for an [n x k] weight (the caller sizes the FP32 partial
// buffer as splits * batch * n floats when the result is > 1).
extern "C" int ws_decode_gemm_splits(int n, int k) {
  // CTAs a split-K launch aims for: one per SM by default; WS_DECODE_SPLIT_CTAS overrides (two CTAs fit per SM
  // with the 4-stage ring)
  static const int target = [] {
    const char* e = std::getenv("WS_DECODE_SPLIT_CTAS");
    const int v = e != nullptr ? std::atoi(e) : 0;
    return v >= 16 && v <= 1184 ? v : 148;
  }();
  const int slabs = (n + dec::TM - 1) / dec::TM;
  const int total_kb = (k + dec::BK - 1) / dec::BK;
  int splits = target / (slabs > 0 ? slabs : 1);
  if (splits < 1) splits = 1;
  while (splits > 1 && total_kb / splits < 4) --splits;
  const int per = (total_kb + splits - 1) / splits;
  return (total_kb + per - 1) / per;  // no split is empty
}

// epilogue: 0 BF16 out [batch, ldo]; 1 FP32 split-K partials [splits, batch, n] (splits from
// ws_decode_gemm_splits); 2 SwiGLU, W is [2n, k] (up rows then gate rows), BF16 out [batch, ldo];
// 3 FP32 out [batch, ldo].  batch <= 128; k % 8 == 0.
// packed != 0: W is the tile-by-tile copy [slabs][ceil(k/64)][128][64] (zero padded; for SwiGLU a tile
// holds 64 up rows followed by their 64 gate rows), so that every TMA load reads 16 contiguous KiB
// instead of 128 row pieces of 128 bytes that lie a full weight row apart.
extern "C" int ws_decode_gemm(const void* w, const void* x, int n, int k, int batch, int epilogue, void* out, int ldo,
                              int* error_flag, int packed, cudaStream_t stream) {
  if (n <= 0 || k <= 0 || batch <= 0 || batch > 128 || k % 8 != 0 || epilogue < 0 || epilogue > 3) return -1;
  if (epilogue == 2 && n % 64 != 0) return -2;
  CUtensorMap tw, tx;
  const int w_rows = epilogue == 2 ? 2 * n : n;
  int rc;
  if (packed) {
    const uint64_t tiles = (uint64_t)(epilogue == 2 ? n / 64 : (n + dec::TM - 1) / dec::TM) * ((k + dec::BK - 1) / dec::BK);
    rc = make_map_bf16(&tw, w, dec::BK, tiles * dec::TM, dec::BK, dec::BK, dec::TM);
  } else {
    rc = make_map_bf16(&tw, w, k, w_rows, k, dec::BK, epilogue == 2 ? 64 : dec::TM);
  }
  if (rc) return rc;
  // The rows of X are padded to what the MMA and its operand's tile take: every CTA reads all of X, so a step of 8 layers is 334 us at 16
  // sequences and, padded to 64, 397 at 17 and 414 at 32; padded to 32 353 and 390, at 48 450 -> 434.
  const int bpad = batch <= 16 ? 16 : batch <= 32 ? 32 : batch <= 48 ? 48 : batch <= 64 ? 64 : batch <= 96 ? 96 : 128;
  rc = make_map_bf16(&tx, x, k, batch, k, dec::BK, bpad);
  if (rc) return rc;
  DecodeGemmParams p;
  p.n = n; p.k = k; p.batch = batch; p.packed = packed; p.out = out; p.ldo = ldo; p.error_flag = error_flag;
  const int total_kb = (k + dec::BK - 1) / dec::BK;
  int splits = 1;
  if (epilogue == 1) splits = ws_decode_gemm_splits(n, k);
  p.kb_per_split = (total_kb + splits - 1) / splits;
  const int slabs = epilogue == 2 ? n / 64 : (n + dec::TM - 1) / dec::TM;
  const dim3 grid(slabs, splits);
  switch (bpad) {
    case 16: return launch_decode_epilogue<16>(epilogue, tw, tx, p, grid, stream);
    case 32: return launch_decode_epilogue<32>(epilogue, tw, tx, p, grid, stream);
    case 48: return launch_decode_epilogue<48>(epilogue, tw, tx, p, grid, stream);
    case 64: return launch_decode_epilogue<64>(epilogue, tw, tx, p, grid, stream);
    case 96: return launch_decode_epilogue<96>(epilogue, tw, tx, p, grid, stream);
    default: return launch_decode_epilogue<128>(epilogue, tw, tx, p, grid, stream);
  }
}

extern "C" int ws_decode_reduce_norm(float* x, const float* partial, int splits, const long long* token,
                                     const float* table, int vocab, const float* scale, const float* bias,
                                     const float* w, float eps, int d, int batch, void* out, cudaStream_t stream) {
  if (d % 4 != 0 || batch <= 0 || (splits > 0 && partial == nullptr)) return -1;
  const bool brief = d <= 2048;
  const cudaError_t err = launch_chained(brief ? decode_reduce_norm_short_kernel : decode_reduce_norm_kernel, dim3(batch),
                                         dim3(brief ? 512 : 256), 0, stream, x, partial, splits,
                                         token, table, vocab, scale, bias, w, eps, d, batch,
                                         static_cast<__nv_bfloat16*>(out));
  ws_count_launch();
  return err == cudaSuccess ? 0 : -21;
}

extern "C" int ws_decode_norm_gemm(const float* x, float* x_out, const float* partial, int splits, const long long* token,
                                   const float* table, int vocab, const float* scale, const float* bias, const float* norm, float eps,
                                   const void* w, int n, int d, int epilogue, void* out, int ldo, int* error_flag, int packed,
                                   cudaStream_t stream) {
  if (d < dec::BK || d > 4 * NORM_WORKERS || d % dec::BK != 0 || n <= 0 || splits < 0 ||
      (epilogue != 0 && epilogue != 2 && epilogue != 3) || (splits > 0 && partial == nullptr) || x_out == x)
    return -1;
  if (epilogue == 2 && n % 64 != 0) return -2;
  const int slabs = epilogue == 2 ? n / 64 : (n + dec::TM - 1) / dec::TM;
  CUtensorMap tw;
  const int rc = packed ? make_map_bf16(&tw, w, dec::BK, (uint64_t)slabs * (d / dec::BK) * dec::TM, dec::BK, dec::BK, dec::TM)
                        : make_map_bf16(&tw, w, d, epilogue == 2 ? 2 * n : n, d, dec::BK, epilogue == 2 ? 64 : dec::TM);
  if (rc) return rc;
  DecodeGemmParams p;
  p.n = n; p.k = d; p.batch = 1; p.kb_per_split = d / dec::BK; p.packed = packed; p.out = out; p.ldo = ldo; p.error_flag = error_flag;
  DecodeNormParams q;
  q.x = x; q.x_out = x_out; q.partial = partial; q.splits = splits; q.token = token; q.table = table; q.vocab = vocab;
  q.scale = scale; q.bias = bias; q.w = norm; q.eps = eps;
  switch (epilogue) {
    case 0: return launch_norm_gemm<0>(tw, p, q, slabs, stream);
    case 2: return launch_norm_gemm<2>(tw, p, q, slabs, stream);
    default: return launch_norm_gemm<3>(tw, p, q, slabs, stream);
  }
}

extern "C" int ws_decode_attn(const void* qkvgu, void* kc, void* vc, void* uc, const void* mixed, const float* rope,
                              const long long* pos, int batch, int H, int d, void* y, int early, cudaStream_t stream) {
  if (d != H * 64 || batch <= 0) return -1;
  // WS_DECODE_ATTN=rows selects the row-per-thread form of the kernel
  static const bool rows_form = [] {
    const char* e = std::getenv("WS_DECODE_ATTN");
    return e != nullptr && e[0] == 'r';
  }();
  const int items = batch * H;
  cudaError_t err;
  // (the warp form stores eight outputs at a time)
  if (!rows_form && items > 2 * ATTN_ROUND && reinterpret_cast<uintptr_t>(y) % 16 == 0)
    err = launch_chained(decode_attn_warp_kernel, dim3((items + ATTN_WARPS - 1) / ATTN_WARPS), dim3(32 * ATTN_WARPS), 0, stream,
                         static_cast<const __nv_bfloat16*>(qkvgu), static_cast<__nv_bfloat16*>(kc), static_cast<__nv_bfloat16*>(vc),
                         static_cast<__nv_bfloat16*>(uc), static_cast<const __nv_bfloat16*>(mixed), reinterpret_cast<const float2*>(rope), pos,
                         H, d, items, static_cast<__nv_bfloat16*>(y), early != 0);
  else
    err = launch_chained(
        rows_form ? decode_attn_rows_kernel : decode_attn_kernel, dim3(items), dim3(128), 0, stream,
        static_cast<const __nv_bfloat16*>(qkvgu),
        static_cast<__nv_bfloat16*>(kc), static_cast<__nv_bfloat16*>(vc), static_cast<__nv_bfloat16*>(uc),
        static_cast<const __nv_bfloat16*>(mixed), reinterpret_cast<const float2*>(rope), pos, H, d,
        static_cast<__nv_bfloat16*>(y), early != 0);
  ws_count_launch();
  return err == cudaSuccess ? 0 : -21;
}

// token [batch] int64 = argmax(logits [batch, vocab] FP32); also stored in history[:, cursor[0]] (history may be
// NULL); then pos[0] += 1 and cursor[0] += 1.  cursor is two int64 words: the column, and a word of scratch (zero).
extern "C" int ws_decode_pick(const float* logits, int batch, int vocab, long long* token, long long* history,
                              int capacity, long long* cursor, long long* pos, cudaStream_t stream) {
  if (batch <= 0 || vocab <= 0 || vocab % 4 != 0) return -1;
  const cudaError_t err = launch_chained(decode_pick_kernel, dim3(batch), dim3(256), 0, stream, logits, vocab, token, history,
                                         capacity, cursor, pos);
  ws_count_launch();
  return err == cudaSuccess ? 0 : -21;
}

extern "C" int ws_decode_chunk_end(const void* kc, const void* uc, float* fast, float* slow, void* mixed,
                                   const float* fast_keep, const float* slow_keep, const float* mix, int batch, int H,
                                   cudaStream_t stream) {
  if (batch <= 0 || H <= 0) return -1;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(decode_chunk_end_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHUNK_END_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  const cudaError_t err = launch_chained(decode_chunk_end_kernel, dim3(batch * H), dim3(256), CHUNK_END_SMEM, stream,
                                         static_cast<const __nv_bfloat16*>(kc), static_cast<const __nv_bfloat16*>(uc), fast,
                                         slow, static_cast<__nv_bfloat16*>(mixed), fast_keep, slow_keep, mix, H);
  ws_count_launch();
  return err == cudaSuccess ? 0 : -21;
}
