// Backward kernels of the middle of a WarpState core (chunk 128, head_dim 64).
//
//   dstate_kernel       : dState[b,n,h] = rope(Q)^T (dy * (1 - sigmoid(g)) / 8)           (64x64)
//   memory_scan_bwd     : reverse scan over chunks: dState -> dWrites (BF16) and the partial
//                         gradients of the three per-head scalars (decays, mix); FP32, fixed order
//   attn_bwd_kernel     : per (batch, chunk, head) tile recomputes S / P / O / Mem, then
//                            dP = dlocal V^T, dV = P^T dlocal, dS = P*(dP - D)/8,
//                            dQr = dS Kr + dmem State^T, dKr = dS^T Qr,
//                            dtK = tU dW^T, dtU = tK dW   (write path),
//                         and writes the packed gradient [tokens, 5d] = (dQ, dK, dV, dGate, dU)
//                         with the RoPE transpose and the tanh / sigmoid derivatives applied --
//                         the region the reference handles with flash-attention backward plus
//                         its "paired backward layout" kernels (ops/backward_layout.py:114-210).
//
// All ten matrix products of the tile run on tcgen05 with accumulators in TMEM; two threads share
// a token row in every element-wise stage.
#include <type_traits>
#include "ws_ptx.cuh"
#include "ws_api.h"
#include "ws_launch.h"
#include "attention_common.cuh"

namespace ws {

extern "C" void ws_count_launch(void);

// =============================================================================== dState
// smem: Qr 16K | dy -> dmem/8 16K | gate, then the FP32 result 16K | bars
constexpr int DS_SMEM = 3 * TILE_BYTES + 1024 + 128;

__global__ void __launch_bounds__(128, 4)
dstate_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_dy,
              const __grid_constant__ CUtensorMap tm_out, const float2* rope, int T, int H, int d,
              int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem;
  uint8_t* sD = smem + TILE_BYTES;
  uint8_t* sG = smem + 2 * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 3 * TILE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int n_chunks = T / CHUNK;
  const int tile = blockIdx.x;
  const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
  const int row0 = b * T + n * CHUNK;

  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 64);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  if (tid == 0) {
    mbar_expect_tx(&bars[0], 3 * TILE_BYTES);
    tma_load_2d(sQ, &tm_qkvgu, &bars[0], h * HD, row0);
    tma_load_2d(sD, &tm_dy, &bars[0], h * HD, row0);
    tma_load_2d(sG, &tm_qkvgu, &bars[0], 3 * d + h * HD, row0);
  }
  bool ok = mbar_wait(&bars[0], 0, abort_flag);
  if (ok) {
    rope_tanh_row(sQ, tid, rope, true, false);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint4* p = reinterpret_cast<uint4*>(tile_chunk(sD, tid, j));
      uint4 v = *p;
      const uint4 gq = *reinterpret_cast<const uint4*>(tile_chunk(sG, tid, j));
      uint32_t* w = reinterpret_cast<uint32_t*>(&v);
      const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gq);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 dyv = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w[t]));
        const float2 gf = __bfloat1622float2(gb[t]);
        w[t] = pack_bf16x2(dyv.x * (1.f - sigmoid_f(gf.x)) * 0.125f, dyv.y * (1.f - sigmoid_f(gf.y)) * 0.125f);
      }
      *p = v;
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (warp == 0 && elect_one() && ok) {
    constexpr uint32_t idesc = make_idesc_bf16(128, 64, true, true);
#pragma unroll
    for (int k = 0; k < CHUNK / 16; ++k)
      umma_bf16(tmem, make_smem_desc_sw128(smem_u32(sQ) + k * 2048, 0, 1024),
                make_smem_desc_sw128(smem_u32(sD) + k * 2048, 0, 1024), idesc, k > 0);
    umma_commit(&bars[1]);
  }
  ok = ok && mbar_wait(&bars[1], 0, abort_flag);
  tc_fence_after_sync();
  if (warp < 2) {
    // Row `tid` of the [64 x 64] FP32 result goes to two swizzled [64 x 32] half tiles (the gate tile's
    // space), and each warp stores its 32 rows of both halves by TMA.
#pragma unroll
    for (int c = 0; c < HD; c += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const int col = c + j;
        uint8_t* dst = sG + (col >> 5) * 8192 + tid * 128 + ((((col & 31) >> 2) ^ (tid & 7)) << 4);
        *reinterpret_cast<float4*>(dst) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]),
                                                      __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if ((tid & 31) == 0) {
      if (ok) {
        tma_store_2d(&tm_out, sG + warp * 4096, 0, tile * HD + warp * 32);
        tma_store_2d(&tm_out, sG + 8192 + warp * 4096, 32, tile * HD + warp * 32);
        tma_store_commit();
      }
      tma_store_wait_read0();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 4);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 64);
  }
}

// =============================================================================== dState, streaming form
// dstate_kernel as one persistent CTA per SM with specialised warps, exactly as chunk_writes_stream_kernel
// (attention_fwd.cu): producer warp with a 3-stage ring of (Q, dy, gate) tiles, 512 workers that turn Q into rope(Q)
// and dy into dy (1 - sigmoid(gate)) / 8 in place, MMA issue into a double-buffered accumulator, two epilogue warps
// that store the FP32 [64 x 64] result by TMA.  Bit-identical to dstate_kernel.
constexpr int DSS_STAGES = 3;
constexpr int DSS_THREADS = 19 * 32;
constexpr int DSS_SMEM = DSS_STAGES * 3 * TILE_BYTES + 2 * 16384 + 1024 + 256;

__global__ void __launch_bounds__(DSS_THREADS, 1)
dstate_stream_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_dy,
                     const __grid_constant__ CUtensorMap tm_out, const float2* rope, int T, int H, int d,
                     int tiles, int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* ring = smem;                                   // stage s: Q, dy, gate at s * 48 KiB
  uint8_t* staging = smem + DSS_STAGES * 3 * TILE_BYTES;  // two FP32 [64 x 64] tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + 2 * 16384);
  uint64_t* full = bars;                    // [4] tile landed
  uint64_t* empty = bars + DSS_STAGES;       // [4] MMAs have read the stage
  uint64_t* tfull = bars + 2 * DSS_STAGES;   // [2] accumulator complete
  uint64_t* tempty = tfull + 2;             // [2] accumulator read by both epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_chunks = T / CHUNK;

  if (tid == 0) {
    for (int s = 0; s < DSS_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 2);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_qkvgu);
    tma_prefetch_desc(&tm_dy);
    tma_prefetch_desc(&tm_out);
  }
  if (warp == 16) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  const int first = blockIdx.x, step = gridDim.x;
  if (warp == 18) {
    if (lane == 0) {
      int i = 0;
      for (int tile = first; tile < tiles; tile += step, ++i) {
        const int s = i % DSS_STAGES;
        if (!mbar_wait(&empty[s], ((i / DSS_STAGES) & 1) ^ 1, abort_flag)) break;
        const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
        const int row0 = b * T + n * CHUNK;
        mbar_expect_tx(&full[s], 3 * TILE_BYTES);
        tma_load_2d(ring + s * 3 * TILE_BYTES, &tm_qkvgu, &full[s], h * HD, row0);
        tma_load_2d(ring + s * 3 * TILE_BYTES + TILE_BYTES, &tm_dy, &full[s], h * HD, row0);
        tma_load_2d(ring + s * 3 * TILE_BYTES + 2 * TILE_BYTES, &tm_qkvgu, &full[s], 3 * d + h * HD, row0);
      }
    }
  } else if (warp < 16) {
    const int r = tid & 127, q = tid >> 7;   // row, and which two of its eight pieces
    float2 cs[8];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int t = 0; t < 4; ++t) cs[j * 4 + t] = rope[((q * 2 + j) * 4 + t) * CHUNK + r];
    int i = 0;
    for (int tile = first; tile < tiles; tile += step, ++i) {
      const int s = i % DSS_STAGES;
      uint8_t* sQ = ring + s * 3 * TILE_BYTES;
      uint8_t* sD = sQ + TILE_BYTES;
      uint8_t* sGate = sD + TILE_BYTES;
      const bool ok = mbar_wait(&full[s], (i / DSS_STAGES) & 1, abort_flag);
      if (ok) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint4* pq = reinterpret_cast<uint4*>(tile_chunk(sQ, r, q * 2 + j));
          uint4* pd = reinterpret_cast<uint4*>(tile_chunk(sD, r, q * 2 + j));
          uint4 qv = *pq, dv = *pd;
          const uint4 gv = *reinterpret_cast<const uint4*>(tile_chunk(sGate, r, q * 2 + j));
          uint32_t* qw = reinterpret_cast<uint32_t*>(&qv);
          uint32_t* dw = reinterpret_cast<uint32_t*>(&dv);
          const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&qw[t]));
            const float2 c = cs[j * 4 + t];
            const float2 qr = rope_rotate(x, c);
            qw[t] = pack_bf16x2(qr.x, qr.y);
            const float2 dyv = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&dw[t]));
            const float2 gf = __bfloat1622float2(gb[t]);
            dw[t] = pack_bf16x2(dyv.x * (1.f - sigmoid_f(gf.x)) * 0.125f, dyv.y * (1.f - sigmoid_f(gf.y)) * 0.125f);
          }
          *pq = qv;
          *pd = dv;
        }
      }
      fence_proxy_async_smem();
      // the workers' barrier doubles as their vote: if any of them gave up on the tile, all leave together
      uint32_t any_bad;
      asm volatile(
          "{\n"
          ".reg .pred p, q;\n"
          "setp.ne.u32 q, %1, 0;\n"
          "bar.red.or.pred p, 2, 512, q;\n"
          "selp.u32 %0, 1, 0, p;\n"
          "}\n"
          : "=r"(any_bad)
          : "r"(ok ? 0u : 1u)
          : "memory");
      if (any_bad) break;
      if (warp == 0 && elect_one()) {
        const int buf = i & 1;
        if (mbar_wait(&tempty[buf], ((i >> 1) & 1) ^ 1, abort_flag)) {
          tc_fence_after_sync();
          // D[128 x 64]: rows 0..63 = Qr^T (dmem / 8); rows 64..127 repeat them (zero stride between A's atoms)
          constexpr uint32_t idesc = make_idesc_bf16(128, 64, true, true);
#pragma unroll
          for (int k = 0; k < CHUNK / 16; ++k)
            umma_bf16(tmem + buf * 64, make_smem_desc_sw128(smem_u32(sQ) + k * 2048, 0, 1024),
                      make_smem_desc_sw128(smem_u32(sD) + k * 2048, 0, 1024), idesc, k > 0);
          umma_commit(&empty[s]);
          umma_commit(&tfull[buf]);
        }
      }
    }
  } else {  // warps 16, 17: accumulator lanes 0..31 and 32..63
    const int ew = warp - 16, row = ew * 32 + lane;
    int i = 0;
    for (int tile = first; tile < tiles; tile += step, ++i) {
      const int buf = i & 1;
      uint32_t landed = 0;
      if (lane == 0) landed = mbar_wait(&tfull[buf], (i >> 1) & 1, abort_flag) ? 1u : 0u;
      if (__shfl_sync(0xffffffffu, landed, 0) == 0u) break;   // the whole warp leaves together
      tc_fence_after_sync();
      uint8_t* st = staging + buf * 16384;
      if (lane == 0) tma_store_wait_read0();   // the store issued two tiles ago from this buffer has read it
      __syncwarp();
#pragma unroll
      for (int c = 0; c < HD; c += 16) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(tmem + buf * 64 + (static_cast<uint32_t>(ew * 32) << 16) + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const int col = c + j;
          uint8_t* dst = st + (col >> 5) * 8192 + row * 128 + ((((col & 31) >> 2) ^ (row & 7)) << 4);
          *reinterpret_cast<float4*>(dst) =
              make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        }
      }
      tc_fence_before_sync();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&tempty[buf]);   // this warp's 32 lanes of the accumulator have been read
        tma_store_2d(&tm_out, st + ew * 4096, 0, tile * HD + ew * 32);
        tma_store_2d(&tm_out, st + 8192 + ew * 4096, 32, tile * HD + ew * 32);
        tma_store_commit();
      }
    }
    if (lane == 0) tma_store_wait_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 4);
  if (warp == 16) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 128);
  }
}

// =============================================================================== reverse scan
// The reverse scan needs the state every chunk saw.  Those are recomputed from the writes in groups of
// SCAN_GROUP chunks: a first pass keeps the state at every group boundary, then the groups are walked
// from the last to the first, each re-running its forward recurrence into registers before its reverse
// part.  One group (sequences up to 2048 tokens) skips the first pass.
constexpr int SCAN_GROUP = 16;
constexpr int SCAN_MAX_GROUPS = 16;
constexpr int SCAN_MAX_CHUNKS = SCAN_GROUP * SCAN_MAX_GROUPS;  // 32768 tokens per sequence

// dstate [B,N,H,4096] FP32 (gradient of the mixed state read by chunk n), writes [B,N,H,4096] FP32
// -> dwrites [B,N,H,4096] BF16 and partial sums [B*H*16][3] of d(fast decay), d(slow decay), d(mix).
// A thread owns two neighbouring state elements of each unit (SCAN_THREADS threads' worth), one operand of its packed
// instructions.  Bound by DRAM: 10 bytes an element and chunk.  Persistent, three CTAs per SM: while a warp walks one group of
// chunks, what it needs of its next group (the next unit's, after the last) is on its way into its own places in shared memory,
// so no barrier of the block is needed.  Such a copy has to pass L1 by: with 192 KiB taken as shared memory L1 is so small that
// copies through it (8 bytes a thread) waited for its lines, 24.7 us at 4 x 16 chunks x 32 heads.  Now 16.5 us (84 MB, 5.1 TB/s),
// 8 x 16 x 32 29.1 (5.8 TB/s), 2 x 7 x 20 5.0; a block per unit that loaded into registers, computed and left took 27.1, 50.2
// and 5.8.  Which product of a sum is rounded on its own, and the order of the sums, are that form's, bit for bit; it costs nothing (16.6, 29.3, 5.0).
constexpr int SCAN_THREADS = 128;
constexpr int SCAN_VEC = 2;
constexpr int SCAN_SLOT = 2 * SCAN_GROUP * SCAN_THREADS;   // pairs: the writes and the state gradients of a group
constexpr int SCAN_SMEM = 2 * SCAN_SLOT * 8;

// Two FP32 numbers in a register pair, the first in the low half; every operation rounds each of them once.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair2(float lo, float hi) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 halves(f32x2 v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// sum + (x.x y.x + x.y y.y): one chain for both elements, so that the sums, too, are those of the form without packed instructions
__device__ __forceinline__ void add_products(float& sum, float2 x, float2 y) {
  sum = __fadd_rn(sum, __fmaf_rn(x.x, y.x, __fmul_rn(x.y, y.y)));
}

__global__ void __launch_bounds__(SCAN_THREADS, 3)
memory_scan_bwd_kernel(const float* dstate, const float* writes,
                       const float* fast_logit, const float* slow_logit,
                       const float* mix_logit, __nv_bfloat16* __restrict__ dwrites,
                       float* __restrict__ partials, int B, int N, int H) {
  extern __shared__ __align__(16) uint8_t scan_smem[];
  __shared__ float red[2][3][SCAN_THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int units = B * H * 16;
  const int groups = (N + SCAN_GROUP - 1) / SCAN_GROUP;
  const int pieces = 2 * groups - 1;   // of a unit: the first pass over all groups but the last, then every group, the last one first
  const size_t chunk_stride = static_cast<size_t>(H) * 4096;
  f32x2* const mine = reinterpret_cast<f32x2*>(scan_smem) + tid;
  auto place = [&](int unit) {   // chunk 0 of this warp's elements
    const int head = unit >> 4;
    return (static_cast<size_t>(head / H) * N * H + head % H) * 4096 + (unit & 15) * (SCAN_THREADS * SCAN_VEC) + warp * (32 * SCAN_VEC);
  };
  auto group_of = [&](int piece) { return piece < groups - 1 ? piece : pieces - 1 - piece; };
  // a warp fetches its own 64 elements of every chunk, one half of it those of the writes, the other those of the gradients
  const int half = lane >> 4;
  const float* const from = half == 0 ? writes : dstate;
  const uint32_t into = smem_u32(scan_smem) + half * (SCAN_GROUP * SCAN_THREADS * 8) + warp * 256 + (lane & 15) * 16;
  auto request = [&](int unit, int piece, int slot) {
    const int n0 = group_of(piece) * SCAN_GROUP;
    const int count = half == 0 || piece >= groups - 1 ? min(SCAN_GROUP, N - n0) : 0;
    const float* at = from + place(unit) + n0 * chunk_stride + (lane & 15) * 4;
    const uint32_t to = into + slot * (SCAN_SLOT * 8);
#pragma unroll
    for (int i = 0; i < SCAN_GROUP; ++i) {
      if (i < count) cp_async_16(to + i * (SCAN_THREADS * 8), at);
      at += chunk_stride;
      asm volatile("" : "+l"(at));   // one address that moves on, not sixteen kept from unit to unit
    }
  };
  f32x2 start_f[SCAN_MAX_GROUPS], start_s[SCAN_MAX_GROUPS];
  float next_fast = 0.f, next_slow = 0.f, next_mix = 0.f;
  auto request_logits = [&](int unit) {
    const int h = (unit >> 4) % H;
    next_fast = fast_logit[h];
    next_slow = slow_logit[h];
    next_mix = mix_logit[h];
  };
  int slot = 0, turn = 0;
  if (blockIdx.x < units) {
    request_logits(blockIdx.x);
    request(blockIdx.x, 0, 0);
  }
  cp_async_commit();
  for (int unit = blockIdx.x; unit < units; unit += gridDim.x, turn ^= 1) {
    const float df1 = 1.f / (1.f + expf(-next_fast)), ds1 = 1.f / (1.f + expf(-next_slow)), mix1 = 1.f / (1.f + expf(-next_mix));
    const f32x2 df = pair2(df1, df1), ds = pair2(ds1, ds1), mix = pair2(mix1, mix1), minus = pair2(-1.f, -1.f);
    const f32x2 rf = pair2(1.f - df1, 1.f - df1), rs = pair2(1.f - ds1, 1.f - ds1), rm = pair2(1.f - mix1, 1.f - mix1);
    __nv_bfloat16* const out = dwrites + place(unit) + lane * SCAN_VEC;
    f32x2 f = 0, s = 0;
    // a, bb: gradients of the fast and slow state AFTER the chunk being visited (F_{n+1}, S_{n+1})
    f32x2 a = 0, bb = 0;
    float g_df = 0.f, g_ds = 0.f, g_mix = 0.f;
#pragma unroll 1
    for (int piece = 0; piece < pieces; ++piece, slot ^= 1) {
      __syncwarp();   // every lane has done with the slot that is filled next
      const int to_come = piece + 1 < pieces ? unit : unit + static_cast<int>(gridDim.x);
      if (to_come < units) {
        if (to_come != unit) request_logits(to_come);
        request(to_come, to_come == unit ? piece + 1 : 0, slot ^ 1);
      }
      cp_async_commit();
      cp_async_wait<1>();   // this piece is there, the next one on its way
      __syncwarp();         // and the other lanes' part of it
      const int g = group_of(piece), n0 = g * SCAN_GROUP;
      const int count = min(SCAN_GROUP, N - n0);
      const f32x2 *W = mine + slot * SCAN_SLOT, *G = W + SCAN_GROUP * SCAN_THREADS;
      auto advance = [&](f32x2 w) {
        f = fma2(df, f, mul2(rf, w));
        s = fma2(ds, s, mul2(rs, w));
      };
      if (piece < groups - 1) {
        start_f[g] = f;
        start_s[g] = s;
#pragma unroll
        for (int i = 0; i < SCAN_GROUP; ++i) advance(W[i * SCAN_THREADS]);
        continue;
      }
      if (g < groups - 1) {   // the last group goes on from the first pass
        f = start_f[g];
        s = start_s[g];
      }
      auto walk = [&](auto whole) {
        f32x2 F[SCAN_GROUP], S[SCAN_GROUP];
#pragma unroll
        for (int i = 0; i < SCAN_GROUP; ++i) {  // forward: state seen by chunk n0 + i
          if (whole.value || i < count) {
            F[i] = f;
            S[i] = s;
            advance(W[i * SCAN_THREADS]);
          }
        }
        __nv_bfloat16* to = out + (n0 + count - 1) * chunk_stride;
#pragma unroll
        for (int i = SCAN_GROUP - 1; i >= 0; --i) {
          if (whole.value || i < count) {
            const f32x2 w = W[i * SCAN_THREADS], gr = G[i * SCAN_THREADS];
            const float2 dw = halves(fma2(rf, a, mul2(rs, bb)));
            *reinterpret_cast<uint32_t*>(to) = pack_bf16x2(dw.x, dw.y);
            to -= chunk_stride;
            asm volatile("" : "+l"(to));   // as above
            const float2 of_f = halves(a), of_s = halves(bb), of_mix = halves(gr);
            const float2 by_f = halves(fma2(w, minus, F[i])), by_s = halves(fma2(w, minus, S[i])), by_mix = halves(fma2(S[i], minus, F[i]));
            add_products(g_df, of_f, by_f);     // F_{n+1} = df F_n + (1 - df) w_n
            add_products(g_ds, of_s, by_s);
            add_products(g_mix, of_mix, by_mix);
            a = fma2(df, a, mul2(mix, gr));     // gradient of F_n
            bb = fma2(ds, bb, mul2(rm, gr));
          }
        }
      };
      if (count == SCAN_GROUP) walk(std::true_type());
      else walk(std::false_type());
    }
    // block reduction (fixed order)
    const float vals[3] = {g_df, g_ds, g_mix};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      float v = vals[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[turn][q][warp] = v;
    }
    __syncthreads();   // the other half of `red` is written before the next one of these, this half only after it
    if (tid < 3) {
      float v = 0.f;
#pragma unroll
      for (int wi = 0; wi < SCAN_THREADS / 32; ++wi) v += red[turn][tid][wi];
      partials[static_cast<size_t>(unit) * 3 + tid] = v;
    }
  }
}

// Gradients of the decay and mix logits from the scan's partial sums (`logit_grad`).  (A launch in place of the sum, three
// sigmoids and nine products that a framework expression of it takes: 15 launches of 2 us for 3 H numbers.)
__global__ void __launch_bounds__(96)
memory_logit_grads_kernel(const float* partials, const float* fast_logit,
                          const float* slow_logit, const float* mix_logit, int B, int H,
                          float* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  logit_grad(partials, fast_logit, slow_logit, mix_logit, B, H, blockIdx.x, threadIdx.x >> 5, out);
}

// =============================================================================== attention bwd
// Two persistent CTAs of 256 threads per SM walk the (batch, chunk, head) tiles; threads t and t + 128 own row t of the chunk, one
// half of its columns each (of the 128 score columns, every other block of 32, so that the causal triangle is halved too).
// The kernel is a chain of MMA phases with element-wise work between them, so a single
// tile cannot keep an SM busy; what matters is how many tiles an SM holds at once, and how long the element-wise
// stretches of the chain are.  Shared memory is therefore kept to 112 KiB and TMEM to 256 columns, so that TWO CTAs fit
// per SM, and a row is shared by two threads, which exchange its softmax statistics and its D through shared memory.
//
// With a CTA per tile a third of its 30.7 k clocks went before and after the chain: 1.2 k of set-up, 5.4 k until the operands
// had landed, 2.8 k until its stores had read shared memory.  A CTA that goes on to its next tile requests Q and K of that one
// as soon as the last products have read dS, whose buffer they take, and everything else once the stores have drained, behind
// the rotation of Q and K.  The six tile buffers trade places for that, in pairs, from tile to tile.  Element-wise work that
// does not need a product's result runs under it: dmem under S, dlocal under O, the tanhs and dV under dQ and dK.
// 2048 tiles (4 x 2048 tokens, 32 heads): 122.9 us with a CTA per tile, 109 so; 280 tiles (one round) 16.7 and 16.6.  (dlocal (1 - g)
// under O, too, is a microsecond faster, but rounds dGate in another order than the form with a CTA per tile.)  What
// bounds it now is the load and store pipe, which tile traffic, tensor-core operands and TMA share: the gate row read by
// each thread from global memory (16 bytes of 32 rows to an instruction) 117, registers spilled for 0.1 KB 118, four threads to a row 137.
//
//   smem, three pairs of 16 KiB tiles: A = Qr, Kr | B = dy -> dlocal -> tanh(U), V -> tanh(Kr) | P = gate, dmem/8 -> P -> dS -> next A
//         | sSt (8K) | sDW (8K) | barriers.  Gradients leave from where their last operand was: dQ, dK from A, dU, dGate from B,
//         dV from sSt and sDW.  Next tile: A <- P, B <- A, P <- B.
//   TMEM: [0,128) S -> O (first 64) -> dP -> dKr (first 64) + dtK (last 64)
//         [128,192) Mem -> dV -> dtU        [192,256) dQr (memory part, later += attention part)
//
// U is fetched late (into the buffer that dlocal has left), behind the dS phase.  P is stored normalised, so O and dV need no
// row scaling.
constexpr int AB_THREADS = 256;
constexpr int AB_PIECES = 4;   // 16-byte pieces of a 64-column row that a thread owns
// No alignment slack: 2 x (114816 + 1024 reserved) = 231680 <= 233472 bytes of an SM.  The dynamic
// segment is declared 1024-byte aligned (the 128-byte swizzle needs it); the kernel checks.
constexpr int AB_SMEM = 4 * TILE_BYTES + 2 * TILE_BYTES + 2 * 8192 + 128;

// The buffers trade places, so a thread reaches them by 32-bit shared addresses: `at` = its tile + where its four pieces of its row
// begin, piece j of them at `at` ^ 16 j (the swizzle is an exclusive or of the bits that count the pieces).
__device__ __forceinline__ uint4& ab_piece(uint32_t at, int j) {
  return *static_cast<uint4*>(__cvta_shared_to_generic(at ^ (j << 4)));
}
// Rotary embedding of the thread's pieces of a Q and a K row, in place (as rope_tanh_row in attention_common.cuh).
__device__ __forceinline__ void ab_rope(uint32_t q_at, uint32_t k_at, int row, int piece0, const float2* rope) {
#pragma unroll
  for (int j = 0; j < AB_PIECES; ++j) {
    uint4 q = ab_piece(q_at, j), k = ab_piece(k_at, j);
    uint32_t* qw = reinterpret_cast<uint32_t*>(&q);
    uint32_t* kw = reinterpret_cast<uint32_t*>(&k);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 cs = rope[((piece0 + j) * 4 + t) * CHUNK + row];
      const float2 qr = rope_rotate(__bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&qw[t])), cs);
      const float2 kr = rope_rotate(__bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&kw[t])), cs);
      qw[t] = pack_bf16x2(qr.x, qr.y);
      kw[t] = pack_bf16x2(kr.x, kr.y);
    }
    ab_piece(q_at, j) = q;
    ab_piece(k_at, j) = k;
  }
}
__device__ __forceinline__ uint4 tanh_piece(uint4 v) {
  uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w[t]));
    w[t] = pack_bf16x2(tanh_fast(x.x), tanh_fast(x.y));
  }
  return v;
}

__global__ void __launch_bounds__(AB_THREADS, 2)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_state,
                const __grid_constant__ CUtensorMap tm_dy, const __grid_constant__ CUtensorMap tm_dw,
                const __grid_constant__ CUtensorMap tm_dout, const float2* rope, int H, int d,
                int tiles, int* error_flag) {
  extern __shared__ __align__(1024) uint8_t smem_ab[];
  uint8_t* smem = smem_ab;
  if ((smem_u32(smem) & 1023u) != 0u) {  // uniform over the CTA: nothing has been set up yet
    if (threadIdx.x == 0 && error_flag != nullptr) atomicExch(error_flag, 7);
    return;
  }
  uint8_t* sSt = smem + 6 * TILE_BYTES;
  uint8_t* sDW = sSt + 8192;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDW + 8192);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);   // bars: loads 0 Q and K, 7 the other operands, 5 U; products 1 S, 2 A, 3 B, 4 C, 6 D
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, row = tid & 127, half = tid >> 7, quarter = warp & 3;
  const int piece0 = half * AB_PIECES;

  if (tid == 0) {
    for (int i = 0; i < 8; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t t_lo = tmem;          // S / O / dP / dKr+dtK
  const uint32_t t_mid = tmem + 128;   // Mem / dV / dtU
  const uint32_t t_dq = tmem + 192;    // dQr
  const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;

  auto load_qk = [&](int tile, uint32_t to) {
    const int h = tile % H, row0 = tile / H * CHUNK;   // tiles of a chunk lie behind one another, chunks in token order
    mbar_expect_tx(&bars[0], 2 * TILE_BYTES);
    tma_load_2d(__cvta_shared_to_generic(to), &tm_qkvgu, &bars[0], h * HD, row0);
    tma_load_2d(__cvta_shared_to_generic(to + TILE_BYTES), &tm_qkvgu, &bars[0], d + h * HD, row0);
  };
  auto load_rest = [&](int tile, uint32_t to, uint32_t gate_to) {
    const int h = tile % H, row0 = tile / H * CHUNK;
    mbar_expect_tx(&bars[7], 3 * TILE_BYTES + 2 * 8192);
    tma_load_2d(__cvta_shared_to_generic(to), &tm_dy, &bars[7], h * HD, row0);
    tma_load_2d(__cvta_shared_to_generic(gate_to), &tm_qkvgu, &bars[7], 3 * d + h * HD, row0);
    tma_load_2d(sSt, &tm_state, &bars[7], 0, tile * HD);
    tma_load_2d(__cvta_shared_to_generic(to + TILE_BYTES), &tm_qkvgu, &bars[7], 2 * d + h * HD, row0);
    tma_load_2d(sDW, &tm_dw, &bars[7], 0, tile * HD);
  };
  uint32_t sA = smem_u32(smem), sB = sA + 2 * TILE_BYTES, sP = sA + 4 * TILE_BYTES;
  const uint32_t mine_at = row * 128 + ((piece0 ^ (row & 7)) << 4), dv_at = smem_u32(sSt) + mine_at;
  if (tid == 0) {
    load_qk(blockIdx.x, sA);
    load_rest(blockIdx.x, sB, sP);
  }
  bool ok = true;
  uint32_t ph = 0;   // every barrier completes once per tile
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ph ^= 1) {
    const int h = tile % H, row0 = tile / H * CHUNK;
    const uint32_t sQ = sA, sK = sA + TILE_BYTES, sB2 = sB, sB3 = sB + TILE_BYTES;
    // The thread's half of the gate row, of the dGate row and of the dV row stay in registers (4 x 16 bytes each) until
    // the last stage, where all five gradient tiles leave through shared memory and TMA stores.
    uint4 gate_row[AB_PIECES], dgate_row[AB_PIECES], dv_row[AB_PIECES];
    ok = mbar_wait(&bars[0], ph, abort_flag) && ok;
    if (ok) ab_rope(sQ + mine_at, sK + mine_at, row, piece0, rope);
    if (tid < 128 && (tid & 31) == 0) tma_store_wait_read0();   // the gradients of the tile before have left B, P, sSt and sDW
    tc_fence_before_sync();
    fence_proxy_async_smem();
    __syncthreads();
    // ---- MMA S = Qr Kr^T, and the other operands of this tile
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after_sync();
      if (tile != static_cast<int>(blockIdx.x)) load_rest(tile, sB, sP);
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16(t_lo, make_smem_desc_sw128((sQ) + k * 32, 0, 1024),
                  make_smem_desc_sw128((sK) + k * 32, 0, 1024), idesc_s, k > 0);
      umma_commit(&bars[1]);
    }
    ok = mbar_wait(&bars[7], ph, abort_flag) && ok;
#pragma unroll
    for (int j = 0; j < AB_PIECES; ++j) gate_row[j] = ab_piece(sP + mine_at, j);
    if (ok) {
      // dmem/8 = dy * (1 - sigmoid(gate)) / 8  -> the second tile of P
#pragma unroll
      for (int j = 0; j < AB_PIECES; ++j) {
        const uint4 dyq = ab_piece(sB2 + mine_at, j);
        const uint4 gq = gate_row[j];
        const __nv_bfloat162* dyb = reinterpret_cast<const __nv_bfloat162*>(&dyq);
        const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gq);
        uint4 o;
        uint32_t* wo = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 dyv = __bfloat1622float2(dyb[t]);
          const float2 gf = __bfloat1622float2(gb[t]);
          // the sigmoid is rounded before it is taken from 1, as the forward pass has it
          wo[t] = pack_bf16x2(dyv.x * fmaf(sigmoid_f(gf.x), -0.125f, 0.125f), dyv.y * fmaf(sigmoid_f(gf.y), -0.125f, 0.125f));
        }
        ab_piece(sP + TILE_BYTES + mine_at, j) = o;
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    // ---- MMA A: Mem = Qr State, dQr = (dmem/8) State^T
    if (warp == 0 && elect_one() && ok) {
      constexpr uint32_t idesc_m = make_idesc_bf16(128, 64, false, true);
      constexpr uint32_t idesc_kk64 = make_idesc_bf16(128, 64, false, false);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16(t_mid, make_smem_desc_sw128((sQ) + k * 32, 0, 1024),
                  make_smem_desc_sw128(smem_u32(sSt) + k * 2048, 0, 1024), idesc_m, k > 0);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16(t_dq, make_smem_desc_sw128((sP + TILE_BYTES) + k * 32, 0, 1024),
                  make_smem_desc_sw128(smem_u32(sSt) + k * 32, 0, 1024), idesc_kk64, k > 0);
      umma_commit(&bars[2]);
    }
    ok = mbar_wait(&bars[1], ph, abort_flag) && ok;
    tc_fence_after_sync();

    // ---- softmax over this thread's two blocks of columns, {half, half + 2} x 32, held in registers: one TMEM read and
    // one exponential per score.  The two threads of a row meet once, with (max, sum) of their columns, in the State
    // tile's space (the State has been consumed); a block behind the causal mask counts as (-inf, 0), and so does a half
    // whose visible scores are all -inf (a product that overflowed): the other half decides the row.
    const float kScale = 0.125f * 1.4426950408889634f;
    float* meet = reinterpret_cast<float*>(sSt);   // [2][128] max | [2][128] sum | [2][128] D
    float e[2][32];
    float my_max = -INFINITY, my_sum = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int cc = half + 2 * k;
      if (cc <= quarter) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_lo + lane_base + cc * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          e[k][j] = cc * 32 + j <= row ? __uint_as_float(r[j]) : -INFINITY;
          my_max = fmaxf(my_max, e[k][j]);
        }
      } else {   // never read; without a value here they would be kept from tile to tile
#pragma unroll
        for (int j = 0; j < 32; ++j) e[k][j] = 0.f;
      }
    }
    const float from = my_max == -INFINITY ? 0.f : my_max;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (half + 2 * k <= quarter) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          e[k][j] = exp2f((e[k][j] - from) * kScale);
          my_sum += e[k][j];
        }
      }
    }
    ok = mbar_wait(&bars[2], ph, abort_flag) && ok;   // State and dmem have been consumed
    meet[half * 128 + row] = my_max;
    meet[256 + half * 128 + row] = my_sum;
    __syncthreads();
    const float other_max = meet[(half ^ 1) * 128 + row];
    const float row_max = fmaxf(my_max, other_max);
    const float my_share = exp2f((my_max - row_max) * kScale);
    const float row_sum = my_sum * my_share + meet[256 + (half ^ 1) * 128 + row] * exp2f((other_max - row_max) * kScale);
    const float to_p = my_share / row_sum;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int cc = half + 2 * k;
      uint32_t pk[16];
      if (cc <= quarter) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) pk[j >> 1] = pack_bf16x2(e[k][j] * to_p, e[k][j + 1] * to_p);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) pk[j] = 0u;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) ab_piece(sP + k * TILE_BYTES + mine_at, j) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
    }
    tc_fence_before_sync();
    fence_proxy_async_smem();
    __syncthreads();
    // ---- MMA B: O = P V
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after_sync();
      constexpr uint32_t idesc_o = make_idesc_bf16(128, 64, false, true);
#pragma unroll
      for (int k = 0; k < CHUNK / 16; ++k)
        umma_bf16(t_lo, make_smem_desc_sw128((sP) + (k >> 2) * TILE_BYTES + (k & 3) * 32, 0, 1024),
                  make_smem_desc_sw128((sB3) + k * 2048, 0, 1024), idesc_o, k > 0);
      umma_commit(&bars[3]);
    }
    // ---- element-wise stage 1: under the product dlocal = dy * g (in place in B2), behind it dGate = dy (local - memory) g (1 - g),
    // in that order, and D = sum(dlocal * local)
    uint4 dy_row[AB_PIECES];
    float sig[AB_PIECES * 8];
#pragma unroll
    for (int i = 0; i < AB_PIECES; ++i) {
      uint4 dyq = ab_piece(sB2 + mine_at, i);
      dy_row[i] = dyq;
      const uint4 gq = gate_row[i];
      uint32_t* w = reinterpret_cast<uint32_t*>(&dyq);
      const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gq);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 dyv = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w[t]));
        const float2 gf = __bfloat1622float2(gb[t]);
        const int e0 = i * 8 + 2 * t, e1 = e0 + 1;
        sig[e0] = sigmoid_f(gf.x);
        sig[e1] = sigmoid_f(gf.y);
        w[t] = pack_bf16x2(dyv.x * sig[e0], dyv.y * sig[e1]);
      }
      ab_piece(sB2 + mine_at, i) = dyq;
    }
    ok = mbar_wait(&bars[3], ph, abort_flag) && ok;
    tc_fence_after_sync();
    float Drow = 0.f;
#pragma unroll
    for (int i = 0; i < AB_PIECES; i += 2) {
      const int c = (piece0 + i) * 8;
      uint32_t ro[16], rm[16];
      tmem_ld_32x32b_x16(t_lo + lane_base + c, ro);
      tmem_ld_32x32b_x16(t_mid + lane_base + c, rm);
      tmem_ld_wait();
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        const float l0 = __uint_as_float(ro[j]), l1 = __uint_as_float(ro[j + 1]);
        const float m0 = __uint_as_float(rm[j]) * 0.125f, m1 = __uint_as_float(rm[j + 1]) * 0.125f;
        const uint4& dyq = dy_row[i + (j >> 3)];
        const float2 dyv = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&dyq)[(j & 7) >> 1]);
        const float g0 = sig[i * 8 + j], g1 = sig[i * 8 + j + 1];
        const float dl0 = dyv.x * g0, dl1 = dyv.y * g1;
        Drow += dl0 * l0 + dl1 * l1;
        w[j >> 1] = pack_bf16x2(dyv.x * (l0 - m0) * g0 * (1.f - g0), dyv.y * (l1 - m1) * g1 * (1.f - g1));
      }
      dgate_row[i] = make_uint4(w[0], w[1], w[2], w[3]);
      dgate_row[i + 1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    meet[512 + half * 128 + row] = Drow;
    tc_fence_before_sync();
    fence_proxy_async_smem();
    __syncthreads();
    Drow = (Drow + meet[512 + (half ^ 1) * 128 + row]) * 0.125f;
    // ---- MMA C: dP = dlocal V^T, dV = P^T dlocal
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after_sync();
      constexpr uint32_t idesc_kk128 = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_mnmn64 = make_idesc_bf16(128, 64, true, true);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16(t_lo, make_smem_desc_sw128((sB2) + k * 32, 0, 1024),
                  make_smem_desc_sw128((sB3) + k * 32, 0, 1024), idesc_kk128, k > 0);
#pragma unroll
      for (int k = 0; k < CHUNK / 16; ++k)
        umma_bf16(t_mid, make_smem_desc_sw128((sP) + k * 2048, TILE_BYTES, 1024),
                  make_smem_desc_sw128((sB2) + k * 2048, 0, 1024), idesc_mnmn64, k > 0);
      umma_commit(&bars[4]);
    }
    ok = mbar_wait(&bars[4], ph, abort_flag) && ok;
    tc_fence_after_sync();
    if (tid == 0 && ok) {  // B2 (dlocal) has been consumed: fetch U into it behind the dS phase
      mbar_expect_tx(&bars[5], TILE_BYTES);
      tma_load_2d(__cvta_shared_to_generic(sB2), &tm_qkvgu, &bars[5], 4 * d + h * HD, row0);
    }

    // ---- dS = P * (dP - D) / 8 over P
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int cc = half + 2 * k;
      if (cc > quarter) continue;
      uint32_t r[32], pk[16];
      tmem_ld_32x32b_x32(t_lo + lane_base + cc * 32, r);
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(&pk[4 * j]) = ab_piece(sP + k * TILE_BYTES + mine_at, j);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float2 pv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pk[j]));
        const float s0 = pv.x * fmaf(__uint_as_float(r[2 * j]), 0.125f, -Drow);   // (dP - D) / 8
        const float s1 = pv.y * fmaf(__uint_as_float(r[2 * j + 1]), 0.125f, -Drow);
        pk[j] = pack_bf16x2(s0, s1);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) ab_piece(sP + k * TILE_BYTES + mine_at, j) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
    }
    tc_fence_before_sync();
    fence_proxy_async_smem();
    __syncthreads();
    // ---- MMA D, first half: dQr += dS Kr, dKr = dS^T Qr
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after_sync();
      constexpr uint32_t idesc_kmn64 = make_idesc_bf16(128, 64, false, true);
      constexpr uint32_t idesc_mnmn64 = make_idesc_bf16(128, 64, true, true);
#pragma unroll
      for (int k = 0; k < CHUNK / 16; ++k)
        umma_bf16(t_dq, make_smem_desc_sw128((sP) + (k >> 2) * TILE_BYTES + (k & 3) * 32, 0, 1024),
                  make_smem_desc_sw128((sK) + k * 2048, 0, 1024), idesc_kmn64, 1u);
#pragma unroll
      for (int k = 0; k < CHUNK / 16; ++k)
        umma_bf16(t_lo, make_smem_desc_sw128((sP) + k * 2048, TILE_BYTES, 1024),
                  make_smem_desc_sw128((sQ) + k * 2048, 0, 1024), idesc_mnmn64, k > 0);
    }
    // ---- under it: dV out; tanh(Kr) -> B3, tanh(U)
#pragma unroll
    for (int i = 0; i < AB_PIECES; i += 2) {
      uint32_t rv[16];
      tmem_ld_32x32b_x16(t_mid + lane_base + (piece0 + i) * 8, rv);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; j += 8) {
        dv_row[i + (j >> 3)] = make_uint4(pack_bf16x2(__uint_as_float(rv[j]), __uint_as_float(rv[j + 1])),
                                          pack_bf16x2(__uint_as_float(rv[j + 2]), __uint_as_float(rv[j + 3])),
                                          pack_bf16x2(__uint_as_float(rv[j + 4]), __uint_as_float(rv[j + 5])),
                                          pack_bf16x2(__uint_as_float(rv[j + 6]), __uint_as_float(rv[j + 7])));
      }
    }
#pragma unroll
    for (int j = 0; j < AB_PIECES; ++j) ab_piece(sB3 + mine_at, j) = tanh_piece(ab_piece(sK + mine_at, j));   // V is no longer needed
    ok = mbar_wait(&bars[5], ph, abort_flag) && ok;  // U has landed
    if (ok) {
#pragma unroll
      for (int j = 0; j < AB_PIECES; ++j) ab_piece(sB2 + mine_at, j) = tanh_piece(ab_piece(sB2 + mine_at, j));
    }
    tc_fence_before_sync();
    fence_proxy_async_smem();
    __syncthreads();
    // ---- second half: dtK = tU dW^T, dtU = tK dW; the arrival counts for both halves
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after_sync();
      constexpr uint32_t idesc_kmn64 = make_idesc_bf16(128, 64, false, true);
      constexpr uint32_t idesc_kk64 = make_idesc_bf16(128, 64, false, false);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)  // dtK = tU dW^T
        umma_bf16(t_lo + 64, make_smem_desc_sw128((sB2) + k * 32, 0, 1024),
                  make_smem_desc_sw128(smem_u32(sDW) + k * 32, 0, 1024), idesc_kk64, k > 0);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)  // dtU = tK dW
        umma_bf16(t_mid, make_smem_desc_sw128((sB3) + k * 32, 0, 1024),
                  make_smem_desc_sw128(smem_u32(sDW) + k * 2048, 0, 1024), idesc_kmn64, k > 0);
      umma_commit(&bars[6]);
    }
    ok = mbar_wait(&bars[6], ph, abort_flag) && ok;
    tc_fence_after_sync();

    if (tid == 0 && ok && tile + static_cast<int>(gridDim.x) < tiles) load_qk(tile + gridDim.x, sP);   // dS has been consumed

    // ---- final: dQ, dK (RoPE transpose), dU
#pragma unroll
    for (int i = 0; i < AB_PIECES; i += 2) {
      const int c = (piece0 + i) * 8;
      uint32_t rq[16], rk[16], rtk[16], rtu[16];
      tmem_ld_32x32b_x16(t_dq + lane_base + c, rq);
      tmem_ld_32x32b_x16(t_lo + lane_base + c, rk);
      tmem_ld_32x32b_x16(t_lo + 64 + lane_base + c, rtk);
      tmem_ld_32x32b_x16(t_mid + lane_base + c, rtu);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; j += 8) {
        const int mine = i + (j >> 3);
        const uint4 tkq = ab_piece(sB3 + mine_at, mine);
        const uint4 tuq = ab_piece(sB2 + mine_at, mine);
        const __nv_bfloat162* tkb = reinterpret_cast<const __nv_bfloat162*>(&tkq);
        const __nv_bfloat162* tub = reinterpret_cast<const __nv_bfloat162*>(&tuq);
        uint4 o_q, o_k, o_u;
        uint32_t* w_q = reinterpret_cast<uint32_t*>(&o_q);
        uint32_t* w_k = reinterpret_cast<uint32_t*>(&o_k);
        uint32_t* w_u = reinterpret_cast<uint32_t*>(&o_u);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int e0 = j + 2 * t, e1 = e0 + 1;
          const float2 cs = rope[((c + e0) >> 1) * CHUNK + row];
          const float2 tk = __bfloat1622float2(tkb[t]);
          const float2 tu = __bfloat1622float2(tub[t]);
          // y0 = x0 c - x1 s ; y1 = x1 c + x0 s   =>   dx0 = dy0 c + dy1 s ; dx1 = dy1 c - dy0 s
          const float q0 = __uint_as_float(rq[e0]), q1 = __uint_as_float(rq[e1]);
          w_q[t] = pack_bf16x2(q0 * cs.x + q1 * cs.y, q1 * cs.x - q0 * cs.y);
          const float k0 = __uint_as_float(rk[e0]) + __uint_as_float(rtk[e0]) * (1.f / CHUNK) * (1.f - tk.x * tk.x);
          const float k1 = __uint_as_float(rk[e1]) + __uint_as_float(rtk[e1]) * (1.f / CHUNK) * (1.f - tk.y * tk.y);
          w_k[t] = pack_bf16x2(k0 * cs.x + k1 * cs.y, k1 * cs.x - k0 * cs.y);
          w_u[t] = pack_bf16x2(__uint_as_float(rtu[e0]) * (1.f / CHUNK) * (1.f - tu.x * tu.x),
                               __uint_as_float(rtu[e1]) * (1.f / CHUNK) * (1.f - tu.y * tu.y));
        }
        // every operand of the last MMA group has been consumed, and tanh(U) and tanh(Kr) by the thread that takes their place
        ab_piece(sQ + mine_at, mine) = o_q;
        ab_piece(sK + mine_at, mine) = o_k;
        ab_piece(sB2 + mine_at, mine) = o_u;
        ab_piece(sB3 + mine_at, mine) = dgate_row[mine];
        ab_piece(dv_at, mine) = dv_row[mine];
      }
    }
    fence_proxy_async_smem();
    // the two warps that share 32 token rows (immediate barrier numbers: a register would reserve all sixteen)
    if (quarter == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
    else if (quarter == 1) asm volatile("bar.sync 2, 64;" ::: "memory");
    else if (quarter == 2) asm volatile("bar.sync 3, 64;" ::: "memory");
    else asm volatile("bar.sync 4, 64;" ::: "memory");
    if (tid < 128 && (tid & 31) == 0) {  // one store per gradient tile for those rows
      if (ok) {
        const int r = row0 + quarter * 32, off = quarter * 4096;
        tma_store_2d(&tm_dout, __cvta_shared_to_generic(sQ + off), 0 * d + h * HD, r);
        tma_store_2d(&tm_dout, __cvta_shared_to_generic(sK + off), 1 * d + h * HD, r);
        tma_store_2d(&tm_dout, sSt + off, 2 * d + h * HD, r);
        tma_store_2d(&tm_dout, __cvta_shared_to_generic(sB3 + off), 3 * d + h * HD, r);
        tma_store_2d(&tm_dout, __cvta_shared_to_generic(sB2 + off), 4 * d + h * HD, r);
        tma_store_commit();
      }
    }
    const uint32_t next = sP;
    sP = sB;
    sB = sA;
    sA = next;
  }
  if (tid < 128 && (tid & 31) == 0) tma_store_wait_read0();
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 5);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 256);
  }
}

}  // namespace ws

using namespace ws;

extern "C" int ws_attn_dstate(const void* qkvgu, const void* dy, const float* rope, float* dstate, int B, int T,
                              int H, int d, int* error_flag, cudaStream_t stream) {
  if (T % CHUNK != 0 || d != H * HD) return -1;
  CUtensorMap tm, td, to;
  int rc = make_tile_map(&tm, qkvgu, 5 * (uint64_t)d, (uint64_t)B * T, 5 * (uint64_t)d, HD, CHUNK);
  if (rc) return rc;
  rc = make_tile_map(&td, dy, (uint64_t)d, (uint64_t)B * T, (uint64_t)d, HD, CHUNK);
  if (rc) return rc;
  rc = make_map_f32(&to, dstate, HD, (uint64_t)B * (T / CHUNK) * H * HD, HD, 32, 32);
  if (rc) return rc;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(dstate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  const int tiles = B * (T / CHUNK) * H;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(dstate_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DSS_SMEM) != cudaSuccess)
      return -20;
  }
  if (ws_attn_stream_form() != 0)
    launch_dependent(dstate_stream_kernel, dim3(tiles < sms ? tiles : sms), dim3(DSS_THREADS), DSS_SMEM, stream, tm, td, to,
                     reinterpret_cast<const float2*>(rope), T, H, d, tiles, error_flag);
  else
    launch_dependent(dstate_kernel, dim3(tiles), dim3(128), DS_SMEM, stream, tm, td, to, reinterpret_cast<const float2*>(rope), T, H, d,
                     error_flag);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ws_memory_scan_bwd(const float* dstate, const float* writes, const float* fast_logit,
                                  const float* slow_logit, const float* mix_logit, void* dwrites, float* partials,
                                  int B, int N, int H, cudaStream_t stream) {
  if (N > SCAN_MAX_CHUNKS) return -1;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -20;
    sms = n;
  }
  if (!allow_shared_memory<memory_scan_bwd_kernel>(SCAN_SMEM)) return -20;
  const int units = B * H * 16;
  launch_dependent(memory_scan_bwd_kernel, dim3(units < 3 * sms ? units : 3 * sms), dim3(SCAN_THREADS), SCAN_SMEM, stream, dstate, writes,
                   fast_logit, slow_logit, mix_logit, (__nv_bfloat16*)dwrites, partials, B, N, H);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ws_attn_bwd(const void* qkvgu, const void* states, const void* dy, const void* dwrites,
                           const float* rope, void* dqkvgu, int B, int T, int H, int d, int* error_flag,
                           cudaStream_t stream) {
  if (T % CHUNK != 0 || d != H * HD) return -1;
  const int tiles = B * (T / CHUNK) * H;
  CUtensorMap tm, ts, td, tw, to;
  int rc = make_tile_map(&tm, qkvgu, 5 * (uint64_t)d, (uint64_t)B * T, 5 * (uint64_t)d, HD, CHUNK);
  if (rc) return rc;
  rc = make_tile_map(&to, dqkvgu, 5 * (uint64_t)d, (uint64_t)B * T, 5 * (uint64_t)d, HD, 32);
  if (rc) return rc;
  rc = make_tile_map(&ts, states, HD, (uint64_t)tiles * HD, HD, HD, HD);
  if (rc) return rc;
  rc = make_tile_map(&td, dy, (uint64_t)d, (uint64_t)B * T, (uint64_t)d, HD, CHUNK);
  if (rc) return rc;
  rc = make_tile_map(&tw, dwrites, HD, (uint64_t)tiles * HD, HD, HD, HD);
  if (rc) return rc;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AB_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -20;
  }
  launch_dependent(attn_bwd_kernel, dim3(tiles < 2 * sms ? tiles : 2 * sms), dim3(AB_THREADS), AB_SMEM, stream, tm, ts, td, tw, to,
                   reinterpret_cast<const float2*>(rope), H, d, tiles, error_flag);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ws_memory_logit_grads(const float* partials, const float* fast_logit, const float* slow_logit,
                                     const float* mix_logit, int B, int H, float* out, cudaStream_t stream) {
  if (B <= 0 || H <= 0) return -1;
  launch_dependent(memory_logit_grads_kernel, dim3(H), dim3(96), 0, stream, partials, fast_logit, slow_logit, mix_logit, B,
                   H, out);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
