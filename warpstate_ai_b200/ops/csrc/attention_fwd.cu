// Forward kernels of the middle of a WarpState core (everything between in_proj and out_proj;
// reference math: warpstate/model.py:124-176), for chunk_size 128 and head_dim 64.
//
// The packed projection qkvgu [tokens, 5d] (Q,K,V,gate,U) is read in place with TMA, through a map
// over (column, position, sequence): a tile of one (batch, chunk, head) is the box of columns
// [sel*d + h*64, +64) x positions [n*128, +128) of sequence b, with zeros past the sequence's end --
// the reference's chunkify/permute/contiguous copies do not exist here.
//
//   chunk_writes_kernel : W[b,n,h] = tanh(rope(K))^T tanh(U) / 128            (tcgen05, 64x64 out)
//   memory_scan_kernel  : state seen by chunk n = mix*F_n + (1-mix)*S_n with
//                         F_n = d_f F_{n-1} + (1-d_f) W_{n-1}, F_0 = 0 (FP32, O(N) scan)
//   attn_fwd_kernel     : S = rope(Q) rope(K)^T (tcgen05 -> TMEM), causal softmax by one thread
//                         per row straight out of TMEM, O = P V and Mem = rope(Q) state (tcgen05),
//                         y = sigmoid(g) * O/l + (1 - sigmoid(g)) * Mem/8, stored token-major.
//
// One thread owns one token row (= one TMEM lane): no cross-thread reductions anywhere.
#include "ws_ptx.cuh"
#include "ws_api.h"
#include "ws_launch.h"
#include "attention_common.cuh"

#include <cstdlib>
#include <type_traits>

namespace ws {

extern "C" void ws_count_launch(void);

// =============================================================================== writes
// smem: sK 16K | sU 16K | bars
constexpr int WR_SMEM = 2 * TILE_BYTES + 1024 + 128;

__global__ void __launch_bounds__(128, 6)
chunk_writes_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_out,
                    const float2* rope, int T, int H, int d, int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sK = smem;
  uint8_t* sU = smem + TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * TILE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int n_chunks = (T + CHUNK - 1) / CHUNK;
  const int tile = blockIdx.x;
  const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
  const int row0 = n * CHUNK;

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
    mbar_expect_tx(&bars[0], 2 * TILE_BYTES);
    tma_load_3d(sK, &tm_qkvgu, &bars[0], 1 * d + h * HD, row0, b);
    tma_load_3d(sU, &tm_qkvgu, &bars[0], 4 * d + h * HD, row0, b);
  }
  bool ok = mbar_wait(&bars[0], 0, abort_flag);
  if (ok) {
    rope_tanh_row(sK, tid, rope, true, true);    // K -> tanh(rope(K))
    rope_tanh_row(sU, tid, rope, false, true);   // U -> tanh(U)
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (warp == 0 && elect_one() && ok) {
    // D[128 x 64]: rows 0..63 = tK^T tU.  A is read MN-major with a zero stride between its two
    // 64-wide atoms, so rows 64..127 repeat rows 0..63 and are ignored.
    constexpr uint32_t idesc = make_idesc_bf16(128, 64, true, true);
#pragma unroll
    for (int k = 0; k < CHUNK / 16; ++k) {
      const uint64_t da = make_smem_desc_sw128(smem_u32(sK) + k * 2048, 0, 1024);
      const uint64_t db = make_smem_desc_sw128(smem_u32(sU) + k * 2048, 0, 1024);
      umma_bf16(tmem, da, db, idesc, k > 0);
    }
    umma_commit(&bars[1]);
  }
  ok = ok && mbar_wait(&bars[1], 0, abort_flag);
  tc_fence_after_sync();
  if (warp < 2) {  // lanes 0..63 hold the result rows
    // Row `tid` goes to two swizzled [64 x 32] FP32 half tiles in the (consumed) K tile's space; each
    // warp then stores its 32 rows of both halves by TMA.
#pragma unroll
    for (int c = 0; c < HD; c += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const int col = c + j;
        uint8_t* dst = sK + (col >> 5) * 8192 + tid * 128 + ((((col & 31) >> 2) ^ (tid & 7)) << 4);
        *reinterpret_cast<float4*>(dst) =
            make_float4(__uint_as_float(r[j]) * (1.f / CHUNK), __uint_as_float(r[j + 1]) * (1.f / CHUNK),
                        __uint_as_float(r[j + 2]) * (1.f / CHUNK), __uint_as_float(r[j + 3]) * (1.f / CHUNK));
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if ((tid & 31) == 0) {
      if (ok) {
        tma_store_2d(&tm_out, sK + warp * 4096, 0, tile * HD + warp * 32);
        tma_store_2d(&tm_out, sK + 8192 + warp * 4096, 32, tile * HD + warp * 32);
        tma_store_commit();
      }
      tma_store_wait_read0();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 2);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 64);
  }
}

// =============================================================================== writes, streaming form
// The same product as chunk_writes_kernel, as one persistent CTA per SM with specialised warps:
//
//   warp 18      producer: TMA loads of the K and U tiles of tile i into stage i % 4 of a ring (4 x 32 KiB)
//   warps 0..15  workers (512 threads): thread (row r, quarter q) turns two of the eight 16-byte pieces of row r of K
//                into tanh(rope(K)) and of U into tanh(U), in place; its 8 (cos, sin) pairs are loaded once, since
//                they depend on the row and the column only.  (With 8 worker warps the kernel issued an instruction
//                in 33 % of the cycles, each warp waiting 8 cycles between two of its own: four warps per scheduler
//                instead of two hide that.)  Worker thread 0 then issues the tile's eight MMAs into
//                TMEM buffer i % 2; their completion frees the ring stage and hands the buffer to the epilogue.
//   warps 16, 17 epilogue (accumulator lanes 0..63): TMEM -> x 1/128 -> swizzled FP32 staging tile -> TMA store
//
// so the loads of the next three tiles, the element-wise work of the current one and the store of the previous
// one overlap; chunk_writes_kernel gets its overlap from six independent CTAs per SM instead, each of which walks
// the chain load -> element-wise -> MMA -> store alone.  Results are bit-identical (same arithmetic, same MMA order).
constexpr int WS_STAGES = 4;
constexpr int WS_THREADS = 19 * 32;
constexpr int WS_SMEM = WS_STAGES * 2 * TILE_BYTES + 2 * 16384 + 1024 + 256;

__global__ void __launch_bounds__(WS_THREADS, 1)
chunk_writes_stream_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_out,
                           const float2* rope, int T, int H, int d, int tiles, int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* ring = smem;                                   // stage s: K at s * 32 KiB, U 16 KiB behind it
  uint8_t* staging = smem + WS_STAGES * 2 * TILE_BYTES;   // two FP32 [64 x 64] tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + 2 * 16384);
  uint64_t* full = bars;                    // [4] tile landed
  uint64_t* empty = bars + WS_STAGES;       // [4] MMAs have read the stage
  uint64_t* tfull = bars + 2 * WS_STAGES;   // [2] accumulator complete
  uint64_t* tempty = tfull + 2;             // [2] accumulator read by both epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_chunks = (T + CHUNK - 1) / CHUNK;

  if (tid == 0) {
    for (int s = 0; s < WS_STAGES; ++s) {
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
        const int s = i % WS_STAGES;
        if (!mbar_wait(&empty[s], ((i / WS_STAGES) & 1) ^ 1, abort_flag)) break;
        const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
        const int row0 = n * CHUNK;
        mbar_expect_tx(&full[s], 2 * TILE_BYTES);
        tma_load_3d(ring + s * 2 * TILE_BYTES, &tm_qkvgu, &full[s], 1 * d + h * HD, row0, b);
        tma_load_3d(ring + s * 2 * TILE_BYTES + TILE_BYTES, &tm_qkvgu, &full[s], 4 * d + h * HD, row0, b);
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
      const int s = i % WS_STAGES;
      uint8_t* sK = ring + s * 2 * TILE_BYTES;
      uint8_t* sU = sK + TILE_BYTES;
      const bool ok = mbar_wait(&full[s], (i / WS_STAGES) & 1, abort_flag);
      if (ok) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint4* pk = reinterpret_cast<uint4*>(tile_chunk(sK, r, q * 2 + j));
          uint4* pu = reinterpret_cast<uint4*>(tile_chunk(sU, r, q * 2 + j));
          uint4 kv = *pk, uv = *pu;
          uint32_t* kw = reinterpret_cast<uint32_t*>(&kv);
          uint32_t* uw = reinterpret_cast<uint32_t*>(&uv);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&kw[t]));
            const float2 c = cs[j * 4 + t];
            const float2 kr = rope_rotate(x, c);
            kw[t] = pack_bf16x2(tanh_fast(kr.x), tanh_fast(kr.y));
            const float2 u = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&uw[t]));
            uw[t] = pack_bf16x2(tanh_fast(u.x), tanh_fast(u.y));
          }
          *pk = kv;
          *pu = uv;
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
          // D[128 x 64]: rows 0..63 = tK^T tU.  A is read MN-major with a zero stride between its two 64-wide
          // atoms, so rows 64..127 repeat rows 0..63 and are ignored.
          constexpr uint32_t idesc = make_idesc_bf16(128, 64, true, true);
#pragma unroll
          for (int k = 0; k < CHUNK / 16; ++k)
            umma_bf16(tmem + buf * 64, make_smem_desc_sw128(smem_u32(sK) + k * 2048, 0, 1024),
                      make_smem_desc_sw128(smem_u32(sU) + k * 2048, 0, 1024), idesc, k > 0);
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
              make_float4(__uint_as_float(v[j]) * (1.f / CHUNK), __uint_as_float(v[j + 1]) * (1.f / CHUNK),
                          __uint_as_float(v[j + 2]) * (1.f / CHUNK), __uint_as_float(v[j + 3]) * (1.f / CHUNK));
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
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 2);
  if (warp == 16) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 128);
  }
}

// =============================================================================== scan
// writes [B,N,H,4096] FP32 -> states [B,N,H,4096] BF16 (mixed state read by chunk n), and
// optionally the fast / slow states [B,H,4096] FP32 after the first `complete` chunks, with their BF16 mix
// (prefill: a prompt that ends inside a chunk leaves the state of the chunks before it).
// One thread owns four consecutive state elements (16-byte loads, 8-byte stores) and requests the writes of
// SCAN_AHEAD chunks before it runs their recurrence, so a thread keeps 128 bytes in flight instead of 4.
constexpr int SCAN_AHEAD = 8;
constexpr int SCAN_THREADS_FWD = 128;

// What a decode needs of the chunk a prompt ends in: roped K, V and U of its `rest` positions, as the step kernel
// appends them, and zeros behind them (rest = 0 clears the caches).  OPEN_BLOCKS blocks per (sequence, head); 16-byte pieces.  They go
// with the scan's blocks in one launch: neither fills the chip for a few sequences, and a launch of their own was 3 us a layer
// of a 300-token prompt.
constexpr int OPEN_BLOCKS = 4;
struct OpenChunk {
  const __nv_bfloat16* qkvgu;
  const float2* rope;
  int T, rest, H, d;
  __nv_bfloat16 *kc, *vc, *uc;
};
__device__ __forceinline__ void open_chunk(const OpenChunk& o, int block) {
  const int at_head = block / OPEN_BLOCKS, part = block - at_head * OPEN_BLOCKS;
  const int h = at_head % o.H, b = at_head / o.H;
  const size_t cache = static_cast<size_t>(at_head) * CHUNK * HD;
  const __nv_bfloat16* base = o.qkvgu + (static_cast<size_t>(b) * o.T + (o.T - o.rest)) * 5 * o.d + h * HD;
  constexpr int PIECES = CHUNK * 8 / OPEN_BLOCKS;
#pragma unroll
  for (int k0 = 0; k0 < PIECES; k0 += SCAN_THREADS_FWD) {
    const int i = part * PIECES + k0 + threadIdx.x, r = i >> 3, j = i & 7;
    uint4 k = make_uint4(0u, 0u, 0u, 0u), v = k, u = k;
    if (r < o.rest) {
      const __nv_bfloat16* row = base + static_cast<size_t>(r) * 5 * o.d + j * 8;
      k = *reinterpret_cast<const uint4*>(row + o.d);
      v = *reinterpret_cast<const uint4*>(row + 2 * o.d);
      u = *reinterpret_cast<const uint4*>(row + 4 * o.d);
      uint32_t* w = reinterpret_cast<uint32_t*>(&k);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 x = rope_rotate(__bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w[t])),
                                     o.rope[(j * 4 + t) * CHUNK + r]);
        w[t] = pack_bf16x2(x.x, x.y);
      }
    }
    const size_t at = cache + static_cast<size_t>(r) * HD + j * 8;
    *reinterpret_cast<uint4*>(o.kc + at) = k;
    *reinterpret_cast<uint4*>(o.vc + at) = v;
    *reinterpret_cast<uint4*>(o.uc + at) = u;
  }
}

// PROMPT: the blocks past the scan's take the open chunk, and `writes` may be absent where there is no complete chunk.
template <bool PROMPT>
__global__ void __launch_bounds__(SCAN_THREADS_FWD)
memory_scan_kernel(const float* writes, const float* fast_logit,
                   const float* slow_logit, const float* mix_logit,
                   __nv_bfloat16* __restrict__ states, float* __restrict__ final_fast,
                   float* __restrict__ final_slow, __nv_bfloat16* __restrict__ final_mixed,
                   const float* init_fast, const float* init_slow, int B, int N, int complete,
                   int H, const OpenChunk tail) {
  pdl_launch_dependents();
  pdl_wait();
  if constexpr (PROMPT) {
    const int scan_blocks = B * H * (1024 / SCAN_THREADS_FWD);
    if (static_cast<int>(blockIdx.x) >= scan_blocks) {
      open_chunk(tail, blockIdx.x - scan_blocks);
      return;
    }
  }
  const size_t quad = blockIdx.x * static_cast<size_t>(SCAN_THREADS_FWD) + threadIdx.x;  // over B*H*1024 groups of four
  const size_t total = static_cast<size_t>(B) * H * 1024;
  if (quad >= total) return;
  const int e = static_cast<int>(quad % 1024) * 4;
  const int h = (quad / 1024) % H;
  const int b = quad / (1024 * static_cast<size_t>(H));
  const float df = 1.f / (1.f + expf(-fast_logit[h]));
  const float ds = 1.f / (1.f + expf(-slow_logit[h]));
  const float mix = 1.f / (1.f + expf(-mix_logit[h]));
  const size_t flat = quad * 4;
  float4 f = init_fast != nullptr ? *reinterpret_cast<const float4*>(init_fast + flat) : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 s = init_slow != nullptr ? *reinterpret_cast<const float4*>(init_slow + flat) : make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t chunk_stride = static_cast<size_t>(H) * 4096;
  const size_t base = (static_cast<size_t>(b) * N * H + h) * 4096 + e;
  auto mixed = [&]() {
    uint2 o;
    o.x = pack_bf16x2(mix * f.x + (1.f - mix) * s.x, mix * f.y + (1.f - mix) * s.y);
    o.y = pack_bf16x2(mix * f.z + (1.f - mix) * s.z, mix * f.w + (1.f - mix) * s.w);
    return o;
  };
  auto leave = [&]() {
    *reinterpret_cast<float4*>(final_fast + flat) = f;
    *reinterpret_cast<float4*>(final_slow + flat) = s;
    if (final_mixed != nullptr) *reinterpret_cast<uint2*>(final_mixed + flat) = mixed();
  };
  for (int n0 = 0; n0 < N; n0 += SCAN_AHEAD) {
    float4 w[SCAN_AHEAD];
#pragma unroll
    for (int j = 0; j < SCAN_AHEAD; ++j)
      if (n0 + j < (PROMPT ? complete : N)) w[j] = *reinterpret_cast<const float4*>(writes + base + (n0 + j) * chunk_stride);
      else if constexpr (PROMPT) w[j] = make_float4(0.f, 0.f, 0.f, 0.f);   // of the open chunk: nothing reads the state behind it
#pragma unroll
    for (int j = 0; j < SCAN_AHEAD; ++j) {
      if (n0 + j >= N) break;
      if (states != nullptr) *reinterpret_cast<uint2*>(states + base + (n0 + j) * chunk_stride) = mixed();
      if (n0 + j == complete && final_fast != nullptr) leave();
      f.x = df * f.x + (1.f - df) * w[j].x; f.y = df * f.y + (1.f - df) * w[j].y;
      f.z = df * f.z + (1.f - df) * w[j].z; f.w = df * f.w + (1.f - df) * w[j].w;
      s.x = ds * s.x + (1.f - ds) * w[j].x; s.y = ds * s.y + (1.f - ds) * w[j].y;
      s.z = ds * s.z + (1.f - ds) * w[j].z; s.w = ds * s.w + (1.f - ds) * w[j].w;
    }
  }
  if (complete == N && final_fast != nullptr) leave();
}

// =============================================================================== attention
// smem: sQ 16K | sK 16K | sX 16K | sV 16K | sSt 8K | bars  (73 KiB: three CTAs per SM)
// The gate tile arrives by TMA with the other operands (into sX; every thread moves its gate row to
// registers before the softmax) and the blended output leaves by TMA (staged in sQ, one 32-row
// store per warp): a thread that owns a token row would otherwise touch one 16-byte piece of 32
// different cache lines per warp instruction.  P (128 x 128 BF16) overlays sK | sX once S = Q K^T
// is complete.  TMEM: 128 columns; S occupies all of them, and after the softmax has read S, O takes
// columns 0-63 and Mem = Q State columns 64-127, so three CTAs fit the 512 columns of an SM too.
// The kernel is bound by the latency of its dependent chain, so tiles in flight are what counts.
//
// PROMPT: the chunk that a prompt ends in.  A decode step computes such positions with FP32 softmax weights, so here, too,
// no weight is rounded to BF16: it is split into two BF16 terms (2^-17 of it is left out), and O = P_hi V + P_lo V.  The
// low terms wait in registers (64 of them) until the high ones have been consumed, then take their place in shared memory;
// the tiles of complete chunks skip all of it.
constexpr int AF_SMEM = 4 * TILE_BYTES + 8192 + 1024 + 128;

template <bool PROMPT>
__global__ void __launch_bounds__(128, 3)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_state,
                const __grid_constant__ CUtensorMap tm_y, const float2* rope, int T, int H, int d, bool memory,
                int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem;
  uint8_t* sK = smem + TILE_BYTES;
  uint8_t* sG = smem + 2 * TILE_BYTES;   // gate tile, later the second half of P
  uint8_t* sV = smem + 3 * TILE_BYTES;
  uint8_t* sSt = smem + 4 * TILE_BYTES;
  uint8_t* sP = sK;                      // P overlays K | gate
  uint64_t* bars = reinterpret_cast<uint64_t*>(sSt + 8192);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int n_chunks = (T + CHUNK - 1) / CHUNK;
  const int tile = blockIdx.x;
  const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
  const int row0 = n * CHUNK;
  const bool open = PROMPT && row0 + CHUNK > T;

  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_init(&bars[2], 1);
    if (PROMPT) mbar_init(&bars[3], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t t_s = tmem, t_o = tmem, t_m = tmem + 64;  // O and Mem reuse S's columns after the softmax
  const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;

  if (tid == 0) {
    mbar_expect_tx(&bars[0], 4 * TILE_BYTES + (memory ? 8192 : 0));
    tma_load_3d(sQ, &tm_qkvgu, &bars[0], 0 * d + h * HD, row0, b);
    tma_load_3d(sK, &tm_qkvgu, &bars[0], 1 * d + h * HD, row0, b);
    tma_load_3d(sV, &tm_qkvgu, &bars[0], 2 * d + h * HD, row0, b);
    tma_load_3d(sG, &tm_qkvgu, &bars[0], 3 * d + h * HD, row0, b);
    if (memory) tma_load_2d(sSt, &tm_state, &bars[0], 0, tile * HD);
  }
  bool ok = mbar_wait(&bars[0], 0, abort_flag);
  uint4 gate_row[8];  // this thread's gate row: the tile's space becomes half of P
#pragma unroll
  for (int j = 0; j < 8; ++j) gate_row[j] = *reinterpret_cast<const uint4*>(tile_chunk(sG, tid, j));
  if (ok) {
    rope_tanh_row(sQ, tid, rope, true, false);
    rope_tanh_row(sK, tid, rope, true, false);
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (warp == 0 && elect_one() && ok) {
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
#pragma unroll
    for (int k = 0; k < HD / 16; ++k)
      umma_bf16(t_s, make_smem_desc_sw128(smem_u32(sQ) + k * 32, 0, 1024),
                make_smem_desc_sw128(smem_u32(sK) + k * 32, 0, 1024), idesc_s, k > 0);
    umma_commit(&bars[1]);
  }
  ok = ok && mbar_wait(&bars[1], 0, abort_flag);
  tc_fence_after_sync();

  // ---- causal softmax of row `tid` (scores scaled by 1/8); P stays unnormalised
  const float kScale = 0.125f * 1.4426950408889634f;  // fold log2(e)
  float row_max = -INFINITY;
  const int last_chunk = warp;  // columns beyond 32*warp+31 are masked for the whole warp
  for (int cc = 0; cc <= last_chunk; ++cc) {
    uint32_t r[32];
    tmem_ld_32x32b_x32(t_s + lane_base + cc * 32, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (cc * 32 + j <= tid) row_max = fmaxf(row_max, __uint_as_float(r[j]));
  }
  float row_sum = 0.f;
  [[maybe_unused]] uint32_t low[PROMPT ? 4 : 1][16];
#pragma unroll(PROMPT ? 4 : 1)
  for (int cc = 0; cc < 4; ++cc) {
    uint32_t pk[16];
    if (cc <= last_chunk) {
      uint32_t r[32];
      tmem_ld_32x32b_x32(t_s + lane_base + cc * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float p0 = (cc * 32 + j <= tid) ? softmax_term(__uint_as_float(r[j]), row_max, kScale) : 0.f;
        const float p1 = (cc * 32 + j + 1 <= tid) ? softmax_term(__uint_as_float(r[j + 1]), row_max, kScale) : 0.f;
        const __nv_bfloat162 v = __floats2bfloat162_rn(p0, p1);
        const float2 back = __bfloat1622float2(v);
        row_sum += back.x + back.y;  // normalise by what the MMA will actually sum
        pk[j >> 1] = *reinterpret_cast<const uint32_t*>(&v);
        if constexpr (PROMPT) {
          const __nv_bfloat162 l = __floats2bfloat162_rn(p0 - back.x, p1 - back.y);
          const float2 rest = __bfloat1622float2(l);
          if (open) row_sum += rest.x + rest.y;
          low[cc][j >> 1] = *reinterpret_cast<const uint32_t*>(&l);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        pk[j] = 0u;
        if constexpr (PROMPT) low[cc][j] = 0u;
      }
    }
    store_row_chunk32(sP, tid, cc * 32, pk);
  }
  tc_fence_before_sync();  // every thread's reads of S precede the MMAs that overwrite its columns
  fence_proxy_async_smem();
  __syncthreads();
  if (warp == 0 && elect_one() && ok) {
    tc_fence_after_sync();
    constexpr uint32_t idesc_o = make_idesc_bf16(128, 64, false, true);
#pragma unroll
    for (int k = 0; k < CHUNK / 16; ++k)
      umma_bf16(t_o, make_smem_desc_sw128(smem_u32(sP) + (k >> 2) * TILE_BYTES + (k & 3) * 32, 0, 1024),
                make_smem_desc_sw128(smem_u32(sV) + k * 2048, 0, 1024), idesc_o, k > 0);
#pragma unroll
    for (int k = 0; memory && k < HD / 16; ++k)  // Mem = Q State
      umma_bf16(t_m, make_smem_desc_sw128(smem_u32(sQ) + k * 32, 0, 1024),
                make_smem_desc_sw128(smem_u32(sSt) + k * 2048, 0, 1024), idesc_o, k > 0);
    umma_commit(&bars[2]);
  }
  ok = ok && mbar_wait(&bars[2], 0, abort_flag);
  tc_fence_after_sync();
  if constexpr (PROMPT) {
    if (open) {  // O += P_lo V
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) store_row_chunk32(sP, tid, cc * 32, low[cc]);
      fence_proxy_async_smem();
      __syncthreads();
      if (warp == 0 && elect_one() && ok) {
        constexpr uint32_t idesc_o = make_idesc_bf16(128, 64, false, true);
#pragma unroll
        for (int k = 0; k < CHUNK / 16; ++k)
          umma_bf16(t_o, make_smem_desc_sw128(smem_u32(sP) + (k >> 2) * TILE_BYTES + (k & 3) * 32, 0, 1024),
                    make_smem_desc_sw128(smem_u32(sV) + k * 2048, 0, 1024), idesc_o, 1u);
        umma_commit(&bars[3]);
      }
      ok = ok && mbar_wait(&bars[3], 0, abort_flag);
      tc_fence_after_sync();
    }
  }

  // ---- gate blend into the (now idle) Q tile, then one TMA store of the warp's 32 rows
  const float inv_l = 1.f / row_sum;
#pragma unroll
  for (int c = 0; c < HD; c += 16) {
    uint32_t ro[16], rm[16];
    tmem_ld_32x32b_x16(t_o + lane_base + c, ro);
    if (memory) {
      tmem_ld_32x32b_x16(t_m + lane_base + c, rm);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) rm[j] = 0u;
    }
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; j += 8) {
      const int chunk = (c + j) >> 3;
      const uint4 gq = gate_row[chunk];
      const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gq);
      uint4 out;
      uint32_t* ow = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 gf = __bfloat1622float2(gb[t]);
        const float g0 = sigmoid_f(gf.x), g1 = sigmoid_f(gf.y);
        ow[t] = pack_bf16x2(gate_blend(g0, __uint_as_float(ro[j + 2 * t]), inv_l, __uint_as_float(rm[j + 2 * t])),
                            gate_blend(g1, __uint_as_float(ro[j + 2 * t + 1]), inv_l, __uint_as_float(rm[j + 2 * t + 1])));
      }
      *reinterpret_cast<uint4*>(tile_chunk(sQ, tid, chunk)) = out;
    }
  }
  fence_proxy_async_smem();
  __syncwarp();
  if ((tid & 31) == 0) {
    if (ok && row0 + warp * 32 < T) {
      tma_store_3d(&tm_y, sQ + warp * 4096, h * HD, row0 + warp * 32, b);
      tma_store_commit();
    }
    tma_store_wait_read0();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 3);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 128);
  }
}

// =============================================================================== attention, streaming form
// attn_fwd_kernel as one persistent CTA per SM with specialised warps (25 warps):
//
//   warp 24        producer: TMA loads of tile i (Q, K, gate, V, state: 72 KiB) into stage i % 3 of a ring
//   warps 0..7     RoPE workers: thread (row r, half q) rotates four of the eight 16-byte pieces of row r of Q and of
//                  K in place (its 16 (cos, sin) pairs live in registers); worker 0 then issues S = Qr Kr^T and
//                  Mem = Qr State into TMEM set i % 2 -- Mem does not depend on the softmax, so it rides with S
//   warps 8..15    softmax group 0 (tiles 0, 2, 4, ...), warps 16..23 softmax group 1 (tiles 1, 3, ...): two threads per token
//                  row, the first with the front half of the visible blocks of 32 score columns, the second with the rest, each with
//                  half of the output columns; they exchange their maxima and the sum through shared memory.  The sum goes through
//                  the row's columns in order, as one thread has it: the second thread adds its terms to the first one's sum
//                  from P, under the product.  (Two sums added up at the end are 3 to 4 % faster, but change an ulp of
//                  some of a prompt's rows, which every layer behind them multiplies.)  With one thread per row a tile was 14.9 k
//                  clocks of its group, 8192 rows of 32 heads took 50.9 us, 48.7 so; 16 prompts of 1000 tokens with their writes and scan
//                  199 and 172.
//                  As in attn_fwd_kernel: causal softmax straight out of TMEM, unnormalised P (BF16) into
//                  the tile's K and Q space (both dead once S and Mem are complete; the gate tile stays where it is),
//                  O = P V issued by the group's first warp into columns of its own, gate blend from O, Mem
//                  and the gate tile into the Q space, one TMA store per 32 rows; the store's read of the tile releases
//                  the ring stage, the group's last TMEM read releases the TMEM set.
//
// Two tiles are in their softmax / blend phase at any time while a third is being rotated and a fourth loaded;
// attn_fwd_kernel gets its overlap from three independent CTAs per SM, each walking the whole chain alone.
// TMEM: set g = columns [192 g, 192 g + 192): S 128, Mem 64; O of group g = columns [384 + 64 g, 448 + 64 g).  Bit-identical
// results.  PROMPT as in attn_fwd_kernel, but the low terms of P take the place, in TMEM, of the scores that they come from; their product
// reads them there as its first operand.  Formed again from the scores, behind the product of the high ones and into their place in shared
// memory, they were a second pass over the open chunk: 96 tiles of a 300-token prompt (with its writes and scan) 16.8 -> 14.9 us, 4096 tiles of
// 16 x 1000 tokens 172 -> 162 (with a row's sum in two parts).
constexpr int AS_STAGES = 3;
constexpr int AS_THREADS = 25 * 32;
constexpr int AS_STAGE_BYTES = 4 * TILE_BYTES + 8192;
constexpr int AS_MEET = 2 * 3 * 128 * 4;   // per group and row: two maxima, the sum
constexpr int AS_SMEM = AS_STAGES * AS_STAGE_BYTES + AS_MEET + 1024 + 256;

template <bool PROMPT>
__global__ void __launch_bounds__(AS_THREADS, 1)
attn_fwd_stream_kernel(const __grid_constant__ CUtensorMap tm_qkvgu, const __grid_constant__ CUtensorMap tm_state,
                       const __grid_constant__ CUtensorMap tm_y, const float2* rope, int T, int H, int d,
                       int tiles, bool memory, int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  float* meetings = reinterpret_cast<float*>(smem + AS_STAGES * AS_STAGE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AS_STAGES * AS_STAGE_BYTES + AS_MEET);
  uint64_t* full = bars;                     // [3] stage loaded
  uint64_t* empty = bars + AS_STAGES;        // [3] stage released (4 storing warps of the owning group)
  uint64_t* sfull = bars + 2 * AS_STAGES;    // [2] S and Mem complete
  uint64_t* ofull = sfull + 2;               // [2] O complete
  uint64_t* setfree = ofull + 2;             // [2] TMEM set read out (4 storing warps, for two each)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(setfree + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_chunks = (T + CHUNK - 1) / CHUNK;

  if (tid == 0) {
    for (int s = 0; s < AS_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 4);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(&sfull[g], 1);
      mbar_init(&ofull[g], 1);
      mbar_init(&setfree[g], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_qkvgu);
    tma_prefetch_desc(&tm_state);
    tma_prefetch_desc(&tm_y);
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  const int first = blockIdx.x, step = gridDim.x;
  auto stage_ptr = [&](int s) { return smem + s * AS_STAGE_BYTES; };  // Q | K | gate | V | state

  if (warp == 24) {
    if (lane == 0) {
      int i = 0;
      for (int tile = first; tile < tiles; tile += step, ++i) {
        const int s = i % AS_STAGES;
        if (!mbar_wait(&empty[s], ((i / AS_STAGES) & 1) ^ 1, abort_flag)) break;
        const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
        const int row0 = n * CHUNK;
        uint8_t* st = stage_ptr(s);
        mbar_expect_tx(&full[s], memory ? AS_STAGE_BYTES : 4 * TILE_BYTES);
        tma_load_3d(st, &tm_qkvgu, &full[s], 0 * d + h * HD, row0, b);
        tma_load_3d(st + TILE_BYTES, &tm_qkvgu, &full[s], 1 * d + h * HD, row0, b);
        tma_load_3d(st + 2 * TILE_BYTES, &tm_qkvgu, &full[s], 3 * d + h * HD, row0, b);
        tma_load_3d(st + 3 * TILE_BYTES, &tm_qkvgu, &full[s], 2 * d + h * HD, row0, b);
        if (memory) tma_load_2d(st + 4 * TILE_BYTES, &tm_state, &full[s], 0, tile * HD);
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ RoPE workers + S / Mem issue
    const int r = tid & 127, q = tid >> 7;
    float2 cs[16];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int t = 0; t < 4; ++t) cs[j * 4 + t] = rope[((q * 4 + j) * 4 + t) * CHUNK + r];
    int i = 0;
    for (int tile = first; tile < tiles; tile += step, ++i) {
      const int s = i % AS_STAGES, g = i & 1;
      uint8_t* sQ = stage_ptr(s);
      uint8_t* sK = sQ + TILE_BYTES;
      uint8_t* sSt = sQ + 4 * TILE_BYTES;
      const bool ok = mbar_wait(&full[s], (i / AS_STAGES) & 1, abort_flag);
      if (ok) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4* pq = reinterpret_cast<uint4*>(tile_chunk(sQ, r, q * 4 + j));
          uint4* pk = reinterpret_cast<uint4*>(tile_chunk(sK, r, q * 4 + j));
          uint4 qv = *pq, kv = *pk;
          uint32_t* qw = reinterpret_cast<uint32_t*>(&qv);
          uint32_t* kw = reinterpret_cast<uint32_t*>(&kv);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 c = cs[j * 4 + t];
            const float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&qw[t]));
            const float2 qr = rope_rotate(x, c);
            qw[t] = pack_bf16x2(qr.x, qr.y);
            const float2 kr = rope_rotate(__bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&kw[t])), c);
            kw[t] = pack_bf16x2(kr.x, kr.y);
          }
          *pq = qv;
          *pk = kv;
        }
      }
      fence_proxy_async_smem();
      uint32_t any_bad;
      asm volatile(
          "{\n"
          ".reg .pred p, q;\n"
          "setp.ne.u32 q, %1, 0;\n"
          "bar.red.or.pred p, 2, 256, q;\n"
          "selp.u32 %0, 1, 0, p;\n"
          "}\n"
          : "=r"(any_bad)
          : "r"(ok ? 0u : 1u)
          : "memory");
      if (any_bad) break;
      if (warp == 0 && elect_one() && mbar_wait(&setfree[g], ((i >> 1) & 1) ^ 1, abort_flag)) {
        tc_fence_after_sync();
        const uint32_t t_s = tmem + g * 192, t_m = t_s + 128;
        constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
        constexpr uint32_t idesc_m = make_idesc_bf16(128, 64, false, true);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)
          umma_bf16(t_s, make_smem_desc_sw128(smem_u32(sQ) + k * 32, 0, 1024),
                    make_smem_desc_sw128(smem_u32(sK) + k * 32, 0, 1024), idesc_s, k > 0);
#pragma unroll
        for (int k = 0; memory && k < HD / 16; ++k)  // Mem = Qr State
          umma_bf16(t_m, make_smem_desc_sw128(smem_u32(sQ) + k * 32, 0, 1024),
                    make_smem_desc_sw128(smem_u32(sSt) + k * 2048, 0, 1024), idesc_m, k > 0);
        umma_commit(&sfull[g]);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax groups
    const int g = (warp - 8) >> 3;
    const int wq = warp & 3, half = ((warp - 8) >> 2) & 1;   // lane quarter of this warp; which blocks of columns it has
    const int gt = wq * 32 + lane;              // row of the tile = TMEM lane
    const uint32_t t_s = tmem + g * 192, t_o = tmem + 384 + g * 64, t_m = t_s + 128;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const float kScale = 0.125f * 1.4426950408889634f;  // fold log2(e)
    const int last_chunk = wq;  // columns beyond 32*wq+31 are masked for the whole warp
    // this warp's two blocks of 32 columns: the first thread of a row has the front of what is visible (and a block of zeros where that is one)
    const int block0 = half == 0 ? 0 : wq < 2 ? 1 : 2, block1 = half == 0 ? (wq < 2 ? 3 : 1) : block0 + 1;
    float* meet = meetings + g * 384;           // [2][128] maxima | [128] sums
    // whether any of the group's threads is not ok; a barrier of its 256 threads
    auto any_bad = [&](bool ok) {
      uint32_t bad;
      if (g == 0)
        asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 3, 256, q;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(bad) : "r"(ok ? 0u : 1u) : "memory");
      else
        asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 4, 256, q;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(bad) : "r"(ok ? 0u : 1u) : "memory");
      return bad != 0u;
    };
    // the two warps that share 32 rows
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(5 + g * 4 + wq) : "memory"); };
    int i = g;
    for (int tile = first + g * step; tile < tiles; tile += 2 * step, i += 2) {
      const int s = i % AS_STAGES, k2 = i >> 1;
      uint8_t* sQ = stage_ptr(s);
      uint8_t* sK = sQ + TILE_BYTES;
      uint8_t* sG = sQ + 2 * TILE_BYTES;
      uint8_t* sV = sQ + 3 * TILE_BYTES;
      const int h = tile % H, n = (tile / H) % n_chunks, b = tile / (H * n_chunks);
      const int row0 = n * CHUNK;
      const bool open = PROMPT && row0 + CHUNK > T;
      // columns 0..63 of P go to the K tile's space, columns 64..127 to the Q tile's
      auto store_p = [&](int cc, const uint32_t(&pk)[16]) {
        uint8_t* half = (cc < 2) ? sK : sQ;
        const int j0 = (cc & 1) * 4;
#pragma unroll
        for (int w4 = 0; w4 < 4; ++w4)
          *reinterpret_cast<uint4*>(tile_chunk(half, gt, j0 + w4)) =
              make_uint4(pk[4 * w4], pk[4 * w4 + 1], pk[4 * w4 + 2], pk[4 * w4 + 3]);
      };
      auto issue_o = [&] {
        tc_fence_after_sync();
        constexpr uint32_t idesc_o = make_idesc_bf16(128, 64, false, true);
#pragma unroll
        for (int k = 0; k < CHUNK / 16; ++k)
          umma_bf16(t_o, make_smem_desc_sw128(smem_u32((k >> 2) ? sQ : sK) + (k & 3) * 32, 0, 1024),
                    make_smem_desc_sw128(smem_u32(sV) + k * 2048, 0, 1024), idesc_o, k > 0);
        if (open) {   // O += P_lo V
#pragma unroll
          for (int k = 0; k < CHUNK / 16; ++k)
            umma_bf16_ts(t_o, t_s + (k >> 1) * 32 + (k & 1) * 8, make_smem_desc_sw128(smem_u32(sV) + k * 2048, 0, 1024), idesc_o, 1u);
        }
        umma_commit(&ofull[g]);
      };
      uint32_t landed = 0;
      if (lane == 0) landed = mbar_wait(&sfull[g], k2 & 1, abort_flag) ? 1u : 0u;
      bool ok = __shfl_sync(0xffffffffu, landed, 0) != 0u;
      tc_fence_after_sync();
      float row_sum = 0.f, row_max = -INFINITY;
      if (ok) {
        for (int cc = block0; cc <= last_chunk; cc = cc == block0 ? block1 : CHUNK) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_s + lane_base + cc * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (cc * 32 + j <= gt) row_max = fmaxf(row_max, __uint_as_float(v[j]));
        }
      }
      meet[half * 128 + gt] = row_max;
      pair_sync();
      if (ok) {
        row_max = fmaxf(row_max, meet[(half ^ 1) * 128 + gt]);
        // REST: a prompt's open chunk, whose weights are two BF16 terms (a branch per score would cost every tile)
        auto weights = [&](auto rest_too) {
          constexpr bool REST = decltype(rest_too)::value;
          for (int cc = block0; cc < 4; cc = cc == block0 ? block1 : CHUNK) {
            uint32_t pk[16];
            [[maybe_unused]] uint32_t low[16];
            if (cc <= last_chunk) {
              uint32_t v[32];
              tmem_ld_32x32b_x32(t_s + lane_base + cc * 32, v);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                const float p0 = (cc * 32 + j <= gt) ? softmax_term(__uint_as_float(v[j]), row_max, kScale) : 0.f;
                const float p1 = (cc * 32 + j + 1 <= gt) ? softmax_term(__uint_as_float(v[j + 1]), row_max, kScale) : 0.f;
                const __nv_bfloat162 pv = __floats2bfloat162_rn(p0, p1);
                const float2 back = __bfloat1622float2(pv);
                row_sum += back.x + back.y;  // normalise by what the MMA will actually sum
                pk[j >> 1] = *reinterpret_cast<const uint32_t*>(&pv);
                if constexpr (REST) {
                  const __nv_bfloat162 rv = __floats2bfloat162_rn(p0 - back.x, p1 - back.y);
                  const float2 rest = __bfloat1622float2(rv);
                  row_sum += rest.x + rest.y;
                  low[j >> 1] = *reinterpret_cast<const uint32_t*>(&rv);
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) pk[j] = low[j] = 0u;
            }
            store_p(cc, pk);
            if constexpr (REST) tmem_st_32x32b_x16(t_s + lane_base + cc * 32, low);   // over scores that this thread alone reads
          }
          if constexpr (REST) tmem_st_wait();
        };
        if (PROMPT && open) weights(std::integral_constant<bool, PROMPT>{});
        else weights(std::false_type{});
      }
      if (half == 0) meet[256 + gt] = row_sum;
      tc_fence_before_sync();
      fence_proxy_async_smem();
      if (any_bad(ok)) break;
      if (warp == 8 + 8 * g && elect_one()) issue_o();
      if (wq > 0) {   // under the product: behind the first thread's terms the second one's, from P
        if (half == 1) {
          float sum = meet[256 + gt];
          const auto term = [](uint32_t two) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&two));
            return f.x + f.y;
          };
          if (PROMPT && open) tc_fence_after_sync();
#pragma unroll 1
          for (int cc = block0; cc <= last_chunk; ++cc) {
            uint4 p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = *reinterpret_cast<const uint4*>(tile_chunk(cc < 2 ? sK : sQ, gt, (cc & 1) * 4 + j));
            if (PROMPT && open) {
              uint32_t low[16];
              tmem_ld_32x32b_x16(t_s + lane_base + cc * 32, low);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 4; ++j)
                sum = sum + term(p[j].x) + term(low[4 * j]) + term(p[j].y) + term(low[4 * j + 1]) + term(p[j].z) + term(low[4 * j + 2]) +
                      term(p[j].w) + term(low[4 * j + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) sum = sum + term(p[j].x) + term(p[j].y) + term(p[j].z) + term(p[j].w);
            }
          }
          meet[256 + gt] = sum;
        }
        pair_sync();
      }
      row_sum = meet[256 + gt];
      landed = 0;
      if (lane == 0) landed = mbar_wait(&ofull[g], k2 & 1, abort_flag) ? 1u : 0u;
      ok = __shfl_sync(0xffffffffu, landed, 0) != 0u;
      tc_fence_after_sync();
      if (ok) {
        // ---- gate blend into the (now idle) Q tile, then one TMA store of the warp's 32 rows
        const float inv_l = 1.f / row_sum;
#pragma unroll
        for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 16) {
          uint32_t ro[16], rm[16];
          tmem_ld_32x32b_x16(t_o + lane_base + c, ro);
          if (memory) {
            tmem_ld_32x32b_x16(t_m + lane_base + c, rm);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) rm[j] = 0u;
          }
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 8) {
            const int chunk = (c + j) >> 3;
            const uint4 gq = *reinterpret_cast<const uint4*>(tile_chunk(sG, gt, chunk));
            const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gq);
            uint4 out;
            uint32_t* ow = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const float2 gf = __bfloat1622float2(gb[t]);
              const float g0 = sigmoid_f(gf.x), g1 = sigmoid_f(gf.y);
              ow[t] = pack_bf16x2(gate_blend(g0, __uint_as_float(ro[j + 2 * t]), inv_l, __uint_as_float(rm[j + 2 * t])),
                                  gate_blend(g1, __uint_as_float(ro[j + 2 * t + 1]), inv_l, __uint_as_float(rm[j + 2 * t + 1])));
            }
            *reinterpret_cast<uint4*>(tile_chunk(sQ, gt, chunk)) = out;
          }
        }
      }
      tc_fence_before_sync();
      fence_proxy_async_smem();
      pair_sync();
      if (half == 0 && lane == 0) {
        mbar_arrive(&setfree[g]);   // these lanes of S / O / Mem have been read
        if (ok && row0 + wq * 32 < T) {
          tma_store_3d(&tm_y, sQ + wq * 4096, h * HD, row0 + wq * 32, b);
          tma_store_commit();
        }
        tma_store_wait_read0();
        mbar_arrive(&empty[s]);     // neither warp touches these rows of the stage any more
      }
      __syncwarp();
      // a warp that gave up does not leave alone: its next wait fails at once (the abort flag is up), and the
      // group's vote at the next barrier takes all eight warps out together
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0 && error_flag != nullptr) atomicExch(error_flag, 3);
  if (warp == 8) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace ws

using namespace ws;

// Which form the tile kernels of the attention block take: 1 = persistent streaming CTAs, 0 = one tile per CTA,
// -1 = the process default (streaming unless WS_ATTN_STREAM=0 is in the environment).
static int g_attn_stream_mode = -1;
extern "C" void ws_attn_set_stream_mode(int mode) { g_attn_stream_mode = mode; }
extern "C" int ws_attn_stream_form(void) {
  if (g_attn_stream_mode >= 0) return g_attn_stream_mode != 0;
  static const bool from_env = [] {
    const char* e = std::getenv("WS_ATTN_STREAM");
    return e == nullptr || e[0] != '0';
  }();
  return from_env ? 1 : 0;
}

// The tile kernels address tokens as (position, sequence): a chunk that reaches past the end of its sequence reads
// zeros there (the tensor map's fill) and its stores are clipped.  (A prompt of 300 tokens, 28 layers: 65.4 ms when the
// 44 tokens past the second chunk were decode steps, 3.6 in one pass.)  Behind the causal mask those positions change
// nothing of the others, and tanh(0) adds nothing to a write.
static int chunk_writes(const void* qkvgu, const float* rope, float* writes, int B, int T, int H, int d, int* error_flag,
                        cudaStream_t stream) {
  if (T <= 0 || d != H * HD) return -1;
  CUtensorMap tm;
  int rc = make_sequence_map(&tm, qkvgu, 5 * (uint64_t)d, T, B, HD, CHUNK);
  if (rc) return rc;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(chunk_writes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WR_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  const int tiles = B * ((T + CHUNK - 1) / CHUNK) * H;
  CUtensorMap to;
  rc = make_map_f32(&to, writes, HD, (uint64_t)tiles * HD, HD, 32, 32);
  if (rc) return rc;
  const bool stream_form = ws_attn_stream_form() != 0;
  static int sms = 0;
  if (stream_form && sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(chunk_writes_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WS_SMEM) != cudaSuccess)
      return -20;
  }
  if (stream_form)
    launch_dependent(chunk_writes_stream_kernel, dim3(tiles < sms ? tiles : sms), dim3(WS_THREADS), WS_SMEM, stream, tm, to,
                     reinterpret_cast<const float2*>(rope), T, H, d, tiles, error_flag);
  else
    launch_dependent(chunk_writes_kernel, dim3(tiles), dim3(128), WR_SMEM, stream, tm, to, reinterpret_cast<const float2*>(rope), T, H, d,
                     error_flag);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ws_chunk_writes(const void* qkvgu, const float* rope, float* writes, int B, int T, int H, int d,
                               int* error_flag, cudaStream_t stream) {
  return T % CHUNK != 0 ? -1 : chunk_writes(qkvgu, rope, writes, B, T, H, d, error_flag, stream);
}

// `tail`: a prompt's open chunk, which goes along; NULL: none.
static int memory_scan(const float* writes, const float* fast_logit, const float* slow_logit, const float* mix_logit,
                       void* states, float* final_fast, float* final_slow, void* final_mixed, const float* init_fast,
                       const float* init_slow, int B, int N, int complete, int H, const OpenChunk* tail, cudaStream_t stream) {
  const int blocks = B * H * (1024 / SCAN_THREADS_FWD);
  launch_dependent(tail != nullptr ? memory_scan_kernel<true> : memory_scan_kernel<false>,
                   dim3(blocks + (tail != nullptr ? B * H * OPEN_BLOCKS : 0)), dim3(SCAN_THREADS_FWD), 0, stream, writes, fast_logit,
                   slow_logit, mix_logit, (__nv_bfloat16*)states, final_fast, final_slow, (__nv_bfloat16*)final_mixed,
                   init_fast, init_slow, B, N, complete, H, tail != nullptr ? *tail : OpenChunk{});
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ws_memory_scan(const float* writes, const float* fast_logit, const float* slow_logit,
                              const float* mix_logit, void* states, float* final_fast, float* final_slow,
                              const float* init_fast, const float* init_slow, int B, int N, int H,
                              cudaStream_t stream) {
  return memory_scan(writes, fast_logit, slow_logit, mix_logit, states, final_fast, final_slow, nullptr, init_fast,
                     init_slow, B, N, N, H, nullptr, stream);
}

template <bool PROMPT>
static int attn_fwd(const void* qkvgu, const void* states, const float* rope, void* y, int B, int T, int H, int d,
                    int* error_flag, cudaStream_t stream) {
  if (T <= 0 || d != H * HD) return -1;
  const int tiles = B * ((T + CHUNK - 1) / CHUNK) * H;
  CUtensorMap tm, ts, ty;
  int rc = make_sequence_map(&tm, qkvgu, 5 * (uint64_t)d, T, B, HD, CHUNK);
  if (rc) return rc;
  const bool memory = states != nullptr;   // otherwise every position is in a sequence's first chunk, whose memories are empty
  rc = make_tile_map(&ts, memory ? states : qkvgu, HD, (uint64_t)tiles * HD, HD, HD, HD);
  if (rc) return rc;
  rc = make_sequence_map(&ty, y, (uint64_t)d, T, B, HD, 32);
  if (rc) return rc;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attn_fwd_kernel<PROMPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, AF_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(attn_fwd_stream_kernel<PROMPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, AS_SMEM) != cudaSuccess)
      return -20;
  }
  if (ws_attn_stream_form() != 0)
    launch_dependent(attn_fwd_stream_kernel<PROMPT>, dim3(tiles < sms ? tiles : sms), dim3(AS_THREADS), AS_SMEM, stream, tm, ts, ty,
                     reinterpret_cast<const float2*>(rope), T, H, d, tiles, memory, error_flag);
  else
    launch_dependent(attn_fwd_kernel<PROMPT>, dim3(tiles), dim3(128), AF_SMEM, stream, tm, ts, ty,
                     reinterpret_cast<const float2*>(rope), T, H, d, memory, error_flag);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ws_attn_fwd(const void* qkvgu, const void* states, const float* rope, void* y, int B, int T, int H,
                           int d, int* error_flag, cudaStream_t stream) {
  return T % CHUNK != 0 ? -1 : attn_fwd<false>(qkvgu, states, rope, y, B, T, H, d, error_flag, stream);
}

extern "C" int ws_attn_prefill(const void* qkvgu, const float* rope, const float* fast_logit, const float* slow_logit,
                               const float* mix_logit, float* writes, void* states, void* y, float* fast, float* slow,
                               void* mixed, void* kc, void* vc, void* uc, int B, int T, int H, int d, int* error_flag,
                               cudaStream_t stream) {
  const int complete = T / CHUNK, rest = T % CHUNK;
  // A prompt without a complete chunk writes nothing into the memories and reads nothing from them.
  int rc = complete > 0 ? chunk_writes(qkvgu, rope, writes, B, T, H, d, error_flag, stream) : 0;
  const OpenChunk tail{static_cast<const __nv_bfloat16*>(qkvgu), reinterpret_cast<const float2*>(rope), T, rest, H, d,
                       static_cast<__nv_bfloat16*>(kc), static_cast<__nv_bfloat16*>(vc), static_cast<__nv_bfloat16*>(uc)};
  if (!rc)
    rc = memory_scan(writes, fast_logit, slow_logit, mix_logit, complete > 0 ? states : nullptr, fast, slow, mixed, nullptr, nullptr, B,
                     complete + (rest > 0), complete, H, &tail, stream);
  if (!rc) rc = attn_fwd<true>(qkvgu, complete > 0 ? states : nullptr, rope, y, B, T, H, d, error_flag, stream);
  return rc;
}
