// Products of few tokens with the operands' roles exchanged: out[m, n] = x[m, k] W[n, k]^T where a CTA pair's 256-row operand
// is a tile of W and the tokens, padded to 32 (above 256 to 64), are its columns.
//
// What bounds a projection of a few hundred tokens on the pair kernel (gemm2_tcgen05.cu) is its tile of 256 tokens: 128
// of them leave half of it to padding, 300 take two of them, and the 80 or 112 tiles of in_proj or up/gate are then two rounds
// over 74 CTA pairs.  Here 300 tokens are one tile of 320 columns (two accumulators of 160), 40 or 56 tiles, one round.
// k-blocks cost 0.28 us per 256 columns on the tensor cores and 16 KiB of W plus 64 bytes per column of an SM's intake.
//
// The accumulator has features in its lanes and tokens in its columns: results are transposed on their way through shared
// memory and leave as 32 x 32 tiles by TMA.  SwiGLU: a CTA's 128 rows are 64 of up and the 64 of gate that belong to them;
// the gate rows' warps hand silu(gate) to the up rows' warps, 32 tokens at a time.
//
// Roles, barriers and bounds are the pair kernel's: warp 0 TMA producer (the leader announces both CTAs' bytes), warp 1 TMEM
// owner and, in the leader, MMA issuer, warps 2-9 epilogue.  Every wait is bounded.
#include "ws_ptx.cuh"
#include "ws_api.h"
#include "ws_tma_host.h"
#include "gemm_epilogue.cuh"
#include "ws_launch.h"

#include <cuda_bf16.h>

#include <cstring>

namespace ws {

extern "C" void ws_count_launch(void);

namespace rowsk {
constexpr int BM = 128, BK = 64, THREADS = 320, MAX_STAGES = 8, MAX_TOKENS = 512;
constexpr int A_BYTES = BM * BK * 2;
constexpr int EXCHANGE = 2 * 2 * 64 * 32 * 4;  // SwiGLU: per warpgroup two blocks of 64 features x 32 tokens, FP32
// Two tiles of 32 x 32 BF16 for each warp that stores: all eight, or the four of the up rows.
template <bool SWIGLU>
constexpr int staging_bytes() { return (SWIGLU ? 4 : 8) * 4096; }
template <bool SWIGLU>
constexpr int ring_bytes() { return (SWIGLU ? 176 : 192) * 1024; }
template <bool SWIGLU>
constexpr int smem_bytes() { return 1024 + ring_bytes<SWIGLU>() + staging_bytes<SWIGLU>() + (SWIGLU ? EXCHANGE : 0); }
static_assert(smem_bytes<false>() <= 231424 && smem_bytes<true>() <= 231424, "");
}  // namespace rowsk

struct alignas(64) RowsProblem {
  CUtensorMap w, x, out;
  int m, n, k;           // n: features of the output
  int blocks, width;     // accumulators per tile, columns of each
  int stages, buffers;
  int wide, ahead;         // ahead: W may be read ahead of the launches in front of this one (WsGemm::b_ahead)
  int* error_flag;
};

template <bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(rowsk::THREADS, 1)
gemm_rows_kernel(const __grid_constant__ RowsProblem p) {
  using namespace rowsk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int half = p.width / 2, b_bytes = p.blocks * half * 128, stages = p.stages, stage_bytes = A_BYTES + b_bytes;
  uint8_t* sA = smem;
  uint8_t* sB = smem + stages * A_BYTES;
  uint8_t* staging = smem + ring_bytes<SWIGLU>();
  [[maybe_unused]] float* exchange = reinterpret_cast<float*>(staging + staging_bytes<SWIGLU>());
  __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES], tfull[2], tempty[2];
  __shared__ uint32_t tmem_address;
  __shared__ int aborted;
  volatile int* abort_flag = &aborted;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 16);   // epilogue warps of both CTAs
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.w);
    tma_prefetch_desc(&p.x);
    tma_prefetch_desc(&p.out);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_address, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_address;
  pdl_launch_dependents();
  if (warp != 0 || !p.ahead) pdl_wait();

  constexpr int FEATURES = SWIGLU ? 128 : 256;   // of a tile; a CTA has half of them
  const int tiles = (p.n + FEATURES - 1) / FEATURES, num_k = (p.k + BK - 1) / BK;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, columns = p.blocks * p.width;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      auto load_weights = [&](int stage, int f0, int kb) {
        const uint32_t bar = mapa_shared(smem_u32(&full[stage]), 0);
        if (leader) mbar_expect_tx(&full[stage], 2 * stage_bytes);
        uint8_t* a = sA + stage * A_BYTES;
        tma_load_2d_pair(a, &p.w, bar, kb * BK, f0);
        if (SWIGLU) tma_load_2d_pair(a + 64 * 128, &p.w, bar, kb * BK, p.n + f0);
      };
      // the weights of the first ring, under the tail of the kernel whose result the tokens are
      int requested = 0;
      if (p.ahead) {
        if (pair < tiles)
          for (; requested < min(num_k, stages); ++requested)
            load_weights(requested, pair * FEATURES + static_cast<int>(rank) * (FEATURES / 2), requested);
        pdl_wait();
      }
      for (int tile = pair; tile < tiles && ok; tile += pairs) {
        const int f0 = tile * FEATURES + static_cast<int>(rank) * (FEATURES / 2);
        for (int kb = 0; kb < num_k; ++kb) {
          if (!mbar_wait(&empty[s], ph, abort_flag)) {
            ok = false;
            break;
          }
          const uint32_t bar = mapa_shared(smem_u32(&full[s]), 0);
          if (tile != pair || kb >= requested) load_weights(s, f0, kb);
          for (int j = 0; j < p.blocks; ++j)
            tma_load_2d_pair(sB + s * b_bytes + j * half * 128, &p.x, bar, kb * BK, j * p.width + static_cast<int>(rank) * half);
          if (++s == stages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (leader && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(2 * BM, p.width, false, false);
      int s = 0, count = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = pair; tile < tiles && ok; tile += pairs, ++count) {
        const int buf = p.buffers == 2 ? count & 1 : 0;
        const uint32_t use = p.buffers == 2 ? count >> 1 : count;
        if (!mbar_wait(&tempty[buf], (use & 1) ^ 1, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem + buf * columns;
        for (int kb = 0; kb < num_k; ++kb) {
          if (!mbar_wait(&full[s], ph, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint64_t a = make_smem_desc_sw128(smem_u32(sA + s * A_BYTES), 0, 1024);
          const uint64_t b = make_smem_desc_sw128(smem_u32(sB + s * b_bytes), 0, 1024);
          for (int j = 0; j < p.blocks; ++j)
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_bf16_pair(acc + j * p.width, a + 2 * k, b + j * (half * 8) + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit_pair_mask(smem_u32(&empty[s]), 3);
          if (++s == stages) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok) umma_commit_pair_mask(smem_u32(&tfull[buf]), 3);
      }
    }
  } else {
    const int quarter = warp & 3, group = (warp - 2) >> 2, chunks = (p.m + 31) / 32;
    const bool gate = SWIGLU && quarter >= 2;
    uint8_t* tile_of = staging + (SWIGLU ? group * 2 + (quarter & 1) : warp - 2) * 4096;
    [[maybe_unused]] float* handed = exchange + group * 2 * 64 * 32;
    int count = 0, sent = 0, step = 0;
    for (int tile = pair; tile < tiles; tile += pairs, ++count) {
      const int buf = p.buffers == 2 ? count & 1 : 0;
      const uint32_t use = p.buffers == 2 ? count >> 1 : count;
      bool ok = mbar_wait_warp(&tfull[buf], use & 1, abort_flag);
      if constexpr (SWIGLU) {   // the group meets at barriers below: if one of its warps gave up, all leave together
        uint32_t bad;
        if (group == 0)
          asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 1, 128, q;\n selp.u32 %0, 1, 0, p;\n}\n"
                       : "=r"(bad) : "r"(ok ? 0u : 1u) : "memory");
        else
          asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 2, 128, q;\n selp.u32 %0, 1, 0, p;\n}\n"
                       : "=r"(bad) : "r"(ok ? 0u : 1u) : "memory");
        ok = bad == 0u;
      }
      if (!ok) break;
      tc_fence_after_sync();
      const int x0 = tile * FEATURES + static_cast<int>(rank) * (FEATURES / 2) + quarter * 32;
      const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + buf * columns;
#pragma unroll 1
      for (int chunk = group; chunk < chunks; chunk += 2, ++step) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + chunk * 32, r);
        tmem_ld_wait();
        if constexpr (SWIGLU) {
          float* block = handed + (step & 1) * 64 * 32;   // [token][feature]; the other block may still be read
          const int f = (quarter & 1) * 32 + lane;
          if (gate) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float g = swiglu_input(__uint_as_float(r[j]), p.wide);
              block[j * 64 + f] = g * sigmoidf_(g);
            }
          }
          if (group == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
          else asm volatile("bar.sync 2, 128;" ::: "memory");
          if (gate) continue;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            r[j] = __float_as_uint(block[j * 64 + f] * swiglu_input(__uint_as_float(r[j]), p.wide));
        }
        uint8_t* t = tile_of + (sent++ & 1) * 2048;
        if (lane == 0) tma_store_wait_read1();   // the store issued from this tile two chunks ago has read it
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j)
          *reinterpret_cast<__nv_bfloat16*>(tile_chunk64(t, j, lane >> 3) + (lane & 7) * 2) = __float2bfloat16_rn(__uint_as_float(r[j]));
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (x0 < p.n) tma_store_2d(&p.out, t, x0, chunk * 32);
          tma_store_commit();
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_relaxed(mapa_shared(smem_u32(&tempty[buf]), 0));
    }
    if (lane == 0) tma_store_wait_all();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 6);
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem, 512);
  }
}

template <bool SWIGLU>
static int launch_rows(const RowsProblem& p, int pairs, cudaStream_t stream) {
  static bool configured = false;
  auto kern = gemm_rows_kernel<SWIGLU>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, rowsk::smem_bytes<SWIGLU>()) != cudaSuccess) return -20;
    configured = true;
  }
  launch_dependent(kern, dim3(2 * pairs), dim3(rowsk::THREADS), rowsk::smem_bytes<SWIGLU>(), stream, p);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

// Columns a tile has for m tokens: a multiple of 32 in one accumulator, of 64 in two.
static int rows_columns(int m) { return m <= 256 ? (m + 31) / 32 * 32 : (m + 63) / 64 * 64; }

}  // namespace ws

using namespace ws;

// Whether a product takes this kernel: few tokens, not so few tiles that it is cut along k, and the rounds over the chip times
// what a k-block takes, in units of 0.28 us (256 x 256 x 64 on a pair), here and on the pair kernel.  The SwiGLU epilogue costs
// 1-2 us more here, with half of its warps waiting for the others, so it needs a wider margin, above all behind a short
// contraction.  Measured with cold weights (pair -> here, us): in_proj of d 2048 at 128 tokens 23.6 -> 20.5, 192 23.6 -> 22.6,
// 256 23.6 -> 23.4, 300 33.8 -> 26.7, 384 33.8 -> 28.7, 448 33.8 -> 30.8, 512 33.8 -> 32.8; up/gate at 128 27.6 -> 24.6, 192
// 27.7 -> 26.7, 224 27.6 -> 28.7, 300 37.9 -> 32.8, 448 37.9 -> 36.9, 512 37.9 -> 41.0; d 1280 in_proj at 128 17.4 -> 16.4, 300
// 17.4 -> 18.5, up/gate at 128 18.5 -> 18.4, 192 18.4 -> 19.5.
// And where the single-CTA kernel would take the product, fewer than twice the rounds that it needs: its tiles of 128 tokens are
// spread over all SMs one by one, so 75 to 148 of them are one round there and two here, 128 x 20480 outputs of k 4096 38.9 ->
// 47.3 us, 128 x 32768 of k 2048 27.7 -> 27.5, SwiGLU 128 x 10752 of k 2048 21.8 -> 28.2; but three rounds for two pay, 128 x 40000 of
// k 1024 26.4 -> 21.3, of k 2048 43.6 -> 37.5, SwiGLU 128 x 27000 of k 2048 43.8 -> 41.5.
// In a chain of launches, over 29 sizes of W (k 1024 to 4096) at 12 token counts: what is taken takes 0.73 to 1.00 of what it did
// as a BF16 product and 0.79 to 1.05 as SwiGLU; the slower ones are 160 to 192 tokens at few tiles, and 160 to 300 at k 3072
// where two rounds are nearly empty.
extern "C" int ws_gemm_rows_takes(int m, int n, int k, int epilogue, int packed, int sms) {
  const bool swiglu = epilogue == WS_EPI_SWIGLU;
  if ((epilogue != WS_EPI_BF16 && !(swiglu && !packed)) || m < 96 || m > rowsk::MAX_TOKENS || n % 8 != 0 || k < 1024 || sms < 2)
    return 0;
  const int plan = ws_gemm_plan(m, n, k, 0, epilogue, packed, sms);
  const int pairs = sms / 2, columns = rows_columns(m), weights = swiglu ? 2 * n : n;
  const int here = ((weights + 255) / 256 + pairs - 1) / pairs;
  const int single = ((m + 127) / 128 * ((weights + 255) / 256) + sms - 1) / sms;
  if (plan > 1 || (plan == 0 && here >= 2 * single)) return 0;
  const int there = ((m + 255) / 256 * ((weights + 255) / 256) + pairs - 1) / pairs;
  const float tensor = columns / 256.f, intake = (16384.f + 64.f * columns) / 32768.f;
  const float margin = !swiglu ? 0.97f : k >= 2048 ? 0.9f : 0.8f;
  return here * (tensor > intake ? tensor : intake) <= margin * there ? 1 : 0;
}

extern "C" int ws_gemm_rows(const WsGemm* g, int sms, cudaStream_t stream) {
  const bool swiglu = g->epilogue == WS_EPI_SWIGLU;
  RowsProblem p;
  memset(&p, 0, sizeof(p));
  p.m = g->m; p.n = g->n; p.k = g->k; p.wide = g->wide; p.ahead = g->b_ahead; p.error_flag = g->error_flag;
  const int columns = rows_columns(g->m);
  p.blocks = columns <= 256 ? 1 : 2;
  p.width = columns / p.blocks;
  p.buffers = columns <= 256 ? 2 : 1;
  const int stage = rowsk::A_BYTES + p.blocks * (p.width / 2) * 128;
  const int ring = swiglu ? rowsk::ring_bytes<true>() : rowsk::ring_bytes<false>();
  p.stages = ring / stage < rowsk::MAX_STAGES ? ring / stage : rowsk::MAX_STAGES;
  int rc = make_map_bf16(&p.w, g->b, g->k, swiglu ? 2 * g->n : g->n, g->ldb, rowsk::BK, swiglu ? 64 : 128);
  if (!rc) rc = make_map_bf16(&p.x, g->a, g->k, g->m, g->lda, rowsk::BK, p.width / 2);
  if (!rc)
    rc = make_map_bf16_swz(&p.out, swiglu ? g->out2 : g->out, g->n, g->m, swiglu ? g->ldo2 : g->ldo, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  if (rc) return rc;
  const int per_tile = swiglu ? 128 : 256, tiles = (g->n + per_tile - 1) / per_tile;
  const int pairs = tiles < sms / 2 ? tiles : sms / 2;
  return swiglu ? launch_rows<true>(p, pairs, stream) : launch_rows<false>(p, pairs, stream);
}
