// LM-head cross-entropy helpers.  The vocabulary projection itself runs in the tcgen05 GEMM with
// the WS_EPI_CE_FWD / WS_EPI_CE_BWD epilogues (gemm2_tcgen05.cu, gemm_tcgen05.cu), so a forward pass that no
// backward pass follows writes no logits; before one it may leave BF16 logits behind.  This file combines the
// per-128-column (max, sum exp) partials of a row into its log-sum-exp and label log-probability, packs the
// labelled rows, and turns kept logits into their gradients.
//
// Replaces the reference's chunked / full LM-head losses (warpstate/model.py:316-334,
// ops/loss_experiment.py:14-19: BF16 head GEMM, FP32 cast of the logits, log-softmax, NLL) and
// the per-sequence log-probability head of DPO (dpo.py:150-161).
#include "ws_ptx.cuh"
#include "ws_api.h"
#include "ws_launch.h"

namespace ws {

extern "C" void ws_count_launch(void);

// One warp per row.  parts: float2 [rows, ld] with `nparts` valid entries per row.
// lse[row] = log sum_j exp(logit_j);  logp[row] = label_logit - lse (0 where label == ignore).
__global__ void __launch_bounds__(256)
ce_combine_kernel(const float2* parts, int ld, int nparts, const float* label_logit,
                  const long long* labels, long long ignore_index, int rows, const int* index,
                  const int* count, float* __restrict__ lse_out, float* __restrict__ logp_out) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + warp;
  if (row >= rows || (count != nullptr && row >= *count)) return;
  const float2* pr = parts + static_cast<size_t>(row) * ld;
  float mx = -INFINITY;
  for (int i = lane; i < nparts; i += 32) mx = fmaxf(mx, pr[i].x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float s = 0.f;
  for (int i = lane; i < nparts; i += 32) {
    const float2 v = pr[i];
    s += v.y * expf(v.x - mx);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const float lse = mx + logf(s);
    lse_out[row] = lse;
    const long long lab = labels[row];
    logp_out[index != nullptr ? index[row] : row] = (lab == ignore_index) ? 0.f : label_logit[row] - lse;
  }
}

// --------------------------------------------------------------------------- labelled rows
// A post-training batch labels the responses only (a quarter to a half of the padded positions), and an unlabelled row
// adds nothing to the loss or to any gradient: the head's GEMMs run over the labelled rows, packed together.  How
// many there are stays on the device (the GEMM reads it), so nothing waits for the host.
//
// One CTA: a thread has SELECT_ITEMS labels in flight, a rank is the count of labelled rows before it (warp ballots,
// then a scan over the warps of the block).  It is one round trip to memory per 16384 rows, whatever the labels are.
// Head forward + backward at 4 x 2048 rows of which 2302 are labelled, d 2048, vocabulary 32768: 3.44 -> 1.20 ms; with
// all of 16384 rows labelled the three small kernels are within the noise of 7.2 ms (nothing is copied).
constexpr int SELECT_THREADS = 1024;
constexpr int SELECT_ITEMS = 16;
constexpr int SELECT_PAD = 256;   // rows of a tile of the CTA-pair GEMM

__global__ void __launch_bounds__(SELECT_THREADS)
select_rows_kernel(const long long* labels, long long ignore_index, int rows, int* __restrict__ index,
                   int* __restrict__ count, long long* __restrict__ labels_sel, float* __restrict__ logp) {
  __shared__ int counts[SELECT_ITEMS * 32];   // labelled rows per (item, warp), then those before it
  __shared__ int total;
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int before = 0;
  for (int base = 0; base < rows; base += SELECT_THREADS * SELECT_ITEMS) {
    long long label[SELECT_ITEMS];
    unsigned taken[SELECT_ITEMS];
#pragma unroll
    for (int i = 0; i < SELECT_ITEMS; ++i) {
      const int row = base + i * SELECT_THREADS + tid;
      label[i] = row < rows ? labels[row] : ignore_index;
    }
#pragma unroll
    for (int i = 0; i < SELECT_ITEMS; ++i) {
      taken[i] = __ballot_sync(0xffffffffu, label[i] != ignore_index);
      if (lane == 0) counts[i * 32 + warp] = __popc(taken[i]);
    }
    __syncthreads();
    if (warp == 0) {   // exclusive scan over the 512 counts, 16 of them per lane
      int own[SELECT_ITEMS], sum = 0;
#pragma unroll
      for (int j = 0; j < SELECT_ITEMS; ++j) {
        own[j] = counts[lane * SELECT_ITEMS + j];
        sum += own[j];
      }
      int run = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
      }
      if (lane == 31) total = run;
      run -= sum;
#pragma unroll
      for (int j = 0; j < SELECT_ITEMS; ++j) {
        counts[lane * SELECT_ITEMS + j] = run;
        run += own[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SELECT_ITEMS; ++i) {
      const int row = base + i * SELECT_THREADS + tid;
      if (row >= rows) continue;
      if (label[i] != ignore_index) {
        const int at = before + counts[i * 32 + warp] + __popc(taken[i] & ((1u << lane) - 1u));
        index[at] = row;
        labels_sel[at] = label[i];
      } else {
        logp[row] = 0.f;
      }
    }
    before += total;
    __syncthreads();
  }
  const int pad = min(rows, (before + SELECT_PAD - 1) / SELECT_PAD * SELECT_PAD);
  for (int r = before + tid; r < pad; r += SELECT_THREADS) {
    index[r] = -1;
    labels_sel[r] = ignore_index;
  }
  if (tid == 0) *count = before;
}

// One warp per row of 16-byte pieces (d % 8 == 0).
__global__ void __launch_bounds__(256)
gather_rows_kernel(const __nv_bfloat16* in, int ld, const int* index,
                   const int* count, int rows, int d, __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  const int n = *count, row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (n == rows || row >= min(rows, (n + SELECT_PAD - 1) / SELECT_PAD * SELECT_PAD)) return;
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * d);
  if (row >= n) {
    for (int i = lane; i < d / 8; i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const uint4* src = reinterpret_cast<const uint4*>(in + static_cast<size_t>(index[row]) * ld);
  constexpr int PIECES = 8;   // per lane in flight: a load does not pass the store of an earlier piece
  for (int i0 = lane; i0 < d / 8; i0 += 32 * PIECES) {
    uint4 piece[PIECES];
#pragma unroll
    for (int q = 0; q < PIECES; ++q)
      if (i0 + 32 * q < d / 8) piece[q] = src[i0 + 32 * q];
#pragma unroll
    for (int q = 0; q < PIECES; ++q)
      if (i0 + 32 * q < d / 8) dst[i0 + 32 * q] = piece[q];
  }
}

__global__ void __launch_bounds__(256)
clear_unlabelled_kernel(const long long* labels, long long ignore_index, int rows, int d,
                        __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows || labels[row] != ignore_index) return;
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * d);
  for (int i = lane; i < d / 8; i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Logit gradients from logits that the forward pass kept: one CTA per row, 16-byte pieces, read and written once.  At
// 8192 x 32768 that is 1 GiB of traffic (0.16 ms at the copy rate) in place of the product that makes the logits again
// (1.1 TFLOP, 0.7 ms).  Head forward + backward at 16384 labelled rows: 7.3 -> 5.8 ms, at 2302: 1.22 -> 0.99 ms.  Same
// arithmetic as the WS_EPI_CE_BWD epilogue on the same BF16 logits: the same bits.
constexpr int DLOGITS_PAD = 64;   // rows per k-block of the weight gradient

__global__ void __launch_bounds__(256)
ce_dlogits_kernel(__nv_bfloat16* logits, int vocab, const long long* labels_sel,
                  const int* index, const float* lse_in, const float* row_weight,
                  const int* count, int start, int rows) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  const int n = min(max(*count - start, 0), rows);
  if (row >= min(rows, (n + DLOGITS_PAD - 1) / DLOGITS_PAD * DLOGITS_PAD)) return;
  uint4* line = reinterpret_cast<uint4*>(logits + static_cast<size_t>(row) * vocab);
  if (row >= n) {
    for (int i = threadIdx.x; i < vocab / 8; i += 256) line[i] = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const float lse = lse_in[row], w = row_weight[index[row]];
  const long long lab = labels_sel[row];
#pragma unroll 4
  for (int i = threadIdx.x; i < vocab / 8; i += 256) {
    uint4 v = line[i];
    uint32_t* q = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q[t]));
      const int col = i * 8 + 2 * t;
      float d0 = __expf(x.x - lse), d1 = __expf(x.y - lse);
      if (col == lab) d0 -= 1.f;
      if (col + 1 == lab) d1 -= 1.f;
      q[t] = pack_bf16x2(d0 * w, d1 * w);
    }
    line[i] = v;
  }
}

}  // namespace ws

using namespace ws;

extern "C" int ws_ce_combine(const void* parts, int ld, int nparts, const float* label_logit,
                             const long long* labels, long long ignore_index, int rows, const int* index,
                             const int* count, float* lse, float* logp, cudaStream_t stream) {
  if (rows <= 0 || nparts <= 0) return -1;
  launch_dependent(ce_combine_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, reinterpret_cast<const float2*>(parts), ld, nparts,
                                                         label_logit, labels, ignore_index, rows, index, count, lse, logp);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_select_rows(const long long* labels, long long ignore_index, int rows, int* index, int* count,
                              long long* labels_sel, float* logp, cudaStream_t stream) {
  if (rows <= 0) return -1;
  launch_dependent(select_rows_kernel, dim3(1), dim3(SELECT_THREADS), 0, stream, labels, ignore_index, rows, index, count,
                   labels_sel, logp);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_gather_rows(const void* in, int ld, const int* index, const int* count, int rows, int d, void* out,
                              cudaStream_t stream) {
  if (rows <= 0 || d % 8 != 0 || ld % 8 != 0) return -1;
  launch_dependent(gather_rows_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream,
                   static_cast<const __nv_bfloat16*>(in), ld, index, count, rows, d, static_cast<__nv_bfloat16*>(out));
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_clear_unlabelled(const long long* labels, long long ignore_index, int rows, int d, void* out,
                                   cudaStream_t stream) {
  if (rows <= 0 || d % 8 != 0) return -1;
  launch_dependent(clear_unlabelled_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, labels, ignore_index, rows, d,
                   static_cast<__nv_bfloat16*>(out));
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int ws_ce_dlogits(void* logits, int vocab, const long long* labels_sel, const int* index, const float* lse,
                             const float* row_weight, const int* count, int start, int rows, cudaStream_t stream) {
  if (rows <= 0 || vocab % 8 != 0) return -1;
  launch_dependent(ce_dlogits_kernel, dim3(rows), dim3(256), 0, stream, static_cast<__nv_bfloat16*>(logits), vocab,
                   labels_sel, index, lse, row_weight, count, start, rows);
  ws_count_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
