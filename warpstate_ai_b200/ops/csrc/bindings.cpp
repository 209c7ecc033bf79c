// torch.ops.ws_b200.* registrations: argument checking and pointer extraction only; all
// device work is in the .cu files behind the C ABI of ws_api.h.
#include <cstdio>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <algorithm>
#include <string>
#include <tuple>
#include <vector>

#include "ws_api.h"

namespace {

cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// The message is built as a std::string first: passing the `const char*` and the int straight
// to TORCH_CHECK's variadic formatter crashed the process (SIGSEGV) instead of throwing.
void check_rc(int rc, const char* what) {
  if (rc != 0) {
    const std::string message = std::string("ws_b200::") + what + " failed with code " + std::to_string(rc);
    TORCH_CHECK(false, message);
  }
}

const void* opt_ptr(const c10::optional<at::Tensor>& t) {
  return t.has_value() && t->defined() ? t->data_ptr() : nullptr;
}
int64_t opt_ld(const c10::optional<at::Tensor>& t) {
  return t.has_value() && t->defined() && t->dim() >= 2 ? t->stride(0) : 0;
}

// Generic GEMM entry.  `a`/`b` are 2-D BF16 tensors whose last dimension is contiguous; the
// caller states how they are to be read (a_mn/b_mn) and the problem size.
void gemm(const at::Tensor& a, const at::Tensor& b, bool a_mn, bool b_mn, int64_t epilogue,
          int64_t m, int64_t n, int64_t k, c10::optional<at::Tensor> out_, c10::optional<at::Tensor> out2,
          c10::optional<at::Tensor> aux, c10::optional<at::Tensor> row_scale, double alpha,
          double beta, c10::optional<at::Tensor> error_flag, bool wide) {
  // the packed (up | gate) matrix of the SwiGLU epilogue is optional: only a backward pass reads it
  const bool has_out = out_.has_value() && out_->defined();
  TORCH_CHECK(has_out || (out2.has_value() && out2->defined()), "gemm: an output is required");
  TORCH_CHECK(has_out || epilogue == WS_EPI_SWIGLU, "gemm: out required");
  const at::Tensor& out = has_out ? *out_ : *out2;
  TORCH_CHECK(a.is_cuda() && b.is_cuda() && out.is_cuda(), "gemm: CUDA tensors required");
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16,
              "gemm: BF16 operands required");
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1,
              "gemm: operands must be 2-D with a contiguous last dimension");
  TORCH_CHECK(out.dim() == 2 && out.stride(1) == 1, "gemm: out must be 2-D row-major");
  // TMA needs 16-byte aligned bases and row pitches (8 BF16 elements).
  TORCH_CHECK(a.stride(0) % 8 == 0 && b.stride(0) % 8 == 0 &&
              reinterpret_cast<uintptr_t>(a.data_ptr()) % 16 == 0 && reinterpret_cast<uintptr_t>(b.data_ptr()) % 16 == 0,
              "gemm: operand row pitches must be multiples of 8 elements and bases 16-byte aligned");
  const int64_t b_rows = epilogue == WS_EPI_SWIGLU ? 2 * n : n;
  if (!a_mn) { TORCH_CHECK(a.size(0) == m && a.size(1) == k, "gemm: A must be [m,k]"); }
  else { TORCH_CHECK(a.size(0) == k && a.size(1) == m, "gemm: A must be [k,m]"); }
  if (!b_mn) { TORCH_CHECK(b.size(0) == b_rows && b.size(1) == k, "gemm: B must be [n,k]"); }
  else { TORCH_CHECK(b.size(0) == k && b.size(1) == b_rows, "gemm: B must be [k,n]"); }
  const bool f32_out = epilogue == WS_EPI_RESID_F32 || epilogue == WS_EPI_ACC_F32 || epilogue == WS_EPI_F32;
  TORCH_CHECK(out.scalar_type() == (f32_out ? at::kFloat : at::kBFloat16), "gemm: wrong out dtype");
  const int64_t out_cols = has_out && (epilogue == WS_EPI_SWIGLU || epilogue == WS_EPI_SWIGLU_BWD) ? 2 * n : n;
  TORCH_CHECK(out.size(0) == m && out.size(1) == out_cols, "gemm: wrong out shape");
  if (row_scale.has_value() && row_scale->defined()) {
    TORCH_CHECK(row_scale->scalar_type() == at::kFloat && row_scale->numel() == m && row_scale->is_contiguous(),
                "gemm: row_scale must be float32 [m]");
  }
  if (epilogue == WS_EPI_RESID_F32) {
    TORCH_CHECK(aux.has_value() && aux->scalar_type() == at::kFloat && aux->size(0) == m && aux->size(1) == n,
                "gemm: residual must be float32 [m,n]");
  }
  if (epilogue == WS_EPI_RESID_BF16) {
    TORCH_CHECK(aux.has_value() && aux->scalar_type() == at::kBFloat16 && aux->size(0) == m && aux->size(1) == n,
                "gemm: residual must be bfloat16 [m,n]");
  }
  if (epilogue == WS_EPI_SWIGLU_BWD) {
    TORCH_CHECK(aux.has_value() && aux->scalar_type() == at::kBFloat16 && aux->size(0) == m && aux->size(1) == 2 * n,
                "gemm: packed (up|gate) must be bfloat16 [m,2n]");
  }
  if (epilogue == WS_EPI_SWIGLU) {
    TORCH_CHECK(out2.has_value() && out2->scalar_type() == at::kBFloat16 && out2->size(0) == m && out2->size(1) == n,
                "gemm: activation output must be bfloat16 [m,n]");
  }

  c10::cuda::CUDAGuard guard(a.device());
  WsGemm g = {};
  g.a = a.data_ptr(); g.b = b.data_ptr();
  g.m = (int)m; g.n = (int)n; g.k = (int)k;
  g.lda = (int)a.stride(0); g.ldb = (int)b.stride(0);
  g.a_mn = a_mn; g.b_mn = b_mn; g.epilogue = (int)epilogue;
  g.out = has_out ? out.data_ptr() : nullptr; g.ldo = has_out ? (int)out.stride(0) : 0;
  g.out2 = const_cast<void*>(opt_ptr(out2)); g.ldo2 = (int)opt_ld(out2);
  g.aux = opt_ptr(aux); g.ldaux = (int)opt_ld(aux);
  g.row_scale = reinterpret_cast<const float*>(opt_ptr(row_scale));
  g.row_vec = nullptr;
  g.alpha = (float)alpha; g.beta = (float)beta;
  g.error_flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  g.wide = wide;
  const int splits = ws_gemm_splits(&g);
  int rc;
  if (splits > 1) {
    at::Tensor part = at::empty({splits, m, n}, out.options().dtype(at::kFloat));
    rc = ws_gemm_split(&g, splits, part.data_ptr<float>(), cur_stream());
  } else {
    rc = ws_gemm(&g, cur_stream());
  }
  if (rc != 0) {  // name the problem: a bare code is of little use for a tensor-map or shape refusal
    char what[256];
    snprintf(what, sizeof(what), "gemm (m=%lld n=%lld k=%lld a_mn=%d b_mn=%d epilogue=%lld lda=%d ldb=%d ldo=%d)",
             (long long)m, (long long)n, (long long)k, (int)a_mn, (int)b_mn, (long long)epilogue, g.lda, g.ldb, g.ldo);
    check_rc(rc, what);
  }
}

// grads[i] = beta[i] * grads[i] + dy[i]^T x[i]  (FP32), all problems in one persistent launch
// when the CTA-pair kernel can take them (up to four with >= 256 output rows each).
void grad_weight_group(at::TensorList dys, at::TensorList xs, at::TensorList grads,
                       at::ArrayRef<double> betas, c10::optional<at::Tensor> error_flag) {
  const size_t count = dys.size();
  TORCH_CHECK(count > 0 && xs.size() == count && grads.size() == count && betas.size() == count,
              "grad_weight_group: list lengths differ");
  std::vector<WsGemm> items(count);
  for (size_t i = 0; i < count; ++i) {
    const at::Tensor& dy = dys[i];
    const at::Tensor& x = xs[i];
    const at::Tensor& grad = grads[i];
    TORCH_CHECK(dy.is_cuda() && x.is_cuda() && grad.is_cuda() && dy.device() == dys[0].device(),
                "grad_weight_group: CUDA tensors on one device required");
    TORCH_CHECK(dy.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16 && grad.scalar_type() == at::kFloat,
                "grad_weight_group: BF16 operands and FP32 gradients required");
    TORCH_CHECK(dy.dim() == 2 && x.dim() == 2 && grad.dim() == 2 && dy.stride(1) == 1 && x.stride(1) == 1 &&
                grad.stride(1) == 1, "grad_weight_group: 2-D tensors with a contiguous last dimension required");
    TORCH_CHECK(dy.size(0) == x.size(0) && grad.size(0) == dy.size(1) && grad.size(1) == x.size(1),
                "grad_weight_group: shapes must be dy [T,N], x [T,K], grad [N,K]");
    TORCH_CHECK(dy.stride(0) % 8 == 0 && x.stride(0) % 8 == 0 &&
                reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16 == 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0,
                "grad_weight_group: operand row pitches must be multiples of 8 elements and bases 16-byte aligned");
    WsGemm& g = items[i];
    g.a = dy.data_ptr(); g.b = x.data_ptr();
    g.m = (int)dy.size(1); g.n = (int)x.size(1); g.k = (int)dy.size(0);
    g.lda = (int)dy.stride(0); g.ldb = (int)x.stride(0);
    g.a_mn = true; g.b_mn = true; g.epilogue = WS_EPI_ACC_F32;
    g.out = grad.data_ptr(); g.ldo = (int)grad.stride(0);
    g.out2 = nullptr; g.ldo2 = 0;
    g.aux = nullptr; g.ldaux = 0;
    g.row_scale = nullptr; g.row_vec = nullptr;
    g.alpha = 1.0f; g.beta = (float)betas[i];
    g.error_flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  }
  c10::cuda::CUDAGuard guard(dys[0].device());
  check_rc(ws_gemm_group(items.data(), (int)count, cur_stream()), "grad_weight_group");
}

// ----------------------------------------------------------------------------- row kernels
std::tuple<at::Tensor, at::Tensor, at::Tensor> rmsnorm_fwd(const at::Tensor& x,
                                                           const c10::optional<at::Tensor>& col_scale,
                                                           const c10::optional<at::Tensor>& col_bias,
                                                           const at::Tensor& w, double eps, bool want_xmod) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous(), "rmsnorm_fwd: x must be contiguous [rows,d]");
  TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16, "rmsnorm_fwd: x dtype");
  TORCH_CHECK(w.device() == x.device() && w.scalar_type() == at::kFloat && w.is_contiguous() && w.numel() == x.size(1), "rmsnorm_fwd: w");
  c10::cuda::CUDAGuard guard(x.device());
  const int rows = (int)x.size(0), d = (int)x.size(1);
  const bool mod = col_scale.has_value() && col_scale->defined();
  if (mod) {
    TORCH_CHECK(col_scale->device() == x.device() && col_scale->scalar_type() == at::kFloat && col_scale->is_contiguous() &&
                col_scale->numel() == d && col_bias.has_value() && col_bias->device() == x.device() && col_bias->scalar_type() == at::kFloat &&
                col_bias->is_contiguous() && col_bias->numel() == d, "rmsnorm_fwd: depth modulation vectors must be float32 [d] on the device of x");
  }
  at::Tensor z = at::empty({rows, d}, x.options().dtype(at::kBFloat16));
  at::Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  at::Tensor xmod = (mod && want_xmod) ? at::empty_like(x) : at::Tensor();
  check_rc(ws_rmsnorm_fwd(x.data_ptr(), x.scalar_type() == at::kBFloat16,
                          mod ? col_scale->data_ptr<float>() : nullptr,
                          mod ? col_bias->data_ptr<float>() : nullptr, w.data_ptr<float>(), (float)eps, rows, d,
                          xmod.defined() ? xmod.data_ptr() : nullptr, z.data_ptr(), rstd.data_ptr<float>(), 0,
                          cur_stream()), "rmsnorm_fwd");
  return {z, rstd, xmod.defined() ? xmod : x};
}

// -> (dx, its BF16 copy where asked for, the partial rows [parts, d] of the weight's gradient)
std::tuple<at::Tensor, at::Tensor, at::Tensor> rmsnorm_bwd_partial(const at::Tensor& dz, const at::Tensor& x,
                                                                   const at::Tensor& rstd, const at::Tensor& w,
                                                                   const c10::optional<at::Tensor>& dres,
                                                                   const c10::optional<at::Tensor>& out_scale,
                                                                   bool want_bf16) {
  TORCH_CHECK(dz.is_cuda() && dz.scalar_type() == at::kBFloat16 && dz.is_contiguous(), "rmsnorm_bwd: dz");
  TORCH_CHECK(x.is_contiguous() && x.sizes() == dz.sizes(), "rmsnorm_bwd: x");
  c10::cuda::CUDAGuard guard(x.device());
  const int rows = (int)x.size(0), d = (int)x.size(1);
  const bool has_res = dres.has_value() && dres->defined();
  if (has_res) { TORCH_CHECK(dres->scalar_type() == x.scalar_type() && dres->is_contiguous() && dres->sizes() == x.sizes(), "rmsnorm_bwd: dres"); }
  const bool has_scale = out_scale.has_value() && out_scale->defined();
  at::Tensor dx = at::empty_like(x);
  at::Tensor dxb = want_bf16 ? at::empty({rows, d}, x.options().dtype(at::kBFloat16)) : at::Tensor();
  const int parts = ws_rmsnorm_bwd_parts(rows);
  at::Tensor partial = at::empty({parts, d}, x.options().dtype(at::kFloat));
  check_rc(ws_rmsnorm_bwd(dz.data_ptr(), x.data_ptr(), x.scalar_type() == at::kBFloat16, rstd.data_ptr<float>(),
                          w.data_ptr<float>(), has_res ? dres->data_ptr() : nullptr,
                          has_scale ? out_scale->data_ptr<float>() : nullptr, rows, d, dx.data_ptr(),
                          want_bf16 ? dxb.data_ptr() : nullptr, partial.data_ptr<float>(), cur_stream()),
           "rmsnorm_bwd");
  return {dx, dxb, partial};
}

// The same with dw [d], their sum, in the place of the partial rows.
std::tuple<at::Tensor, at::Tensor, at::Tensor> rmsnorm_bwd(const at::Tensor& dz, const at::Tensor& x,
                                                           const at::Tensor& rstd, const at::Tensor& w,
                                                           const c10::optional<at::Tensor>& dres,
                                                           const c10::optional<at::Tensor>& out_scale,
                                                           bool want_bf16) {
  auto [dx, dxb, partial] = rmsnorm_bwd_partial(dz, x, rstd, w, dres, out_scale, want_bf16);
  c10::cuda::CUDAGuard guard(x.device());
  const int parts = (int)partial.size(0), d = (int)partial.size(1);
  at::Tensor dw = at::empty({d}, x.options().dtype(at::kFloat));
  check_rc(ws_colsum_finalize(partial.data_ptr<float>(), parts, d, nullptr, 0.f, dw.data_ptr<float>(), cur_stream()),
           "colsum_finalize");
  return {dx, dxb, dw};
}

// The norm behind a depth modulation (FP32 stream): -> (dx, the gradients of w, of the bias, of the scale: FP32 [3, d] where they are
// `summed`, otherwise the partial rows [3, parts, d] that they are made of).  From the modulation's input x; a caller that has only its
// output xmod gets x back as (xmod - bias) / (1 + scale), 0 where scale is -1, with an error of an ulp of xmod over 1 + scale.
std::tuple<at::Tensor, at::Tensor> rmsnorm_bwd_modulated(const at::Tensor& dz, const c10::optional<at::Tensor>& xmod,
                                                         const at::Tensor& rstd, const at::Tensor& w, const at::Tensor& dres,
                                                         const at::Tensor& scale, const at::Tensor& bias,
                                                         const c10::optional<at::Tensor>& x_, bool summed) {
  const bool given = x_.has_value() && x_->defined();
  TORCH_CHECK(given || (xmod.has_value() && xmod->defined()), "rmsnorm_bwd_mod: x or xmod");
  TORCH_CHECK(dz.is_cuda() && dz.scalar_type() == at::kBFloat16 && dz.is_contiguous(), "rmsnorm_bwd_mod: dz");
  const at::Tensor x = given ? *x_ : ((*xmod - bias) / (1.0 + scale)).masked_fill_(scale == -1.0, 0.0);
  for (const at::Tensor* t : {&x, &dres})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->sizes() == dz.sizes(),
                "rmsnorm_bwd_mod: x and dres must be FP32 [rows, d]");
  const int rows = (int)x.size(0), d = (int)x.size(1);
  for (const at::Tensor* t : {&w, &scale, &bias})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == d, "rmsnorm_bwd_mod: vectors must be FP32 [d]");
  TORCH_CHECK(rstd.scalar_type() == at::kFloat && rstd.is_contiguous() && rstd.numel() == rows, "rmsnorm_bwd_mod: rstd");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor dx = at::empty_like(x);
  at::Tensor partial = at::empty({3, ws_rmsnorm_bwd_mod_parts(rows), d}, x.options());
  at::Tensor grads = summed ? at::empty({3, d}, x.options()) : at::Tensor();
  check_rc(ws_rmsnorm_bwd_mod(dz.data_ptr(), x.data_ptr<float>(), rstd.data_ptr<float>(), w.data_ptr<float>(),
                              dres.data_ptr<float>(), scale.data_ptr<float>(), bias.data_ptr<float>(), rows, d,
                              dx.data_ptr<float>(), partial.data_ptr<float>(), summed ? grads.data_ptr<float>() : nullptr, cur_stream()),
           "rmsnorm_bwd_mod");
  return {dx, summed ? grads : partial};
}

std::tuple<at::Tensor, at::Tensor> rmsnorm_bwd_mod(const at::Tensor& dz, const c10::optional<at::Tensor>& xmod,
                                                   const at::Tensor& rstd, const at::Tensor& w, const at::Tensor& dres,
                                                   const at::Tensor& scale, const at::Tensor& bias, const c10::optional<at::Tensor>& x) {
  return rmsnorm_bwd_modulated(dz, xmod, rstd, w, dres, scale, bias, x, true);
}

// (sum_rows a / (1+inv_scale), sum_rows a*b / (1+inv_scale))
std::tuple<at::Tensor, at::Tensor> colsum2(const at::Tensor& a, const at::Tensor& b,
                                           const c10::optional<at::Tensor>& inv_scale) {
  TORCH_CHECK(a.is_cuda() && a.is_contiguous() && b.is_contiguous() && a.sizes() == b.sizes() &&
              a.scalar_type() == b.scalar_type(), "colsum2: a, b");
  c10::cuda::CUDAGuard guard(a.device());
  const int rows = (int)a.size(0), d = (int)a.size(1);
  const int parts = ws_colsum_parts(rows);
  at::Tensor pa = at::empty({parts, d}, a.options().dtype(at::kFloat));
  at::Tensor pab = at::empty({parts, d}, a.options().dtype(at::kFloat));
  check_rc(ws_colsum2(a.data_ptr(), b.data_ptr(), a.scalar_type() == at::kBFloat16, rows, d, pa.data_ptr<float>(),
                      pab.data_ptr<float>(), cur_stream()), "colsum2");
  at::Tensor sa = at::empty({d}, a.options().dtype(at::kFloat));
  at::Tensor sab = at::empty({d}, a.options().dtype(at::kFloat));
  const float* inv = inv_scale.has_value() && inv_scale->defined() ? inv_scale->data_ptr<float>() : nullptr;
  check_rc(ws_colsum_finalize(pa.data_ptr<float>(), parts, d, inv, 0.f, sa.data_ptr<float>(), cur_stream()), "colsum_finalize");
  check_rc(ws_colsum_finalize(pab.data_ptr<float>(), parts, d, inv, 0.f, sab.data_ptr<float>(), cur_stream()), "colsum_finalize");
  return {sa, sab};
}

at::Tensor cast_bf16(const at::Tensor& x, c10::optional<at::Tensor> out) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.is_contiguous(), "cast_bf16: x");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor o = out.has_value() && out->defined() ? *out : at::empty(x.sizes(), x.options().dtype(at::kBFloat16));
  TORCH_CHECK(o.scalar_type() == at::kBFloat16 && o.is_contiguous() && o.numel() == x.numel(), "cast_bf16: out");
  if (x.numel() % 4 == 0 && (reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0) &&
      (reinterpret_cast<uintptr_t>(o.data_ptr()) % 8 == 0)) {
    check_rc(ws_cast_f32_bf16(x.data_ptr<float>(), o.data_ptr(), (size_t)x.numel(), cur_stream()), "cast_bf16");
  } else {
    o.copy_(x);
  }
  return o;
}

at::Tensor embed_fwd(const at::Tensor& ids, const at::Tensor& table, bool out_bf16) {
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous(), "embed_fwd: ids");
  TORCH_CHECK(table.dim() == 2 && table.is_contiguous(), "embed_fwd: table");
  c10::cuda::CUDAGuard guard(table.device());
  const int rows = (int)ids.numel(), d = (int)table.size(1);
  at::Tensor out = at::empty({rows, d}, table.options().dtype(out_bf16 ? at::kBFloat16 : at::kFloat));
  check_rc(ws_embed_fwd(ids.data_ptr<int64_t>() ? reinterpret_cast<const long long*>(ids.data_ptr<int64_t>()) : nullptr,
                        table.data_ptr(), table.scalar_type() == at::kBFloat16, rows, d, (int)table.size(0),
                        out.data_ptr(), out_bf16, cur_stream()), "embed_fwd");
  return out;
}

// grad_table [V,d] FP32 += scatter of dx rows by token id, deterministic (sorted segments).
void embed_bwd(const at::Tensor& dx, const at::Tensor& ids, at::Tensor grad_table) {
  TORCH_CHECK(dx.is_cuda() && dx.dim() == 2 && dx.is_contiguous(), "embed_bwd: dx");
  TORCH_CHECK(grad_table.scalar_type() == at::kFloat && grad_table.is_contiguous(), "embed_bwd: grad_table");
  c10::cuda::CUDAGuard guard(dx.device());
  const int rows = (int)dx.size(0), d = (int)dx.size(1);
  at::Tensor flat = ids.reshape({-1});
  auto sorted = flat.sort(/*stable=*/true, /*dim=*/0, /*descending=*/false);
  at::Tensor sorted_ids = std::get<0>(sorted).contiguous();
  at::Tensor order = std::get<1>(sorted).contiguous();
  TORCH_CHECK(grad_table.dim() == 2 && grad_table.size(1) == d && flat.numel() == rows, "embed_bwd: shapes");
  // the runs of equal ids are found by the kernel: no host-side count, no device-to-host read
  check_rc(ws_embed_bwd(dx.data_ptr(), dx.scalar_type() == at::kBFloat16,
                        reinterpret_cast<const long long*>(sorted_ids.data_ptr<int64_t>()),
                        reinterpret_cast<const long long*>(order.data_ptr<int64_t>()), rows, d,
                        (int)grad_table.size(0), grad_table.data_ptr<float>(), cur_stream()), "embed_bwd");
}

// ----------------------------------------------------------------------------- attention / memory
void check_qkvgu(const at::Tensor& qkvgu, int64_t B, int64_t T, int64_t H) {
  TORCH_CHECK(qkvgu.is_cuda() && qkvgu.scalar_type() == at::kBFloat16 && qkvgu.is_contiguous() && qkvgu.dim() == 2,
              "attention: qkvgu must be contiguous BF16 [B*T, 5d]");
  TORCH_CHECK(qkvgu.size(0) == B * T && qkvgu.size(1) == 5 * H * 64 && T % 128 == 0,
              "attention: shape mismatch (chunk 128, head_dim 64)");
}

at::Tensor chunk_writes(const at::Tensor& qkvgu, const at::Tensor& rope, int64_t B, int64_t T, int64_t H,
                        const c10::optional<at::Tensor>& error_flag) {
  check_qkvgu(qkvgu, B, T, H);
  TORCH_CHECK(rope.scalar_type() == at::kFloat && rope.is_contiguous() && rope.numel() == 128 * 64, "rope table");
  c10::cuda::CUDAGuard guard(qkvgu.device());
  at::Tensor writes = at::empty({B, T / 128, H, 64, 64}, qkvgu.options().dtype(at::kFloat));
  check_rc(ws_chunk_writes(qkvgu.data_ptr(), rope.data_ptr<float>(), writes.data_ptr<float>(), (int)B, (int)T,
                           (int)H, (int)(H * 64), reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))),
                           cur_stream()), "chunk_writes");
  return writes;
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> memory_scan(const at::Tensor& writes, const at::Tensor& fast_logit,
                                                           const at::Tensor& slow_logit, const at::Tensor& mix_logit,
                                                           bool want_states, bool want_final,
                                                           const c10::optional<at::Tensor>& init_fast,
                                                           const c10::optional<at::Tensor>& init_slow) {
  TORCH_CHECK(writes.is_cuda() && writes.scalar_type() == at::kFloat && writes.is_contiguous() && writes.dim() == 5,
              "memory_scan: writes must be FP32 [B,N,H,64,64]");
  const int B = (int)writes.size(0), N = (int)writes.size(1), H = (int)writes.size(2);
  for (const at::Tensor* t : {&fast_logit, &slow_logit, &mix_logit})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == H, "memory_scan: logits");
  c10::cuda::CUDAGuard guard(writes.device());
  at::Tensor states = want_states ? at::empty(writes.sizes(), writes.options().dtype(at::kBFloat16)) : at::Tensor();
  at::Tensor ff = want_final ? at::empty({B, H, 64, 64}, writes.options()) : at::Tensor();
  at::Tensor fs = want_final ? at::empty({B, H, 64, 64}, writes.options()) : at::Tensor();
  const float* i_f = init_fast.has_value() && init_fast->defined() ? init_fast->data_ptr<float>() : nullptr;
  const float* i_s = init_slow.has_value() && init_slow->defined() ? init_slow->data_ptr<float>() : nullptr;
  check_rc(ws_memory_scan(writes.data_ptr<float>(), fast_logit.data_ptr<float>(), slow_logit.data_ptr<float>(),
                          mix_logit.data_ptr<float>(), want_states ? states.data_ptr() : nullptr,
                          want_final ? ff.data_ptr<float>() : nullptr, want_final ? fs.data_ptr<float>() : nullptr,
                          i_f, i_s, B, N, H, cur_stream()), "memory_scan");
  return {states, ff, fs};
}

// Without states every sequence is one chunk, whose memories are empty.
at::Tensor attn_fwd(const at::Tensor& qkvgu, const c10::optional<at::Tensor>& states, const at::Tensor& rope, int64_t B, int64_t T,
                    int64_t H, const c10::optional<at::Tensor>& error_flag) {
  check_qkvgu(qkvgu, B, T, H);
  const bool memory = states.has_value() && states->defined();
  TORCH_CHECK(memory ? states->scalar_type() == at::kBFloat16 && states->is_contiguous() && states->numel() == B * (T / 128) * H * 4096
                     : T == 128, "attn_fwd: states");
  c10::cuda::CUDAGuard guard(qkvgu.device());
  at::Tensor y = at::empty({B * T, H * 64}, qkvgu.options());
  check_rc(ws_attn_fwd(qkvgu.data_ptr(), memory ? states->data_ptr() : nullptr, rope.data_ptr<float>(), y.data_ptr(), (int)B, (int)T,
                       (int)H, (int)(H * 64), reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))),
                       cur_stream()), "attn_fwd");
  return y;
}

// Prompts of any length: y [B*T, d]; the decode state of the layer is written in place.
at::Tensor attn_prefill(const at::Tensor& qkvgu, const at::Tensor& rope, const at::Tensor& fast_logit,
                        const at::Tensor& slow_logit, const at::Tensor& mix_logit, int64_t B, int64_t T, int64_t H,
                        at::Tensor fast, at::Tensor slow, at::Tensor mixed, at::Tensor kc, at::Tensor vc, at::Tensor uc,
                        const c10::optional<at::Tensor>& error_flag) {
  TORCH_CHECK(qkvgu.is_cuda() && qkvgu.scalar_type() == at::kBFloat16 && qkvgu.is_contiguous() && qkvgu.dim() == 2 &&
              B >= 1 && T >= 1 && qkvgu.size(0) == B * T && qkvgu.size(1) == 5 * H * 64,
              "attn_prefill: qkvgu must be contiguous BF16 [B*T, 5*H*64]");
  TORCH_CHECK(rope.scalar_type() == at::kFloat && rope.is_contiguous() && rope.numel() == 128 * 64, "attn_prefill: rope table");
  for (const at::Tensor* t : {&fast_logit, &slow_logit, &mix_logit})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == H, "attn_prefill: logits");
  for (const at::Tensor* t : {&fast, &slow})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == B * H * 4096,
                "attn_prefill: fast and slow must be contiguous FP32 [B, H, 64, 64]");
  TORCH_CHECK(mixed.is_cuda() && mixed.scalar_type() == at::kBFloat16 && mixed.is_contiguous() && mixed.numel() == B * H * 4096,
              "attn_prefill: mixed must be contiguous BF16 [B, H, 64, 64]");
  for (const at::Tensor* t : {&kc, &vc, &uc})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->numel() == B * H * 128 * 64,
                "attn_prefill: caches must be contiguous BF16 [B, H, 128, 64]");
  c10::cuda::CUDAGuard guard(qkvgu.device());
  const int64_t chunks = (T + 127) / 128;
  at::Tensor writes = at::empty({B, chunks, H, 64, 64}, qkvgu.options().dtype(at::kFloat));
  at::Tensor states = at::empty({B, chunks, H, 64, 64}, qkvgu.options());
  at::Tensor y = at::empty({B * T, H * 64}, qkvgu.options());
  check_rc(ws_attn_prefill(qkvgu.data_ptr(), rope.data_ptr<float>(), fast_logit.data_ptr<float>(),
                           slow_logit.data_ptr<float>(), mix_logit.data_ptr<float>(), writes.data_ptr<float>(),
                           states.data_ptr(), y.data_ptr(), fast.data_ptr<float>(), slow.data_ptr<float>(),
                           mixed.data_ptr(), kc.data_ptr(), vc.data_ptr(), uc.data_ptr(), (int)B, (int)T, (int)H,
                           (int)(H * 64), reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))), cur_stream()),
           "attn_prefill");
  return y;
}

// returns (dqkvgu [M,5d] BF16, partials [B*H*16,3] FP32)
std::tuple<at::Tensor, at::Tensor> attn_bwd(const at::Tensor& qkvgu, const at::Tensor& dy, const at::Tensor& states,
                                            const at::Tensor& writes, const at::Tensor& rope,
                                            const at::Tensor& fast_logit, const at::Tensor& slow_logit,
                                            const at::Tensor& mix_logit, int64_t B, int64_t T, int64_t H,
                                            const c10::optional<at::Tensor>& error_flag) {
  check_qkvgu(qkvgu, B, T, H);
  const int64_t d = H * 64, N = T / 128;
  TORCH_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.is_contiguous() && dy.numel() == B * T * d,
              "attn_bwd: dy must be contiguous BF16 [B*T, d]");
  TORCH_CHECK(states.scalar_type() == at::kBFloat16 && states.is_contiguous() && states.numel() == B * N * H * 4096,
              "attn_bwd: states");
  TORCH_CHECK(writes.scalar_type() == at::kFloat && writes.is_contiguous() && writes.numel() == B * N * H * 4096,
              "attn_bwd: writes");
  TORCH_CHECK(N <= 256, "attn_bwd: at most 256 chunks (32768 tokens) per sequence");
  c10::cuda::CUDAGuard guard(qkvgu.device());
  int* err = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  at::Tensor dstate = at::empty({B, N, H, 64, 64}, qkvgu.options().dtype(at::kFloat));
  check_rc(ws_attn_dstate(qkvgu.data_ptr(), dy.data_ptr(), rope.data_ptr<float>(), dstate.data_ptr<float>(), (int)B,
                          (int)T, (int)H, (int)d, err, cur_stream()), "attn_dstate");
  at::Tensor dwrites = at::empty({B, N, H, 64, 64}, qkvgu.options());
  at::Tensor partials = at::empty({B * H * 16, 3}, qkvgu.options().dtype(at::kFloat));
  // the scan fetches 16 bytes at a time
  const at::Tensor aligned = reinterpret_cast<uintptr_t>(writes.data_ptr()) % 16 == 0 ? writes : writes.clone();
  check_rc(ws_memory_scan_bwd(dstate.data_ptr<float>(), aligned.data_ptr<float>(), fast_logit.data_ptr<float>(),
                              slow_logit.data_ptr<float>(), mix_logit.data_ptr<float>(), dwrites.data_ptr(),
                              partials.data_ptr<float>(), (int)B, (int)N, (int)H, cur_stream()), "memory_scan_bwd");
  at::Tensor dqkvgu = at::empty_like(qkvgu);
  check_rc(ws_attn_bwd(qkvgu.data_ptr(), states.data_ptr(), dy.data_ptr(), dwrites.data_ptr(), rope.data_ptr<float>(),
                       dqkvgu.data_ptr(), (int)B, (int)T, (int)H, (int)d, err, cur_stream()), "attn_bwd");
  return {dqkvgu, partials};
}

// partials [B*H*16, 3] of attn_bwd -> FP32 [3, H]: gradients of the fast decay, slow decay and mix logits
at::Tensor memory_logit_grads(const at::Tensor& partials, const at::Tensor& fast_logit, const at::Tensor& slow_logit,
                              const at::Tensor& mix_logit, int64_t B) {
  const int64_t H = fast_logit.numel();
  TORCH_CHECK(partials.is_cuda() && partials.scalar_type() == at::kFloat && partials.is_contiguous() &&
              partials.numel() == B * H * 48, "memory_logit_grads: partials must be contiguous FP32 [B*H*16, 3]");
  for (const at::Tensor* t : {&fast_logit, &slow_logit, &mix_logit})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == H, "memory_logit_grads: logits");
  c10::cuda::CUDAGuard guard(partials.device());
  at::Tensor out = at::empty({3, H}, partials.options());
  check_rc(ws_memory_logit_grads(partials.data_ptr<float>(), fast_logit.data_ptr<float>(), slow_logit.data_ptr<float>(),
                                 mix_logit.data_ptr<float>(), (int)B, (int)H, out.data_ptr<float>(), cur_stream()),
           "memory_logit_grads");
  return out;
}

// ----------------------------------------------------------------------------- whole blocks
// The kernel sequences of one block (ops/fused.py) as one call each.  A block is eight to twelve launches of 2-20 us in
// a short sequence, and issued one by one from Python the host takes longer than the device below a few thousand rows;
// here a launch costs its allocation, its tensor maps and the launch.  Same arithmetic in the same order; one launch fewer where
// out_proj is cut along k.
// Smoke model (d 256, 4 depths, 2 x 512 tokens), forward + backward: 2.53 -> 2.03 ms.
at::Tensor project(const at::Tensor& x, const at::Tensor& w, bool b_mn, int64_t epilogue, int64_t n, at::Tensor out,
                   const c10::optional<at::Tensor>& out2, const c10::optional<at::Tensor>& aux,
                   const c10::optional<at::Tensor>& flag) {
  gemm(x, w, false, b_mn, epilogue, x.size(0), n, x.size(1), out, out2, aux, c10::nullopt, 1.0, 0.0, flag, false);
  return out;
}
at::Tensor project_bf16(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& flag) {
  return project(x, w, false, WS_EPI_BF16, w.size(0), at::empty({x.size(0), w.size(0)}, x.options()), c10::nullopt, c10::nullopt, flag);
}
at::Tensor project_residual(const at::Tensor& x, const at::Tensor& w, const at::Tensor& resid,
                            const c10::optional<at::Tensor>& flag) {
  return project(x, w, false, resid.scalar_type() == at::kFloat ? WS_EPI_RESID_F32 : WS_EPI_RESID_BF16, w.size(0),
                 at::empty_like(resid), c10::nullopt, resid, flag);
}
at::Tensor input_grad(const at::Tensor& dy, const at::Tensor& w, const c10::optional<at::Tensor>& flag) {
  return project(dy, w, true, WS_EPI_BF16, w.size(1), at::empty({dy.size(0), w.size(1)}, dy.options()), c10::nullopt, c10::nullopt, flag);
}

// (x + y W^T, its RMSNorm in BF16, the norm's factors).  Where the product is cut along k, the kernel that adds the pieces
// does the norm as well.
std::tuple<at::Tensor, at::Tensor, at::Tensor> project_residual_norm(const at::Tensor& y, const at::Tensor& w, const at::Tensor& resid,
                                                                     const at::Tensor& norm, double eps,
                                                                     const c10::optional<at::Tensor>& flag) {
  const int64_t m = y.size(0), n = w.size(0), k = y.size(1);
  const auto aligned = [&](const at::Tensor& t) { return t.device() == y.device() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; };
  if (y.is_cuda() && resid.scalar_type() == at::kFloat && n % 128 == 0 && n <= 2048 && k % 8 == 0 && w.dim() == 2 && w.size(1) == k && y.is_contiguous() &&
      w.is_contiguous() && resid.is_contiguous() && resid.size(0) == m && resid.size(1) == n && aligned(y) && aligned(w) && aligned(resid) &&
      y.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && norm.scalar_type() == at::kFloat && norm.is_contiguous() &&
      norm.numel() == n && aligned(norm)) {
    WsGemm g = {};
    g.a = y.data_ptr(); g.b = w.data_ptr();
    g.m = (int)m; g.n = (int)n; g.k = (int)k; g.lda = (int)k; g.ldb = (int)k;
    g.epilogue = WS_EPI_RESID_F32;
    g.aux = resid.data_ptr(); g.ldaux = (int)n; g.ldo = (int)n;
    g.alpha = 1.f;
    g.error_flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(flag)));
    c10::cuda::CUDAGuard guard(y.device());
    const int splits = ws_gemm_splits(&g);
    if (splits > 1) {
      at::Tensor part = at::empty({splits, m, n}, resid.options()), x2 = at::empty_like(resid), z = at::empty({m, n}, y.options());
      at::Tensor rstd = at::empty({m}, resid.options());
      g.out = x2.data_ptr();
      check_rc(ws_gemm_split_norm(&g, splits, part.data_ptr<float>(), nullptr, nullptr, norm.data_ptr<float>(), (float)eps, z.data_ptr(),
                                  rstd.data_ptr<float>(), cur_stream()), "gemm_split_norm");
      return {x2, z, rstd};
    }
  }
  at::Tensor x2 = project_residual(y, w, resid, flag);
  auto [z, rstd, unchanged] = rmsnorm_fwd(x2, c10::nullopt, c10::nullopt, norm, eps, false);
  return {x2, z, rstd};
}

// x2 = xmod + out_proj(y), then x2 + down(swiglu(up_gate(norm2 x2))).  -> (x2, rstd2, z2, packed, act, x3); packed only
// with `keep` (the backward pass reads it), x3 only with `want_output`.
struct BlockTail { at::Tensor x2, rstd2, z2, packed, act, x3; };
BlockTail block_tail(const at::Tensor& y, const at::Tensor& xmod, const at::Tensor& w_out, const at::Tensor& n2,
                     const at::Tensor& w_ug, const at::Tensor& w_down, double eps, bool keep, bool want_output,
                     const c10::optional<at::Tensor>& flag) {
  BlockTail t;
  std::tie(t.x2, t.z2, t.rstd2) = project_residual_norm(y, w_out, xmod, n2, eps, flag);
  const int64_t h = w_ug.size(0) / 2;
  if (keep) t.packed = at::empty({y.size(0), 2 * h}, y.options());
  t.act = at::empty({y.size(0), h}, y.options());
  project(t.z2, w_ug, false, WS_EPI_SWIGLU, h, t.packed, t.act, c10::nullopt, flag);
  if (want_output) t.x3 = project_residual(t.act, w_down, t.x2, flag);
  return t;
}

// -> (x3, xmod, rstd1, z1, qkvgu, y, x2, rstd2, z2, packed, act, writes, states); x3 and packed may be undefined.
std::vector<at::Tensor> block_fwd(const at::Tensor& x, const c10::optional<at::Tensor>& scale,
                                  const c10::optional<at::Tensor>& bias, const at::Tensor& n1, const at::Tensor& w_in,
                                  const at::Tensor& w_out, const at::Tensor& n2, const at::Tensor& w_ug,
                                  const at::Tensor& w_down, const at::Tensor& fast_logit, const at::Tensor& slow_logit,
                                  const at::Tensor& mix_logit, const at::Tensor& rope, double eps, int64_t B, int64_t T,
                                  int64_t H, bool keep, bool want_output, const c10::optional<at::Tensor>& flag) {
  auto [z1, rstd1, xmod] = rmsnorm_fwd(x, scale, bias, n1, eps, true);
  at::Tensor qkvgu = project_bf16(z1, w_in, flag);
  at::Tensor writes = chunk_writes(qkvgu, rope, B, T, H, flag);
  at::Tensor states = std::get<0>(memory_scan(writes, fast_logit, slow_logit, mix_logit, true, false, c10::nullopt, c10::nullopt));
  at::Tensor y = attn_fwd(qkvgu, states, rope, B, T, H, flag);
  BlockTail t = block_tail(y, xmod, w_out, n2, w_ug, w_down, eps, keep, want_output, flag);
  at::Tensor none = at::empty({0}, x.options());
  return {want_output ? t.x3 : none, xmod, rstd1, z1, qkvgu, y, t.x2, t.rstd2, t.z2, keep ? t.packed : none, t.act, writes, states};
}

// Blocks that nothing differentiates, one after another in one call: scoring (one block) and prompts (all of them).  What passes
// between the kernels lies in one allocation (or six) instead of fifteen a block, and goes from kernel to kernel by address; the
// launches are those of `block_fwd`, but that the kernel which adds the pieces of a cut down projection forms the next
// block's modulation and norm as well, and that one-chunk sequences, whose memories are empty, have no launches for them.
// Scoring 128 tokens by a block of width 2048 95 -> 75 us, a prompt of 300 tokens in 28 blocks 2.92 -> 2.84 ms.
class ForwardBlocks {
 public:
  struct Weights { const at::Tensor *in, *out, *ug, *down; };

  // `wide`: prompts, whose (up, gate) stay FP32 until the activation.
  ForwardBlocks(int64_t B, int64_t T, int64_t H, int64_t h, const at::Tensor& rope, double eps, const c10::optional<at::Tensor>& flag, bool wide,
                const at::TensorOptions& f32)
      : B_(B), T_(T), H_(H), M_(B * T), d_(H * 64), h_(h), rope_(rope.data_ptr<float>()), eps_((float)eps),
        flag_(reinterpret_cast<int*>(const_cast<void*>(opt_ptr(flag)))), wide_(wide), stream_(cur_stream()) {
    TORCH_CHECK(rope.device() == f32.device() && rope.scalar_type() == at::kFloat && rope.is_contiguous() && rope.numel() == 128 * 64,
                "blocks: rope table");
    TORCH_CHECK(B >= 1 && T >= 1 && H >= 1 && d_ % 128 == 0 && h % 8 == 0 && h > 0, "blocks: no rows, or d not a multiple of 128, or an FFN width that is not one of 8");
    const int64_t chunks = (T + 127) / 128, memories = B * chunks * H * 4096;
    // the second half of a block lies where the first one's packed projections and memories were
    const int64_t front = aligned(10 * M_ * d_) + aligned(4 * memories) + aligned(2 * memories);
    pieces_out_ = streamed() ? ws_decode_gemm_splits((int)d_, (int)d_) : pieces(residual(nullptr, nullptr, nullptr, nullptr, d_));
    pieces_down_ = streamed() ? ws_decode_gemm_splits((int)d_, (int)h_) : pieces(residual(nullptr, nullptr, nullptr, nullptr, h_));
    const int64_t cut = std::max(pieces_out_, pieces_down_);
    const int64_t back = aligned(4 * M_ * d_) + aligned(2 * M_ * h_) + (cut > 1 || streamed() ? aligned(4 * cut * M_ * d_) : 0);
    // One allocation for scoring, whose time is the host's.  A prompt's are hundreds of megabytes, and the pool gives them back when a
    // new engine captures its step (a graph's capture empties the pool's cache): as one piece that cost the first pass of 64 x 128 tokens
    // with 40 steps a millisecond more than in parts, 35.0 and 33.8 ms.
    const int64_t shared = std::max(front, back);
    if (!wide) scratch_.push_back(at::empty({aligned(4 * M_ * d_) + aligned(2 * M_ * d_) * 2 + aligned(4 * M_) + shared}, f32.dtype(at::kByte)));
    uint8_t* at = wide ? nullptr : scratch_.back().data_ptr<uint8_t>();
    const auto take = [&](int64_t bytes) {
      if (wide) {
        scratch_.push_back(at::empty({aligned(bytes)}, f32.dtype(at::kByte)));
        return scratch_.back().data_ptr<uint8_t>();
      }
      uint8_t* p = at;
      at += aligned(bytes);
      return p;
    };
    x_ = wide ? reinterpret_cast<float*>(take(4 * M_ * d_)) : nullptr;   // between blocks; scoring is one block
    xmod_ = reinterpret_cast<float*>(take(4 * M_ * d_));
    z_ = take(2 * M_ * d_);
    y_ = take(2 * M_ * d_);
    rstd_ = reinterpret_cast<float*>(take(4 * M_));
    qkvgu_ = take(shared);
    writes_ = reinterpret_cast<float*>(qkvgu_ + aligned(10 * M_ * d_));
    states_ = qkvgu_ + aligned(10 * M_ * d_) + aligned(4 * memories);
    x2_ = reinterpret_cast<float*>(qkvgu_);
    act_ = qkvgu_ + aligned(4 * M_ * d_);
    part_ = reinterpret_cast<float*>(act_ + aligned(2 * M_ * h_));
  }

  // FP32 [d] (aligned to 16 bytes) or [H], in place or as a copy, one per tensor, that lives as long as this object.  All of them
  // before `begin`: launches of the chain read norms and modulations ahead of their turn, so no launch in it may write them.
  const float* vector(const at::Tensor& t, int64_t n) {
    TORCH_CHECK(t.device() == scratch_[0].device() && t.numel() == n,
                "blocks: norms and modulation must have d elements, logits one per head, on the device of x");
    const auto usable = [&](const at::Tensor& v) { return n == H_ || reinterpret_cast<uintptr_t>(v.data_ptr()) % 16 == 0; };
    if (t.scalar_type() == at::kFloat && t.is_contiguous() && usable(t)) return t.data_ptr<float>();
    for (const auto& [source, copy] : copies_)
      if (source == t.unsafeGetTensorImpl()) return copy.data_ptr<float>();
    TORCH_INTERNAL_ASSERT(residual_ == nullptr, "blocks: a copy of a vector behind the start of the chain");
    at::Tensor copy = t.detach().to(at::kFloat).contiguous();
    if (copy.data_ptr() == t.data_ptr()) copy = copy.clone();
    copies_.emplace_back(t.unsafeGetTensorImpl(), std::move(copy));
    return copies_.back().second.data_ptr<float>();
  }
  // norms [d] and logits [H] of a block
  struct Vectors { const float *n1, *n2, *fast, *slow, *mix; };
  Vectors vectors(const at::Tensor& n1, const at::Tensor& n2, const at::Tensor& fast, const at::Tensor& slow, const at::Tensor& mix) {
    return {vector(n1, d_), vector(n2, d_), vector(fast, H_), vector(slow, H_), vector(mix, H_)};
  }

  void check_weights(const Weights& w) {
    const int64_t rows[4] = {5 * d_, d_, 2 * h_, d_}, cols[4] = {d_, d_, d_, h_};
    const at::Tensor* t[4] = {w.in, w.out, w.ug, w.down};
    for (int i = 0; i < 4; ++i)
      TORCH_CHECK(t[i]->device() == scratch_[0].device() && t[i]->scalar_type() == at::kBFloat16 && t[i]->dim() == 2 && t[i]->size(0) == rows[i] &&
                  t[i]->size(1) == cols[i] && t[i]->stride(1) == 1 && t[i]->stride(0) % 8 == 0 &&
                  reinterpret_cast<uintptr_t>(t[i]->data_ptr()) % 16 == 0 && (!streamed() || t[i]->is_contiguous()),
                  "blocks: BF16 CUDA weights [5d, d], [d, d], [2 ffn, d], [d, ffn]");
  }

  // The first block's modulation (scale may be NULL) and norm of x [M, d].  For prompts it is launched behind everything before it:
  // nothing writes weights after that, and every product of the chain reads its own ahead of the launches in front of it (28 blocks at 300
  // tokens 2843 -> 2814 us; for one block the start costs as much as that gives).
  void begin(const float* x, const float* scale, const float* bias, const float* n1) {
    check_rc(ws_rmsnorm_fwd(x, 0, scale, bias, n1, eps_, (int)M_, (int)d_, scale != nullptr ? xmod_ : nullptr, z_, rstd_, wide_,
                            stream_), "rmsnorm_fwd");
    residual_ = scale != nullptr ? xmod_ : x;
  }

  void project_in(const Weights& w) {
    if (streamed()) return stream(*w.in, z_, 5 * d_, d_, 0, qkvgu_, "in_proj");
    WsGemm g = product(z_, d_, *w.in, 5 * d_, WS_EPI_BF16);
    g.out = qkvgu_; g.ldo = (int)(5 * d_);
    run(g, 1, "in_proj");
  }

  void attention(const Vectors& v) {
    const bool memory = T_ > 128;
    if (memory) {
      check_rc(ws_chunk_writes(qkvgu_, rope_, writes_, (int)B_, (int)T_, (int)H_, (int)d_, flag_, stream_), "chunk_writes");
      check_rc(ws_memory_scan(writes_, v.fast, v.slow, v.mix, states_, nullptr, nullptr, nullptr, nullptr, (int)B_, (int)(T_ / 128), (int)H_, stream_),
               "memory_scan");
    }
    check_rc(ws_attn_fwd(qkvgu_, memory ? states_ : nullptr, rope_, y_, (int)B_, (int)T_, (int)H_, (int)d_, flag_, stream_), "attn_fwd");
  }

  void attention_prompt(const Vectors& v, const at::Tensor* state) {
    check_rc(ws_attn_prefill(qkvgu_, rope_, v.fast, v.slow, v.mix, writes_, states_, y_, state[0].data_ptr<float>(),
                             state[1].data_ptr<float>(), state[2].data_ptr(), state[3].data_ptr(), state[4].data_ptr(), state[5].data_ptr(),
                             (int)B_, (int)T_, (int)H_, (int)d_, flag_, stream_), "attn_prefill");
  }

  // From out_proj to the output of the block: into `out`, or into this object with the next block's modulation and norm.
  void finish(const Weights& w, const float* n2, float* out, const float* next_scale = nullptr, const float* next_bias = nullptr,
              const float* next_n1 = nullptr) {
    if (streamed()) return finish_streamed(w, n2, next_scale, next_bias, next_n1);
    residual_norm(residual(y_, w.out, residual_, x2_, d_), pieces_out_, nullptr, nullptr, n2, "out_proj");
    WsGemm g = product(z_, d_, *w.ug, h_, WS_EPI_SWIGLU);
    g.out2 = act_; g.ldo2 = (int)h_;
    run(g, 1, "up_gate");
    if (out != nullptr) {
      run(residual(act_, w.down, x2_, out, h_), pieces_down_, "down");
    } else {
      residual_norm(residual(act_, w.down, x2_, next_scale != nullptr ? xmod_ : x_, h_), pieces_down_, next_scale, next_bias, next_n1, "down");
      residual_ = next_scale != nullptr ? xmod_ : x_;
    }
  }

  const float* stream_rows() const { return residual_; }
  const void* attention_rows() const { return y_; }

 private:
  // A prompt of few tokens is the rows of a decode step as far as its projections go: their time is that of the weights, which
  // the step's kernels stream (decode.cu), and the rounding of (up, gate) is the step's too.  12 blocks, with the products' own kernels ->
  // so, us at 64, 96, 97, 112 and 128 tokens: width 2048 1570 -> 800, 927 -> 859, 940 -> 966, 950 -> 908, 1065 -> 950; 1792 1448 -> 709,
  // 866 -> 790, 875 -> 920, 880 -> 856, 956 -> 887; 1536 1331 -> 647, 782 -> 745, 793 -> 879, 794 -> 840, 862 -> 870; 1280 1160 -> 595,
  // 713 -> 688, 723 -> 746, 728 -> 760, 790 -> 814.  16 blocks: 1024 1288 -> 728, 946 -> 870, 961 -> 935, 962 -> 898, 1029 -> 974; 768 1180 -> 711,
  // 877 -> 830, 887 -> 922, 900 -> 902, 973 -> 916; 512 998 -> 657, 785 -> 792, 794 -> 862, 814 -> 889, 893 -> 949; at 5 tokens 855 -> 650 and, at
  // 1280, 1405 -> 660.  So up to 96 tokens, and past them, where the products have whole tiles, only the widest.  Narrower blocks have
  // projections of a few k-blocks, which there is nothing to stream of.
  // Weights are read as they lie, row behind row, and the chain starts behind everything before it, as those kernels demand.
  bool streamed() const { return wide_ && M_ <= (d_ >= 2048 ? 128 : 96) && d_ >= 512 && h_ % 64 == 0; }

  void stream(const at::Tensor& w, const void* x, int64_t n, int64_t k, int epilogue, void* out, const char* what) {
    check_rc(ws_decode_gemm(w.data_ptr(), x, (int)n, (int)k, (int)M_, epilogue, out, (int)n, flag_, 0, stream_), what);
  }
  void finish_streamed(const Weights& w, const float* n2, const float* next_scale, const float* next_bias, const float* next_n1) {
    // the residual stream is added to in place: the first block's modulated rows are this object's own
    float* const x = const_cast<float*>(residual_);
    stream(*w.out, y_, d_, d_, 1, part_, "out_proj");
    check_rc(ws_decode_reduce_norm(x, part_, (int)pieces_out_, nullptr, nullptr, 0, nullptr, nullptr, n2, eps_, (int)d_, (int)M_, z_, stream_),
             "decode_reduce_norm");
    stream(*w.ug, z_, h_, d_, 2, act_, "up_gate");
    stream(*w.down, act_, d_, h_, 1, part_, "down");
    check_rc(ws_decode_reduce_norm(x, part_, (int)pieces_down_, nullptr, nullptr, 0, next_scale, next_bias, next_n1, eps_, (int)d_, (int)M_, z_,
                                   stream_), "decode_reduce_norm");
  }

  static int64_t aligned(int64_t bytes) { return (bytes + 1023) / 1024 * 1024; }

  WsGemm product(const void* a, int64_t k, const at::Tensor& w, int64_t n, int epilogue) const {
    WsGemm g = {};
    g.a = a; g.b = w.data_ptr(); g.m = (int)M_; g.n = (int)n; g.k = (int)k; g.lda = (int)k; g.ldb = (int)w.stride(0);
    g.epilogue = epilogue; g.alpha = 1.f; g.error_flag = flag_; g.wide = wide_; g.b_ahead = wide_;
    return g;
  }
  WsGemm residual(const void* a, const at::Tensor* w, const float* aux, float* out, int64_t k) const {
    WsGemm g = {};
    g.a = a; g.b = w != nullptr ? w->data_ptr() : nullptr; g.m = (int)M_; g.n = (int)d_; g.k = (int)k;
    g.lda = (int)k; g.ldb = w != nullptr ? (int)w->stride(0) : (int)k;
    g.epilogue = WS_EPI_RESID_F32; g.alpha = 1.f; g.error_flag = flag_; g.b_ahead = wide_;
    g.aux = aux; g.ldaux = (int)d_; g.out = out; g.ldo = (int)d_;
    return g;
  }
  // Into how many pieces a residual product of these sizes is cut: the plan looks at sizes, and its checks at addresses.
  static int64_t pieces(WsGemm g) {
    g.a = g.b = g.aux = g.out = reinterpret_cast<void*>(16);
    return ws_gemm_splits(&g);
  }
  void run(const WsGemm& g, int64_t cut, const char* what) {
    check_rc(cut > 1 ? ws_gemm_split(&g, (int)cut, part_, stream_) : ws_gemm(&g, stream_), what);
  }
  // g.out = residual + product, modulated where a scale is given; z_ = its norm.
  void residual_norm(WsGemm g, int64_t cut, const float* scale, const float* bias, const float* norm, const char* what) {
    if (cut > 1 && d_ <= 2048) {
      check_rc(ws_gemm_split_norm(&g, (int)cut, part_, scale, bias, norm, eps_, z_, rstd_, stream_), what);
      return;
    }
    float* const to = static_cast<float*>(g.out);
    if (scale != nullptr) g.out = x_;
    run(g, cut, what);
    check_rc(ws_rmsnorm_fwd(g.out, 0, scale, bias, norm, eps_, (int)M_, (int)d_, scale != nullptr ? to : nullptr, z_, rstd_, 0,
                            stream_), "rmsnorm_fwd");
  }

  const int64_t B_, T_, H_, M_, d_, h_;
  const float* rope_;
  const float eps_;
  int* flag_;
  const bool wide_;
  cudaStream_t stream_;
  int64_t pieces_out_ = 1, pieces_down_ = 1;
  std::vector<at::Tensor> scratch_;
  std::vector<std::pair<const c10::TensorImpl*, at::Tensor>> copies_;   // of vectors that the caller holds meanwhile
  float *x_, *xmod_, *rstd_, *writes_, *x2_, *part_;
  const float* residual_ = nullptr;
  uint8_t *z_, *y_, *qkvgu_, *states_, *act_;
};

// Backward up to the gradient of the block's input; the weight gradients follow as one group (grad_weight_group).
// -> (dx, dx3 BF16, dpacked, dx2 BF16, dqkvgu, g_norm2, logit gradients [3, H], first norm's [3, d] or [1, d]): w, and
// behind an FP32 depth modulation its bias and scale.  x: the norm's input, or behind an FP32 modulation that one's.
std::vector<at::Tensor> block_bwd(const at::Tensor& dx3, const at::Tensor& x, const at::Tensor& rstd1,
                                  const at::Tensor& qkvgu, const at::Tensor& x2, const at::Tensor& rstd2,
                                  const at::Tensor& packed, const at::Tensor& writes, const at::Tensor& states,
                                  const c10::optional<at::Tensor>& scale, const c10::optional<at::Tensor>& bias,
                                  const at::Tensor& n1, const at::Tensor& n2, const at::Tensor& w_in, const at::Tensor& w_out,
                                  const at::Tensor& w_ug, const at::Tensor& w_down, const at::Tensor& fast_logit,
                                  const at::Tensor& slow_logit, const at::Tensor& mix_logit, const at::Tensor& rope, int64_t B, int64_t T, int64_t H,
                                  const c10::optional<at::Tensor>& flag) {
  const bool bf16_stream = dx3.scalar_type() == at::kBFloat16;
  at::Tensor dx3b = bf16_stream ? dx3 : cast_bf16(dx3, c10::nullopt);
  const int64_t h = w_down.size(1);
  at::Tensor dpacked = project(dx3b, w_down, true, WS_EPI_SWIGLU_BWD, h, at::empty({dx3b.size(0), 2 * h}, dx3b.options()),
                               c10::nullopt, packed, flag);
  auto [dx2, dx2b, second] = rmsnorm_bwd_partial(input_grad(dpacked, w_ug, flag), x2, rstd2, n2, dx3, c10::nullopt, !bf16_stream);
  if (bf16_stream) dx2b = dx2;
  auto [dqkvgu, scan] = attn_bwd(qkvgu, input_grad(dx2b, w_out, flag), states, writes, rope, fast_logit, slow_logit,
                                 mix_logit, B, T, H, flag);
  at::Tensor dz1 = input_grad(dqkvgu, w_in, flag), dx, first;
  const bool modulated = scale.has_value() && scale->defined() && !bf16_stream;
  if (modulated)
    std::tie(dx, first) = rmsnorm_bwd_modulated(dz1, c10::nullopt, rstd1, n1, dx2, *scale, *bias, x, false);
  else
    std::tie(dx, std::ignore, first) = rmsnorm_bwd_partial(dz1, x, rstd1, n1, dx2, scale, false);
  c10::cuda::CUDAGuard guard(dx.device());
  const int64_t d = x2.size(1), sums = modulated ? 3 : 1;
  const at::TensorOptions floats = second.options();
  at::Tensor g_n2 = at::empty({d}, floats), logits = at::empty({3, H}, floats), norm = at::empty({sums, d}, floats);
  for (const at::Tensor* t : {&fast_logit, &slow_logit, &mix_logit})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == H, "block_bwd: logits");
  check_rc(ws_block_sums(second.data_ptr<float>(), (int)second.size(0), g_n2.data_ptr<float>(), first.data_ptr<float>(),
                         (int)first.size(modulated ? 1 : 0), (int)sums, norm.data_ptr<float>(), scan.data_ptr<float>(), fast_logit.data_ptr<float>(),
                         slow_logit.data_ptr<float>(), mix_logit.data_ptr<float>(), (int)B, (int)H, logits.data_ptr<float>(), (int)d, cur_stream()),
           "block_sums");
  return {dx, dx3b, dpacked, dx2b, dqkvgu, g_n2, logits, norm};
}

// One block as one autograd node whose two directions never enter Python: `ops.fused.CoreFn` for an FP32 stream and weights
// whose gradients go straight into their FP32 buffers (or no backward pass at all).  What CoreFn finds by attribute at each
// pass comes along here.  Calls bound by the host: scoring 128 tokens by a block of width 2048 128 -> 102 us (its kernels take 97), a training pass
// of 2 x 896 tokens at width 1280 520 -> 460, the smoke model's micro-batch (four depths) 2060 -> 1750.
struct BlockSpec {
  at::Tensor bf16[4];   // in_proj, out_proj, up/gate, down
  at::Tensor main[4];   // their FP32 gradients; undefined without a backward pass
  at::Tensor rope;
  c10::optional<at::Tensor> flag;
  at::Tensor hooked;    // CPU word: a hook on finished gradients is set
  int64_t core;         // its number for the core
  bool notify;
  double eps;
  int64_t H;
  bool keep;
};
// Into Python (ops/fused.py): the small gradients are added to their buffers there, and the hook is called.
bool core_finished(int64_t core, bool notify, at::TensorList small) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("ws_b200::core_finished", "")
                             .typed<bool(int64_t, bool, at::TensorList)>();
  return op.call(core, notify, small);
}

std::vector<at::Tensor> differentiated_block_bwd(
    const at::Tensor& dx3, const at::Tensor& x, const at::Tensor& rstd1, const at::Tensor& qkvgu, const at::Tensor& x2,
    const at::Tensor& rstd2, const at::Tensor& packed, const at::Tensor& writes, const at::Tensor& states,
    const c10::optional<at::Tensor>& scale, const c10::optional<at::Tensor>& bias, const at::Tensor& n1, const at::Tensor& n2,
    const at::Tensor& w_in, const at::Tensor& w_out, const at::Tensor& w_ug, const at::Tensor& w_down, const at::Tensor& fast_logit,
    const at::Tensor& slow_logit, const at::Tensor& mix_logit, const at::Tensor& rope, int64_t B, int64_t T, int64_t H,
    const c10::optional<at::Tensor>& flag) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("ws_b200::block_bwd", "").typed<decltype(block_bwd)>();
  return op.call(dx3, x, rstd1, qkvgu, x2, rstd2, packed, writes, states, scale, bias, n1, n2, w_in, w_out, w_ug, w_down, fast_logit,
                 slow_logit, mix_logit, rope, B, T, H, flag);
}

struct BlockFn : public torch::autograd::Function<BlockFn> {
  static at::Tensor vector(const at::Tensor& t) { return t.defined() ? t.detach().to(at::kFloat).contiguous() : t; }
  static c10::optional<at::Tensor> maybe(const at::Tensor& t) { return t.defined() ? c10::optional<at::Tensor>(t) : c10::nullopt; }

  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& x, const c10::optional<at::Tensor>& scale,
                            const c10::optional<at::Tensor>& bias, const at::Tensor& n1, const at::Tensor& n2, const at::Tensor& w_in,
                            const at::Tensor& w_out, const at::Tensor& w_ug, const at::Tensor& w_down, const at::Tensor& fast,
                            const at::Tensor& slow, const at::Tensor& mix, const BlockSpec* spec) {
    const int64_t B = x.size(0), T = x.size(1), d = x.size(2);
    const at::Tensor x_in = x.reshape({B * T, d}).contiguous(), sc = vector(scale.value_or(at::Tensor())), bi = vector(bias.value_or(at::Tensor()));
    if (!spec->keep) {
      c10::cuda::CUDAGuard guard(x_in.device());
      const ForwardBlocks::Weights w{&spec->bf16[0], &spec->bf16[1], &spec->bf16[2], &spec->bf16[3]};
      TORCH_CHECK(x_in.is_cuda() && d == spec->H * 64 && T % 128 == 0 && w.ug->dim() == 2, "block: x must be a CUDA tensor [B, T, d], T whole chunks");
      ForwardBlocks blocks(B, T, spec->H, w.ug->size(0) / 2, spec->rope, spec->eps, spec->flag, false, x_in.options());
      blocks.check_weights(w);
      at::Tensor out = at::empty({B, T, d}, x_in.options());
      const ForwardBlocks::Vectors v = blocks.vectors(n1, n2, fast, slow, mix);
      blocks.begin(x_in.data_ptr<float>(), sc.defined() ? blocks.vector(sc, d) : nullptr, bi.defined() ? blocks.vector(bi, d) : nullptr, v.n1);
      blocks.project_in(w);
      blocks.attention(v);
      blocks.finish(w, v.n2, out.data_ptr<float>());
      return out;
    }
    const at::Tensor logits[3] = {vector(fast), vector(slow), vector(mix)};
    std::vector<at::Tensor> s = block_fwd(x_in, maybe(sc), maybe(bi), vector(n1), spec->bf16[0], spec->bf16[1], vector(n2),
                                          spec->bf16[2], spec->bf16[3], logits[0], logits[1], logits[2], spec->rope, spec->eps,
                                          B, T, spec->H, true, true, spec->flag);
    // x3, xmod, rstd1, z1, qkvgu, y, x2, rstd2, z2, packed, act, writes, states
    const at::Tensor none = s[2];
    ctx->save_for_backward({x_in, sc.defined() ? sc : none, bi.defined() ? bi : none, n1, n2, s[2], s[3], s[4], s[5], s[6],
                            s[7], s[8], s[9], s[10]});
    auto& data = ctx->saved_data;
    data["attention"] = std::vector<at::Tensor>{s[11], s[12]};
    data["weights"] = std::vector<at::Tensor>(spec->bf16, spec->bf16 + 4);
    data["gradients"] = std::vector<at::Tensor>(spec->main, spec->main + 4);
    data["logits"] = std::vector<at::Tensor>(logits, logits + 3);
    data["rope"] = spec->rope;
    data["flag"] = spec->flag.has_value() ? *spec->flag : at::Tensor();
    data["hooked"] = spec->hooked;
    data["shape"] = std::vector<int64_t>{B, T, d, spec->H, sc.defined() ? 1 : 0, spec->core, spec->notify ? 1 : 0};
    return s[0].view({B, T, d});
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto t = ctx->get_saved_variables();   // x, scale, bias, n1, n2, rstd1, z1, qkvgu, y, x2, rstd2, z2, packed, act
    auto& data = ctx->saved_data;
    const std::vector<int64_t> shape = data["shape"].toIntVector();
    const int64_t B = shape[0], T = shape[1], d = shape[2];
    const bool modulated = shape[4] != 0;
    const auto attention = data["attention"].toTensorVector(), w = data["weights"].toTensorVector(),
               main = data["gradients"].toTensorVector(), logits = data["logits"].toTensorVector();
    const at::Tensor flag_tensor = data["flag"].toTensor();
    const c10::optional<at::Tensor> flag = maybe(flag_tensor);
    const at::Tensor dx3 = grads[0].reshape({B * T, d}).contiguous();
    const auto scale = modulated ? c10::optional<at::Tensor>(t[1]) : c10::nullopt, bias = modulated ? c10::optional<at::Tensor>(t[2]) : c10::nullopt;
    // With create_graph the call goes through the dispatcher, which marks its results as having no second derivative.
    std::vector<at::Tensor> r = (at::GradMode::is_enabled() ? differentiated_block_bwd : block_bwd)(
        dx3, t[0], t[5], t[7], t[9], t[10], t[12], attention[0], attention[1], scale, bias, vector(t[3]), vector(t[4]), w[0], w[1],
        w[2], w[3], logits[0], logits[1], logits[2], data["rope"].toTensor(), B, T, shape[3], flag);
    // r: dx, dx3 BF16, dpacked, dx2 BF16, dqkvgu, g_norm2, logit gradients, first norm's (and bias and scale)
    const at::Tensor dys[4] = {r[1], r[2], r[3], r[4]}, xs[4] = {t[13], t[11], t[8], t[6]};
    const at::Tensor into[4] = {main[3], main[2], main[1], main[0]};
    const double betas[4] = {1.0, 1.0, 1.0, 1.0};
    grad_weight_group(dys, xs, into, betas, flag);
    // Whether the hook on finished gradients is set counts now, not when the forward pass ran.
    const at::Tensor none;
    std::vector<at::Tensor> small = {r[7].select(0, 0), r[5], r[6].select(0, 0), r[6].select(0, 1), r[6].select(0, 2)};
    if (*data["hooked"].toTensor().data_ptr<int>() != 0 && core_finished(shape[5], shape[6] != 0, small)) small.assign(5, none);
    return {r[0].view({B, T, d}), modulated ? r[7].select(0, 2) : none, modulated ? r[7].select(0, 1) : none, small[0],
            small[1], none, none, none, none, small[2], small[3], small[4], none};
  }
};

at::Tensor block(const at::Tensor& x, const c10::optional<at::Tensor>& scale, const c10::optional<at::Tensor>& bias,
                 const at::Tensor& n1, const at::Tensor& n2, at::TensorList weights, at::TensorList bf16, at::TensorList main,
                 const at::Tensor& fast, const at::Tensor& slow, const at::Tensor& mix, const at::Tensor& rope, double eps,
                 int64_t H, const c10::optional<at::Tensor>& flag, const at::Tensor& hooked, int64_t core, bool notify) {
  TORCH_CHECK(x.dim() == 3 && x.scalar_type() == at::kFloat && weights.size() == 4 && bf16.size() == 4 &&
              (main.size() == 4 || (main.empty() && !at::GradMode::is_enabled())) && scale.has_value() == bias.has_value(),
              "block: FP32 x [B, T, d], four weights, their BF16 copies and FP32 gradients");
  TORCH_CHECK(hooked.is_cpu() && hooked.scalar_type() == at::kInt && hooked.numel() == 1, "block: hooked must be one int32 on the CPU");
  BlockSpec spec;
  for (int i = 0; i < 4; ++i) {
    spec.bf16[i] = bf16[i];
    if (!main.empty()) spec.main[i] = main[i];
  }
  spec.rope = rope; spec.flag = flag; spec.eps = eps; spec.H = H; spec.keep = at::GradMode::is_enabled();
  spec.hooked = hooked; spec.core = core; spec.notify = notify;
  return BlockFn::apply(x, scale, bias, n1, n2, weights[0], weights[1], weights[2],
                        weights[3], fast, slow, mix, static_cast<const BlockSpec*>(&spec));
}

// All blocks over prompts of any length x [B*T, d] FP32: per block weights in, out, up/gate, down (BF16), vectors n1, n2 and the three
// logits, and what a decode continues from, fast, slow, mixed, k, v, u (written); depth_scale and depth_bias [blocks, d].
// -> (residual input, attention output) of the last block at the final position of every sequence, [B, d] each.
std::tuple<at::Tensor, at::Tensor> blocks_prefill(const at::Tensor& x, const at::Tensor& depth_scale, const at::Tensor& depth_bias,
                                                  at::TensorList weights, at::TensorList vectors, at::TensorList states, const at::Tensor& rope,
                                                  double eps, int64_t B, int64_t T, int64_t H, const c10::optional<at::Tensor>& flag) {
  const int64_t n = (int64_t)weights.size() / 4, d = H * 64;
  TORCH_CHECK(n >= 1 && weights.size() == 4 * (size_t)n && vectors.size() == 5 * (size_t)n && states.size() == 6 * (size_t)n,
              "blocks_prefill: four weights, five vectors and six states a block");
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.is_contiguous() && x.dim() == 2 && x.size(0) == B * T && x.size(1) == d &&
              reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0, "blocks_prefill: x must be contiguous FP32 [B*T, d]");
  for (const at::Tensor* t : {&depth_scale, &depth_bias})
    TORCH_CHECK(t->device() == x.device() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->dim() == 2 && t->size(0) == n && t->size(1) == d &&
                reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0, "blocks_prefill: depth modulation must be contiguous FP32 [blocks, d]");
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(weights[2].dim() == 2, "blocks_prefill: weights");
  ForwardBlocks blocks(B, T, H, weights[2].size(0) / 2, rope, eps, flag, true, x.options());
  const auto of = [&](int64_t i) { return ForwardBlocks::Weights{&weights[4 * i], &weights[4 * i + 1], &weights[4 * i + 2], &weights[4 * i + 3]}; };
  const float *scale = depth_scale.data_ptr<float>(), *bias = depth_bias.data_ptr<float>();
  for (int64_t i = 0; i < n; ++i) {
    blocks.check_weights(of(i));
    const at::Tensor* st = &states[6 * i];
    for (int j = 0; j < 6; ++j)
      TORCH_CHECK(st[j].device() == x.device() && st[j].is_contiguous() && st[j].scalar_type() == (j < 2 ? at::kFloat : at::kBFloat16) &&
                  st[j].numel() == B * H * (j < 3 ? 4096 : 8192), "blocks_prefill: FP32 memories, BF16 mix and caches");
  }
  std::vector<ForwardBlocks::Vectors> v;
  for (int64_t i = 0; i < n; ++i) {
    const at::Tensor* t = &vectors[5 * i];
    v.push_back(blocks.vectors(t[0], t[1], t[2], t[3], t[4]));
  }
  blocks.begin(x.data_ptr<float>(), scale, bias, v[0].n1);
  for (int64_t i = 0; i < n; ++i) {
    blocks.project_in(of(i));
    blocks.attention_prompt(v[i], &states[6 * i]);
    if (i + 1 < n) blocks.finish(of(i), v[i].n2, nullptr, scale + (i + 1) * d, bias + (i + 1) * d, v[i + 1].n1);
  }
  at::Tensor last = at::empty({B, d}, x.options()), y = at::empty({B, d}, x.options().dtype(at::kBFloat16));
  const auto rows = [&](at::Tensor& to, const void* from, size_t element) {
    const size_t bytes = d * element;
    const cudaError_t err = cudaMemcpy2DAsync(to.data_ptr(), bytes, static_cast<const uint8_t*>(from) + (T - 1) * bytes, T * bytes, bytes, B,
                                              cudaMemcpyDeviceToDevice, cur_stream());
    TORCH_CHECK(err == cudaSuccess, "blocks_prefill: copy of the last rows failed");
  };
  rows(last, blocks.stream_rows(), 4);
  rows(y, blocks.attention_rows(), 2);
  return {last, y};
}

// ----------------------------------------------------------------------------- optimizer
static const int* opt_status(const c10::optional<at::Tensor>& status) {
  if (!status.has_value() || !status->defined()) return nullptr;
  TORCH_CHECK(status->is_cuda() && status->scalar_type() == at::kInt && status->numel() >= 1, "status: int32 CUDA tensor");
  return status->data_ptr<int>();
}
static const float* opt_f32(const c10::optional<at::Tensor>& t, const char* what) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->numel() >= 1, what);
  return t->data_ptr<float>();
}

// -> stats [8] FP32: norm, clip coefficient, norm^2, skip flag (the rest is zero)
at::Tensor grad_norm_clip(const at::Tensor& g, double max_norm, const c10::optional<at::Tensor>& extra_sumsq,
                          const c10::optional<at::Tensor>& status) {
  TORCH_CHECK(g.is_cuda() && g.scalar_type() == at::kFloat && g.is_contiguous() && g.numel() % 4 == 0,
              "grad_norm_clip: flat float32 buffer with numel % 4 == 0 required");
  c10::cuda::CUDAGuard guard(g.device());
  at::Tensor partial = at::empty({ws_sumsq_parts()}, g.options());
  at::Tensor stats = at::zeros({8}, g.options());
  check_rc(ws_grad_norm_clip(g.data_ptr<float>(), (size_t)g.numel(), partial.data_ptr<float>(),
                             opt_f32(extra_sumsq, "grad_norm_clip: extra_sumsq"), (float)max_norm, opt_status(status),
                             stats.data_ptr<float>(), cur_stream()), "grad_norm_clip");
  return stats;
}

at::Tensor clip_from_partials(const at::Tensor& partial, double max_norm, const c10::optional<at::Tensor>& extra_sumsq,
                              const c10::optional<at::Tensor>& status) {
  TORCH_CHECK(partial.is_cuda() && partial.scalar_type() == at::kFloat && partial.is_contiguous() && partial.numel() >= 1,
              "clip_from_partials: float32 CUDA partial sums required");
  c10::cuda::CUDAGuard guard(partial.device());
  at::Tensor stats = at::zeros({8}, partial.options());
  check_rc(ws_clip_from_partials(partial.data_ptr<float>(), (int)partial.numel(),
                                 opt_f32(extra_sumsq, "clip_from_partials: extra_sumsq"), (float)max_norm,
                                 opt_status(status), stats.data_ptr<float>(), cur_stream()), "clip_from_partials");
  return stats;
}

void adamw_step(at::Tensor p, const at::Tensor& g, at::Tensor m, at::Tensor v, c10::optional<at::Tensor> p_bf16,
                double lr, double beta1, double beta2, double eps, double wd, int64_t step,
                const c10::optional<at::Tensor>& grad_scale, double grad_scale_const,
                const c10::optional<at::Tensor>& skip) {
  TORCH_CHECK(p.is_cuda() && p.scalar_type() == at::kFloat && p.is_contiguous(), "adamw_step: p");
  TORCH_CHECK(g.numel() == p.numel() && m.numel() == p.numel() && v.numel() == p.numel(), "adamw_step: sizes");
  TORCH_CHECK(g.scalar_type() == at::kFloat && m.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat &&
              g.is_contiguous() && m.is_contiguous() && v.is_contiguous(), "adamw_step: float32 contiguous");
  c10::cuda::CUDAGuard guard(p.device());
  void* pb = nullptr;
  if (p_bf16.has_value() && p_bf16->defined()) {
    TORCH_CHECK(p_bf16->scalar_type() == at::kBFloat16 && p_bf16->numel() == p.numel() && p_bf16->is_contiguous(),
                "adamw_step: p_bf16");
    pb = p_bf16->data_ptr();
  }
  const float* gs = grad_scale.has_value() && grad_scale->defined() ? grad_scale->data_ptr<float>() : nullptr;
  check_rc(ws_adamw(p.data_ptr<float>(), g.data_ptr<float>(), m.data_ptr<float>(), v.data_ptr<float>(), pb,
                    (size_t)p.numel(), (float)lr, (float)beta1, (float)beta2, (float)eps, (float)wd, (int)step, gs,
                    (float)grad_scale_const, opt_f32(skip, "adamw_step: skip"), cur_stream()), "adamw_step");
}

int64_t launch_count() { return (int64_t)ws_launch_count(); }

// ----------------------------------------------------------------------------- LM head
// (lse [rows], logp [rows]) of hidden @ weight.T against labels; logits stay on chip.
std::tuple<at::Tensor, at::Tensor> lm_head_fwd(const at::Tensor& hidden, const at::Tensor& weight,
                                               const at::Tensor& labels, int64_t ignore_index,
                                               const c10::optional<at::Tensor>& error_flag) {
  TORCH_CHECK(hidden.is_cuda() && hidden.scalar_type() == at::kBFloat16 && hidden.dim() == 2 && hidden.stride(1) == 1,
              "lm_head_fwd: hidden must be BF16 [rows, d]");
  TORCH_CHECK(weight.scalar_type() == at::kBFloat16 && weight.dim() == 2 && weight.is_contiguous() &&
              weight.size(1) == hidden.size(1), "lm_head_fwd: weight must be BF16 [vocab, d]");
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == hidden.size(0),
              "lm_head_fwd: labels must be int64 [rows]");
  c10::cuda::CUDAGuard guard(hidden.device());
  const int rows = (int)hidden.size(0), d = (int)hidden.size(1), vocab = (int)weight.size(0);
  const int nparts = 2 * ((vocab + 255) / 256) - (((vocab % 256) != 0 && (vocab % 256) <= 128) ? 1 : 0);
  const int ld = 2 * ((vocab + 255) / 256);
  at::Tensor parts = at::empty({rows, ld, 2}, hidden.options().dtype(at::kFloat));
  at::Tensor label_logit = at::zeros({rows}, hidden.options().dtype(at::kFloat));
  WsGemm g = {};
  g.a = hidden.data_ptr(); g.b = weight.data_ptr();
  g.m = rows; g.n = vocab; g.k = d;
  g.lda = (int)hidden.stride(0); g.ldb = (int)weight.stride(0);
  g.a_mn = 0; g.b_mn = 0; g.epilogue = WS_EPI_CE_FWD;
  g.out = parts.data_ptr(); g.ldo = ld;
  g.out2 = label_logit.data_ptr(); g.ldo2 = 0;
  g.aux = labels.data_ptr(); g.ldaux = 0;
  g.row_scale = nullptr; g.row_vec = nullptr; g.alpha = 1.f; g.beta = 0.f;
  g.error_flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  check_rc(ws_gemm(&g, cur_stream()), "lm_head_fwd gemm");
  at::Tensor lse = at::empty({rows}, hidden.options().dtype(at::kFloat));
  at::Tensor logp = at::empty({rows}, hidden.options().dtype(at::kFloat));
  check_rc(ws_ce_combine(parts.data_ptr(), ld, nparts, label_logit.data_ptr<float>(),
                         reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()), (long long)ignore_index, rows,
                         nullptr, nullptr, lse.data_ptr<float>(), logp.data_ptr<float>(), cur_stream()), "ce_combine");
  return {lse, logp};
}

// The same over the labelled rows only, which are packed together on the device (see lmhead.cu).  Returns
// (logp [rows], lse of the packed rows, index, count, hidden packed, labels packed, BF16 logits of the first keep_rows
// packed rows); what backward needs of them goes to lm_head_bwd_labelled.
std::vector<at::Tensor> lm_head_fwd_labelled(const at::Tensor& hidden, const at::Tensor& weight, const at::Tensor& labels,
                                             int64_t ignore_index, int64_t keep_rows,
                                             const c10::optional<at::Tensor>& error_flag) {
  TORCH_CHECK(keep_rows >= 0 && keep_rows <= hidden.size(0) && (keep_rows == 0 || weight.size(0) % 8 == 0),
              "lm_head_fwd_labelled: keep_rows");
  TORCH_CHECK(hidden.is_cuda() && hidden.scalar_type() == at::kBFloat16 && hidden.dim() == 2 && hidden.is_contiguous() &&
              hidden.size(1) % 8 == 0 && reinterpret_cast<uintptr_t>(hidden.data_ptr()) % 16 == 0,
              "lm_head_fwd_labelled: hidden must be contiguous BF16 [rows, d], d % 8 == 0");
  TORCH_CHECK(weight.scalar_type() == at::kBFloat16 && weight.dim() == 2 && weight.is_contiguous() &&
              weight.size(1) == hidden.size(1), "lm_head_fwd_labelled: weight must be BF16 [vocab, d]");
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == hidden.size(0),
              "lm_head_fwd_labelled: labels must be int64 [rows]");
  c10::cuda::CUDAGuard guard(hidden.device());
  const int rows = (int)hidden.size(0), d = (int)hidden.size(1), vocab = (int)weight.size(0);
  const int ld = 2 * ((vocab + 255) / 256);
  const int nparts = ld - (((vocab % 256) != 0 && (vocab % 256) <= 128) ? 1 : 0);
  const auto f32 = hidden.options().dtype(at::kFloat);
  at::Tensor index = at::empty({rows}, hidden.options().dtype(at::kInt));
  at::Tensor count = at::empty({1}, hidden.options().dtype(at::kInt));
  at::Tensor labels_sel = at::empty({rows}, labels.options());
  at::Tensor packed = at::empty_like(hidden);
  at::Tensor logp = at::empty({rows}, f32);
  at::Tensor parts = at::empty({rows, ld, 2}, f32);
  at::Tensor per_row = at::zeros({2, rows}, f32);   // label logits, log-sum-exps (0 in the padding rows)
  float* label_logit = per_row.data_ptr<float>();
  at::Tensor lse = per_row.select(0, 1);
  const long long* lab = reinterpret_cast<const long long*>(labels_sel.data_ptr<int64_t>());
  check_rc(ws_select_rows(reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()), (long long)ignore_index, rows,
                          index.data_ptr<int>(), count.data_ptr<int>(),
                          reinterpret_cast<long long*>(labels_sel.data_ptr<int64_t>()), logp.data_ptr<float>(),
                          cur_stream()), "select_rows");
  check_rc(ws_gather_rows(hidden.data_ptr(), d, index.data_ptr<int>(), count.data_ptr<int>(), rows, d, packed.data_ptr(),
                          cur_stream()), "gather_rows");
  WsGemm g = {};
  g.a = packed.data_ptr(); g.b = weight.data_ptr();
  g.m = rows; g.n = vocab; g.k = d;
  g.lda = d; g.ldb = d;
  g.epilogue = WS_EPI_CE_FWD;
  g.out = parts.data_ptr(); g.ldo = ld;
  g.out2 = label_logit;
  g.aux = lab;
  g.alpha = 1.f;
  g.error_flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  g.limit = count.data_ptr<int>();
  g.whole = hidden.data_ptr(); g.whole_rows = rows; g.ldwhole = d;
  at::Tensor logits = at::empty({keep_rows, vocab}, hidden.options());
  if (keep_rows > 0) { g.keep = logits.data_ptr(); g.keep_rows = (int)keep_rows; }
  check_rc(ws_gemm(&g, cur_stream()), "lm_head_fwd_labelled gemm");
  check_rc(ws_ce_combine(parts.data_ptr(), ld, nparts, label_logit, lab, (long long)ignore_index, rows,
                         index.data_ptr<int>(), count.data_ptr<int>(), lse.data_ptr<float>(), logp.data_ptr<float>(),
                         cur_stream()), "ce_combine");
  return {logp, lse, index, count, packed, labels_sel, logits};
}

// dhidden [rows, d] (every row written) and grad_weight [vocab, d] += of sum(row_weight * -logp), the rows in blocks of
// `block`: the logit gradients, from the kept logits in place (`logits` is consumed) or past its rows from logits that
// are computed again, then the two products.  row_weight is per row before the selection.
void lm_head_bwd_labelled(const at::Tensor& hidden, const at::Tensor& packed, const at::Tensor& weight,
                          const at::Tensor& labels, const at::Tensor& labels_sel, const at::Tensor& index,
                          const at::Tensor& count, const at::Tensor& lse, const at::Tensor& row_weight,
                          int64_t ignore_index, int64_t block, at::Tensor logits, at::Tensor dhidden,
                          at::Tensor grad_weight, const c10::optional<at::Tensor>& error_flag) {
  const int rows = (int)hidden.size(0), d = (int)hidden.size(1), vocab = (int)weight.size(0);
  TORCH_CHECK(hidden.is_cuda() && hidden.scalar_type() == at::kBFloat16 && hidden.is_contiguous() &&
              packed.scalar_type() == at::kBFloat16 && packed.is_contiguous() && packed.sizes() == hidden.sizes() &&
              weight.scalar_type() == at::kBFloat16 && weight.is_contiguous() && weight.size(1) == d && vocab % 8 == 0,
              "lm_head_bwd_labelled: operands");
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == rows &&
              labels_sel.scalar_type() == at::kLong && labels_sel.is_contiguous() && labels_sel.numel() == rows &&
              index.scalar_type() == at::kInt && index.is_contiguous() && index.numel() == rows &&
              count.scalar_type() == at::kInt && count.numel() == 1 && lse.scalar_type() == at::kFloat &&
              lse.is_contiguous() && lse.numel() == rows && row_weight.scalar_type() == at::kFloat &&
              row_weight.is_contiguous() && row_weight.numel() == rows, "lm_head_bwd_labelled: per-row vectors");
  TORCH_CHECK(dhidden.scalar_type() == at::kBFloat16 && dhidden.is_contiguous() && dhidden.sizes() == hidden.sizes() &&
              grad_weight.scalar_type() == at::kFloat && grad_weight.dim() == 2 && grad_weight.stride(1) == 1 &&
              grad_weight.size(0) == vocab && grad_weight.size(1) == d && block > 0 && block % 256 == 0,
              "lm_head_bwd_labelled: outputs");
  c10::cuda::CUDAGuard guard(hidden.device());
  check_rc(ws_clear_unlabelled(reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()), (long long)ignore_index,
                               rows, d, dhidden.data_ptr(), cur_stream()), "clear_unlabelled");
  const int64_t kept = logits.numel() / vocab;
  TORCH_CHECK(logits.scalar_type() == at::kBFloat16 && logits.is_contiguous() && logits.numel() == kept * vocab &&
              (kept == rows || (kept < rows && kept % 256 == 0)),
              "lm_head_bwd_labelled: logits must be contiguous BF16 [kept rows, vocab]");
  at::Tensor scratch;
  int* flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  for (int start = 0, here = 0; start < rows; start += here) {
    const bool have = start < kept;   // the kept rows are one block: the weight gradient is read and written once for them
    here = have ? (int)kept : std::min((int)block, rows - start);
    const auto from_start = [&](const at::Tensor& t) { return t.data_ptr<at::BFloat16>() + static_cast<int64_t>(start) * d; };
    void* dlogits;
    if (have) {
      dlogits = logits.data_ptr<at::BFloat16>() + static_cast<int64_t>(start) * vocab;
      check_rc(ws_ce_dlogits(dlogits, vocab, reinterpret_cast<const long long*>(labels_sel.data_ptr<int64_t>()) + start,
                             index.data_ptr<int>() + start, lse.data_ptr<float>() + start, row_weight.data_ptr<float>(),
                             count.data_ptr<int>(), start, here, cur_stream()), "ce_dlogits");
    } else {
      if (!scratch.defined()) scratch = at::empty({here, vocab}, hidden.options());   // the first block is the largest
      dlogits = scratch.data_ptr();
      WsGemm g = {};
      g.a = from_start(packed); g.b = weight.data_ptr();
      g.m = here; g.n = vocab; g.k = d;
      g.lda = d; g.ldb = d;
      g.epilogue = WS_EPI_CE_BWD;
      g.out = dlogits; g.ldo = vocab;
      g.aux = labels_sel.data_ptr<int64_t>() + start;
      g.row_scale = row_weight.data_ptr<float>(); g.row_vec = lse.data_ptr<float>() + start;
      g.row_map = index.data_ptr<int>() + start;
      g.alpha = 1.f;
      g.error_flag = flag;
      g.limit = count.data_ptr<int>(); g.limit_from = start;
      g.whole = from_start(hidden); g.whole_rows = rows; g.ldwhole = d;
      check_rc(ws_gemm(&g, cur_stream()), "lm_head_bwd_labelled dlogits");
    }
    WsGemm x = {};
    x.a = dlogits; x.b = weight.data_ptr();
    x.m = here; x.n = d; x.k = vocab;
    x.lda = vocab; x.ldb = d;
    x.b_mn = 1;
    x.epilogue = WS_EPI_BF16;
    x.out = dhidden.data_ptr(); x.ldo = d;
    x.row_map = index.data_ptr<int>() + start;
    x.alpha = 1.f;
    x.error_flag = flag;
    x.limit = count.data_ptr<int>(); x.limit_from = start;
    check_rc(ws_gemm(&x, cur_stream()), "lm_head_bwd_labelled dhidden");
    WsGemm w = {};
    w.a = dlogits; w.b = from_start(packed);
    w.m = vocab; w.n = d; w.k = here;
    w.lda = vocab; w.ldb = d;
    w.a_mn = 1; w.b_mn = 1;
    w.epilogue = WS_EPI_ACC_F32;
    w.out = grad_weight.data_ptr(); w.ldo = (int)grad_weight.stride(0);
    w.alpha = 1.f; w.beta = 1.f;
    w.error_flag = flag;
    w.limit = count.data_ptr<int>(); w.limit_from = start;
    w.whole = from_start(hidden); w.whole_rows = rows; w.ldwhole = d;
    check_rc(ws_gemm(&w, cur_stream()), "lm_head_bwd_labelled dweight");
  }
}

bool gemm_pair_available() { return ws_gemm_pair_available() != 0; }

// dlogits [rows, vocab] BF16 = (softmax(hidden @ weight.T) - onehot(labels)) * row_weight
at::Tensor lm_head_dlogits(const at::Tensor& hidden, const at::Tensor& weight, const at::Tensor& labels,
                           const at::Tensor& lse, const at::Tensor& row_weight,
                           const c10::optional<at::Tensor>& error_flag) {
  TORCH_CHECK(hidden.is_cuda() && hidden.scalar_type() == at::kBFloat16 && hidden.dim() == 2 && hidden.stride(1) == 1,
              "lm_head_dlogits: hidden");
  TORCH_CHECK(weight.scalar_type() == at::kBFloat16 && weight.is_contiguous() && weight.size(1) == hidden.size(1) &&
              weight.size(0) % 8 == 0, "lm_head_dlogits: weight must be BF16 [vocab, d] with vocab % 8 == 0");
  const int rows = (int)hidden.size(0), d = (int)hidden.size(1), vocab = (int)weight.size(0);
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == rows &&
              lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.numel() == rows &&
              row_weight.scalar_type() == at::kFloat && row_weight.is_contiguous() && row_weight.numel() == rows,
              "lm_head_dlogits: per-row vectors");
  c10::cuda::CUDAGuard guard(hidden.device());
  at::Tensor out = at::empty({rows, vocab}, hidden.options());
  WsGemm g = {};
  g.a = hidden.data_ptr(); g.b = weight.data_ptr();
  g.m = rows; g.n = vocab; g.k = d;
  g.lda = (int)hidden.stride(0); g.ldb = (int)weight.stride(0);
  g.a_mn = 0; g.b_mn = 0; g.epilogue = WS_EPI_CE_BWD;
  g.out = out.data_ptr(); g.ldo = vocab;
  g.out2 = nullptr; g.ldo2 = 0;
  g.aux = labels.data_ptr(); g.ldaux = 0;
  g.row_scale = row_weight.data_ptr<float>(); g.row_vec = lse.data_ptr<float>(); g.alpha = 1.f; g.beta = 0.f;
  g.error_flag = reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag)));
  check_rc(ws_gemm(&g, cur_stream()), "lm_head_dlogits gemm");
  return out;
}

// ----------------------------------------------------------------------------- communication
std::vector<unsigned long long> ptr_table(at::IntArrayRef v) {
  std::vector<unsigned long long> out;
  for (int64_t p : v) out.push_back(static_cast<unsigned long long>(p));
  return out;
}

void grad_allreduce(at::IntArrayRef grad_ptrs, at::IntArrayRef flag_ptrs, int64_t mc_grad, int64_t rank,
                    int64_t world, int64_t start, int64_t count, int64_t bucket, int64_t seq, double scale, bool push,
                    int64_t ctas, c10::optional<at::Tensor> sumsq_out, at::Tensor status, double budget_seconds) {
  TORCH_CHECK((int64_t)grad_ptrs.size() == world && (int64_t)flag_ptrs.size() == world, "grad_allreduce: peer tables");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 8, "grad_allreduce: status");
  c10::cuda::CUDAGuard guard(status.device());
  float* ss = nullptr;
  if (sumsq_out.has_value() && sumsq_out->defined()) {
    TORCH_CHECK(sumsq_out->scalar_type() == at::kFloat && sumsq_out->numel() >= ctas, "grad_allreduce: sumsq_out");
    ss = sumsq_out->data_ptr<float>();
  }
  auto g = ptr_table(grad_ptrs), f = ptr_table(flag_ptrs);
  check_rc(ws_grad_allreduce(g.data(), f.data(), (unsigned long long)mc_grad, (int)rank, (int)world, (size_t)start,
                             (size_t)count, (int)bucket, (unsigned)seq, (float)scale, push ? 1 : 0, (int)ctas, ss,
                             status.data_ptr<int>(), budget_seconds, cur_stream()), "grad_allreduce");
}

void wait_probe(const at::Tensor& flag, int64_t expected, at::Tensor status, double budget_seconds) {
  TORCH_CHECK(flag.is_cuda() && flag.scalar_type() == at::kInt && status.scalar_type() == at::kInt &&
              status.numel() >= 8, "wait_probe: int32 CUDA tensors required");
  c10::cuda::CUDAGuard guard(flag.device());
  check_rc(ws_wait_probe(reinterpret_cast<const unsigned*>(flag.data_ptr<int>()), (unsigned)expected,
                         status.data_ptr<int>(), budget_seconds, cur_stream()), "wait_probe");
}

void grad_reduce_segments(at::IntArrayRef grad_ptrs, at::IntArrayRef flag_ptrs, int64_t mc_grad, int64_t rank,
                          int64_t world, at::IntArrayRef starts, at::IntArrayRef counts, at::IntArrayRef push,
                          int64_t bucket, int64_t seq, double scale, int64_t ctas, c10::optional<at::Tensor> sumsq_out,
                          at::Tensor status, double budget_seconds) {
  TORCH_CHECK((int64_t)grad_ptrs.size() == world && (int64_t)flag_ptrs.size() == world, "grad_reduce_segments: peer tables");
  TORCH_CHECK(starts.size() == counts.size() && starts.size() == push.size() && !starts.empty() && starts.size() <= 6,
              "grad_reduce_segments: 1..6 segments with start, count and push each");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 8, "grad_reduce_segments: status");
  c10::cuda::CUDAGuard guard(status.device());
  float* ss = nullptr;
  if (sumsq_out.has_value() && sumsq_out->defined()) {
    TORCH_CHECK(sumsq_out->scalar_type() == at::kFloat && sumsq_out->numel() >= ctas && sumsq_out->is_contiguous(),
                "grad_reduce_segments: sumsq_out");
    ss = sumsq_out->data_ptr<float>();
  }
  size_t st[6], ct[6];
  int pu[6];
  for (size_t i = 0; i < starts.size(); ++i) {
    TORCH_CHECK(starts[i] >= 0 && counts[i] >= 0, "grad_reduce_segments: negative range");
    st[i] = (size_t)starts[i]; ct[i] = (size_t)counts[i]; pu[i] = push[i] ? 1 : 0;
  }
  auto g = ptr_table(grad_ptrs), f = ptr_table(flag_ptrs);
  check_rc(ws_grad_reduce_segments(g.data(), f.data(), (unsigned long long)mc_grad, (int)rank, (int)world, st, ct, pu,
                                   (int)starts.size(), (int)bucket, (unsigned)seq, (float)scale, (int)ctas, ss,
                                   status.data_ptr<int>(), budget_seconds, cur_stream()), "grad_reduce_segments");
}

// -> stats [8] FP32: global norm, clip coefficient, norm^2, skip flag, loss summed over ranks
at::Tensor norm_exchange(at::IntArrayRef flag_ptrs, int64_t rank, int64_t world, int64_t base_word, int64_t seq,
                         const at::Tensor& partial, const c10::optional<at::Tensor>& local_loss, double max_norm,
                         at::Tensor status, double budget_seconds) {
  TORCH_CHECK((int64_t)flag_ptrs.size() == world, "norm_exchange: peer table");
  TORCH_CHECK(partial.is_cuda() && partial.scalar_type() == at::kFloat && partial.is_contiguous() && partial.numel() >= 1,
              "norm_exchange: partial");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 8, "norm_exchange: status");
  c10::cuda::CUDAGuard guard(partial.device());
  at::Tensor stats = at::zeros({8}, partial.options());
  auto f = ptr_table(flag_ptrs);
  check_rc(ws_norm_exchange(f.data(), (int)rank, (int)world, (int)base_word, (unsigned)seq, partial.data_ptr<float>(),
                            (int)partial.numel(), opt_f32(local_loss, "norm_exchange: local_loss"), (float)max_norm,
                            status.data_ptr<int>(), stats.data_ptr<float>(), budget_seconds, cur_stream()),
           "norm_exchange");
  return stats;
}

void node_barrier(at::IntArrayRef flag_ptrs, int64_t rank, int64_t world, int64_t base_word, int64_t seq,
                  at::Tensor status, double budget_seconds) {
  TORCH_CHECK((int64_t)flag_ptrs.size() == world, "node_barrier: peer table");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 8, "node_barrier: status");
  c10::cuda::CUDAGuard guard(status.device());
  auto f = ptr_table(flag_ptrs);
  check_rc(ws_node_barrier(f.data(), (int)rank, (int)world, (int)base_word, (unsigned)seq, status.data_ptr<int>(),
                           budget_seconds, cur_stream()), "node_barrier");
}

// wb [n, k] BF16 (local) = cast of the row-sharded FP32 weight (shard addresses as mapped in this process)
void gather_cast(std::vector<int64_t> shard_ptrs, int64_t rows_per_shard, at::Tensor wb, int64_t ctas) {
  TORCH_CHECK(wb.is_cuda() && wb.scalar_type() == at::kBFloat16 && wb.is_contiguous() && wb.dim() == 2,
              "gather_cast: wb must be contiguous BF16 [n, k]");
  const int64_t world = (int64_t)shard_ptrs.size();
  TORCH_CHECK(world >= 1 && world <= 8, "gather_cast: 1..8 shards");
  const void* shards[8] = {};
  for (int64_t r = 0; r < world; ++r) shards[r] = reinterpret_cast<const void*>(static_cast<uintptr_t>(shard_ptrs[r]));
  c10::cuda::CUDAGuard guard(wb.device());
  check_rc(ws_gather_cast(shards, (int)world, (int)rows_per_shard, (int)wb.size(0), (int)wb.size(1), wb.data_ptr(),
                          (int)ctas, cur_stream()), "gather_cast");
}

void adamw_shard_push(at::IntArrayRef master_ptrs, at::IntArrayRef bf16_ptrs, int64_t rank, int64_t world,
                      const at::Tensor& g, at::Tensor m, at::Tensor v, int64_t lo, int64_t n, double lr, double beta1,
                      double beta2, double eps, double wd, int64_t step, const c10::optional<at::Tensor>& grad_scale,
                      bool push_master, const c10::optional<at::Tensor>& skip) {
  TORCH_CHECK((int64_t)master_ptrs.size() == world && (int64_t)bf16_ptrs.size() == world, "adamw_shard_push: tables");
  TORCH_CHECK(g.is_cuda() && g.scalar_type() == at::kFloat && g.is_contiguous() && g.numel() >= lo + n, "adamw_shard_push: g");
  TORCH_CHECK(m.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat && m.numel() == n && v.numel() == n &&
              m.is_contiguous() && v.is_contiguous(), "adamw_shard_push: moments");
  c10::cuda::CUDAGuard guard(g.device());
  auto mp = ptr_table(master_ptrs), bp = ptr_table(bf16_ptrs);
  const float* gs = grad_scale.has_value() && grad_scale->defined() ? grad_scale->data_ptr<float>() : nullptr;
  check_rc(ws_adamw_shard_push(mp.data(), bp.data(), (int)rank, (int)world, g.data_ptr<float>(), m.data_ptr<float>(),
                               v.data_ptr<float>(), (size_t)lo, (size_t)n, (float)lr, (float)beta1, (float)beta2,
                               (float)eps, (float)wd, (int)step, gs, push_master ? 1 : 0,
                               opt_f32(skip, "adamw_shard_push: skip"), cur_stream()),
           "adamw_shard_push");
}

// ----------------------------------------------------------------------------- sharded-weight linear
// y = x @ W^T where W [n, k] is FP32 and row-sharded over `shard_ptrs.size()` ranks (addresses as mapped in
// this process: the local shard and the peers' symmetric-memory shards).  One launch gathers, casts and
// multiplies; `wb` receives the BF16 copy of the whole weight as a by-product.
std::tuple<at::Tensor, at::Tensor> gather_cast_linear(const at::Tensor& x, std::vector<int64_t> shard_ptrs, int64_t n,
                                                      int64_t rows_per_shard, at::Tensor wb, at::Tensor flags,
                                                      c10::optional<at::Tensor> error_flag, double budget_seconds,
                                                      bool swiglu, bool want_packed) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.is_contiguous(),
              "gather_cast_linear: x must be contiguous BF16 [m, k]");
  const int64_t m = x.size(0), k = x.size(1);
  const int64_t world = (int64_t)shard_ptrs.size();
  const int64_t w_rows = swiglu ? 2 * n : n;
  TORCH_CHECK(world >= 1 && world <= 8, "gather_cast_linear: 1..8 shards");
  TORCH_CHECK(k % 8 == 0 && n > 0 && n % 8 == 0 && rows_per_shard > 0 && rows_per_shard % 8 == 0 &&
              rows_per_shard * world >= w_rows,
              "gather_cast_linear: k, n and rows_per_shard must be multiples of 8 and the shards must cover the weight");
  TORCH_CHECK(!swiglu || n % 128 == 0, "gather_cast_linear: the SwiGLU form needs a hidden width that is a multiple of 128");
  TORCH_CHECK(wb.is_cuda() && wb.scalar_type() == at::kBFloat16 && wb.is_contiguous() && wb.numel() == w_rows * k,
              "gather_cast_linear: wb must be contiguous BF16 with the weight's shape");
  TORCH_CHECK(flags.is_cuda() && flags.scalar_type() == at::kInt && flags.is_contiguous() && flags.numel() >= (w_rows + 127) / 128 + 1,
              "gather_cast_linear: flags must be int32 with one word per 128 weight rows and one more");
  const void* shards[8] = {};
  for (int64_t r = 0; r < world; ++r) {
    TORCH_CHECK(shard_ptrs[r] != 0 && shard_ptrs[r] % 16 == 0, "gather_cast_linear: null or misaligned shard address");
    shards[r] = reinterpret_cast<const void*>(static_cast<uintptr_t>(shard_ptrs[r]));
  }
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor out, act;
  if (swiglu) {
    act = at::empty({m, n}, x.options());
    if (want_packed) out = at::empty({m, 2 * n}, x.options());
  } else {
    out = at::empty({m, n}, x.options());
  }
  check_rc(ws_gather_gemm(x.data_ptr(), (int)m, (int)n, (int)k, shards, (int)world, (int)rows_per_shard, wb.data_ptr(),
                          flags.data_ptr(), swiglu ? WS_EPI_SWIGLU : WS_EPI_BF16, out.defined() ? out.data_ptr() : nullptr,
                          (int)w_rows, swiglu ? act.data_ptr() : nullptr, (int)n,
                          reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))), (float)budget_seconds, 0,
                          cur_stream()), "gather_cast_linear");
  if (!out.defined()) out = at::empty({0}, x.options());
  if (!act.defined()) act = at::empty({0}, x.options());
  return std::make_tuple(out, act);
}

// ----------------------------------------------------------------------------- decode step
int64_t decode_gemm_splits(int64_t n, int64_t k) { return ws_decode_gemm_splits((int)n, (int)k); }
// Raises the library's error for a non-zero status of a C entry point (what every binding does
// with the codes it gets back); callable without a GPU, so the error path itself is testable.
int64_t raise_for_status(int64_t code) {
  check_rc((int)code, "status");
  return code;
}

void decode_gemm(const at::Tensor& w, const at::Tensor& x, int64_t n, int64_t epilogue, at::Tensor out,
                 c10::optional<at::Tensor> error_flag, bool packed) {
  TORCH_CHECK(w.is_cuda() && x.is_cuda() && out.is_cuda(), "decode_gemm: CUDA tensors required");
  TORCH_CHECK(w.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16 && w.is_contiguous() &&
              x.is_contiguous() && x.dim() == 2, "decode_gemm: contiguous BF16 W and x [batch, k] required");
  const int64_t k = x.size(1), batch = x.size(0);
  TORCH_CHECK(batch >= 1 && batch <= 64 && k % 8 == 0, "decode_gemm: batch must be 1..64 and k a multiple of 8");
  TORCH_CHECK(epilogue >= 0 && epilogue <= 3 && n > 0, "decode_gemm: epilogue 0..3 and n > 0 required");
  if (packed) {
    const int64_t slabs = epilogue == 2 ? n / 64 : (n + 127) / 128;
    TORCH_CHECK(w.dim() == 4 && w.size(0) == slabs && w.size(1) == (k + 63) / 64 && w.size(2) == 128 && w.size(3) == 64,
                "decode_gemm: a packed W must be [slabs, ceil(k/64), 128, 64]");
  } else {
    TORCH_CHECK(w.dim() == 2 && w.size(1) == k && w.size(0) == (epilogue == 2 ? 2 * n : n),
                "decode_gemm: W must be [rows, k] with rows matching n");
  }
  TORCH_CHECK(reinterpret_cast<uintptr_t>(w.data_ptr()) % 16 == 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0,
              "decode_gemm: 16-byte aligned operands required");
  TORCH_CHECK(out.is_contiguous(), "decode_gemm: contiguous out required");
  if (epilogue == 1) {
    TORCH_CHECK(out.scalar_type() == at::kFloat && out.numel() == decode_gemm_splits(n, k) * batch * n,
                "decode_gemm: partial buffer must be FP32 [splits, batch, n]");
  } else {
    TORCH_CHECK(out.scalar_type() == (epilogue == 3 ? at::kFloat : at::kBFloat16) && out.dim() == 2 &&
                out.size(0) == batch && out.size(1) == n, "decode_gemm: out must be [batch, n] of the epilogue's dtype");
  }
  c10::cuda::CUDAGuard guard(w.device());
  check_rc(ws_decode_gemm(w.data_ptr(), x.data_ptr(), (int)n, (int)k, (int)batch, (int)epilogue, out.data_ptr(), (int)n,
                          reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))), packed ? 1 : 0, cur_stream()),
           "decode_gemm");
}

void decode_reduce_norm(at::Tensor x, const c10::optional<at::Tensor>& partial, const c10::optional<at::Tensor>& token,
                        const c10::optional<at::Tensor>& table, const c10::optional<at::Tensor>& scale,
                        const c10::optional<at::Tensor>& bias, const at::Tensor& w, double eps,
                        c10::optional<at::Tensor> out) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 2 && x.is_contiguous(), "decode_reduce_norm: x");
  const int64_t batch = x.size(0), d = x.size(1);
  TORCH_CHECK(d % 4 == 0 && w.scalar_type() == at::kFloat && w.numel() == d && w.is_contiguous(), "decode_reduce_norm: w");
  int splits = 0;
  const float* pp = nullptr;
  if (partial.has_value() && partial->defined()) {
    TORCH_CHECK(partial->scalar_type() == at::kFloat && partial->is_contiguous() && partial->numel() % (batch * d) == 0,
                "decode_reduce_norm: partial must be FP32 [splits, batch, d]");
    splits = (int)(partial->numel() / (batch * d));
    pp = partial->data_ptr<float>();
  }
  const long long* tok = nullptr;
  const float* tab = nullptr;
  int vocab = 0;
  if (token.has_value() && token->defined()) {
    TORCH_CHECK(table.has_value() && token->scalar_type() == at::kLong && token->numel() == batch && token->is_contiguous() &&
                table->scalar_type() == at::kFloat && table->is_contiguous() && table->size(1) == d && splits == 0,
                "decode_reduce_norm: token [batch] int64 with an FP32 table [vocab, d], and no partials");
    tok = reinterpret_cast<const long long*>(token->data_ptr<int64_t>());
    tab = table->data_ptr<float>();
    vocab = (int)table->size(0);
  }
  const bool mod = scale.has_value() && scale->defined();
  if (mod) {
    TORCH_CHECK(bias.has_value() && scale->scalar_type() == at::kFloat && bias->scalar_type() == at::kFloat &&
                scale->numel() == d && bias->numel() == d && scale->is_contiguous() && bias->is_contiguous(),
                "decode_reduce_norm: modulation vectors must be FP32 [d]");
  }
  void* op = nullptr;
  if (out.has_value() && out->defined()) {
    TORCH_CHECK(out->scalar_type() == at::kBFloat16 && out->is_contiguous() && out->numel() == batch * d, "decode_reduce_norm: out");
    op = out->data_ptr();
  }
  c10::cuda::CUDAGuard guard(x.device());
  check_rc(ws_decode_reduce_norm(x.data_ptr<float>(), pp, splits, tok, tab, vocab, mod ? scale->data_ptr<float>() : nullptr,
                                 mod ? bias->data_ptr<float>() : nullptr, w.data_ptr<float>(), (float)eps, (int)d,
                                 (int)batch, op, cur_stream()), "decode_reduce_norm");
}

// One sequence: decode_reduce_norm and the decode_gemm that reads its result as one launch; x_out takes the residual that the former leaves in x.
void decode_norm_gemm(const at::Tensor& x, const c10::optional<at::Tensor>& x_out, const c10::optional<at::Tensor>& partial,
                      const c10::optional<at::Tensor>& token, const c10::optional<at::Tensor>& table, const c10::optional<at::Tensor>& scale,
                      const c10::optional<at::Tensor>& bias, const at::Tensor& norm, double eps, const at::Tensor& w, int64_t n,
                      int64_t epilogue, at::Tensor out, const c10::optional<at::Tensor>& error_flag, bool packed) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 2 && x.is_contiguous(), "decode_norm_gemm: x must be contiguous FP32 [1, d]");
  const int64_t d = x.size(1);
  TORCH_CHECK(x.size(0) == 1 && d % 64 == 0 && d >= 64 && d <= 2048, "decode_norm_gemm: one sequence, d a multiple of 64 up to 2048");
  const auto vector = [&](const at::Tensor& t, const char* what) {
    TORCH_CHECK(t.device() == x.device() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() == d &&
                reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, what);
    return t.data_ptr<float>();
  };
  const float* nw = vector(norm, "decode_norm_gemm: norm must be FP32 [d]");
  const bool mod = scale.has_value() && scale->defined();
  TORCH_CHECK(mod == (bias.has_value() && bias->defined()), "decode_norm_gemm: modulation needs scale and bias");
  const float* sc = mod ? vector(*scale, "decode_norm_gemm: scale must be FP32 [d]") : nullptr;
  const float* bi = mod ? vector(*bias, "decode_norm_gemm: bias must be FP32 [d]") : nullptr;
  float* xo = nullptr;
  if (x_out.has_value() && x_out->defined()) {
    TORCH_CHECK(x_out->device() == x.device() && x_out->scalar_type() == at::kFloat && x_out->is_contiguous() && x_out->sizes() == x.sizes() &&
                x_out->data_ptr() != x.data_ptr(), "decode_norm_gemm: x_out must be a buffer of its own like x");
    xo = x_out->data_ptr<float>();
  }
  int splits = 0;
  const float* pp = nullptr;
  if (partial.has_value() && partial->defined()) {
    TORCH_CHECK(partial->device() == x.device() && partial->scalar_type() == at::kFloat && partial->is_contiguous() &&
                partial->numel() % d == 0, "decode_norm_gemm: partial must be FP32 [splits, 1, d]");
    splits = (int)(partial->numel() / d);
    pp = partial->data_ptr<float>();
  }
  const long long* tok = nullptr;
  const float* tab = nullptr;
  int vocab = 0;
  if (token.has_value() && token->defined()) {
    TORCH_CHECK(table.has_value() && token->device() == x.device() && token->scalar_type() == at::kLong && token->numel() == 1 &&
                token->is_contiguous() && table->device() == x.device() && table->scalar_type() == at::kFloat && table->is_contiguous() &&
                table->dim() == 2 && table->size(1) == d && splits == 0,
                "decode_norm_gemm: token [1] int64 with an FP32 table [vocab, d], and no partials");
    tok = reinterpret_cast<const long long*>(token->data_ptr<int64_t>());
    tab = table->data_ptr<float>();
    vocab = (int)table->size(0);
  }
  TORCH_CHECK(epilogue == 0 || epilogue == 2 || epilogue == 3, "decode_norm_gemm: epilogue 0, 2 or 3");
  TORCH_CHECK(w.device() == x.device() && w.scalar_type() == at::kBFloat16 && w.is_contiguous() && n > 0 &&
              reinterpret_cast<uintptr_t>(w.data_ptr()) % 16 == 0, "decode_norm_gemm: contiguous BF16 W");
  if (packed) {
    TORCH_CHECK(w.dim() == 4 && w.size(0) == (epilogue == 2 ? n / 64 : (n + 127) / 128) && w.size(1) == d / 64 && w.size(2) == 128 && w.size(3) == 64,
                "decode_norm_gemm: a packed W must be [slabs, d / 64, 128, 64]");
  } else {
    TORCH_CHECK(w.dim() == 2 && w.size(1) == d && w.size(0) == (epilogue == 2 ? 2 * n : n), "decode_norm_gemm: W must be [rows, d] with rows matching n");
  }
  TORCH_CHECK(out.device() == x.device() && out.is_contiguous() && out.scalar_type() == (epilogue == 3 ? at::kFloat : at::kBFloat16) &&
              out.dim() == 2 && out.size(0) == 1 && out.size(1) == n, "decode_norm_gemm: out must be [1, n] of the epilogue's dtype");
  c10::cuda::CUDAGuard guard(x.device());
  check_rc(ws_decode_norm_gemm(x.data_ptr<float>(), xo, pp, splits, tok, tab, vocab, sc, bi, nw, (float)eps, w.data_ptr(), (int)n, (int)d,
                               (int)epilogue, out.data_ptr(), (int)n, reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))),
                               packed ? 1 : 0, cur_stream()), "decode_norm_gemm");
}

void decode_attn(const at::Tensor& qkvgu, at::Tensor kc, at::Tensor vc, at::Tensor uc, const at::Tensor& mixed,
                 const at::Tensor& rope, const at::Tensor& pos, int64_t H, at::Tensor y, bool early) {
  TORCH_CHECK(qkvgu.is_cuda() && qkvgu.scalar_type() == at::kBFloat16 && qkvgu.dim() == 2 && qkvgu.is_contiguous(),
              "decode_attn: qkvgu must be contiguous BF16 [batch, 5d]");
  const int64_t batch = qkvgu.size(0), d = qkvgu.size(1) / 5;
  TORCH_CHECK(d == H * 64, "decode_attn: head_dim must be 64");
  for (const at::Tensor* t : {&kc, &vc, &uc}) {
    TORCH_CHECK(t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->numel() == batch * H * 128 * 64,
                "decode_attn: caches must be contiguous BF16 [batch, H, 128, 64]");
  }
  TORCH_CHECK(mixed.scalar_type() == at::kBFloat16 && mixed.is_contiguous() && mixed.numel() == batch * H * 64 * 64,
              "decode_attn: mixed state must be contiguous BF16 [batch, H, 64, 64]");
  TORCH_CHECK(rope.scalar_type() == at::kFloat && rope.is_contiguous() && rope.numel() == 128 * 32 * 2, "decode_attn: rope table");
  TORCH_CHECK(pos.scalar_type() == at::kLong && pos.numel() == 1 && pos.is_cuda(), "decode_attn: pos must be a CUDA int64 scalar");
  TORCH_CHECK(y.scalar_type() == at::kBFloat16 && y.is_contiguous() && y.numel() == batch * d, "decode_attn: y");
  c10::cuda::CUDAGuard guard(qkvgu.device());
  check_rc(ws_decode_attn(qkvgu.data_ptr(), kc.data_ptr(), vc.data_ptr(), uc.data_ptr(), mixed.data_ptr(),
                          rope.data_ptr<float>(), reinterpret_cast<const long long*>(pos.data_ptr<int64_t>()), (int)batch,
                          (int)H, (int)d, y.data_ptr(), early, cur_stream()), "decode_attn");
}

void decode_layer_tail(const at::Tensor& w_out, const at::Tensor& w_ug, const at::Tensor& w_down,
                       const c10::optional<at::Tensor>& w_in_next, const at::Tensor& y, at::Tensor x, at::Tensor part_out,
                       at::Tensor part_down, at::Tensor n, at::Tensor act, at::Tensor qkvgu, const at::Tensor& w_norm2,
                       const c10::optional<at::Tensor>& next_scale, const c10::optional<at::Tensor>& next_bias,
                       const at::Tensor& w_norm_next, double eps, at::Tensor barrier, const c10::optional<at::Tensor>& error_flag,
                       const c10::optional<at::Tensor>& trace) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 2 && x.is_contiguous(), "decode_layer_tail: x");
  const int64_t batch = x.size(0), d = x.size(1);
  TORCH_CHECK(w_down.dim() == 2 && w_down.size(0) == d, "decode_layer_tail: w_down must be [d, ffn]");
  const int64_t ffn = w_down.size(1);
  auto bf16 = [](const at::Tensor& t, int64_t rows, int64_t cols, const char* what) {
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.dim() == 2 && t.size(0) == rows &&
                t.size(1) == cols && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, what);
  };
  bf16(w_out, d, d, "decode_layer_tail: w_out must be contiguous BF16 [d, d]");
  bf16(w_ug, 2 * ffn, d, "decode_layer_tail: w_ug must be contiguous BF16 [2 ffn, d]");
  bf16(w_down, d, ffn, "decode_layer_tail: w_down must be contiguous BF16 [d, ffn]");
  if (w_in_next.has_value()) bf16(*w_in_next, 5 * d, d, "decode_layer_tail: w_in_next must be contiguous BF16 [5 d, d]");
  bf16(y, batch, d, "decode_layer_tail: y must be contiguous BF16 [batch, d]");
  bf16(n, batch, d, "decode_layer_tail: n must be contiguous BF16 [batch, d]");
  bf16(act, batch, ffn, "decode_layer_tail: act must be contiguous BF16 [batch, ffn]");
  bf16(qkvgu, batch, 5 * d, "decode_layer_tail: qkvgu must be contiguous BF16 [batch, 5 d]");
  TORCH_CHECK(part_out.scalar_type() == at::kFloat && part_out.is_contiguous() &&
              part_out.numel() == decode_gemm_splits(d, d) * batch * d, "decode_layer_tail: part_out [splits, batch, d] FP32");
  TORCH_CHECK(part_down.scalar_type() == at::kFloat && part_down.is_contiguous() &&
              part_down.numel() == decode_gemm_splits(d, ffn) * batch * d, "decode_layer_tail: part_down [splits, batch, d] FP32");
  for (const at::Tensor* t : {&w_norm2, &w_norm_next}) {
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == d,
                "decode_layer_tail: norm weights must be FP32 [d]");
  }
  TORCH_CHECK(next_scale.has_value() == next_bias.has_value(), "decode_layer_tail: modulation needs scale and bias");
  if (next_scale.has_value()) {
    TORCH_CHECK(next_scale->scalar_type() == at::kFloat && next_scale->numel() == d && next_scale->is_contiguous() &&
                next_bias->scalar_type() == at::kFloat && next_bias->numel() == d && next_bias->is_contiguous(),
                "decode_layer_tail: modulation vectors must be FP32 [d]");
  }
  TORCH_CHECK(barrier.is_cuda() && barrier.scalar_type() == at::kInt && barrier.is_contiguous() && barrier.numel() >= 2,
              "decode_layer_tail: barrier must hold two int32 words");
  long long* stamps = nullptr;
  if (trace.has_value()) {
    const int sms = at::cuda::getDeviceProperties(x.device().index())->multiProcessorCount;
    TORCH_CHECK(trace->is_cuda() && trace->scalar_type() == at::kLong && trace->is_contiguous() && trace->numel() >= 16 * sms,
                "decode_layer_tail: trace must be int64 [SMs, 16]");
    stamps = reinterpret_cast<long long*>(trace->data_ptr<int64_t>());
  }
  c10::cuda::CUDAGuard guard(x.device());
  check_rc(ws_decode_layer_tail(w_out.data_ptr(), w_ug.data_ptr(), w_down.data_ptr(),
                                w_in_next.has_value() ? w_in_next->data_ptr() : nullptr, y.data_ptr(), x.data_ptr<float>(),
                                part_out.data_ptr<float>(), part_down.data_ptr<float>(), n.data_ptr(), act.data_ptr(),
                                qkvgu.data_ptr(), w_norm2.data_ptr<float>(),
                                next_scale.has_value() ? next_scale->data_ptr<float>() : nullptr,
                                next_bias.has_value() ? next_bias->data_ptr<float>() : nullptr, w_norm_next.data_ptr<float>(),
                                (float)eps, (int)batch, (int)d, (int)ffn, reinterpret_cast<unsigned*>(barrier.data_ptr<int>()),
                                reinterpret_cast<int*>(const_cast<void*>(opt_ptr(error_flag))), stamps, cur_stream()), "decode_layer_tail");
}

void decode_chunk_end(const at::Tensor& kc, const at::Tensor& uc, at::Tensor fast, at::Tensor slow, at::Tensor mixed,
                      const at::Tensor& fast_keep, const at::Tensor& slow_keep, const at::Tensor& mix) {
  TORCH_CHECK(kc.is_cuda() && kc.dim() == 4 && kc.size(2) == 128 && kc.size(3) == 64, "decode_chunk_end: caches must be [batch, H, 128, 64]");
  const int64_t batch = kc.size(0), H = kc.size(1);
  for (const at::Tensor* t : {&kc, &uc})
    TORCH_CHECK(t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->numel() == batch * H * 8192, "decode_chunk_end: BF16 caches");
  for (const at::Tensor* t : {&fast, &slow})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == batch * H * 4096, "decode_chunk_end: FP32 memories");
  TORCH_CHECK(mixed.scalar_type() == at::kBFloat16 && mixed.is_contiguous() && mixed.numel() == batch * H * 4096,
              "decode_chunk_end: mixed must be BF16 [batch, H, 64, 64]");
  for (const at::Tensor* t : {&fast_keep, &slow_keep, &mix})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == H, "decode_chunk_end: per-head FP32 values");
  c10::cuda::CUDAGuard guard(kc.device());
  check_rc(ws_decode_chunk_end(kc.data_ptr(), uc.data_ptr(), fast.data_ptr<float>(), slow.data_ptr<float>(), mixed.data_ptr(),
                               fast_keep.data_ptr<float>(), slow_keep.data_ptr<float>(), mix.data_ptr<float>(), (int)batch,
                               (int)H, cur_stream()), "decode_chunk_end");
}

void decode_pick(const at::Tensor& logits, at::Tensor token, const c10::optional<at::Tensor>& history, at::Tensor cursor,
                 at::Tensor pos) {
  TORCH_CHECK(logits.is_cuda() && logits.scalar_type() == at::kFloat && logits.dim() == 2 && logits.is_contiguous() &&
              logits.size(1) % 4 == 0, "decode_pick: logits must be contiguous FP32 [batch, vocab], vocab a multiple of 4");
  const int64_t batch = logits.size(0);
  TORCH_CHECK(token.is_cuda() && token.scalar_type() == at::kLong && token.is_contiguous() && token.numel() == batch,
              "decode_pick: token must be int64 [batch]");
  TORCH_CHECK(cursor.is_cuda() && cursor.scalar_type() == at::kLong && cursor.is_contiguous() && cursor.numel() == 2,
              "decode_pick: cursor must be two int64 words");
  TORCH_CHECK(pos.is_cuda() && pos.scalar_type() == at::kLong && pos.numel() == 1, "decode_pick: pos must be an int64 scalar");
  long long* hist = nullptr;
  int capacity = 0;
  if (history.has_value()) {
    TORCH_CHECK(history->is_cuda() && history->scalar_type() == at::kLong && history->is_contiguous() && history->dim() == 2 &&
                history->size(0) == batch, "decode_pick: history must be contiguous int64 [batch, capacity]");
    hist = reinterpret_cast<long long*>(history->data_ptr<int64_t>());
    capacity = (int)history->size(1);
  }
  c10::cuda::CUDAGuard guard(logits.device());
  check_rc(ws_decode_pick(logits.data_ptr<float>(), (int)batch, (int)logits.size(1),
                          reinterpret_cast<long long*>(token.data_ptr<int64_t>()), hist, capacity,
                          reinterpret_cast<long long*>(cursor.data_ptr<int64_t>()),
                          reinterpret_cast<long long*>(pos.data_ptr<int64_t>()), cur_stream()), "decode_pick");
}

}  // namespace

TORCH_LIBRARY(ws_b200, m) {
  m.def("decode_gemm_splits(int n, int k) -> int");
  m.def("gather_cast_linear(Tensor x, int[] shard_ptrs, int n, int rows_per_shard, Tensor(a!) wb, Tensor(b!) flags, "
        "Tensor(c!)? error_flag, float budget_seconds, bool swiglu=False, bool want_packed=True) -> (Tensor, Tensor)");
  m.def("raise_for_status(int code) -> int");
  m.def("decode_gemm(Tensor w, Tensor x, int n, int epilogue, Tensor(a!) out, Tensor(b!)? error_flag, bool packed=False) -> ()");
  m.def("decode_reduce_norm(Tensor(a!) x, Tensor? partial, Tensor? token, Tensor? table, Tensor? scale, Tensor? bias, "
        "Tensor w, float eps, Tensor(b!)? out) -> ()");
  m.def("decode_norm_gemm(Tensor x, Tensor(a!)? x_out, Tensor? partial, Tensor? token, Tensor? table, Tensor? scale, Tensor? bias, "
        "Tensor norm, float eps, Tensor w, int n, int epilogue, Tensor(b!) out, Tensor(c!)? error_flag, bool packed=False) -> ()");
  m.def("decode_layer_tail(Tensor w_out, Tensor w_ug, Tensor w_down, Tensor? w_in_next, Tensor y, Tensor(a!) x, "
        "Tensor(b!) part_out, Tensor(c!) part_down, Tensor(d!) n, Tensor(e!) act, Tensor(f!) qkvgu, Tensor w_norm2, "
        "Tensor? next_scale, Tensor? next_bias, Tensor w_norm_next, float eps, Tensor(g!) barrier, Tensor(h!)? error_flag, "
        "Tensor(i!)? trace=None) -> ()");
  m.def("decode_chunk_end(Tensor kc, Tensor uc, Tensor(a!) fast, Tensor(b!) slow, Tensor(c!) mixed, Tensor fast_keep, "
        "Tensor slow_keep, Tensor mix) -> ()");
  m.def("decode_pick(Tensor logits, Tensor(a!) token, Tensor(b!)? history, Tensor(c!) cursor, Tensor(d!) pos) -> ()");
  m.def("decode_attn(Tensor qkvgu, Tensor(a!) kc, Tensor(b!) vc, Tensor(c!) uc, Tensor mixed, Tensor rope, Tensor pos, "
        "int H, Tensor(d!) y, bool early=False) -> ()");
  m.def("rmsnorm_fwd(Tensor x, Tensor? col_scale, Tensor? col_bias, Tensor w, float eps, bool want_xmod) -> (Tensor, Tensor, Tensor)");
  m.def("rmsnorm_bwd(Tensor dz, Tensor x, Tensor rstd, Tensor w, Tensor? dres, Tensor? out_scale, bool want_bf16) -> (Tensor, Tensor, Tensor)");
  m.def("rmsnorm_bwd_mod(Tensor dz, Tensor? xmod, Tensor rstd, Tensor w, Tensor dres, Tensor scale, Tensor bias, "
        "Tensor? x=None) -> (Tensor, Tensor)");
  m.def("colsum2(Tensor a, Tensor b, Tensor? inv_scale) -> (Tensor, Tensor)");
  m.def("cast_bf16(Tensor x, Tensor(a!)? out) -> Tensor");
  m.def("embed_fwd(Tensor ids, Tensor table, bool out_bf16) -> Tensor");
  m.def("embed_bwd(Tensor dx, Tensor ids, Tensor(a!) grad_table) -> ()");
  m.def("launch_count() -> int");
  m.def("lm_head_fwd(Tensor hidden, Tensor weight, Tensor labels, int ignore_index, Tensor(a!)? error_flag) -> (Tensor, Tensor)");
  m.def("lm_head_fwd_labelled(Tensor hidden, Tensor weight, Tensor labels, int ignore_index, int keep_rows, "
        "Tensor(a!)? error_flag) -> Tensor[]");
  m.def("lm_head_bwd_labelled(Tensor hidden, Tensor packed, Tensor weight, Tensor labels, Tensor labels_sel, Tensor index, "
        "Tensor count, Tensor lse, Tensor row_weight, int ignore_index, int block, Tensor(a!) logits, "
        "Tensor(b!) dhidden, Tensor(c!) grad_weight, Tensor(d!)? error_flag) -> ()");
  m.def("gemm_pair_available() -> bool");
  m.def("lm_head_dlogits(Tensor hidden, Tensor weight, Tensor labels, Tensor lse, Tensor row_weight, Tensor(a!)? error_flag) -> Tensor");
  m.def("grad_allreduce(int[] grad_ptrs, int[] flag_ptrs, int mc_grad, int rank, int world, int start, int count, "
        "int bucket, int seq, float scale, bool push, int ctas, Tensor(a!)? sumsq_out, Tensor(b!) status, "
        "float budget_seconds) -> ()");
  m.def("wait_probe(Tensor flag, int expected, Tensor(a!) status, float budget_seconds) -> ()");
  m.def("adamw_shard_push(int[] master_ptrs, int[] bf16_ptrs, int rank, int world, Tensor g, Tensor(a!) m, "
        "Tensor(b!) v, int lo, int n, float lr, float beta1, float beta2, float eps, float wd, int step, "
        "Tensor? grad_scale, bool push_master, Tensor? skip=None) -> ()");
  m.def("attn_bwd(Tensor qkvgu, Tensor dy, Tensor states, Tensor writes, Tensor rope, Tensor fast_logit, "
        "Tensor slow_logit, Tensor mix_logit, int B, int T, int H, Tensor(a!)? error_flag) -> (Tensor, Tensor)");
  m.def("chunk_writes(Tensor qkvgu, Tensor rope, int B, int T, int H, Tensor(a!)? error_flag) -> Tensor");
  m.def("memory_scan(Tensor writes, Tensor fast_logit, Tensor slow_logit, Tensor mix_logit, bool want_states, "
        "bool want_final, Tensor? init_fast, Tensor? init_slow) -> (Tensor, Tensor, Tensor)");
  m.def("attn_fwd(Tensor qkvgu, Tensor? states, Tensor rope, int B, int T, int H, Tensor(a!)? error_flag) -> Tensor");
  m.def("attn_prefill(Tensor qkvgu, Tensor rope, Tensor fast_logit, Tensor slow_logit, Tensor mix_logit, int B, int T, "
        "int H, Tensor(a!) fast, Tensor(b!) slow, Tensor(c!) mixed, Tensor(d!) kc, Tensor(e!) vc, Tensor(f!) uc, "
        "Tensor(g!)? error_flag) -> Tensor");
  m.def("memory_logit_grads(Tensor partials, Tensor fast_logit, Tensor slow_logit, Tensor mix_logit, int B) -> Tensor");
  m.def("block_fwd(Tensor x, Tensor? scale, Tensor? bias, Tensor n1, Tensor w_in, Tensor w_out, Tensor n2, Tensor w_ug, "
        "Tensor w_down, Tensor fast_logit, Tensor slow_logit, Tensor mix_logit, Tensor rope, float eps, int B, int T, int H, "
        "bool keep, bool want_output, Tensor(a!)? flag) -> Tensor[]");
  m.def("block_bwd(Tensor dx3, Tensor x, Tensor rstd1, Tensor qkvgu, Tensor x2, Tensor rstd2, Tensor packed, Tensor writes, "
        "Tensor states, Tensor? scale, Tensor? bias, Tensor n1, Tensor n2, Tensor w_in, Tensor w_out, Tensor w_ug, Tensor w_down, "
        "Tensor fast_logit, Tensor slow_logit, Tensor mix_logit, Tensor rope, int B, int T, int H, Tensor(a!)? flag) -> Tensor[]");
  m.def("block(Tensor x, Tensor? scale, Tensor? bias, Tensor n1, Tensor n2, Tensor[] weights, Tensor[] bf16, Tensor(a!)[] main, "
        "Tensor fast_logit, Tensor slow_logit, Tensor mix_logit, Tensor rope, float eps, int H, Tensor(b!)? error_flag, Tensor hooked, "
        "int core, bool notify) -> Tensor");
  m.def("core_finished(int core, bool notify, Tensor[] small) -> bool");
  m.def("blocks_prefill(Tensor x, Tensor depth_scale, Tensor depth_bias, Tensor[] weights, Tensor[] vectors, Tensor(a!)[] states, Tensor rope, "
        "float eps, int B, int T, int H, Tensor(b!)? flag) -> (Tensor, Tensor)");
  m.def("grad_norm_clip(Tensor g, float max_norm, Tensor? extra_sumsq, Tensor? status=None) -> Tensor");
  m.def("clip_from_partials(Tensor partial, float max_norm, Tensor? extra_sumsq=None, Tensor? status=None) -> Tensor");
  m.def("grad_reduce_segments(int[] grad_ptrs, int[] flag_ptrs, int mc_grad, int rank, int world, int[] starts, "
        "int[] counts, int[] push, int bucket, int seq, float scale, int ctas, Tensor(a!)? sumsq_out, "
        "Tensor(b!) status, float budget_seconds) -> ()");
  m.def("norm_exchange(int[] flag_ptrs, int rank, int world, int base_word, int seq, Tensor partial, "
        "Tensor? local_loss, float max_norm, Tensor(a!) status, float budget_seconds) -> Tensor");
  m.def("node_barrier(int[] flag_ptrs, int rank, int world, int base_word, int seq, Tensor(a!) status, "
        "float budget_seconds) -> ()");
  m.def("gather_cast(int[] shard_ptrs, int rows_per_shard, Tensor(a!) wb, int ctas) -> ()");
  m.def("adamw_step(Tensor(a!) p, Tensor g, Tensor(b!) m, Tensor(c!) v, Tensor(d!)? p_bf16, float lr, float beta1, "
        "float beta2, float eps, float wd, int step, Tensor? grad_scale, float grad_scale_const, "
        "Tensor? skip=None) -> ()");
  m.def("gemm(Tensor a, Tensor b, bool a_mn, bool b_mn, int epilogue, int m, int n, int k, "
        "Tensor(a!)? out, Tensor(b!)? out2, Tensor? aux, Tensor? row_scale, float alpha, float beta, "
        "Tensor(c!)? error_flag, bool wide=False) -> ()");
  m.def("grad_weight_group(Tensor[] dys, Tensor[] xs, Tensor(a!)[] grads, float[] betas, Tensor(b!)? error_flag) -> ()");
}

TORCH_LIBRARY_IMPL(ws_b200, CompositeImplicitAutograd, m) { m.impl("block", &block); }

TORCH_LIBRARY_IMPL(ws_b200, CompositeExplicitAutograd, m) {
  m.impl("gemm_pair_available", &gemm_pair_available);
  m.impl("launch_count", &launch_count);
  m.impl("decode_gemm_splits", &decode_gemm_splits);
  m.impl("raise_for_status", &raise_for_status);
}

TORCH_LIBRARY_IMPL(ws_b200, CUDA, m) {
  m.impl("gemm", &gemm);
  m.impl("decode_gemm", &decode_gemm);
  m.impl("gather_cast_linear", &gather_cast_linear);
  m.impl("decode_reduce_norm", &decode_reduce_norm);
  m.impl("decode_norm_gemm", &decode_norm_gemm);
  m.impl("decode_attn", &decode_attn);
  m.impl("decode_chunk_end", &decode_chunk_end);
  m.impl("decode_pick", &decode_pick);
  m.impl("decode_layer_tail", &decode_layer_tail);
  m.impl("grad_weight_group", &grad_weight_group);
  m.impl("rmsnorm_fwd", &rmsnorm_fwd);
  m.impl("rmsnorm_bwd", &rmsnorm_bwd);
  m.impl("rmsnorm_bwd_mod", &rmsnorm_bwd_mod);
  m.impl("colsum2", &colsum2);
  m.impl("cast_bf16", &cast_bf16);
  m.impl("embed_fwd", &embed_fwd);
  m.impl("embed_bwd", &embed_bwd);
  m.impl("grad_norm_clip", &grad_norm_clip);
  m.impl("clip_from_partials", &clip_from_partials);
  m.impl("grad_reduce_segments", &grad_reduce_segments);
  m.impl("norm_exchange", &norm_exchange);
  m.impl("node_barrier", &node_barrier);
  m.impl("gather_cast", &gather_cast);
  m.impl("attn_bwd", &attn_bwd);
  m.impl("chunk_writes", &chunk_writes);
  m.impl("memory_scan", &memory_scan);
  m.impl("memory_logit_grads", &memory_logit_grads);
  m.impl("block_fwd", &block_fwd);
  m.impl("block_bwd", &block_bwd);
  m.impl("blocks_prefill", &blocks_prefill);
  m.impl("attn_fwd", &attn_fwd);
  m.impl("attn_prefill", &attn_prefill);
  m.impl("adamw_step", &adamw_step);
  m.impl("lm_head_fwd", &lm_head_fwd);
  m.impl("lm_head_dlogits", &lm_head_dlogits);
  m.impl("lm_head_fwd_labelled", &lm_head_fwd_labelled);
  m.impl("lm_head_bwd_labelled", &lm_head_bwd_labelled);
  m.impl("grad_allreduce", &grad_allreduce);
  m.impl("wait_probe", &wait_probe);
  m.impl("adamw_shard_push", &adamw_shard_push);
}
