// Python bindings of the native layer: tensor-checked wrappers around the C launch interface of
// the sm_100a kernels (csrc/kernels/kernels.h), the multi-GPU kernels (csrc/comm/comm.h) and the
// host runtime (csrc/runtime/runtime.h).  Nothing here allocates on the hot path except the
// per-device status word, created once.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <array>
#include <cmath>
#include <string>
#include <tuple>
#include <vector>

#include "comm/comm.h"
#include "kernels/kernels.h"
#include "runtime/runtime.h"

namespace {

int dt(const at::Tensor& t) {
  if (t.scalar_type() == at::kFloat) return kItbF32;
  if (t.scalar_type() == at::kBFloat16) return kItbBF16;
  TORCH_CHECK(false, "infinitrain_b200: unsupported dtype ", t.scalar_type());
}
cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }
void check_rc(int rc, const char* what) {
  TORCH_CHECK(rc == 0, "infinitrain_b200 kernel '", what, "' failed with code ", rc,
              rc > 0 ? std::string(" (") + cudaGetErrorString(static_cast<cudaError_t>(rc)) + ")"
                     : std::string(" (bad argument: alignment / shape / dtype)"));
}
const void* optr(const c10::optional<at::Tensor>& t) {
  return t.has_value() && t->defined() ? t->data_ptr() : nullptr;
}

// Per-device status word that kernels with bounded waits write on time-out.
at::Tensor& status_word(int device) {
  static std::vector<at::Tensor> words(64);
  if (!words[device].defined())
    words[device] = torch::zeros({4}, torch::dtype(torch::kInt32).device(torch::kCUDA, device));
  return words[device];
}

int64_t kernel_status() {
  int dev = at::cuda::current_device();
  return status_word(dev).cpu()[0].item<int64_t>();
}
void kernel_status_reset() {
  int dev = at::cuda::current_device();
  status_word(dev).zero_();
}

// ------------------------------------------------------------------ GEMM
// Kernel choice: 0 = one CTA per 128 x 256 tile, 1 = CTA pairs on 256 x 256 tiles.  An output whose 128 x 64 tiles
// run all at once (itb_gemm_is_small) is computed by those in either mode.
int g_gemm_mode = 1;
void set_gemm_mode(int64_t mode) { g_gemm_mode = static_cast<int>(mode); }
int64_t get_gemm_mode() { return g_gemm_mode; }
// bit 0: attention backward on tcgen05, bit 1: attention forward on tcgen05 (flash_attn_tc.cu);
// a cleared bit selects the mma.sync kernel of flash_attn.cu for that pass.
int g_attn_mode = 3;
void set_attn_mode(int64_t mode) { g_attn_mode = static_cast<int>(mode); }
int64_t get_attn_mode() { return g_attn_mode; }

// C[M,N] = A . B^T-like product; see kernels.h for the layout flags.
void gemm(const at::Tensor& a, bool a_mn, const at::Tensor& b, bool b_mn, int64_t M, int64_t N,
          int64_t K, at::Tensor& c, const c10::optional<at::Tensor>& c2,
          const c10::optional<at::Tensor>& bias, const c10::optional<at::Tensor>& residual,
          const c10::optional<at::Tensor>& aux, int64_t flags, int64_t split_k) {
  TORCH_CHECK(a.is_cuda() && b.is_cuda() && c.is_cuda(), "gemm: CUDA tensors required");
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16,
              "gemm: bf16 operands required");
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && c.dim() == 2, "gemm: 2-D tensors required");
  TORCH_CHECK(a.stride(1) == 1 && b.stride(1) == 1 && c.stride(1) == 1,
              "gemm: innermost dimension must be contiguous");
  c10::cuda::CUDAGuard guard(a.device());
  ItbGemmArgs g{};
  g.M = static_cast<int>(M);
  g.N = static_cast<int>(N);
  g.K = static_cast<int>(K);
  g.A = a.data_ptr();
  g.lda = a.stride(0);
  g.a_mn_major = a_mn;
  g.B = b.data_ptr();
  g.ldb = b.stride(0);
  g.b_mn_major = b_mn;
  TORCH_CHECK(a_mn ? (a.size(0) == K && a.size(1) == M) : (a.size(0) == M && a.size(1) == K),
              "gemm: A shape mismatch");
  TORCH_CHECK(b_mn ? (b.size(0) == K && b.size(1) == N) : (b.size(0) == N && b.size(1) == K),
              "gemm: B shape mismatch");
  TORCH_CHECK(c.size(0) == M && c.size(1) >= N, "gemm: C shape mismatch");
  const bool f32 = flags & kGemmOutF32;
  TORCH_CHECK(c.scalar_type() == (f32 ? at::kFloat : at::kBFloat16), "gemm: C dtype mismatch");
  g.C = c.data_ptr();
  g.ldc = c.stride(0);
  if (flags & kGemmGeluDual) {
    TORCH_CHECK(c2.has_value() && c2->scalar_type() == at::kBFloat16 &&
                    c2->stride(0) == c.stride(0) && !f32,
                "gemm: gelu dual output needs a bf16 C2 with C's layout");
    g.C2 = c2->data_ptr();
  }
  if (flags & kGemmBias) {
    TORCH_CHECK(bias.has_value() && bias->scalar_type() == at::kFloat && bias->numel() >= N,
                "gemm: fp32 bias of length N required");
    g.bias = static_cast<const float*>(bias->data_ptr());
  }
  if (flags & kGemmResidual) {
    TORCH_CHECK(residual.has_value() && residual->scalar_type() == c.scalar_type() &&
                    residual->stride(1) == 1,
                "gemm: residual must have C's dtype");
    g.residual = residual->data_ptr();
    g.ldr = residual->stride(0);
  }
  if (flags & kGemmDGelu) {
    TORCH_CHECK(aux.has_value() && aux->scalar_type() == at::kBFloat16 && aux->stride(1) == 1,
                "gemm: bf16 aux required");
    g.aux = aux->data_ptr();
    g.ld_aux = aux->stride(0);
  }
  g.flags = static_cast<int>(flags);
  g.split_k = static_cast<int>(split_k);
  g.err = status_word(a.get_device()).data_ptr<int>();
  if (g_gemm_mode == 1 && M > 128)
    check_rc(itb_gemm_bf16_pair(&g, cur_stream()), "gemm_bf16_tcgen05_pair");
  else
    check_rc(itb_gemm_bf16(&g, cur_stream()), "gemm_bf16_tcgen05");
}

// ------------------------------------------------------------------ norms
// `statistics`: what the backward pass needs; without it mean and rstd are undefined.
std::vector<at::Tensor> layernorm_fwd(const at::Tensor& x, const at::Tensor& gamma,
                                      const c10::optional<at::Tensor>& beta, double eps,
                                      at::ScalarType out_dtype, bool statistics) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous(), "layernorm: contiguous input required");
  const int C = x.size(-1);
  const int rows = x.numel() / C;
  auto y = torch::empty_like(x, x.options().dtype(out_dtype));
  at::Tensor mean, rstd;
  if (statistics) {
    mean = torch::empty({rows}, x.options().dtype(at::kFloat));
    rstd = torch::empty({rows}, x.options().dtype(at::kFloat));
  }
  check_rc(itb_layernorm_fwd(x.data_ptr(), dt(x), gamma.data_ptr<float>(),
                             static_cast<const float*>(optr(beta)), y.data_ptr(), dt(y),
                             statistics ? mean.data_ptr<float>() : nullptr,
                             statistics ? rstd.data_ptr<float>() : nullptr, rows, C,
                             static_cast<float>(eps), cur_stream()),
           "layernorm_fwd");
  return {y, mean, rstd};
}
// dres (optional): gradient of the residual stream past the norm, added to dx in the same pass;
// dgamma_out / dbeta_out / dres_sum_out (optional fp32 [C]): gradients are ACCUMULATED into these
// tensors (views of a flat gradient buffer) instead of being returned; want_dres_sum without an
// output tensor returns the column sums of dres as a fresh tensor.
std::vector<at::Tensor> layernorm_bwd(const at::Tensor& dy, const at::Tensor& x,
                                      const at::Tensor& gamma, const at::Tensor& mean,
                                      const at::Tensor& rstd, bool has_beta,
                                      const c10::optional<at::Tensor>& dres,
                                      const c10::optional<at::Tensor>& dgamma_out,
                                      const c10::optional<at::Tensor>& dbeta_out,
                                      const c10::optional<at::Tensor>& dres_sum_out, bool want_dres_sum) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous() && dy.is_contiguous(), "layernorm_bwd: contiguous tensors required");
  const int C = x.size(-1);
  const int rows = x.numel() / C;
  auto dx = torch::empty_like(x);
  if (dres) TORCH_CHECK(dres->is_contiguous() && dres->scalar_type() == dx.scalar_type() && dres->numel() == x.numel(),
                        "layernorm_bwd: dres must match dx");
  int acc = 0;
  auto f32 = x.options().dtype(at::kFloat);
  at::Tensor dgamma = dgamma_out ? *dgamma_out : torch::empty({C}, f32);
  at::Tensor dbeta = dbeta_out ? *dbeta_out : torch::empty({C}, f32);
  at::Tensor dsum;
  if (dres && (dres_sum_out || want_dres_sum)) dsum = dres_sum_out ? *dres_sum_out : torch::empty({C}, f32);
  if (dgamma_out) acc |= 1;
  if (dbeta_out) acc |= 2;
  if (dres_sum_out) acc |= 4;
  for (const at::Tensor* t : {&dgamma, &dbeta})
    TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == C, "layernorm_bwd: fp32 [C] outputs");
  auto partial = torch::empty({itb_norm_partial_rows(rows), 3 * C}, f32);
  check_rc(itb_layernorm_bwd_res(dy.data_ptr(), dt(dy), x.data_ptr(), dt(x), gamma.data_ptr<float>(),
                                 mean.data_ptr<float>(), rstd.data_ptr<float>(), dres ? dres->data_ptr() : nullptr,
                                 dx.data_ptr(), dt(dx), dgamma.data_ptr<float>(), dbeta.data_ptr<float>(),
                                 dsum.defined() ? dsum.data_ptr<float>() : nullptr, partial.data_ptr<float>(), rows, C,
                                 acc, cur_stream()),
           "layernorm_bwd");
  return {dx, dgamma, dbeta, dsum};
}
std::vector<at::Tensor> rmsnorm_fwd(const at::Tensor& x, const at::Tensor& gamma, double eps,
                                    at::ScalarType out_dtype, bool statistics) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous(), "rmsnorm: contiguous input required");
  const int C = x.size(-1);
  const int rows = x.numel() / C;
  auto y = torch::empty_like(x, x.options().dtype(out_dtype));
  at::Tensor rstd;
  if (statistics) rstd = torch::empty({rows}, x.options().dtype(at::kFloat));
  check_rc(itb_rmsnorm_fwd(x.data_ptr(), dt(x), gamma.data_ptr<float>(), y.data_ptr(), dt(y),
                           statistics ? rstd.data_ptr<float>() : nullptr, rows, C, static_cast<float>(eps), cur_stream()),
           "rmsnorm_fwd");
  return {y, rstd};
}
std::vector<at::Tensor> rmsnorm_bwd(const at::Tensor& dy, const at::Tensor& x,
                                    const at::Tensor& gamma, const at::Tensor& rstd,
                                    const c10::optional<at::Tensor>& dres,
                                    const c10::optional<at::Tensor>& dgamma_out,
                                    const c10::optional<at::Tensor>& dres_sum_out, bool want_dres_sum) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous() && dy.is_contiguous(), "rmsnorm_bwd: contiguous tensors required");
  const int C = x.size(-1);
  const int rows = x.numel() / C;
  auto dx = torch::empty_like(x);
  if (dres) TORCH_CHECK(dres->is_contiguous() && dres->scalar_type() == dx.scalar_type() && dres->numel() == x.numel(),
                        "rmsnorm_bwd: dres must match dx");
  auto f32 = x.options().dtype(at::kFloat);
  at::Tensor dgamma = dgamma_out ? *dgamma_out : torch::empty({C}, f32);
  TORCH_CHECK(dgamma.scalar_type() == at::kFloat && dgamma.is_contiguous() && dgamma.numel() == C, "rmsnorm_bwd: fp32 [C] output");
  at::Tensor dsum;
  if (dres && (dres_sum_out || want_dres_sum)) dsum = dres_sum_out ? *dres_sum_out : torch::empty({C}, f32);
  const int acc = (dgamma_out ? 1 : 0) | (dres_sum_out ? 4 : 0);
  auto partial = torch::empty({itb_norm_partial_rows(rows), 3 * C}, f32);
  check_rc(itb_rmsnorm_bwd_res(dy.data_ptr(), dt(dy), x.data_ptr(), dt(x), gamma.data_ptr<float>(),
                               rstd.data_ptr<float>(), dres ? dres->data_ptr() : nullptr, dx.data_ptr(), dt(dx),
                               dgamma.data_ptr<float>(), dsum.defined() ? dsum.data_ptr<float>() : nullptr,
                               partial.data_ptr<float>(), rows, C, acc, cur_stream()),
           "rmsnorm_bwd");
  return {dx, dgamma, dsum};
}

// ------------------------------------------------------------------ activations
at::Tensor gelu_fwd(const at::Tensor& x) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous(), "gelu: contiguous input required");
  auto y = torch::empty_like(x);
  check_rc(itb_gelu_fwd(x.data_ptr(), y.data_ptr(), dt(x), x.numel(), cur_stream()), "gelu_fwd");
  return y;
}
at::Tensor gelu_bwd(const at::Tensor& dy, const at::Tensor& x) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous() && dy.is_contiguous() && dy.scalar_type() == x.scalar_type(),
              "gelu_bwd: contiguous tensors of one dtype required");
  auto dx = torch::empty_like(x);
  check_rc(itb_gelu_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dt(x), x.numel(), cur_stream()),
           "gelu_bwd");
  return dx;
}
// a, b: [rows, F] views (row stride ld, unit column stride) -> out [rows, F] contiguous
at::Tensor swiglu_fwd(const at::Tensor& a, const at::Tensor& b) {
  c10::cuda::CUDAGuard guard(a.device());
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1 &&
                  a.stride(0) == b.stride(0) && a.scalar_type() == b.scalar_type(),
              "swiglu: 2-D views with equal row strides required");
  auto out = torch::empty({a.size(0), a.size(1)}, a.options());
  check_rc(itb_swiglu_fwd(a.data_ptr(), b.data_ptr(), a.stride(0), out.data_ptr(), out.stride(0),
                          dt(a), a.size(0), a.size(1), cur_stream()),
           "swiglu_fwd");
  return out;
}
// Returns dab [rows, 2F]: columns [0,F) = da, [F,2F) = db.
at::Tensor swiglu_bwd(const at::Tensor& dout, const at::Tensor& a, const at::Tensor& b) {
  c10::cuda::CUDAGuard guard(a.device());
  TORCH_CHECK(dout.dim() == 2 && dout.stride(1) == 1 && a.stride(1) == 1 && b.stride(1) == 1 &&
                  a.stride(0) == b.stride(0),
              "swiglu_bwd: bad layout");
  const int64_t F = a.size(1);
  auto dab = torch::empty({a.size(0), 2 * F}, a.options());
  check_rc(itb_swiglu_bwd(dout.data_ptr(), dout.stride(0), a.data_ptr(), b.data_ptr(), a.stride(0),
                          dab.data_ptr(), static_cast<char*>(dab.data_ptr()) + F * dab.element_size(),
                          dab.stride(0), dt(a), a.size(0), F, cur_stream()),
           "swiglu_bwd");
  return dab;
}

// ------------------------------------------------------------------ rope
void rope_inplace(at::Tensor& qkv, const at::Tensor& freqs, int64_t B, int64_t T, int64_t n_heads,
                  int64_t D, int64_t row_stride, int64_t pos0, bool inverse) {
  c10::cuda::CUDAGuard guard(qkv.device());
  TORCH_CHECK(freqs.scalar_type() == at::kFloat && freqs.is_contiguous(), "rope: fp32 table");
  TORCH_CHECK(freqs.size(0) >= pos0 + T, "rope: table too short");
  check_rc(itb_rope_inplace(qkv.data_ptr(), dt(qkv), freqs.data_ptr<float>(), B, T, n_heads, D,
                            row_stride, pos0, inverse, cur_stream()),
           "rope");
}

// ------------------------------------------------------------------ embedding
at::Tensor embedding_fwd(const at::Tensor& idx, const at::Tensor& wte,
                         const c10::optional<at::Tensor>& wpe, int64_t pos0, int64_t vocab_start,
                         at::ScalarType out_dtype) {
  c10::cuda::CUDAGuard guard(wte.device());
  TORCH_CHECK(idx.scalar_type() == at::kLong && idx.is_contiguous() && idx.dim() == 2,
              "embedding: int64 [B,T] indices");
  const int B = idx.size(0), T = idx.size(1), C = wte.size(1);
  auto out = torch::empty({B, T, C}, wte.options().dtype(out_dtype));
  check_rc(itb_embedding_fwd(idx.data_ptr<int64_t>() ? reinterpret_cast<const long long*>(idx.data_ptr<int64_t>()) : nullptr,
                             wte.data_ptr(), optr(wpe), dt(wte), out.data_ptr(), dt(out), B, T, C,
                             pos0, vocab_start, vocab_start + wte.size(0), cur_stream()),
           "embedding_fwd");
  return out;
}
void embedding_bwd(const at::Tensor& idx, const at::Tensor& dout,
                   const c10::optional<at::Tensor>& dwte, const c10::optional<at::Tensor>& dwpe,
                   int64_t pos0, int64_t vocab_start) {
  c10::cuda::CUDAGuard guard(dout.device());
  TORCH_CHECK(dout.is_contiguous() && dout.dim() == 3, "embedding_bwd: contiguous [B,T,C]");
  auto aligned = [](const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; };
  TORCH_CHECK(aligned(dout), "embedding_bwd: a gradient on a 16-byte boundary");
  for (const auto* table : {&dwte, &dwpe})
    TORCH_CHECK(!table->has_value() || ((*table)->is_cuda() && (*table)->scalar_type() == at::kFloat && (*table)->dim() >= 2 &&
                                        (*table)->size(-1) == dout.size(2) && (*table)->is_contiguous() && aligned(**table)),
                "embedding_bwd: contiguous fp32 tables as wide as the gradient, on a 16-byte boundary");
  const int B = dout.size(0), T = dout.size(1), C = dout.size(2);
  int64_t vend = vocab_start + (dwte.has_value() ? dwte->size(0) : 0);
  check_rc(itb_embedding_bwd(reinterpret_cast<const long long*>(idx.data_ptr<int64_t>()),
                             dout.data_ptr(), dt(dout),
                             dwte.has_value() ? dwte->data_ptr<float>() : nullptr,
                             dwpe.has_value() ? dwpe->data_ptr<float>() : nullptr, B, T, C, pos0,
                             vocab_start, vend, cur_stream()),
           "embedding_bwd");
}

// ------------------------------------------------------------------ cross entropy
// logits [rows, ld] (first V columns valid).  Returns {loss_mean[1], lse[rows], row_loss[rows]}.
std::vector<at::Tensor> ce_fwd(const at::Tensor& logits, const at::Tensor& target, int64_t V) {
  c10::cuda::CUDAGuard guard(logits.device());
  TORCH_CHECK(logits.dim() == 2 && logits.stride(1) == 1, "ce: 2-D logits");
  TORCH_CHECK(target.scalar_type() == at::kLong && target.is_contiguous(), "ce: int64 targets");
  const int rows = logits.size(0);
  auto f32 = logits.options().dtype(at::kFloat);
  auto loss = torch::zeros({1}, f32);
  auto lse = torch::empty({rows}, f32);
  auto row_loss = torch::empty({rows}, f32);
  check_rc(itb_ce_fwd(logits.data_ptr(), dt(logits), logits.stride(0),
                      reinterpret_cast<const long long*>(target.data_ptr<int64_t>()),
                      row_loss.data_ptr<float>(), lse.data_ptr<float>(), loss.data_ptr<float>(),
                      rows, V, cur_stream()),
           "ce_fwd");
  return {loss, lse, row_loss};
}
void ce_bwd(at::Tensor& logits, const at::Tensor& target, const at::Tensor& lse,
            const at::Tensor& grad_out, int64_t V, bool ignore_oob) {
  c10::cuda::CUDAGuard guard(logits.device());
  TORCH_CHECK(grad_out.scalar_type() == at::kFloat && grad_out.numel() == 1, "ce_bwd: fp32 scalar");
  check_rc(itb_ce_bwd(logits.data_ptr(), dt(logits), logits.stride(0),
                      reinterpret_cast<const long long*>(target.data_ptr<int64_t>()),
                      lse.data_ptr<float>(), grad_out.data_ptr<float>(), logits.size(0), V,
                      ignore_oob, cur_stream()),
           "ce_bwd");
}

// ------------------------------------------------------------------ optimizer
void adamw(at::Tensor& p, const at::Tensor& g, at::Tensor& m, at::Tensor& v,
           const c10::optional<at::Tensor>& shadow, double lr, double b1, double b2, double eps,
           double wd, double bc1, double bc2, double grad_scale,
           const c10::optional<at::Tensor>& dev_hyper) {
  c10::cuda::CUDAGuard guard(p.device());
  TORCH_CHECK(!dev_hyper.has_value() || (dev_hyper->scalar_type() == at::kFloat && dev_hyper->numel() >= 3 &&
                                         dev_hyper->is_cuda()),
              "adamw: dev_hyper must be a CUDA fp32 tensor [lr, 1/bc1, 1/bc2]");
  TORCH_CHECK(p.is_contiguous() && g.is_contiguous() && m.is_contiguous() && v.is_contiguous(),
              "adamw: contiguous flat buffers required");
  TORCH_CHECK(p.scalar_type() == at::kFloat && m.scalar_type() == at::kFloat &&
                  v.scalar_type() == at::kFloat,
              "adamw: fp32 master weights and state required");
  TORCH_CHECK(g.numel() == p.numel() && m.numel() == p.numel() && v.numel() == p.numel(),
              "adamw: size mismatch");
  check_rc(itb_adamw(p.data_ptr<float>(), g.data_ptr(), dt(g), m.data_ptr<float>(),
                     v.data_ptr<float>(), const_cast<void*>(optr(shadow)), p.numel(), lr, b1, b2,
                     eps, wd, bc1, bc2, grad_scale, static_cast<const float*>(optr(dev_hyper)),
                     cur_stream()),
           "adamw");
}
void adam_advance(at::Tensor& hyper, double b1, double b2) {
  c10::cuda::CUDAGuard guard(hyper.device());
  TORCH_CHECK(hyper.is_cuda() && hyper.scalar_type() == at::kFloat && hyper.numel() >= 4, "adam_advance: fp32[4]");
  check_rc(itb_adam_advance(hyper.data_ptr<float>(), b1, b2, cur_stream()), "adam_advance");
}
void sgd(at::Tensor& p, const at::Tensor& g, const c10::optional<at::Tensor>& shadow, double lr,
         double grad_scale) {
  c10::cuda::CUDAGuard guard(p.device());
  TORCH_CHECK(p.is_contiguous() && g.is_contiguous() && p.scalar_type() == at::kFloat,
              "sgd: contiguous fp32 weights required");
  check_rc(itb_sgd(p.data_ptr<float>(), g.data_ptr(), dt(g), const_cast<void*>(optr(shadow)),
                   p.numel(), lr, grad_scale, cur_stream()),
           "sgd");
}

// ------------------------------------------------------------------ utilities
void cast_into(const at::Tensor& src, at::Tensor& dst) {
  c10::cuda::CUDAGuard guard(src.device());
  TORCH_CHECK(src.is_contiguous() && dst.is_contiguous() && src.numel() == dst.numel(),
              "cast: contiguous tensors of equal size required");
  check_rc(itb_cast(src.data_ptr(), dt(src), dst.data_ptr(), dt(dst), src.numel(), cur_stream()),
           "cast");
}
// Column sums of a [rows, N] matrix; with `into` (fp32 [N]) the sums are ADDED to that tensor (a view
// of a flat gradient buffer) and it is returned.
at::Tensor colsum(const at::Tensor& x, const c10::optional<at::Tensor>& into) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 2 && x.stride(1) == 1, "colsum: 2-D row-major input");
  const int rows = x.size(0), N = x.size(1);
  at::Tensor out = into ? *into : torch::empty({N}, x.options().dtype(at::kFloat));
  TORCH_CHECK(out.scalar_type() == at::kFloat && out.is_contiguous() && out.numel() == N, "colsum: fp32 [N] output");
  auto partial = torch::empty({itb_colsum_partial_rows(rows), N}, x.options().dtype(at::kFloat));
  check_rc(itb_colsum(x.data_ptr(), dt(x), x.stride(0), out.data_ptr<float>(),
                      partial.data_ptr<float>(), rows, N, into ? 1 : 0, cur_stream()),
           "colsum");
  return out;
}

// ------------------------------------------------------------------ attention
// q [B,T,H,D], k/v [B,T,KV,D] (views with unit stride on D, head stride D) -> {o [B,T,H,D], lse}
ItbAttnArgs attn_args(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, double scale,
                      bool causal) {
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "attention: [B,T,H,D] tensors");
  TORCH_CHECK(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 &&
                  v.scalar_type() == at::kBFloat16,
              "attention: bf16 required");
  const int64_t D = q.size(3);
  TORCH_CHECK(q.stride(3) == 1 && k.stride(3) == 1 && v.stride(3) == 1 && q.stride(2) == D &&
                  k.stride(2) == D && v.stride(2) == D,
              "attention: heads must be packed along the last two dimensions");
  ItbAttnArgs a{};
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.q_row_stride = q.stride(1);
  a.k_row_stride = k.stride(1);
  a.v_row_stride = v.stride(1);
  a.q_batch_stride = q.stride(0);
  a.k_batch_stride = k.stride(0);
  a.v_batch_stride = v.stride(0);
  a.B = q.size(0);
  a.T = q.size(1);
  a.H = q.size(2);
  a.KV = k.size(2);
  a.D = D;
  a.scale = static_cast<float>(scale);
  a.causal = causal;
  return a;
}
std::vector<at::Tensor> flash_attn_fwd(const at::Tensor& q, const at::Tensor& k,
                                       const at::Tensor& v, double scale, bool causal) {
  c10::cuda::CUDAGuard guard(q.device());
  ItbAttnArgs a = attn_args(q, k, v, scale, causal);
  auto o = torch::empty({a.B, a.T, a.H, a.D}, q.options());
  auto lse = torch::empty({a.B, a.H, a.T}, q.options().dtype(at::kFloat));
  a.o = o.data_ptr();
  a.o_row_stride = o.stride(1);
  a.o_batch_stride = o.stride(0);
  a.lse = lse.data_ptr<float>();
  if (g_attn_mode & 2)
    check_rc(itb_flash_attn_fwd_tc(&a, status_word(q.get_device()).data_ptr<int>(), cur_stream()),
             "flash_attn_fwd_tc");
  else
    check_rc(itb_flash_attn_fwd(&a, cur_stream()), "flash_attn_fwd");
  return {o, lse};
}
// dq/dk/dv are written into caller-provided views (e.g. column blocks of one packed dqkv buffer).
void flash_attn_bwd(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                    const at::Tensor& v, const at::Tensor& o, const at::Tensor& lse, at::Tensor& dq,
                    at::Tensor& dk, at::Tensor& dv, double scale, bool causal) {
  c10::cuda::CUDAGuard guard(q.device());
  ItbAttnArgs a = attn_args(q, k, v, scale, causal);
  TORCH_CHECK(o.is_contiguous() && dout.is_contiguous(), "attention bwd: contiguous o and dout");
  TORCH_CHECK(dq.strides() == q.strides() && dk.strides() == k.strides() &&
                  dv.strides() == v.strides(),
              "attention bwd: gradient views must share the strides of q/k/v");
  a.o = o.data_ptr();
  a.o_row_stride = o.stride(1);
  a.o_batch_stride = o.stride(0);
  a.lse = lse.data_ptr<float>();
  a.dout = dout.data_ptr();
  a.dq = dq.data_ptr();
  a.dk = dk.data_ptr();
  a.dv = dv.data_ptr();
  auto f32 = q.options().dtype(at::kFloat);
  auto delta = torch::empty({a.B, a.H, a.T}, f32);
  auto dq_accum = torch::empty({a.B, a.T, a.H, a.D}, f32);
  a.delta = delta.data_ptr<float>();
  a.dq_accum = dq_accum.data_ptr<float>();
  at::Tensor dkv_accum;
  const int parts = (g_attn_mode & 1) ? itb_flash_attn_bwd_parts(a.B, a.T, a.H, a.KV, a.causal) : 1;
  if (parts > 1) {
    dkv_accum = torch::empty({parts, 2, a.B, a.T, a.KV, a.D}, f32);
    a.dkv_accum = dkv_accum.data_ptr<float>();
  }
  if (g_attn_mode & 1)
    check_rc(itb_flash_attn_bwd_tc(&a, status_word(q.get_device()).data_ptr<int>(), cur_stream()),
             "flash_attn_bwd_tc");
  else
    check_rc(itb_flash_attn_bwd(&a, cur_stream()), "flash_attn_bwd");
}

// ------------------------------------------------------------------ whole passes of an op in one call
// What an op's forward or backward does around its launches (shapes, strides, allocations) costs the host as much as the
// launches themselves when each step is a call from Python: 87 ops on 1 x 96 tokens of GPT-2 124M took 2.3 ms of host time.
using OptTensor = c10::optional<at::Tensor>;

// Whether the rows of a matrix are one row expanded (the gradient of a sum over rows): a tensor map needs a pitch.
bool one_row(const at::Tensor& x) { return x.size(0) > 1 && x.stride(0) == 0; }

// `x` as a bf16 matrix whose rows TMA can read: unit column stride, rows and base on 16 bytes.
at::Tensor bf16_rows(const at::Tensor& x) {
  at::Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  if (x2.scalar_type() != at::kBFloat16) x2 = x2.to(at::kBFloat16);
  if (x2.stride(1) != 1 || one_row(x2) || (x2.stride(0) % 8) || (reinterpret_cast<uintptr_t>(x2.data_ptr()) % 16))
    x2 = x2.contiguous();
  if (x2.stride(0) % 8) {        // the gradient of a rank-4 product's rows are not a multiple of 16 bytes apart
    const int64_t cols = x2.size(1);
    at::Tensor padded = at::empty({x2.size(0), (cols + 7) / 8 * 8}, x2.options());
    at::Tensor view = padded.narrow(1, 0, cols);
    view.copy_(x2);
    x2 = view;
  }
  return x2;
}

// The leading dimensions of `x` with `last` in the place of its last one.
std::vector<int64_t> sizes_with_last(const at::Tensor& x, int64_t last) {
  std::vector<int64_t> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = last;
  return sizes;
}

// A fresh output of `rows` x N, shaped like `x` but for its last dimension; its rows are `ld` elements apart.
at::Tensor output_like(const at::Tensor& x, int64_t rows, int64_t N, int64_t ld, at::ScalarType dtype, void** data) {
  if (ld == N) {
    at::Tensor y = at::empty(sizes_with_last(x, N), x.options().dtype(dtype));
    *data = y.data_ptr();
    return y;
  }
  at::Tensor out = at::empty({rows, ld}, x.options().dtype(dtype));
  *data = out.data_ptr();
  return out.narrow(1, 0, N).view(sizes_with_last(x, N));
}

struct Gemm : ItbGemmArgs {
  at::Tensor kept;        // a copy that the launch reads
  Gemm(const at::Tensor& a, bool a_mn, const at::Tensor& b, bool b_mn, int64_t m, int64_t n, int64_t k) : ItbGemmArgs{} {
    TORCH_CHECK(a.is_cuda() && b.is_cuda() && a.device() == b.device(), "gemm: operands on one CUDA device required");
    TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "gemm: bf16 operands required");
    TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1,
                "gemm: matrices with a contiguous innermost dimension required");
    TORCH_CHECK(a_mn ? (a.size(0) == k && a.size(1) == m) : (a.size(0) == m && a.size(1) == k), "gemm: A shape mismatch");
    TORCH_CHECK(b_mn ? (b.size(0) == k && b.size(1) == n) : (b.size(0) == n && b.size(1) == k), "gemm: B shape mismatch");
    M = static_cast<int>(m), N = static_cast<int>(n), K = static_cast<int>(k);
    A = a.data_ptr(), lda = a.stride(0), a_mn_major = a_mn;
    B = b.data_ptr(), ldb = b.stride(0), b_mn_major = b_mn;
    err = status_word(a.get_device()).data_ptr<int>();
  }
  Gemm& into(void* c, int64_t ld, int more_flags = 0) {
    C = c, ldc = ld, flags |= more_flags;
    return *this;
  }
  Gemm& add_bias(const OptTensor& b) {
    if (b && b->defined()) {
      TORCH_CHECK(b->is_cuda() && b->scalar_type() == at::kFloat && b->numel() >= N, "gemm: fp32 bias of length N required");
      kept = b->contiguous();
      bias = kept.data_ptr<float>();
      flags |= kGemmBias;
    }
    return *this;
  }
  void run() {
    if (g_gemm_mode == 1 && M > 128)
      check_rc(itb_gemm_bf16_pair(this, cur_stream()), "gemm_bf16_tcgen05_pair");
    else
      check_rc(itb_gemm_bf16(this, cur_stream()), "gemm_bf16_tcgen05");
  }
};

// Adds a residual to a GEMM's output (`keep` holds the matrix that the launch reads).
void add_residual(Gemm& g, const OptTensor& residual, bool out_f32, at::Tensor* keep) {
  if (!residual || !residual->defined()) return;
  TORCH_CHECK(residual->scalar_type() == (out_f32 ? at::kFloat : at::kBFloat16), "gemm: residual must have C's dtype");
  *keep = residual->reshape({g.M, g.N});
  if (keep->stride(1) != 1 || one_row(*keep)) *keep = keep->contiguous();
  g.residual = keep->data_ptr();
  g.ldr = keep->stride(0);
  g.flags |= kGemmResidual;
}

// Whether a kernel may add the gradient of the leaf `p` to `slot` in autograd's place: `slot` is its whole .grad, in fp32 and
// on the boundary that the kernels' vector accesses need, and no hook of the leaf or of its accumulator waits for the sum.
bool adds_in_place(const at::Tensor& p, const at::Tensor& slot) {
  const at::Tensor& grad = p.grad();
  if (!grad.defined() || grad.data_ptr() != slot.data_ptr() || slot.scalar_type() != at::kFloat ||
      grad.scalar_type() != at::kFloat || slot.sizes() != p.sizes() || grad.sizes() != p.sizes() || !slot.is_contiguous() ||
      !grad.is_contiguous() || reinterpret_cast<uintptr_t>(slot.data_ptr()) % 16)
    return false;
  const auto node = torch::autograd::impl::try_get_grad_accumulator(p);
  return !node || (node->tensor_pre_hooks().empty() && node->pre_hooks().empty() && node->post_hooks().empty() &&
                   !node->tensor_post_acc_grad_hooks());
}

bool is_f32(const OptTensor& t) { return t && t->defined() && t->scalar_type() == at::kFloat; }

// y = x w^T (+ bias) (+ residual) or gelu(x w^T + bias): {y, x as a matrix, pre-activation (rows padded to 64 elements)}
std::tuple<at::Tensor, at::Tensor, OptTensor> linear_fwd(const at::Tensor& x, const at::Tensor& w, const OptTensor& bias,
                                                         const OptTensor& residual, bool gelu) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t K = x.size(-1), N = w.size(0), ld = (N + 63) / 64 * 64;
  at::Tensor x2 = bf16_rows(x), kept;
  const int64_t M = x2.size(0);
  const bool f32 = is_f32(residual);
  Gemm g(x2, false, w, false, M, N, K);
  void* data;
  at::Tensor y = output_like(x, M, N, ld, f32 ? at::kFloat : at::kBFloat16, &data);
  OptTensor pre;
  g.add_bias(bias);
  if (gelu) {
    pre = at::empty({M, ld}, x2.options());
    g.into(pre->data_ptr(), ld, kGemmGeluDual);
    g.C2 = data;
  } else {
    g.into(data, ld, f32 ? kGemmOutF32 : 0);
    add_residual(g, residual, f32, &kept);
  }
  g.run();
  return {y, x2, pre};
}

// Called as soon as the kernel that adds a gradient to its slot has been launched, ahead of the pass's other launches, so
// that a reduction of the bucket the gradient completes starts under them; nothing when it is None.
using Ready = pybind11::object;
void call(const Ready& ready) {
  if (!ready.is_none()) ready();
}

// dW [N, K] = dy^T x in fp32, added to `main` (a slot of a flat gradient buffer) or as a fresh tensor.
OptTensor weight_grad(const at::Tensor& dy2, const at::Tensor& x2, const OptTensor& main, const Ready& ready) {
  const int64_t N = dy2.size(1), K = x2.size(1), M = x2.size(0);
  OptTensor dw;
  if (!main) dw = at::empty({N, K}, dy2.options().dtype(at::kFloat));
  const at::Tensor& out = main ? *main : *dw;
  TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kFloat && out.dim() == 2 && out.size(0) == N && out.size(1) >= K &&
                  out.stride(1) == 1,
              "linear: the weight's gradient slot must be an fp32 [N, K] matrix");
  Gemm g(dy2, true, x2, true, N, K, M);
  g.into(out.data_ptr(), out.stride(0), kGemmOutF32 | kGemmAtomic | (main ? 0 : kGemmFresh)).run();
  if (main) call(ready);
  return dw;
}

// Column sums of dy, added to `main` or as a fresh tensor.  Matrices that the kernel cannot read are summed by torch, and
// then not into `main`.
OptTensor bias_grad(const at::Tensor& dy2, const OptTensor& main, const Ready& ready) {
  if (dy2.size(1) % 8 == 0 && reinterpret_cast<uintptr_t>(dy2.data_ptr()) % 16 == 0) {
    at::Tensor out = colsum(dy2, main);
    if (!main) return out;
    call(ready);
    return {};
  }
  return dy2.to(at::kFloat).sum(0);
}

// {dx, dw, db} of linear_fwd; what was added to a slot comes back as None.  `pre` (rows of any pitch) when the output went
// through GELU, `w` when dx is wanted.
std::tuple<OptTensor, OptTensor, OptTensor> linear_bwd(const at::Tensor& dy, const at::Tensor& x2, const OptTensor& w,
                                                       const OptTensor& pre, bool want_dw, const OptTensor& main_dw,
                                                       const Ready& dw_ready, bool want_db, const OptTensor& main_db,
                                                       const Ready& db_ready) {
  c10::cuda::CUDAGuard guard(dy.device());
  at::Tensor dy2 = bf16_rows(dy);
  const int64_t M = x2.size(0), N = dy2.size(1), K = x2.size(1);
  if (pre) dy2 = bf16_rows(gelu_bwd(dy2.contiguous(), pre->narrow(1, 0, N).contiguous()));
  OptTensor dx, dw, db;
  if (w) {
    dx = at::empty(sizes_with_last(dy, K), dy2.options());
    Gemm(dy2, false, *w, true, M, K, N).into(dx->data_ptr(), K, kGemmMaySplit).run();
  }
  if (want_dw) dw = weight_grad(dy2, x2, main_dw, dw_ready);
  if (want_db) db = bias_grad(dy2, main_db, db_ready);
  return {dx, dw, db};
}

// residual + gelu(x w_fc^T + b_fc) w_proj^T + b_proj: {y, x as a matrix, pre-activation, activation}
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> mlp_gelu_fwd(const at::Tensor& x, const at::Tensor& w_fc,
                                                                        const OptTensor& b_fc, const at::Tensor& w_proj,
                                                                        const OptTensor& b_proj, const OptTensor& residual) {
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor x2 = bf16_rows(x), kept;
  const int64_t M = x2.size(0), C = x2.size(1), F = w_fc.size(0);
  at::Tensor h = at::empty({M, F}, x2.options()), act = at::empty({M, F}, x2.options());
  Gemm up(x2, false, w_fc, false, M, F, C);
  up.add_bias(b_fc).into(h.data_ptr(), F, kGemmGeluDual);
  up.C2 = act.data_ptr();
  up.run();
  const bool f32 = is_f32(residual);
  at::Tensor y = at::empty(x.sizes(), x2.options().dtype(f32 ? at::kFloat : at::kBFloat16));
  Gemm down(act, false, w_proj, false, M, C, F);
  down.add_bias(b_proj).into(y.data_ptr(), C, f32 ? kGemmOutF32 : 0);
  add_residual(down, residual, f32, &kept);
  down.run();
  return {y, x2, h, act};
}

// {dx, dw_fc, db_fc, dw_proj, db_proj}; see linear_bwd.
std::tuple<OptTensor, OptTensor, OptTensor, OptTensor, OptTensor> mlp_gelu_bwd(
    const at::Tensor& dy, const at::Tensor& x2, const at::Tensor& h, const at::Tensor& act, const at::Tensor& w_fc,
    const at::Tensor& w_proj, bool want_dx, bool want_dw_fc, const OptTensor& main_fc, const Ready& fc_ready,
    bool want_db_fc, const OptTensor& main_b_fc, const Ready& b_fc_ready, bool want_dw_proj, const OptTensor& main_proj,
    const Ready& proj_ready, bool want_db_proj, const OptTensor& main_b_proj, const Ready& b_proj_ready) {
  c10::cuda::CUDAGuard guard(dy.device());
  at::Tensor dy2 = bf16_rows(dy);
  const int64_t M = x2.size(0), C = x2.size(1), F = h.size(1);
  at::Tensor dh = at::empty({M, F}, dy2.options());
  Gemm g(dy2, false, w_proj, true, M, F, C);      // the derivative is applied in the epilogue
  g.into(dh.data_ptr(), F, kGemmDGelu | kGemmMaySplit);
  g.aux = h.data_ptr();
  g.ld_aux = h.stride(0);
  g.run();
  OptTensor dx, dw_fc, db_fc, dw_proj, db_proj;
  if (want_dw_proj) dw_proj = weight_grad(dy2, act, main_proj, proj_ready);
  if (want_db_proj) db_proj = bias_grad(dy2, main_b_proj, b_proj_ready);
  if (want_dx) {
    dx = at::empty(sizes_with_last(dy, C), dy2.options());
    Gemm(dh, false, w_fc, true, M, C, F).into(dx->data_ptr(), C, kGemmMaySplit).run();
  }
  if (want_dw_fc) dw_fc = weight_grad(dh, x2, main_fc, fc_ready);
  if (want_db_fc) db_fc = bias_grad(dh, main_b_fc, b_fc_ready);
  return {dx, dw_fc, db_fc, dw_proj, db_proj};
}

// Views of the query, key and value heads of a packed [B, T, (H + 2 KV) D] projection.
std::array<at::Tensor, 3> packed_heads(const at::Tensor& qkv, int64_t H, int64_t KV, int64_t D) {
  at::Tensor heads = qkv.view({qkv.size(0), qkv.size(1), H + 2 * KV, D});
  return {heads.narrow(2, 0, H), heads.narrow(2, H, KV), heads.narrow(2, H + KV, KV)};
}

// Attention over a packed projection, with RoPE applied to it in place first: {o [B, T, H D], lse, the projection as
// attention read it}
std::tuple<at::Tensor, at::Tensor, at::Tensor> attention_packed_fwd(const at::Tensor& packed, int64_t H, int64_t KV, int64_t D,
                                                                    const OptTensor& freqs, int64_t pos0, bool causal) {
  TORCH_CHECK(packed.dim() == 3, "attention: [B, T, (H + 2 KV) D] projection");
  at::Tensor qkv = packed.scalar_type() == at::kBFloat16 ? packed : packed.to(at::kBFloat16);
  if (freqs) {
    if (!qkv.is_contiguous()) qkv = qkv.clone(at::MemoryFormat::Contiguous);      // (a transposed one keeps its order otherwise)
    rope_inplace(qkv, *freqs, qkv.size(0), qkv.size(1), H + KV, D, qkv.stride(1), pos0, false);
  }
  auto [q, k, v] = packed_heads(qkv, H, KV, D);
  std::vector<at::Tensor> out = flash_attn_fwd(q, k, v, 1.0 / std::sqrt(static_cast<double>(D)), causal);
  return {out[0].view({qkv.size(0), qkv.size(1), H * D}), out[1], qkv};
}

at::Tensor attention_packed_bwd(const at::Tensor& dout, const at::Tensor& qkv, const at::Tensor& o, const at::Tensor& lse,
                                int64_t H, int64_t KV, int64_t D, const OptTensor& freqs, int64_t pos0, bool causal) {
  const int64_t B = qkv.size(0), T = qkv.size(1);
  auto [q, k, v] = packed_heads(qkv, H, KV, D);
  at::Tensor dqkv = at::empty_like(qkv);
  auto [dq, dk, dv] = packed_heads(dqkv, H, KV, D);
  at::Tensor d = dout.reshape({B, T, H, D});
  if (d.scalar_type() != at::kBFloat16) d = d.to(at::kBFloat16);
  flash_attn_bwd(d.contiguous(), q, k, v, o.view({B, T, H, D}), lse, dq, dk, dv, 1.0 / std::sqrt(static_cast<double>(D)), causal);
  if (freqs) rope_inplace(dqkv, *freqs, B, T, H + KV, D, dqkv.stride(1), pos0, true);
  return dqkv;
}

}  // namespace

void bind_comm(pybind11::module_& m);
void bind_runtime(pybind11::module_& m);

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "infinitrain_b200 native layer (sm_100a kernels, NVLink kernels, host runtime)";
  m.attr("GEMM_OUT_F32") = static_cast<int>(kGemmOutF32);
  m.attr("GEMM_ATOMIC") = static_cast<int>(kGemmAtomic);
  m.attr("GEMM_FRESH") = static_cast<int>(kGemmFresh);
  m.attr("GEMM_MAY_SPLIT") = static_cast<int>(kGemmMaySplit);
  m.attr("GEMM_ACCUM") = static_cast<int>(kGemmAccum);
  m.attr("GEMM_BIAS") = static_cast<int>(kGemmBias);
  m.attr("GEMM_RESIDUAL") = static_cast<int>(kGemmResidual);
  m.attr("GEMM_GELU_DUAL") = static_cast<int>(kGemmGeluDual);
  m.attr("GEMM_DGELU") = static_cast<int>(kGemmDGelu);
  m.attr("GEMM_PROBE_NO_LOAD") = static_cast<int>(kGemmProbeNoLoad);
  m.attr("GEMM_PROBE_NO_MMA") = static_cast<int>(kGemmProbeNoMma);
  m.def("kernel_status", &kernel_status);
  m.def("kernel_status_reset", &kernel_status_reset);
  m.def("gemm", &gemm);
  m.def("set_gemm_mode", &set_gemm_mode);
  m.def("set_attn_mode", &set_attn_mode);
  m.def("get_attn_mode", &get_attn_mode);
  m.def("get_gemm_mode", &get_gemm_mode);
  m.def("layernorm_fwd", &layernorm_fwd, pybind11::arg("x"), pybind11::arg("gamma"), pybind11::arg("beta"),
        pybind11::arg("eps"), pybind11::arg("out_dtype"), pybind11::arg("statistics") = true);
  m.def("layernorm_bwd", &layernorm_bwd, pybind11::arg("dy"), pybind11::arg("x"), pybind11::arg("gamma"),
        pybind11::arg("mean"), pybind11::arg("rstd"), pybind11::arg("has_beta"), pybind11::arg("dres") = pybind11::none(),
        pybind11::arg("dgamma_out") = pybind11::none(), pybind11::arg("dbeta_out") = pybind11::none(),
        pybind11::arg("dres_sum_out") = pybind11::none(), pybind11::arg("want_dres_sum") = false);
  m.def("rmsnorm_fwd", &rmsnorm_fwd, pybind11::arg("x"), pybind11::arg("gamma"), pybind11::arg("eps"),
        pybind11::arg("out_dtype"), pybind11::arg("statistics") = true);
  m.def("rmsnorm_bwd", &rmsnorm_bwd, pybind11::arg("dy"), pybind11::arg("x"), pybind11::arg("gamma"), pybind11::arg("rstd"),
        pybind11::arg("dres") = pybind11::none(), pybind11::arg("dgamma_out") = pybind11::none(),
        pybind11::arg("dres_sum_out") = pybind11::none(), pybind11::arg("want_dres_sum") = false);
  m.def("gelu_fwd", &gelu_fwd);
  m.def("gelu_bwd", &gelu_bwd);
  m.def("swiglu_fwd", &swiglu_fwd);
  m.def("swiglu_bwd", &swiglu_bwd);
  m.def("rope_inplace", &rope_inplace);
  m.def("embedding_fwd", &embedding_fwd);
  m.def("embedding_bwd", &embedding_bwd);
  m.def("ce_fwd", &ce_fwd);
  m.def("ce_bwd", &ce_bwd);
  m.def("adamw", &adamw, pybind11::arg("p"), pybind11::arg("g"), pybind11::arg("m"), pybind11::arg("v"),
        pybind11::arg("shadow"), pybind11::arg("lr"), pybind11::arg("b1"), pybind11::arg("b2"),
        pybind11::arg("eps"), pybind11::arg("wd"), pybind11::arg("bc1"), pybind11::arg("bc2"),
        pybind11::arg("grad_scale"), pybind11::arg("dev_hyper") = pybind11::none());
  m.def("adam_advance", &adam_advance);
  m.def("sgd", &sgd);
  m.def("cast_into", &cast_into);
  m.def("colsum", &colsum, pybind11::arg("x"), pybind11::arg("into") = pybind11::none());
  m.def("flash_attn_fwd", &flash_attn_fwd);
  m.def("flash_attn_bwd", &flash_attn_bwd);
  m.def("bf16_rows", &bf16_rows);
  m.def("adds_in_place", &adds_in_place);
  m.def("linear_fwd", &linear_fwd);
  m.def("linear_bwd", &linear_bwd);
  m.def("mlp_gelu_fwd", &mlp_gelu_fwd);
  m.def("mlp_gelu_bwd", &mlp_gelu_bwd);
  m.def("attention_packed_fwd", &attention_packed_fwd);
  m.def("attention_packed_bwd", &attention_packed_bwd);
  bind_comm(m);
  bind_runtime(m);
}
