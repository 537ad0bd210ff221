// torch_ops.cpp -- the torch side of the model kernels: argument checks, allocation of results
// and scratch, launches on the current stream, and the autograd functions of the operators that
// a model calls several times per layer.  In Python a forward and backward of a norm cost the
// host 85 us, more than the kernels of 4096 x 4096 take (41); from here 73.  The same of rope and
// SwiGLU, and of torch's own x * 2, is 50 to 53: the rest are the third launch, the scratch and the
// second input and output of the norm (forward 9.7 against 7, backward 51.7 against 37.7, and 4 for
// what the graph holds in between).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>

#include "fused_elementwise.h"

namespace {

// The address of a tensor's elements for a kernel.  Asking with the element type is refused where
// there is no memory (fake and meta tensors); asked without, they give a null pointer.
void *data(const at::Tensor &t) { return t.numel() ? t.data_ptr<at::BFloat16>() : nullptr; }

void *checkBf16(const at::Tensor &t, const char *name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous(), name,
              " must be a contiguous CUDA bfloat16 tensor");
  void *p = data(t);
  TORCH_CHECK(((uintptr_t)p & 15) == 0, name, " must be 16-byte aligned");
  return p;
}

void checkLaunch(cudaError_t e) {
  if (e != cudaSuccess) C10_CUDA_CHECK(e);
}

int smCount() { return at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }

std::vector<at::Tensor> rmsnorm_fwd(const at::Tensor &x, const at::Tensor &w, double eps) {
  checkBf16(x, "x");
  checkBf16(w, "weight");
  const int H = (int)x.size(-1);
  TORCH_CHECK(H % 8 == 0 && H <= 8 * 512 * 4 && w.numel() == H, "rmsnorm: hidden size must be a multiple of 8, at most 16384");
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = x.numel() / H;
  auto y = at::empty_like(x);
  auto rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  if (rows > 0)
    checkLaunch(fcxops::rmsnormForward(data(x), data(w), data(y), rstd.data_ptr<float>(), rows, H, (float)eps,
                                          at::cuda::getCurrentCUDAStream()));
  return {y, rstd};
}

// `add`, when given, has x's shape and is added to dx inside the kernel (the gradient that
// reaches x through a residual connection around the norm).
std::vector<at::Tensor> rmsnorm_bwd(const at::Tensor &g, const at::Tensor &x, const at::Tensor &w,
                                    const at::Tensor &rstd, const c10::optional<at::Tensor> &add) {
  checkBf16(g, "grad");
  if (add.has_value()) {
    checkBf16(*add, "add");
    TORCH_CHECK(add->numel() == x.numel(), "rmsnorm_bwd: `add` must have x's shape");
  }
  checkBf16(x, "x");
  checkBf16(w, "weight");
  const int H = (int)x.size(-1);
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = x.numel() / H;
  auto dx = at::empty_like(x);
  TORCH_CHECK(H % 8 == 0 && H <= 8 * 512 * 4 && w.numel() == H, "rmsnorm: hidden size must be a multiple of 8, at most 16384");
  const int sms = smCount();
  auto partial = at::empty({fcxops::rmsnormPartials(rows, H, sms), H}, x.options().dtype(at::kFloat));
  auto dw = at::empty({H}, x.options());
  if (rows == 0) {
    dw.zero_();
    return {dx, dw};
  }
  checkLaunch(fcxops::rmsnormBackward(data(g), data(x), data(w), rstd.data_ptr<float>(),
                                         add.has_value() ? data(*add) : nullptr, data(dx), data(dw),
                                         partial.data_ptr<float>(), rows, H, sms, at::cuda::getCurrentCUDAStream()));
  return {dx, dw};
}

void rope_inplace(at::Tensor &x, const c10::optional<at::Tensor> &positions, double theta, bool backward) {
  checkBf16(x, "x");
  TORCH_CHECK(x.dim() >= 3, "rope: expected [..., heads, head_dim]");
  const int D = (int)x.size(-1), heads = (int)x.size(-2);
  TORCH_CHECK(D % 16 == 0, "rope: head_dim must be a multiple of 16");
  const int64_t tokens = x.numel() / ((int64_t)D * heads);
  const int *pos = nullptr;
  if (positions.has_value()) {
    TORCH_CHECK(positions->scalar_type() == at::kInt && positions->numel() == tokens && positions->is_cuda(), "rope: bad positions");
    pos = positions->data_ptr<int>();
  }
  const c10::cuda::CUDAGuard guard(x.device());
  checkLaunch(fcxops::rope(data(x), pos, (int)tokens, heads, D, logf((float)theta), backward ? -1.f : 1.f,
                              at::cuda::getCurrentCUDAStream()));
}

// qkv: [tokens, (ropeHeads + otherHeads) * D]; returns a new tensor of the same shape.
at::Tensor rope_fused_qkv(const at::Tensor &qkv, int64_t ropeHeads, int64_t totalHeads, int64_t D, double theta,
                          bool backward) {
  checkBf16(qkv, "qkv");
  TORCH_CHECK(D % 16 == 0 && qkv.size(-1) == totalHeads * D && ropeHeads <= totalHeads, "rope_fused_qkv: bad shape");
  const int64_t tokens = qkv.numel() / (totalHeads * D);
  const c10::cuda::CUDAGuard guard(qkv.device());
  auto out = at::empty_like(qkv);
  if (qkv.numel() == 0) return out;
  checkLaunch(fcxops::ropeQkv(data(qkv), data(out), (int)tokens, (int)ropeHeads, (int)totalHeads, (int)D,
                                 logf((float)theta), backward ? -1.f : 1.f, at::cuda::getCurrentCUDAStream()));
  return out;
}

at::Tensor swiglu_fwd(const at::Tensor &ab) {
  checkBf16(ab, "ab");
  const int F = (int)ab.size(-1) / 2;
  TORCH_CHECK(F % 8 == 0, "swiglu: width must be a multiple of 8");
  const c10::cuda::CUDAGuard guard(ab.device());
  auto sizes = ab.sizes().vec();
  sizes.back() = F;
  auto out = at::empty(sizes, ab.options());
  size_t T = ab.numel() / (2 * (size_t)F);
  checkLaunch(fcxops::swigluForward(data(ab), data(out), T, F, at::cuda::getCurrentCUDAStream()));
  return out;
}

at::Tensor swiglu_bwd(const at::Tensor &g, const at::Tensor &ab) {
  checkBf16(g, "grad");
  checkBf16(ab, "ab");
  const int F = (int)ab.size(-1) / 2;
  const c10::cuda::CUDAGuard guard(ab.device());
  auto dab = at::empty_like(ab);
  size_t T = ab.numel() / (2 * (size_t)F);
  checkLaunch(fcxops::swigluBackward(data(g), data(ab), data(dab), T, F,
                                        at::cuda::getCurrentCUDAStream()));
  return dab;
}

// Returns per-row losses; `logits` now holds gradScale * dLoss/dlogits.
at::Tensor cross_entropy_fwd_bwd_(at::Tensor &logits, const at::Tensor &targets, double gradScale) {
  checkBf16(logits, "logits");
  TORCH_CHECK(targets.is_cuda() && targets.scalar_type() == at::kLong && targets.is_contiguous(), "targets must be int64 CUDA");
  const int V = (int)logits.size(-1);
  TORCH_CHECK(V % 8 == 0, "cross-entropy: vocabulary must be a multiple of 8");
  const int64_t rows = logits.numel() / V;
  TORCH_CHECK(targets.numel() == rows, "cross-entropy: one target per row");
  const c10::cuda::CUDAGuard guard(logits.device());
  auto loss = at::empty({rows}, logits.options().dtype(at::kFloat));
  if (rows == 0) return loss;
  checkLaunch(fcxops::crossEntropy(data(logits), targets.data_ptr<int64_t>(), loss.data_ptr<float>(), rows, V,
                                      (float)gradScale, smCount(), at::cuda::getCurrentCUDAStream()));
  return loss;
}

void adamw_flat_(at::Tensor &p, const at::Tensor &g, at::Tensor &m, at::Tensor &v, double lr, double beta1, double beta2,
                 double eps, double wd, int64_t step) {
  void *pp = checkBf16(p, "param"), *pg = checkBf16(g, "grad"), *pm = checkBf16(m, "exp_avg"), *pv = checkBf16(v, "exp_avg_sq");
  TORCH_CHECK(p.numel() == g.numel() && p.numel() == m.numel() && p.numel() == v.numel(), "adamw: size mismatch");
  const c10::cuda::CUDAGuard guard(p.device());
  const size_t n = p.numel();
  if (n == 0) return;
  float bc1 = 1.f - (float)std::pow(beta1, (double)step), bc2 = 1.f - (float)std::pow(beta2, (double)step);
  checkLaunch(fcxops::adamw(pp, pg, pm, pv, n, (float)lr, (float)beta1, (float)beta2,
                               (float)eps, (float)wd, bc1, bc2, at::cuda::getCurrentCUDAStream()));
}

// ---- autograd functions -------------------------------------------------------------------
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

std::atomic<int64_t> launches{0}; // operator kernels launched through the functions below

struct RmsNormFunction : public Function<RmsNormFunction> {
  static at::Tensor forward(AutogradContext *ctx, const at::Tensor &x, const at::Tensor &w, double eps) {
    auto r = rmsnorm_fwd(x, w, eps);
    ++launches;
    ctx->save_for_backward({x, w, r[1]});
    return r[0];
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    auto r = rmsnorm_bwd(g[0].contiguous(), s[0], s[1], s[2], c10::nullopt);
    ++launches;
    return {r[0], r[1], at::Tensor()};
  }
};

// (norm(x), x): the gradient of the second output is added in the norm's backward kernel.
struct RmsNormBranchFunction : public Function<RmsNormBranchFunction> {
  static variable_list forward(AutogradContext *ctx, const at::Tensor &x, const at::Tensor &w, double eps) {
    auto r = rmsnorm_fwd(x, w, eps);
    ++launches;
    ctx->save_for_backward({x, w, r[1]});
    return {r[0], x.view_as(x)};
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    auto s = ctx->get_saved_variables(); // an output that was not used has a gradient of zeros here
    auto r = rmsnorm_bwd(g[0].contiguous(), s[0], s[1], s[2], g[1].contiguous());
    ++launches;
    return {r[0], r[1], at::Tensor()};
  }
};

struct RopeQkvFunction : public Function<RopeQkvFunction> {
  static at::Tensor forward(AutogradContext *ctx, const at::Tensor &qkv, int64_t ropeHeads, int64_t totalHeads, int64_t D,
                            double theta) {
    ctx->saved_data["ropeHeads"] = ropeHeads;
    ctx->saved_data["totalHeads"] = totalHeads;
    ctx->saved_data["D"] = D;
    ctx->saved_data["theta"] = theta;
    ++launches;
    return rope_fused_qkv(qkv, ropeHeads, totalHeads, D, theta, false);
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    ++launches;
    return {rope_fused_qkv(g[0].contiguous(), ctx->saved_data["ropeHeads"].toInt(), ctx->saved_data["totalHeads"].toInt(),
                           ctx->saved_data["D"].toInt(), ctx->saved_data["theta"].toDouble(), true),
            at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

struct SwigluFunction : public Function<SwigluFunction> {
  static at::Tensor forward(AutogradContext *ctx, const at::Tensor &abIn) {
    auto ab = abIn.contiguous();
    ctx->save_for_backward({ab});
    ++launches;
    return swiglu_fwd(ab);
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    ++launches;
    return {swiglu_bwd(g[0].contiguous(), s[0])};
  }
};

at::Tensor rmsnorm(const at::Tensor &x, const at::Tensor &w, double eps) {
  return RmsNormFunction::apply(x.contiguous(), w, eps);
}
std::tuple<at::Tensor, at::Tensor> rmsnorm_branch(const at::Tensor &x, const at::Tensor &w, double eps) {
  auto r = RmsNormBranchFunction::apply(x.contiguous(), w, eps);
  return {r[0], r[1]};
}
at::Tensor rope_qkv(const at::Tensor &qkv, int64_t ropeHeads, int64_t totalHeads, int64_t D, double theta) {
  return RopeQkvFunction::apply(qkv.contiguous(), ropeHeads, totalHeads, D, theta);
}
at::Tensor swiglu(const at::Tensor &ab) { return SwigluFunction::apply(ab); }
int64_t launch_count() { return launches.load(); }

} // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("rmsnorm_fwd", &rmsnorm_fwd);
  m.def("rmsnorm_bwd", &rmsnorm_bwd, py::arg("g"), py::arg("x"), py::arg("w"), py::arg("rstd"), py::arg("add") = py::none());
  m.def("rope_inplace", &rope_inplace);
  m.def("rope_fused_qkv", &rope_fused_qkv);
  m.def("swiglu_fwd", &swiglu_fwd);
  m.def("swiglu_bwd", &swiglu_bwd);
  m.def("cross_entropy_fwd_bwd_", &cross_entropy_fwd_bwd_);
  m.def("adamw_flat_", &adamw_flat_);
  m.def("rmsnorm", &rmsnorm);
  m.def("rmsnorm_branch", &rmsnorm_branch);
  m.def("rope_qkv", &rope_qkv);
  m.def("swiglu", &swiglu);
  m.def("launch_count", &launch_count);
}
