// A whole pre-norm block (norm, recurrent mixer, norm with the residual, feed-forward, residual) in one call from Python, forward and
// backward, on the launchers of its parts.
//
// A layer's pass is 12 (forward) to 44 launches (both directions) whose device time is 70 to 230 us for small batches and chat turns;
// issued from Python, one autograd function or op after the other, the host needs 240 to 950 us for them. From here it needs about a third.
// The launches, their order and their numbers are those of the modules, except where a gradient joins another one in the epilogue of
// the kernel that forms it: the residual branch's in the norm's backward pass (one rounding and one pass less).
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../gemm/tc_gemm.cuh"
#include "launch.h"

namespace {

using torch::Tensor;
using Opt = c10::optional<Tensor>;

// A block's parameters in the order that Python passes them.
enum { NORM1 = 0, QKVG, BETA, OUT, NORM2, UP, UP_BIAS, DOWN, DOWN_BIAS, PARAMS };

struct Shape {
  int64_t B, T, d, H, D, HD, rows;
};

Shape shape_of(const Tensor& x, const std::vector<Opt>& p, int64_t H, int64_t D) {
  TORCH_CHECK(p.size() == PARAMS && x.dim() == 3 && x.is_contiguous() && x.size(1) > 1, "block: x [B, T > 1, dim] and nine parameters");
  for (int i : {NORM1, QKVG, OUT, NORM2, UP, DOWN}) TORCH_CHECK(p[i].has_value(), "block: parameter ", i, " is missing");
  Shape s{x.size(0), x.size(1), x.size(2), H, D, H * D, x.size(0) * x.size(1)};
  TORCH_CHECK(p[QKVG]->dim() == 2 && p[QKVG]->size(0) == 4 * s.HD && p[QKVG]->size(1) == s.d && p[OUT]->size(0) == s.d && p[OUT]->size(1) == s.HD &&
                  p[DOWN]->size(0) == s.d && p[UP]->size(1) == s.d,
              "block: projection shapes");
  return s;
}

// out (or a new bf16 matrix) = alpha a b^T with the epilogue that the flags and operands ask for.
Tensor product(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, double alpha = 1.0, const Opt& bias = {}, int64_t flags = 0, const Opt& aux_in = {},
               const Opt& aux_out = {}, const Opt& into = {}) {
  Tensor c = into ? *into : torch::empty({a_mn ? a.size(1) : a.size(0), b_mn ? b.size(1) : b.size(0)}, a.options());
  tb_launch::tc_gemm(a, b, c, a_mn, b_mn, tb::GEMM_DENSE, flags, alpha, bias, aux_in, aux_out, {}, {}, {}, {}, 1.0, {});
  return c;
}

// The first D / 2 columns of rows [at, at + T) of a rotary table, in place.
Opt table_rows(const Opt& t, int64_t at, int64_t T, int64_t D) {
  if (!t) return {};
  TORCH_CHECK(t->dim() == 2 && t->is_contiguous() && at >= 0 && at + T <= t->size(0) && t->size(1) == D, "block: rotary tables do not cover the call");
  return t->slice(0, at, at + T).slice(1, 0, D / 2);
}

// Without gradients -> [y, state after the tokens, status or nothing].
std::vector<Tensor> block_infer(const Tensor& x, const std::vector<Opt>& p, const Opt& cos, const Opt& sin, int64_t offset, const Opt& init,
                                int64_t H, int64_t D, double eps1, double eps2, double out_scale, bool delta, bool gated) {
  const Shape s = shape_of(x, p, H, D);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor x2 = x.view({s.rows, s.d});
  Tensor n1 = tb_launch::rmsnorm_fwd(x2, {}, *p[NORM1], eps1)[0];
  Tensor qkvg = product(n1, *p[QKVG], false, false);
  Tensor qk = tb_launch::qk_prep_fwd(qkvg, s.HD, table_rows(cos, offset, s.T, D), table_rows(sin, offset, s.T, D), s.T, H, D).view({s.rows, 2 * s.HD});
  Tensor o = torch::empty({s.rows, s.HD}, x.options()), state, status;
  if (delta) {
    Opt beta;
    if (p[BETA]) beta = tb_launch::strength_fwd(n1, *p[BETA]);
    auto f32 = x.options().dtype(at::kFloat);
    state = torch::empty({s.B, H, D, D}, f32);
    if (init) state.copy_(*init);
    else state.zero_();
    tb_launch::gdn_recurrent(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, beta, state, o, 0, s.B, s.T, H, D, true, 1.0);
  } else {
    auto r = tb_launch::gla_fwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, o, 0, init, s.B, s.T, H, true, D);
    state = r[2].view({s.B, H, D, D});
    status = r[3];
  }
  Tensor a = product(o, *p[OUT], false, false, out_scale);
  auto r = tb_launch::rmsnorm_fwd(a, x2, *p[NORM2], eps2);
  Tensor h;
  if (gated) {
    h = torch::empty({s.rows, p[UP]->size(0) / 2}, x.options());
    tb_launch::tc_gemm_swiglu(r[0], *p[UP], h, {}, 0, {}, 0.0, 0.0);
  } else {
    h = product(r[0], *p[UP], false, false, 1.0, p[UP_BIAS], tb::GF_GELU);
  }
  Tensor y = product(h, *p[DOWN], false, false, 1.0, p[DOWN_BIAS]);
  at::add_out(y, r[2], y);
  return {y.view(x.sizes()), state, status};
}

// With gradients, from the first token on (GELU feed-forward). Returns [y, saved tensors for block_backward ..., status].
std::vector<Tensor> block_forward(const Tensor& x, const std::vector<Opt>& p, const Opt& cos, const Opt& sin, int64_t H, int64_t D, double eps1,
                                  double eps2, double out_scale, bool delta) {
  const Shape s = shape_of(x, p, H, D);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor x2 = x.view({s.rows, s.d});
  auto n1 = tb_launch::rmsnorm_fwd(x2, {}, *p[NORM1], eps1);
  Tensor qkvg = product(n1[0], *p[QKVG], false, false);
  Tensor qk = tb_launch::qk_prep_fwd(qkvg, s.HD, table_rows(cos, 0, s.T, D), table_rows(sin, 0, s.T, D), s.T, H, D).view({s.rows, 2 * s.HD});
  Tensor o = torch::empty({s.rows, s.HD}, x.options()), beta, status;
  std::vector<Tensor> mixer;
  if (delta) {
    if (p[BETA]) beta = tb_launch::strength_fwd(n1[0], *p[BETA]);
    mixer = tb_launch::gdn_chunk_fwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, beta.defined() ? Opt(beta) : Opt(), {}, o, 0, s.B, s.T, H, D, true,
                                     1.0, beta.defined());
    status = mixer[9];
    mixer.resize(9);
  } else {
    mixer = tb_launch::gla_fwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, o, 0, {}, s.B, s.T, H, true, D);
    status = mixer[3];
    mixer = {mixer[0], mixer[1], mixer.size() > 4 ? mixer[4] : Tensor()};
  }
  Tensor a = product(o, *p[OUT], false, false, out_scale);
  auto n2 = tb_launch::rmsnorm_fwd(a, x2, *p[NORM2], eps2);
  Tensor slope = torch::empty({s.rows, p[UP]->size(0)}, x.options());
  Tensor h = product(n2[0], *p[UP], false, false, 1.0, p[UP_BIAS], tb::GF_GELU, {}, slope);
  Tensor y = torch::empty(x.sizes(), x.options()), y2 = y.view({s.rows, s.d});  // no view: a caller may write into it
  product(h, *p[DOWN], false, false, 1.0, p[DOWN_BIAS], 0, {}, {}, y2);
  at::add_out(y2, n2[2], y2);
  std::vector<Tensor> r{y, n1[0], n1[1], qkvg, qk, o, n2[2], n2[0], n2[1], slope, h, beta};
  r.insert(r.end(), mixer.begin(), mixer.end());
  r.push_back(status);
  return r;
}

// `saved`: what block_forward returned between y and the status. `into`: fp32 buffers that weight gradients are added to, where a
// parameter has one. `want`: x and the nine parameters, whose gradients are formed. Returns their gradients (undefined where not
// wanted or added) and the status.
std::vector<Tensor> block_backward(const Tensor& dy_, const Tensor& x, const std::vector<Opt>& p, const std::vector<Opt>& into,
                                   const std::vector<bool>& want, const Opt& cos, const Opt& sin, const std::vector<Opt>& saved, int64_t H, int64_t D,
                                   double out_scale, bool delta) {
  const Shape s = shape_of(x, p, H, D);
  TORCH_CHECK(into.size() == PARAMS && want.size() == PARAMS + 1 && saved.size() >= 14, "block_backward: lists");
  c10::cuda::CUDAGuard guard(x.device());
  auto sv = [&](size_t i) { return saved[i] ? *saved[i] : Tensor(); };
  const Tensor n1 = sv(0), rstd1 = sv(1), qkvg = sv(2), qk = sv(3), o = sv(4), sum = sv(5), n2 = sv(6), rstd2 = sv(7), slope = sv(8), h = sv(9),
               beta = sv(10);
  std::vector<Tensor> grad(PARAMS + 1);
  auto weight = [&](int i, const Tensor& dout, const Tensor& in, double alpha = 1.0) {  // dW = alpha dout^T in
    if (!want[i + 1]) return;
    if (into[i]) product(dout, in, true, true, alpha, {}, tb::GF_ACCUMULATE, {}, {}, into[i]);
    else grad[i + 1] = product(dout, in, true, true, alpha);
  };
  auto bias = [&](int i, const Tensor& dout) {
    if (!want[i + 1]) return;
    Tensor g = tb_launch::colsum(dout, into[i], !into[i]);
    if (!into[i]) grad[i + 1] = g;
  };
  Tensor dy = dy_.reshape({s.rows, s.d}).contiguous();
  if ((reinterpret_cast<uintptr_t>(dy.data_ptr()) & 15) != 0) dy = dy.clone();

  Tensor dpre = product(dy, *p[DOWN], false, true, 1.0, {}, tb::GF_DGELU, slope);
  weight(DOWN, dy, h);
  bias(DOWN_BIAS, dy);
  Tensor dn2 = product(dpre, *p[UP], false, true);
  weight(UP, dpre, n2);
  bias(UP_BIAS, dpre);
  auto norm = [&](int i, const Tensor& in, const Tensor& dn, const Tensor& rstd, const Tensor& dres) {
    auto r = tb_launch::rmsnorm_bwd(in, *p[i], dn, rstd, dres, into[i], !into[i]);
    if (want[i + 1] && !into[i]) grad[i + 1] = r[1];
    return r[0];
  };
  Tensor ds = norm(NORM2, sum, dn2, rstd2, dy);  // of the stream after the mixer
  Tensor dout = product(ds, *p[OUT], false, true, out_scale);
  weight(OUT, ds, o, out_scale);

  Tensor dqk = torch::empty_like(qk), dqkvg = torch::empty_like(qkvg), dbeta, status;
  if (delta) {
    std::vector<Tensor> mixer;
    for (size_t i = 11; i < 20; ++i) mixer.push_back(sv(i));
    auto r = tb_launch::gdn_chunk_bwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, dout, 0, beta.defined() ? Opt(beta) : Opt(), {}, mixer, dqk, 0, dqk,
                                      s.HD, dqkvg, 2 * s.HD, dqkvg, 3 * s.HD, s.B, s.T, H, D, true, 1.0);
    dbeta = r[0];
    status = r[2];
  } else {
    status = tb_launch::gla_bwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, dout, 0, sv(11), sv(12), dqk, 0, dqk, s.HD, dqkvg, 2 * s.HD, dqkvg,
                                3 * s.HD, s.B, s.T, H, true, {}, {}, D, saved[13])[0];
  }
  tb_launch::qk_prep_bwd(qkvg, s.HD, dqk.view({s.rows, 2, H, D}), dqkvg, table_rows(cos, 0, s.T, D), table_rows(sin, 0, s.T, D), s.T, H, D);
  weight(QKVG, dqkvg, n1);
  Tensor strengths;
  if (beta.defined()) {
    auto r = tb_launch::strength_bwd(dbeta, beta, n1, *p[BETA]);
    strengths = r[0];
    if (want[BETA + 1]) grad[BETA + 1] = r[1];
  }
  if (want[0] || want[NORM1 + 1]) {
    Tensor dn1 = product(dqkvg, *p[QKVG], false, true);
    if (strengths.defined()) dn1.add_(strengths);
    Tensor dx = norm(NORM1, x.view({s.rows, s.d}), dn1, rstd1, ds);
    if (want[0]) grad[0] = dx.view(x.sizes());
  }
  grad.push_back(status);
  return grad;
}

}  // namespace

void register_block(pybind11::module& m) {
  m.def("block_infer", &block_infer);
  m.def("block_forward", &block_forward);
  m.def("block_backward", &block_backward);
}
