// A whole pre-norm block (norm, recurrent mixer, norm with the residual, feed-forward, residual) on the launchers of its parts: one call from
// Python without gradients; one in each direction with them where the host is waited for, and else two (the norm and the mixer; all that
// follows), so that what the feed-forward saved is given back before the mixer's gradients are formed.
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

// A block's parameters in the order that Python passes them: those up to the mixer, those after it.
enum { NORM1 = 0, QKVG, BETA, MIXER_PARAMS };
enum { OUT = 0, NORM2, UP, UP_BIAS, DOWN, DOWN_BIAS, REST_PARAMS };

struct Shape {
  int64_t B, T, d, H, D, HD, rows;
};

Shape shape_of(const Tensor& x, const std::vector<Opt>& p, int64_t H, int64_t D) {
  TORCH_CHECK(p.size() == MIXER_PARAMS && x.dim() == 3 && x.is_contiguous() && x.size(1) > 1 && p[NORM1].has_value() && p[QKVG].has_value(),
              "block: x [B, T > 1, dim], norm and projection of the mixer");
  Shape s{x.size(0), x.size(1), x.size(2), H, D, H * D, x.size(0) * x.size(1)};
  TORCH_CHECK(p[QKVG]->dim() == 2 && p[QKVG]->size(0) == 4 * s.HD && p[QKVG]->size(1) == s.d, "block: projection shapes");
  return s;
}

// [rows, dim] of contiguous [B, T, dim], whose mixer output is `o`.
Tensor rest_rows(const Tensor& x, const Tensor& o, const std::vector<Opt>& f) {
  TORCH_CHECK(f.size() == REST_PARAMS && x.dim() == 3 && x.is_contiguous(), "block: x [B, T, dim] and six parameters");
  for (int i : {OUT, NORM2, UP, DOWN}) TORCH_CHECK(f[i].has_value(), "block: parameter ", i, " after the mixer is missing");
  Tensor rows = x.view({x.size(0) * x.size(1), x.size(2)});
  TORCH_CHECK(o.dim() == 2 && o.size(0) == rows.size(0) && f[OUT]->dim() == 2 && f[OUT]->size(0) == rows.size(1) && f[OUT]->size(1) == o.size(1) &&
                  f[UP]->dim() == 2 && f[UP]->size(1) == rows.size(1) && f[DOWN]->dim() == 2 && f[DOWN]->size(0) == rows.size(1),
              "block: projection shapes");
  return rows;
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

// h w^T + bias + stream, in a tensor of the stream's shape that is no view (a caller may write into it).
Tensor down_and_residual(const Tensor& h, const std::vector<Opt>& f, const Tensor& stream, at::IntArrayRef sizes) {
  Tensor y = torch::empty(sizes, h.options()), y2 = y.view(stream.sizes());
  product(h, *f[DOWN], false, false, 1.0, f[DOWN_BIAS], 0, {}, {}, y2);
  at::add_out(y2, stream, y2);
  return y;
}

// Every intermediate is let go of where its last reader has been launched, as it is between the modules.

// Without gradients -> [y, state after the tokens, status or nothing].
std::vector<Tensor> block_infer(const Tensor& x, const std::vector<Opt>& p, const std::vector<Opt>& f, const Opt& cos, const Opt& sin, int64_t offset,
                                const Opt& init, int64_t H, int64_t D, double eps1, double eps2, double out_scale, bool delta, bool gated) {
  const Shape s = shape_of(x, p, H, D);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor x2 = x.view({s.rows, s.d}), o, state, status;
  {
    Tensor n1 = tb_launch::rmsnorm_fwd(x2, {}, *p[NORM1], eps1)[0];
    Tensor qkvg = product(n1, *p[QKVG], false, false);
    Opt beta;
    if (delta && p[BETA]) beta = tb_launch::strength_fwd(n1, *p[BETA]);
    n1.reset();
    Tensor qk = tb_launch::qk_prep_fwd(qkvg, s.HD, table_rows(cos, offset, s.T, D), table_rows(sin, offset, s.T, D), s.T, H, D).view({s.rows, 2 * s.HD});
    o = torch::empty({s.rows, s.HD}, x.options());
    if (delta) {
      state = torch::empty({s.B, H, D, D}, x.options().dtype(at::kFloat));
      if (init) state.copy_(*init);
      else state.zero_();
      status = tb_launch::gdn_recurrent(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, beta, state, o, 0, s.B, s.T, H, D, true, 1.0);
    } else {
      auto r = tb_launch::gla_fwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, o, 0, init, s.B, s.T, H, true, D);
      state = r[2].view({s.B, H, D, D});
      status = r[3];
    }
  }
  rest_rows(x, o, f);
  Tensor a = product(o, *f[OUT], false, false, out_scale);
  o.reset();
  auto r = tb_launch::rmsnorm_fwd(a, x2, *f[NORM2], eps2);
  a.reset();
  Tensor h;
  if (gated) {
    h = torch::empty({s.rows, f[UP]->size(0) / 2}, x.options());
    tb_launch::tc_gemm_swiglu(r[0], *f[UP], h, {}, 0, {}, 0.0, 0.0);
  } else {
    h = product(r[0], *f[UP], false, false, 1.0, f[UP_BIAS], tb::GF_GELU);
  }
  r[0].reset();
  return {down_and_residual(h, f, r[2], x.sizes()), state, status};
}

// With gradients, from the first token on: norm and mixer. Returns [output of the mixer, saved tensors for mixer_backward ..., status].
std::vector<Tensor> mixer_forward(const Tensor& x, const std::vector<Opt>& p, const Opt& cos, const Opt& sin, int64_t H, int64_t D, double eps1,
                                  bool delta) {
  const Shape s = shape_of(x, p, H, D);
  c10::cuda::CUDAGuard guard(x.device());
  auto n1 = tb_launch::rmsnorm_fwd(x.view({s.rows, s.d}), {}, *p[NORM1], eps1);
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
  std::vector<Tensor> r{o, n1[0], n1[1], qkvg, qk, beta};
  r.insert(r.end(), mixer.begin(), mixer.end());
  r.push_back(status);
  return r;
}

// Output projection, residual, norm, GELU feed-forward, residual -> [y, saved tensors for rest_backward ...].
std::vector<Tensor> rest_forward(const Tensor& o, const Tensor& x, const std::vector<Opt>& f, double eps2, double out_scale) {
  c10::cuda::CUDAGuard guard(x.device());
  Tensor x2 = rest_rows(x, o, f);
  auto n2 = tb_launch::rmsnorm_fwd(product(o, *f[OUT], false, false, out_scale), x2, *f[NORM2], eps2);
  Tensor slope = torch::empty({x2.size(0), f[UP]->size(0)}, x.options());
  Tensor h = product(n2[0], *f[UP], false, false, 1.0, f[UP_BIAS], tb::GF_GELU, {}, slope);
  return {down_and_residual(h, f, n2[2], x.sizes()), n2[2], n2[0], n2[1], slope, h};
}

// Gradients of parameters: into fp32 buffers that they are added to (`into`), where a parameter has one, or returned. `want`: which.
struct Grads {
  const std::vector<Opt>& into;
  const std::vector<bool>& want;
  std::vector<Tensor> out;

  Grads(const std::vector<Opt>& into_, const std::vector<bool>& want_, size_t n) : into(into_), want(want_), out(n) {
    TORCH_CHECK(into.size() == n && want.size() == n, "block: a buffer and a wish for each parameter");
  }
  void weight(int i, const Tensor& dout, const Tensor& in, double alpha = 1.0) {  // dW = alpha dout^T in
    if (!want[i]) return;
    if (into[i]) product(dout, in, true, true, alpha, {}, tb::GF_ACCUMULATE, {}, {}, into[i]);
    else out[i] = product(dout, in, true, true, alpha);
  }
  void bias(int i, const Tensor& dout) {
    if (!want[i]) return;
    Tensor g = tb_launch::colsum(dout, into[i], !into[i]);
    if (!into[i]) out[i] = g;
  }
  Tensor norm(int i, const Tensor& in, const Tensor& w, const Tensor& dn, const Tensor& rstd, const Tensor& dres) {
    auto r = tb_launch::rmsnorm_bwd(in, w, dn, rstd, dres, into[i], !into[i]);
    if (want[i] && !into[i]) out[i] = r[1];
    return r[0];
  }
};

Tensor aligned_rows(const Tensor& t, int64_t d) {
  Tensor r = t.reshape({-1, d}).contiguous();
  return (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15) == 0 ? r : r.clone();
}

// `saved`: what rest_forward returned after y. Returns the gradients of the mixer's output, of x and of the six parameters.
std::vector<Tensor> rest_backward(const Tensor& dy_, const Tensor& o, const Tensor& x, const std::vector<Opt>& f, const std::vector<Opt>& into,
                                  const std::vector<bool>& want, const std::vector<Tensor>& saved, double out_scale) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(saved.size() == 5, "rest_backward: saved tensors");
  const Tensor &stream = saved[0], &n2 = saved[1], &rstd2 = saved[2], &slope = saved[3], &h = saved[4];
  const int64_t d = rest_rows(x, o, f).size(1);
  Tensor dy = dy_.reshape({-1, d}).contiguous();
  if ((reinterpret_cast<uintptr_t>(dy.data_ptr()) & 15) != 0) dy = dy.clone();
  Grads g(into, want, REST_PARAMS);
  Tensor dpre = product(dy, *f[DOWN], false, true, 1.0, {}, tb::GF_DGELU, slope);
  g.weight(DOWN, dy, h);
  g.bias(DOWN_BIAS, dy);
  Tensor dn2 = product(dpre, *f[UP], false, true);
  g.weight(UP, dpre, n2);
  g.bias(UP_BIAS, dpre);
  dpre.reset();
  Tensor ds = g.norm(NORM2, stream, *f[NORM2], dn2, rstd2, dy);  // of the stream after the mixer
  dn2.reset();
  Tensor dout = product(ds, *f[OUT], false, true, out_scale);
  g.weight(OUT, ds, o, out_scale);
  g.out.insert(g.out.begin(), {dout, ds.view(x.sizes())});
  return g.out;
}

// `saved`: what mixer_forward returned between the mixer's output and the status. `dout`, `ds`: gradients of the mixer's output and, from all that
// follows, of x. Returns the gradients of x (where wanted) and the three parameters, and the status.
std::vector<Tensor> mixer_backward(const Tensor& dout, const Tensor& ds, const Tensor& x, const std::vector<Opt>& p, const std::vector<Opt>& into,
                                   bool want_x, const std::vector<bool>& want, const Opt& cos, const Opt& sin, const std::vector<Opt>& saved, int64_t H,
                                   int64_t D, bool delta) {
  const Shape s = shape_of(x, p, H, D);
  TORCH_CHECK(saved.size() == (delta ? 14 : 8), "mixer_backward: saved tensors");
  c10::cuda::CUDAGuard guard(x.device());
  auto sv = [&](size_t i) { return saved[i] ? *saved[i] : Tensor(); };
  const Tensor n1 = sv(0), rstd1 = sv(1), qkvg = sv(2), qk = sv(3), beta = sv(4);
  Grads g(into, want, MIXER_PARAMS);
  Tensor dqk = torch::empty_like(qk), dqkvg = torch::empty_like(qkvg), dbeta, status;
  if (delta) {
    std::vector<Tensor> mixer;
    for (size_t i = 5; i < 14; ++i) mixer.push_back(sv(i));
    auto r = tb_launch::gdn_chunk_bwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, dout, 0, beta.defined() ? Opt(beta) : Opt(), {}, mixer, dqk, 0, dqk,
                                      s.HD, dqkvg, 2 * s.HD, dqkvg, 3 * s.HD, s.B, s.T, H, D, true, 1.0);
    dbeta = r[0];
    status = r[2];
  } else {
    status = tb_launch::gla_bwd(qk, 0, qk, s.HD, qkvg, 2 * s.HD, qkvg, 3 * s.HD, dout, 0, sv(5), sv(6), dqk, 0, dqk, s.HD, dqkvg, 2 * s.HD, dqkvg,
                                3 * s.HD, s.B, s.T, H, true, {}, {}, D, saved[7])[0];
  }
  tb_launch::qk_prep_bwd(qkvg, s.HD, dqk.view({s.rows, 2, H, D}), dqkvg, table_rows(cos, 0, s.T, D), table_rows(sin, 0, s.T, D), s.T, H, D);
  dqk.reset();
  g.weight(QKVG, dqkvg, n1);
  Tensor strengths;
  if (beta.defined()) {
    auto r = tb_launch::strength_bwd(dbeta, beta, n1, *p[BETA]);
    strengths = r[0];
    if (want[BETA]) g.out[BETA] = r[1];
  }
  Tensor dx;
  if (want_x || want[NORM1]) {
    Tensor dn1 = product(dqkvg, *p[QKVG], false, true);
    if (strengths.defined()) dn1.add_(strengths);
    dx = g.norm(NORM1, x.view({s.rows, s.d}), *p[NORM1], dn1, rstd1, ds.view({s.rows, s.d}));
  }
  g.out.insert(g.out.begin(), want_x ? dx.view(x.sizes()) : Tensor());
  g.out.push_back(status);
  return g.out;
}

// Both halves in one call, for blocks that wait for the host.

// -> [y, output of the mixer, five tensors of rest_forward, those of mixer_forward ..., status].
std::vector<Tensor> block_forward(const Tensor& x, const std::vector<Opt>& p, const std::vector<Opt>& f, const Opt& cos, const Opt& sin, int64_t H,
                                  int64_t D, double eps1, double eps2, double out_scale, bool delta) {
  auto m = mixer_forward(x, p, cos, sin, H, D, eps1, delta);
  auto r = rest_forward(m[0], x, f, eps2, out_scale);
  std::vector<Tensor> out{r[0], m[0]};
  out.insert(out.end(), r.begin() + 1, r.end());
  out.insert(out.end(), m.begin() + 1, m.end());
  return out;
}

// `saved`: what block_forward returned between y and the status; `into` and `want` of the nine parameters. Returns the gradients of x and the
// parameters, and the status.
std::vector<Tensor> block_backward(const Tensor& dy, const Tensor& x, const std::vector<Opt>& p, const std::vector<Opt>& f, const std::vector<Opt>& into,
                                   bool want_x, const std::vector<bool>& want, const Opt& cos, const Opt& sin, const std::vector<Opt>& saved, int64_t H,
                                   int64_t D, double out_scale, bool delta) {
  TORCH_CHECK(into.size() == MIXER_PARAMS + REST_PARAMS && want.size() == into.size() && saved.size() > 6, "block_backward: lists");
  std::vector<Tensor> second;
  for (int i = 1; i < 6; ++i) second.push_back(*saved[i]);
  auto r = rest_backward(dy, *saved[0], x, f, {into.begin() + MIXER_PARAMS, into.end()}, {want.begin() + MIXER_PARAMS, want.end()}, second, out_scale);
  auto m = mixer_backward(r[0], r[1], x, p, {into.begin(), into.begin() + MIXER_PARAMS}, want_x, {want.begin(), want.begin() + MIXER_PARAMS}, cos, sin,
                          {saved.begin() + 6, saved.end()}, H, D, delta);
  m.insert(m.end() - 1, r.begin() + 2, r.end());
  return m;
}

}  // namespace

void register_block(pybind11::module& m) {
  m.def("block_infer", &block_infer);
  m.def("block_forward", &block_forward);
  m.def("block_backward", &block_backward);
  m.def("mixer_forward", &mixer_forward);
  m.def("rest_forward", &rest_forward);
  m.def("rest_backward", &rest_backward);
  m.def("mixer_backward", &mixer_backward);
}
