// Python bindings of the GLA kernels.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cmath>

#include "../block/launch.h"
#include "../elementwise/elementwise.cuh"
#include "gla.cuh"

namespace {
using torch::Tensor;

inline cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// view of columns [col0, col0 + H*64) of a 2-D bf16 matrix with contiguous rows
tb::GlaMat mat(const Tensor& t, int64_t col0) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.stride(1) == 1,
              "expected a 2-D CUDA bf16 matrix with contiguous rows");
  TORCH_CHECK(t.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, "rows must be 16-byte aligned");
  return tb::GlaMat{t.data_ptr(), t.stride(0), (int)col0};
}

// A state or its gradient as the kernels read it: fp32 [.., D, D], contiguous, on the device of the rows `q`.
Tensor state_of(const Tensor& t, const Tensor& q, int64_t numel, const char* what) {
  TORCH_CHECK(t.is_cuda() && t.get_device() == q.get_device() && t.numel() == numel, what, ": [B, H, D, D] on the device of the rows");
  return t.to(at::kFloat).contiguous();
}

}  // namespace

namespace tb_launch {

// Forward over [B*T] rows: whole chunks of 64 tokens on the chunk kernels, the T % 64 tokens after them one by one in fp32
// (all of them where T < 64, and then without the chunk kernels' clamp of the log decay, which that case never had).
// Returns (states bf16 [BH*NT,D,D], decay fp32 [BH*NT,D], final_state fp32 [BH,D,D], status) and, where there are both
// chunks and further tokens, the state between them (fp32 [BH,D,D]); writes out.
std::vector<Tensor> gla_fwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol,
                            const Tensor& g, int64_t gcol, Tensor& out, int64_t ocol, const c10::optional<Tensor>& init,
                            int64_t B, int64_t T, int64_t H, bool gate_logits, int64_t D) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(D == 64 || D == 128, "gla_fwd: head dimension 64 or 128");
  const int64_t NT = T / 64, BH = B * H, rest = T % 64;
  auto f32 = q.options().dtype(at::kFloat);
  Tensor decay = torch::empty({BH * NT, D}, f32);
  Tensor states = torch::empty({BH * NT, D, D}, q.options());
  Tensor fin = torch::empty({BH, D, D}, f32);
  Tensor status = NT > 0 ? torch::zeros({1}, q.options().dtype(at::kInt)) : torch::empty({0}, q.options().dtype(at::kInt));
  auto s = cur_stream();
  const float* ip = nullptr;
  Tensor initc, mid;
  if (init.has_value() && init->defined()) {
    initc = state_of(*init, q, BH * D * D, "gla_fwd: initial state");
    ip = initc.data_ptr<float>();
  }
  if (NT > 0) {
    Tensor kv = torch::empty({BH * NT, D, D}, f32);
    Tensor after = rest > 0 ? (mid = torch::empty({BH, D, D}, f32)) : fin;
    const tb::GlaDims d{(int)B, (int)(NT * 64), (int)H, gate_logits, (int)D, (int)T};
    tb::launch_gla_chunk_outer(0, mat(k, kcol), mat(v, vcol), mat(g, gcol), kv.data_ptr<float>(), decay.data_ptr<float>(), d,
                               status.data_ptr<int>(), s);
    tb::launch_gla_scan(kv.data_ptr<float>(), decay.data_ptr<float>(), ip, reinterpret_cast<__nv_bfloat16*>(states.data_ptr()),
                        after.data_ptr<float>(), (int)BH, (int)NT, (int)D, false, s);
    tb::launch_gla_fwd_out(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol),
                           reinterpret_cast<const __nv_bfloat16*>(states.data_ptr()), mat(out, ocol), d,
                           status.data_ptr<int>(), s);
    ip = after.data_ptr<float>();
  }
  if (rest > 0) {
    const tb::GlaTail t{(int)B, (int)H, (int)D, (int)T, (int)(NT * 64), (int)rest, gate_logits, NT > 0 ? tb::GLA_MIN_LOG_DECAY : -INFINITY};
    tb::launch_gla_tail_fwd(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), mat(out, ocol), ip, fin.data_ptr<float>(), t, s);
  }
  std::vector<Tensor> r{states, decay, fin, status};
  if (NT > 0 && rest > 0) r.push_back(mid);
  return r;
}

// Backward: writes dq, dk, dv, dg into the given matrices. With `dfin` (gradient of the final state, fp32
// [BH,D,D]) and `fin` (the final state itself) the reverse scan starts from dfin instead of zero and the gate
// gradient receives rowsum(dfin * fin). `before_rest`: the state before the T % 64 last tokens (the initial state where
// T < 64; none: zero). Returns (status, gradient of the initial state [BH,D,D] fp32).
std::vector<Tensor> gla_bwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g,
               int64_t gcol, const Tensor& dout, int64_t docol, const Tensor& states, const Tensor& decay, Tensor& dq,
               int64_t dqcol, Tensor& dk, int64_t dkcol, Tensor& dv, int64_t dvcol, Tensor& dg, int64_t dgcol, int64_t B,
               int64_t T, int64_t H, bool gate_logits, const c10::optional<Tensor>& dfin,
               const c10::optional<Tensor>& fin, int64_t D, const c10::optional<Tensor>& before_rest) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(D == 64 || D == 128, "gla_bwd: head dimension 64 or 128");
  const int64_t NT = T / 64, BH = B * H, rest = T % 64;
  auto f32 = q.options().dtype(at::kFloat);
  Tensor dnext, end_term;  // gradient of the state after the tokens in hand, its rowsum with that state
  Tensor dinit = torch::empty({BH, D, D}, f32);
  if (dfin.has_value() && dfin->defined()) {
    TORCH_CHECK(fin.has_value() && fin->defined(), "the final state is needed with its gradient");
    dnext = state_of(*dfin, q, BH * D * D, "gla_bwd: gradient of the final state").reshape({BH, D, D});
    end_term = (dnext * state_of(*fin, q, BH * D * D, "gla_bwd: final state").reshape({BH, D, D})).sum(-1).contiguous();
  }
  auto fp = [](const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; };
  auto s = cur_stream();
  if (rest > 0) {
    const tb::GlaTail t{(int)B, (int)H, (int)D, (int)T, (int)(NT * 64), (int)rest, gate_logits, NT > 0 ? tb::GLA_MIN_LOG_DECAY : -INFINITY};
    Tensor from, dmid = NT > 0 ? torch::empty({BH, D, D}, f32) : dinit, emid = torch::empty({BH, D}, f32);
    if (before_rest.has_value() && before_rest->defined()) {
      from = state_of(*before_rest, q, BH * D * D, "gla_bwd: state before the last tokens");
    }
    TORCH_CHECK(NT == 0 || from.defined(), "gla_bwd: the state after the whole chunks is needed");
    tb::launch_gla_tail_bwd(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), mat(dout, docol), mat(dq, dqcol), mat(dk, dkcol),
                            mat(dv, dvcol), mat(dg, dgcol), fp(from), fp(dnext), fp(end_term), dmid.data_ptr<float>(),
                            emid.data_ptr<float>(), t, s);
    dnext = dmid;
    end_term = emid;
  }
  Tensor status = NT > 0 ? torch::zeros({1}, q.options().dtype(at::kInt)) : torch::empty({0}, q.options().dtype(at::kInt));
  if (NT == 0) return {status, dinit};
  Tensor m = torch::empty({BH * NT, D, D}, f32);
  Tensor dstates = torch::empty({BH * NT, D, D}, q.options());
  Tensor dgl = torch::empty({B * T, H * D}, f32);
  Tensor tot = torch::empty({BH * (D / 64) * NT, 64}, f32);
  const tb::GlaDims d{(int)B, (int)(NT * 64), (int)H, gate_logits, (int)D, (int)T};
  tb::launch_gla_chunk_outer(1, mat(q, qcol), mat(dout, docol), mat(g, gcol), m.data_ptr<float>(), nullptr, d,
                             status.data_ptr<int>(), s);
  tb::launch_gla_scan(m.data_ptr<float>(), decay.data_ptr<float>(), fp(dnext), reinterpret_cast<__nv_bfloat16*>(dstates.data_ptr()),
                      dinit.data_ptr<float>(), (int)BH, (int)NT, (int)D, true, s);
  tb::launch_gla_bwd_main(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), mat(dout, docol),
                          reinterpret_cast<const __nv_bfloat16*>(states.data_ptr()),
                          reinterpret_cast<const __nv_bfloat16*>(dstates.data_ptr()), mat(dq, dqcol), mat(dk, dkcol),
                          mat(dv, dvcol), dgl.data_ptr<float>(), tot.data_ptr<float>(), d, status.data_ptr<int>(), s);
  tb::launch_gla_dg_finalize(dgl.data_ptr<float>(), tot.data_ptr<float>(), mat(g, gcol), mat(dg, dgcol), d, s, fp(end_term));
  return {status, dinit};
}

static void gla_decode(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g,
                int64_t gcol, Tensor& state, Tensor& out, int64_t ocol, int64_t B, int64_t H, bool gate_logits) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(state.scalar_type() == at::kFloat && state.is_contiguous(), "state must be fp32 contiguous [B,H,64,64]");
  tb::launch_gla_decode_step(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), state.data_ptr<float>(), mat(out, ocol),
                             (int)B, (int)H, gate_logits, cur_stream());
}

// One decoding step: qkvg [B, 4 H D] -> (out [B, H D], state after the step). `inplace`: the state is updated where it is.
static std::vector<Tensor> mixer_step(const Tensor& qkvg, const c10::optional<Tensor>& cos, const c10::optional<Tensor>& sin,
                               const c10::optional<Tensor>& pos, int64_t pos_host, const Tensor& state, bool inplace, bool delta,
                               const c10::optional<Tensor>& x, const c10::optional<Tensor>& beta_w) {
  c10::cuda::CUDAGuard guard(qkvg.device());
  const auto m = mat(qkvg, 0);
  TORCH_CHECK(state.is_cuda() && state.scalar_type() == at::kFloat && state.is_contiguous() && state.dim() == 4 &&
                  state.size(2) == state.size(3) && state.size(0) == qkvg.size(0) && state.get_device() == qkvg.get_device() &&
                  4 * state.size(1) * state.size(2) == qkvg.size(1),
              "mixer_step: state [B, H, D, D] fp32 contiguous for qkvg [B, 4 H D]");
  const int64_t B = state.size(0), H = state.size(1), D = state.size(2);
  tb::MixerStep p{};
  p.qkvg = reinterpret_cast<const __nv_bfloat16*>(m.ptr);
  p.ld = m.ld;
  p.H = (int)H;
  if (cos.has_value() && cos->defined()) {
    for (const Tensor& t : {*cos, *sin})
      TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.dim() == 2 && t.size(1) == D && t.size(0) > 0 &&
                      t.size(0) == cos->size(0),
                  "mixer_step: rotary tables [rows, D] fp32");
    p.cos = cos->data_ptr<float>();
    p.sin = sin->data_ptr<float>();
    p.table_rows = cos->size(0);
  }
  if (pos.has_value() && pos->defined()) {
    TORCH_CHECK(pos->is_cuda() && pos->scalar_type() == at::kLong && pos->numel() >= 1, "mixer_step: position int64 on the device");
    p.pos = reinterpret_cast<const long long*>(pos->data_ptr<int64_t>());
  }
  p.pos_host = pos_host;
  if (beta_w.has_value() && beta_w->defined()) {
    TORCH_CHECK(x.has_value() && x->defined(), "mixer_step: the write strength needs the input rows");
    const auto xm = mat(*x, 0), wm = mat(*beta_w, 0);
    TORCH_CHECK(beta_w->is_contiguous() && beta_w->size(0) == H && beta_w->size(1) == x->size(1) && x->size(0) == B && x->size(1) % 8 == 0,
                "mixer_step: beta weight [H, dim] for input rows [B, dim]");
    p.x = reinterpret_cast<const __nv_bfloat16*>(xm.ptr);
    p.ldx = xm.ld;
    p.beta_w = reinterpret_cast<const __nv_bfloat16*>(wm.ptr);
    p.dim = (int)x->size(1);
  }
  Tensor out = torch::empty({B, H * D}, qkvg.options());
  Tensor next = inplace ? state : torch::empty_like(state);
  p.state_in = state.data_ptr<float>();
  p.state_out = next.data_ptr<float>();
  p.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  tb::launch_mixer_step(p, (int)B, (int)D, delta, cur_stream());
  return {out, next};
}

// Gated DeltaNet recurrence (no gradient): q,k,v,g as [B*T, ld] matrices whose columns col0 + h*D.. hold head h. Returns the status of
// the kernel that takes prompts in blocks (empty where the token kernel ran, which waits for nothing).
Tensor gdn_recurrent(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol,
                     const Tensor& g, int64_t gcol, const c10::optional<Tensor>& beta, Tensor& state, Tensor& out,
                     int64_t ocol, int64_t B, int64_t T, int64_t H, int64_t D, bool gate_logits, double scale) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(state.scalar_type() == at::kFloat && state.is_contiguous() && state.numel() == B * H * D * D,
              "state must be fp32 contiguous [B,H,D,D]");
  const float* bp = nullptr;
  int mode = 0;
  if (beta.has_value() && beta->defined()) {
    TORCH_CHECK(beta->scalar_type() == at::kFloat && beta->is_contiguous(), "beta must be fp32 contiguous");
    if (beta->numel() == B * T * H) mode = 1;
    else if (beta->numel() == B * T * H * D) mode = 2;
    else TORCH_CHECK(false, "beta must be [B,T,H] or [B,T,H,D]");
    bp = beta->data_ptr<float>();
  }
  const int64_t ws = tb::gdn_block_workspace_floats((int)B, (int)T, (int)H, (int)D);
  Tensor status = torch::empty({ws > 0 ? 1 : 0}, state.options().dtype(at::kInt));
  if (ws > 0) {
    Tensor work = torch::empty({ws}, state.options());
    tb::launch_gdn_blocks(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), bp, mode, state.data_ptr<float>(), mat(out, ocol),
                          (int)B, (int)T, (int)H, (int)D, gate_logits, (float)scale, work.data_ptr<float>(), status.data_ptr<int>(),
                          cur_stream());
    return status;
  }
  tb::launch_gdn_recurrent(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), bp, mode, state.data_ptr<float>(),
                           mat(out, ocol), (int)B, (int)T, (int)H, (int)D, gate_logits, (float)scale, cur_stream());
  return status;
}
static const __nv_bfloat16* bfc(const Tensor& t) { return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr()); }
static __nv_bfloat16* bfp(Tensor& t) { return reinterpret_cast<__nv_bfloat16*>(t.data_ptr()); }

// Chunk-parallel Gated DeltaNet forward. q, k, v, g: [B*T, ld] bf16 matrices with head h at columns col + h*D;
// beta fp32 [B*T, H] or None; init fp32 [B*H, D, D] or None. Writes `out`; returns
// [U0, W, Tm, Kend, decay, Lraw (empty when not kept), U, states, fin, status].
std::vector<Tensor> gdn_chunk_fwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v,
                                  int64_t vcol, const Tensor& g, int64_t gcol, const c10::optional<Tensor>& beta,
                                  const c10::optional<Tensor>& init, Tensor& out, int64_t ocol, int64_t B, int64_t T,
                                  int64_t H, int64_t D, bool gate_logits, double scale, bool keep_scores) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(T > 0 && (D == 64 || D == 128), "gdn_chunk_fwd: tokens and D in {64, 128}");
  const int64_t NT = (T + 63) / 64, BH = B * H, n = BH * NT;
  auto bf = q.options();
  auto f32 = q.options().dtype(at::kFloat);
  Tensor U0 = torch::empty({n, 64, D}, bf), W = torch::empty({n, 64, D}, bf), Tm = torch::empty({n, 64, 64}, bf),
         Kend = torch::empty({n, 64, D}, bf), decay = torch::empty({n, D}, f32), U = torch::empty({n, 64, D}, bf),
         states = torch::empty({n, D, D}, bf), fin = torch::empty({BH, D, D}, f32);
  Tensor Lraw = keep_scores ? torch::empty({n, 64, 64}, f32) : torch::empty({0}, f32);
  Tensor status = torch::zeros({1}, q.options().dtype(at::kInt));
  const float* bp = nullptr;
  Tensor betac, initc;
  if (beta.has_value() && beta->defined()) {
    betac = beta->to(at::kFloat).contiguous();
    TORCH_CHECK(betac.is_cuda() && betac.get_device() == q.get_device() && betac.numel() == B * T * H, "beta must be [B*T, H] on the device of the rows");
    bp = betac.data_ptr<float>();
  }
  const float* ip = nullptr;
  if (init.has_value() && init->defined()) {
    initc = state_of(*init, q, BH * D * D, "gdn_chunk_fwd: initial state");
    ip = initc.data_ptr<float>();
  }
  tb::GdnScratch w{bfp(U0), bfp(W), bfp(Tm), bfp(Kend), decay.data_ptr<float>(),
                   keep_scores ? Lraw.data_ptr<float>() : nullptr, bfp(U), bfp(states), fin.data_ptr<float>()};
  tb::GdnDims d{(int)B, (int)T, (int)H, (int)D, gate_logits};
  tb::launch_gdn_chunk_fwd(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), bp, ip, mat(out, ocol), w, d,
                           (float)scale, status.data_ptr<int>(), cur_stream());
  return {U0, W, Tm, Kend, decay, Lraw, U, states, fin, status};
}

// Backward. `saved` is the list returned by gdn_chunk_fwd. Writes dq, dk, dv, dg into the given matrices; returns
// [dbeta (fp32 [B*T, H], empty without beta), dS0 (fp32 [B*H, D, D]), status, then the per-chunk intermediates].
std::vector<Tensor> gdn_chunk_bwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v,
                                  int64_t vcol, const Tensor& g, int64_t gcol, const Tensor& dout, int64_t docol,
                                  const c10::optional<Tensor>& beta, const c10::optional<Tensor>& dfin,
                                  std::vector<Tensor> saved, Tensor& dq, int64_t dqcol, Tensor& dk, int64_t dkcol,
                                  Tensor& dv, int64_t dvcol, Tensor& dg, int64_t dgcol, int64_t B, int64_t T, int64_t H,
                                  int64_t D, bool gate_logits, double scale) {
  c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(saved.size() >= 9, "gdn_chunk_bwd: the forward's saved tensors are missing");
  const int64_t NT = (T + 63) / 64, BH = B * H, n = BH * NT, NH = D / 64;
  auto bf = q.options();
  auto f32 = q.options().dtype(at::kFloat);
  Tensor G1 = torch::empty({n, 64, D}, f32), H1 = torch::empty({n, D, D}, f32), dU = torch::empty({n, 64, D}, bf),
         dSend = torch::empty({n, D, D}, bf), dS0 = torch::empty({BH, D, D}, f32), dq1 = torch::empty({n, 64, D}, f32),
         dkw1 = torch::empty({n, 64, D}, f32), dkr1 = torch::empty({n, 64, D}, f32), dW = torch::empty({n, 64, D}, bf),
         dLraw = torch::empty({n, 64, 64}, bf), dgl = torch::empty({B * T, H * D}, f32),
         tot = torch::empty({BH * NH * NT, 64}, f32);
  Tensor status = torch::zeros({1}, q.options().dtype(at::kInt));
  const float* bp = nullptr;
  Tensor betac, dfinc, dbeta = torch::empty({0}, f32);
  if (beta.has_value() && beta->defined()) {
    betac = beta->to(at::kFloat).contiguous();
    bp = betac.data_ptr<float>();
    dbeta = torch::empty({B * T, H}, f32);
    TORCH_CHECK(saved[5].numel() == n * 64 * 64, "gdn_chunk_bwd: the key-key scores were not kept by the forward pass");
  }
  const float* dfp = nullptr;
  if (dfin.has_value() && dfin->defined()) {
    dfinc = dfin->to(at::kFloat).contiguous();
    dfp = dfinc.data_ptr<float>();
  }
  tb::GdnScratch w{bfp(saved[0]), bfp(saved[1]), bfp(saved[2]), bfp(saved[3]), saved[4].data_ptr<float>(),
                   saved[5].numel() > 0 ? saved[5].data_ptr<float>() : nullptr, bfp(saved[6]), bfp(saved[7]),
                   saved[8].data_ptr<float>()};
  tb::GdnBwdScratch x{G1.data_ptr<float>(), H1.data_ptr<float>(), bfp(dU), bfp(dSend), dS0.data_ptr<float>(),
                      dq1.data_ptr<float>(), dkw1.data_ptr<float>(), dkr1.data_ptr<float>(), bfp(dW), bfp(dLraw),
                      bp != nullptr ? dbeta.data_ptr<float>() : nullptr, dgl.data_ptr<float>(), tot.data_ptr<float>()};
  tb::GdnDims d{(int)B, (int)T, (int)H, (int)D, gate_logits};
  auto s = cur_stream();
  tb::launch_gdn_chunk_bwd(mat(q, qcol), mat(k, kcol), mat(v, vcol), mat(g, gcol), mat(dout, docol), bp, dfp, mat(dq, dqcol),
                           mat(dk, dkcol), mat(dv, dvcol), w, x, d, (float)scale, status.data_ptr<int>(), s);
  // the suffix sums over the chunks and the derivative of the clamped log decay: the GLA finalize kernel with every
  // 64-wide slice of a head counted as a head of its own
  Tensor end_term;
  if (dfp != nullptr) end_term = (dfinc.reshape({BH, D, D}) * saved[8].reshape({BH, D, D})).sum(-1).reshape({BH * NH, 64}).contiguous();
  tb::GlaDims gd{(int)B, (int)(NT * 64), (int)(H * NH), gate_logits, 64, (int)T};
  tb::launch_gla_dg_finalize(dgl.data_ptr<float>(), tot.data_ptr<float>(), mat(g, gcol), mat(dg, dgcol), gd, s,
                             end_term.defined() ? end_term.data_ptr<float>() : nullptr);
  // the per-chunk intermediates follow for inspection (stage-by-stage comparison against the PyTorch oracle)
  return {dbeta, dS0, status, G1, H1, dU, dSend, dq1, dkw1, dkr1, dW, dLraw, dgl, tot};
}

static void strength_operands(const Tensor& x, const Tensor& w) {
  (void)mat(x, 0);
  (void)mat(w, 0);
  TORCH_CHECK(w.is_contiguous() && w.size(1) == x.size(1) && w.size(0) <= tb::STRENGTH_MAX_HEADS && x.get_device() == w.get_device(),
              "write strengths: x [rows, dim], w [heads, dim] contiguous, up to 16 heads");
}

// beta [rows, H] fp32 = sigmoid(x w^T)
Tensor strength_fwd(const Tensor& x, const Tensor& w) {
  strength_operands(x, w);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor beta = torch::empty({x.size(0), w.size(0)}, x.options().dtype(at::kFloat));
  tb::launch_strength_fwd(bfc(x), x.stride(0), bfc(w), beta.data_ptr<float>(), (int)x.size(0), (int)x.size(1), (int)w.size(0), cur_stream());
  return beta;
}

// (dx bf16 [rows, dim], dw bf16 [H, dim]) from the gradient of beta (fp32 [rows, H])
std::vector<Tensor> strength_bwd(const Tensor& dbeta, const Tensor& beta, const Tensor& x, const Tensor& w) {
  strength_operands(x, w);
  const int64_t rows = x.size(0), dim = x.size(1), H = w.size(0);
  for (const Tensor* t : {&dbeta, &beta})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == rows * H, "write strengths: fp32 [rows, H]");
  c10::cuda::CUDAGuard guard(x.device());
  Tensor dx = torch::empty({rows, dim}, x.options()), dw = torch::empty({H, dim}, w.options());
  const int parts = tb::strength_bwd_parts((int)rows, (int)dim);
  Tensor partial = torch::empty({parts, H * dim}, x.options().dtype(at::kFloat));
  auto s = cur_stream();
  tb::launch_strength_bwd(dbeta.data_ptr<float>(), beta.data_ptr<float>(), bfc(x), x.stride(0), bfc(w), bfp(dx), partial.data_ptr<float>(),
                          (int)rows, (int)dim, (int)H, s);
  tb::launch_column_parts(partial.data_ptr<float>(), parts, (int)(H * dim), {nullptr, bfp(dw), false}, s);
  return {dx, dw};
}

}  // namespace tb_launch

void register_gla(pybind11::module& m) {
  namespace py = pybind11;
  using namespace tb_launch;
  m.def("gla_fwd", &gla_fwd, py::arg("q"), py::arg("qcol"), py::arg("k"), py::arg("kcol"), py::arg("v"), py::arg("vcol"), py::arg("g"),
        py::arg("gcol"), py::arg("out"), py::arg("ocol"), py::arg("init"), py::arg("B"), py::arg("T"), py::arg("H"),
        py::arg("gate_logits"), py::arg("D") = 64);
  m.def("gla_bwd", &gla_bwd, py::arg("q"), py::arg("qcol"), py::arg("k"), py::arg("kcol"), py::arg("v"), py::arg("vcol"), py::arg("g"),
        py::arg("gcol"), py::arg("dout"), py::arg("docol"), py::arg("states"), py::arg("decay"), py::arg("dq"), py::arg("dqcol"),
        py::arg("dk"), py::arg("dkcol"), py::arg("dv"), py::arg("dvcol"), py::arg("dg"), py::arg("dgcol"), py::arg("B"), py::arg("T"),
        py::arg("H"), py::arg("gate_logits"), py::arg("dfin"), py::arg("fin"), py::arg("D") = 64, py::arg("before_rest") = py::none());
  m.def("gla_decode", &gla_decode);
  m.def("gla_debug_buffer", [](const c10::optional<Tensor>& t) {
    TORCH_CHECK(!t.has_value() || !t->defined() || (t->scalar_type() == at::kLong && t->numel() >= 8), "int64[8] expected");
    tb::gla_set_debug_buffer(t.has_value() && t->defined() ? (long long*)t->data_ptr<int64_t>() : nullptr);
  });
  m.def("mixer_step", &mixer_step);
  m.def("strength_fwd", &strength_fwd);
  m.def("strength_bwd", &strength_bwd);
  m.def("gdn_recurrent", &gdn_recurrent);
  m.def("gdn_chunk_fwd", &gdn_chunk_fwd);
  m.def("gdn_chunk_bwd", &gdn_chunk_bwd);
}
