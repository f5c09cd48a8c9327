// Python binding of the one-launch decoding step: a plan holds the model's tensors, the program and the workspace.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cstring>

#include "dense_step.cuh"

namespace {

using torch::Tensor;
using Opt = c10::optional<Tensor>;

class DenseStepPlan {
 public:
  // layers: [norm, qkvg weight, write-strength weight or None, state, cos or None, sin or None, output weight, norm, up (or gate and up)
  // weight, its bias or None, down weight, its bias or None]; scalars: [eps, output scale, eps] of each.
  DenseStepPlan(const std::vector<std::vector<Opt>>& layers, const std::vector<std::vector<double>>& scalars, const Tensor& embed,
                const Tensor& norm, double eps, const Tensor& head, Tensor token, Tensor out, Tensor pos, Tensor step, bool delta, bool gated)
      : device_(embed.device()) {
    c10::cuda::CUDAGuard guard(device_);
    TORCH_CHECK(!layers.empty() && layers.size() == scalars.size(), "dense_step: layers and scalars");
    const Tensor& state0 = need(layers[0], 3);
    TORCH_CHECK(state0.dim() == 4, "dense_step: state [B, H, D, D]");
    const int64_t B = state0.size(0), H = state0.size(1), D = state0.size(2), hd = H * D, V = embed.size(0), d = embed.size(1);
    TORCH_CHECK(B >= 1 && B <= tb::DENSE_STEP_MAX_ROWS && (D == 64 || D == 128) && d % 32 == 0, "dense_step: sizes");
    rows(embed, V, d);
    TORCH_CHECK(head.dim() == 2 && head.size(0) == V, "dense_step: the head's rows are the embedding's");
    rows(head, V, d);
    TORCH_CHECK(norm.dim() == 1, "dense_step: norm");
    vec(norm, d);
    std::vector<tb::DensePhase> program;
    int64_t widest = std::max(d, hd), hidden = 0;
    for (size_t l = 0; l < layers.size(); ++l) {
      const auto& t = layers[l];
      TORCH_CHECK(t.size() == 12 && scalars[l].size() == 3, "dense_step: twelve tensors and three numbers a layer");
      const int64_t up_rows = need(t, 8).size(0), f = gated ? up_rows / 2 : up_rows;
      TORCH_CHECK(f % 32 == 0 && f > 0 && (!gated || up_rows % 2 == 0), "dense_step: feed-forward width");
      hidden = std::max(hidden, f);
      widest = std::max(widest, f);
      tb::DensePhase ph{};
      ph.kind = tb::DP_PROJECT;
      ph.weight = rows(need(t, 1), 4 * hd, d);
      ph.rows = (int)(4 * hd);
      ph.k = (int)d;
      ph.extra = t[2] ? rows(*t[2], H, d) : nullptr;
      ph.strengths = t[2] ? (int)H : 0;
      ph.norm = vec(need(t, 0), d);
      ph.eps = (float)scalars[l][0];
      program.push_back(ph);
      ph = {};
      ph.kind = tb::DP_MIX;
      const Tensor& st = need(t, 3);
      TORCH_CHECK(own(st).scalar_type() == at::kFloat && st.is_contiguous() && st.sizes() == state0.sizes() && st.size(3) == D,
                  "dense_step: states fp32 [B, H, D, D]");
      ph.state = st.data_ptr<float>();
      ph.delta = delta ? 1 : 0;
      ph.strengths = t[2] ? (int)H : 0;
      TORCH_CHECK(bool(t[4]) == bool(t[5]), "dense_step: both rotary tables or none");
      if (t[4]) {
        for (int j = 4; j < 6; ++j)
          TORCH_CHECK(own(*t[j]).scalar_type() == at::kFloat && t[j]->is_contiguous() && t[j]->dim() == 2 && t[j]->size(1) == D &&
                          t[j]->size(0) == t[4]->size(0),
                      "dense_step: rotary tables fp32 [rows, D]");
        ph.cos = t[4]->data_ptr<float>();
        ph.sin = t[5]->data_ptr<float>();
        ph.table_rows = t[4]->size(0);
      }
      program.push_back(ph);
      ph = {};
      ph.kind = tb::DP_OUT;
      ph.weight = rows(need(t, 6), d, hd);
      ph.rows = (int)d;
      ph.k = (int)hd;
      ph.scale = (float)scalars[l][1];
      program.push_back(ph);
      ph = {};
      ph.kind = gated ? tb::DP_GATE_UP : tb::DP_UP;
      ph.weight = rows(need(t, 8), up_rows, d);
      ph.rows = (int)f;
      ph.k = (int)d;
      ph.norm = vec(need(t, 7), d);
      ph.eps = (float)scalars[l][2];
      ph.bias = t[9] ? vec(*t[9], f) : nullptr;
      program.push_back(ph);
      ph = {};
      ph.kind = tb::DP_DOWN;
      ph.weight = rows(need(t, 10), d, f);
      ph.rows = (int)d;
      ph.k = (int)f;
      ph.bias = t[11] ? vec(*t[11], d) : nullptr;
      program.push_back(ph);
    }
    tb::DensePhase ph{};
    ph.kind = tb::DP_HEAD;
    ph.weight = rows(head, V, d);
    ph.rows = (int)V;
    ph.k = (int)d;
    ph.norm = vec(norm, d);
    ph.eps = (float)eps;
    program.push_back(ph);

    const tb::DenseStepGeom g = tb::dense_step_geom((int)B, (int)widest, (int)d);
    fits_ = g.units > 0;
    for (auto& q : program) {
      if (q.kind == tb::DP_MIX) continue;
      if (q.strengths > g.grid) fits_ = false;  // a CTA forms the write strengths of one head
      if (fits_ && !tb::dense_step_cut(q, g)) fits_ = false;
    }
    if (!fits_) return;
    // blocks and mixer units are dealt on from where the phase before stopped: what is left over of one evens out with the next
    int64_t at = 0, unit = 0;
    for (auto& q : program) {
      if (q.kind == tb::DP_MIX) {
        q.first = (int)(unit % g.grid);
        unit += tb::dense_step_units((int)B, (int)H, (int)D, g.grid);
      } else {
        q.first = (int)(at % g.grid);
        at += q.blocks;
      }
    }
    const auto bytes = torch::TensorOptions().dtype(at::kByte);
    const int64_t size = (int64_t)(program.size() * sizeof(tb::DensePhase));
    Tensor host = torch::empty({size}, bytes);
    std::memcpy(host.data_ptr(), program.data(), size);
    program_ = host.to(device_);
    Tensor maps = torch::zeros({(int64_t)program.size() * 256}, bytes);
    for (size_t i = 0; i < program.size(); ++i)
      if (program[i].kind != tb::DP_MIX) tb::dense_step_maps(program[i], static_cast<char*>(maps.data_ptr()) + i * 256);
    maps_ = maps.to(device_);
    const auto long_ = torch::TensorOptions().dtype(at::kLong).device(device_);
    rows_ = torch::zeros({B * (d + (5 * hd + hidden) / 2 + H)}, long_);
    best_ = torch::empty({g.grid * tb::DENSE_STEP_MAX_ROWS}, long_);
    words_ = torch::zeros({4}, long_.dtype(at::kInt));
    for (const Tensor& x : {token, pos, step, out})
      TORCH_CHECK(own(x).scalar_type() == at::kLong && x.is_contiguous(), "dense_step: token, position, step and output int64 contiguous");
    TORCH_CHECK(token.numel() == B && pos.numel() == 1 && step.numel() == 1 && out.dim() == 2 && out.size(0) == B && out.size(1) > 0,
                "dense_step: token [B, 1], output [B, tokens]");
    p_.program = reinterpret_cast<const tb::DensePhase*>(program_.data_ptr());
    p_.maps = maps_.data_ptr();
    p_.phases = (int)program.size();
    p_.B = (int)B;
    p_.d = (int)d;
    p_.H = (int)H;
    p_.hd = (int)hd;
    p_.act_pitch = g.act_pitch;
    p_.units = g.units;
    p_.slots = g.slots;
    p_.embed = rows(embed, V, d);
    p_.token = reinterpret_cast<long long*>(token.data_ptr<int64_t>());
    p_.out = reinterpret_cast<long long*>(out.data_ptr<int64_t>());
    p_.pos = reinterpret_cast<long long*>(pos.data_ptr<int64_t>());
    p_.step = reinterpret_cast<long long*>(step.data_ptr<int64_t>());
    p_.out_ld = out.size(1);
    auto* w = reinterpret_cast<unsigned long long*>(rows_.data_ptr<int64_t>());  // rows are multiples of 16 words
    p_.stream = w;
    p_.middle = p_.stream + B * d / 2;
    p_.qkvg = p_.middle + B * d / 2;
    p_.mixed = p_.qkvg + B * 2 * hd;
    p_.hidden = p_.mixed + B * hd / 2;
    p_.beta = p_.hidden + B * hidden / 2;
    p_.best = reinterpret_cast<unsigned long long*>(best_.data_ptr<int64_t>());
    p_.sync = reinterpret_cast<unsigned int*>(words_.data_ptr<int>());
    p_.epoch = p_.sync + 3;
    p_.status = words_.data_ptr<int>() + 2;
    grid_ = g.grid;
    smem_ = g.smem;
    head_dim_ = (int)D;
  }

  bool fits() const { return fits_; }
  Tensor status() const { return words_.slice(0, 2, 3); }
  Tensor program() const { return program_; }  // bytes of the DensePhase entries

  // One token of every sequence, on the current stream.
  void replay() {
    TORCH_CHECK(fits_, "dense_step: does not fit");
    c10::cuda::CUDAGuard guard(device_);
    tb::launch_dense_step(p_, grid_, smem_, head_dim_, at::cuda::getCurrentCUDAStream().stream());
  }

 private:
  const Tensor& need(const std::vector<Opt>& t, size_t i) {
    TORCH_CHECK(i < t.size() && t[i].has_value() && t[i]->defined(), "dense_step: tensor ", i, " is missing");
    return *t[i];
  }
  const Tensor& own(const Tensor& t) {  // on this device, and alive as long as the plan
    TORCH_CHECK(t.is_cuda() && t.device() == device_, "dense_step: all tensors on one device");
    held_.push_back(t);
    return t;
  }
  const __nv_bfloat16* rows(const Tensor& t, int64_t n, int64_t k) {
    own(t);
    TORCH_CHECK(t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.size(0) == n && t.size(1) == k && t.is_contiguous() && k % 32 == 0 &&
                    (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0,
                "dense_step: weight bf16 [", n, ", ", k, "], contiguous, 16-byte aligned");
    return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr());
  }
  const __nv_bfloat16* vec(const Tensor& t, int64_t n) {
    own(t);
    TORCH_CHECK(t.scalar_type() == at::kBFloat16 && t.numel() == n && t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0,
                "dense_step: vector bf16 [", n, "], 16-byte aligned");
    return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr());
  }

  c10::Device device_;
  std::vector<Tensor> held_;
  Tensor program_, maps_, rows_, best_, words_;
  tb::DenseStep p_{};
  int grid_ = 0, smem_ = 0, head_dim_ = 0;
  bool fits_ = false;
};

}  // namespace

void register_decode(pybind11::module& m) {
  namespace py = pybind11;
  py::class_<DenseStepPlan>(m, "DenseStepPlan")
      .def(py::init<const std::vector<std::vector<Opt>>&, const std::vector<std::vector<double>>&, const Tensor&, const Tensor&, double,
                    const Tensor&, Tensor, Tensor, Tensor, Tensor, bool, bool>(),
           py::arg("layers"), py::arg("scalars"), py::arg("embed"), py::arg("norm"), py::arg("eps"), py::arg("head"), py::arg("token"),
           py::arg("out"), py::arg("pos"), py::arg("step"), py::arg("delta"), py::arg("gated"))
      .def_property_readonly("fits", &DenseStepPlan::fits)
      .def_property_readonly("status", &DenseStepPlan::status)
      .def_property_readonly("program", &DenseStepPlan::program)
      .def("replay", &DenseStepPlan::replay);
}
