// The checked launchers behind the Python bindings, for native code that runs several of them (block_bind.cpp). Each is documented
// where it is defined.
#pragma once
#include <torch/extension.h>

namespace tb_launch {

using torch::Tensor;
using Opt = c10::optional<Tensor>;

void tc_gemm(const Tensor& a, const Tensor& b, Tensor& c, bool a_mn_major, bool b_mn_major, int64_t mode, int64_t flags, double alpha,
             const Opt& bias, const Opt& aux_in, const Opt& aux_out, const Opt& row_scale, const Opt& tile_group, const Opt& group_offsets,
             const Opt& status, double beta, const Opt& k_runs);
void tc_gemm_swiglu(const Tensor& x, const Tensor& w13, Tensor& h, const Opt& gu, int64_t act, const Opt& bias, double limit, double alpha);
std::vector<Tensor> rmsnorm_fwd(const Tensor& x, const Opt& res, const Tensor& w, double eps);
std::vector<Tensor> rmsnorm_bwd(const Tensor& x, const Tensor& w, const Tensor& dy, const Tensor& rstd, const Opt& dres, const Opt& dw_into,
                                bool dw_bf16);
Tensor qk_prep_fwd(const Tensor& in, int64_t k_off, const Opt& cs, const Opt& sn, int64_t T, int64_t H, int64_t D);
void qk_prep_bwd(const Tensor& in, int64_t k_off, const Tensor& dout, Tensor& d_in, const Opt& cs, const Opt& sn, int64_t T, int64_t H, int64_t D);
Tensor colsum(const Tensor& x, const Opt& out, bool bf16);
std::vector<Tensor> gla_fwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g,
                            int64_t gcol, Tensor& out, int64_t ocol, const Opt& init, int64_t B, int64_t T, int64_t H, bool gate_logits, int64_t D);
std::vector<Tensor> gla_bwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g,
                            int64_t gcol, const Tensor& dout, int64_t docol, const Tensor& states, const Tensor& decay, Tensor& dq, int64_t dqcol,
                            Tensor& dk, int64_t dkcol, Tensor& dv, int64_t dvcol, Tensor& dg, int64_t dgcol, int64_t B, int64_t T, int64_t H,
                            bool gate_logits, const Opt& dfin, const Opt& fin, int64_t D, const Opt& before_rest);
Tensor gdn_recurrent(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g, int64_t gcol,
                     const Opt& beta, Tensor& state, Tensor& out, int64_t ocol, int64_t B, int64_t T, int64_t H, int64_t D, bool gate_logits,
                     double scale);
std::vector<Tensor> gdn_chunk_fwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g,
                                  int64_t gcol, const Opt& beta, const Opt& init, Tensor& out, int64_t ocol, int64_t B, int64_t T, int64_t H,
                                  int64_t D, bool gate_logits, double scale, bool keep_scores);
std::vector<Tensor> gdn_chunk_bwd(const Tensor& q, int64_t qcol, const Tensor& k, int64_t kcol, const Tensor& v, int64_t vcol, const Tensor& g,
                                  int64_t gcol, const Tensor& dout, int64_t docol, const Opt& beta, const Opt& dfin, std::vector<Tensor> saved,
                                  Tensor& dq, int64_t dqcol, Tensor& dk, int64_t dkcol, Tensor& dv, int64_t dvcol, Tensor& dg, int64_t dgcol,
                                  int64_t B, int64_t T, int64_t H, int64_t D, bool gate_logits, double scale);
Tensor strength_fwd(const Tensor& x, const Tensor& w);
std::vector<Tensor> strength_bwd(const Tensor& dbeta, const Tensor& beta, const Tensor& x, const Tensor& w);

}  // namespace tb_launch
