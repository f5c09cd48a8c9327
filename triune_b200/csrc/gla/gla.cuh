// Launchers of the gated-linear-attention kernels (head_dim 64 or 128, chunk 64, bf16 in, fp32 state).
//
// The sequence is processed in three phases, forward and backward alike:
//   1. per chunk, in parallel:   local state contribution (K~^T V, or Q~^T dO going backward)
//   2. per (batch, head):        inter-chunk recurrence over the chunk states (elementwise scan)
//   3. per chunk, in parallel:   outputs (or input gradients) from the chunk-start state + intra-chunk scores
// Every matrix product runs as tcgen05.mma (M=64) on TMA-fed, 128B-swizzled shared-memory tiles with the
// accumulators in TMEM. Per-dimension decays are kept exact by referencing each 16-token sub-chunk of keys
// to its own first row, so every exponent stays within [-80, 80] given the per-token clamp g >= -5.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tb {

constexpr float GLA_MIN_LOG_DECAY = -5.0f;
// What follows from it: the least decay, and the logit whose log-sigmoid it is, -log(e^5 - 1).
static_assert(GLA_MIN_LOG_DECAY == -5.0f, "the two numbers below are of -5");
constexpr float GLA_MIN_DECAY = 6.7379469990854671e-3f, GLA_MIN_LOGIT = -4.9932392505505110f;

// A [B*T rows] x [D cols] bf16 slice of a wider row-major matrix: element (row, c) = ptr[row*ld + col0 + h*D + c].
struct GlaMat {
  const void* ptr;
  long long ld;
  int col0;
};

struct GlaDims {
  int B, T, H;       // T: tokens per sequence taken by the call, a multiple of 64
  bool gate_logits;  // g holds raw logits (log-sigmoid applied in-kernel) instead of log decays
  int D = 64;        // head dimension (keys and values): 64 or 128
  int rows = 0;      // rows per sequence in the matrices where that is more than T, else 0
};

// mode 0: kv[bh,c] = (k * exp(b_last - b))^T v and decay[bh,c] = exp(b_last);  mode 1: kv = (q * exp(b))^T dO.
void launch_gla_chunk_outer(int mode, GlaMat X, GlaMat Y, GlaMat G, float* out_kv, float* out_decay, GlaDims d,
                            int* status, cudaStream_t s);
// forward: states[c] = S before chunk c, S <- decay[c] * S + kv[c];  reverse: states[c] = dS after chunk c.
void launch_gla_scan(const float* kv, const float* decay, const float* init, __nv_bfloat16* states, float* final_state,
                     int BH, int NT, int D, bool reverse, cudaStream_t s);
void launch_gla_fwd_out(GlaMat Q, GlaMat K, GlaMat V, GlaMat G, const __nv_bfloat16* states, GlaMat O, GlaDims d,
                        int* status, cudaStream_t s);
void launch_gla_bwd_main(GlaMat Q, GlaMat K, GlaMat V, GlaMat G, GlaMat dO, const __nv_bfloat16* states,
                         const __nv_bfloat16* dstates, GlaMat dQ, GlaMat dK, GlaMat dV, float* dgl_local,
                         float* chunk_tot, GlaDims d, int* status, cudaStream_t s);
// end_term (optional, fp32 [B*H, D]): rowsum(dS_T * S_T), the gate gradient that reaches every token through a
// differentiated final state.
void launch_gla_dg_finalize(const float* dgl_local, const float* chunk_tot, GlaMat G, GlaMat dG, GlaDims d,
                            cudaStream_t s, const float* end_term = nullptr);
// Fewer than 64 tokens, fp32 throughout (gla_tail.cu): rows [t0, t0 + n) of every sequence of `rows` rows.
struct GlaTail {
  int B, H, D, rows, t0, n;
  bool gate_logits;
  float floor;  // least log decay of a token
};
// state0 / state1: fp32 [B*H, D, D] before (null: zero) and after the tokens; outputs are written to the same rows of O.
void launch_gla_tail_fwd(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaMat& O, const float* state0,
                         float* state1, const GlaTail& t, cudaStream_t s);
// dstate1, end1 (rowsum(dstate1 * state1), fp32 [B*H, D]): null where the state after the tokens has no gradient. Writes the
// tokens' rows of dQ, dK, dV, dG, the gradient of state0 and its rowsum with state0.
void launch_gla_tail_bwd(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaMat& dO, const GlaMat& dQ,
                         const GlaMat& dK, const GlaMat& dV, const GlaMat& dG, const float* state0, const float* dstate1,
                         const float* end1, float* dstate0, float* end0, const GlaTail& t, cudaStream_t s);
// Developer aid: eight int64 counters (device memory) receiving the backward kernel's phase clocks; null disables.
void gla_set_debug_buffer(long long* counters);
// One decode step for B*H heads: state [BH,64,64] fp32 in place; q,k,v,g rows of 64 bf16; out bf16.
void launch_gla_decode_step(GlaMat Q, GlaMat K, GlaMat V, GlaMat G, float* state, GlaMat O, int B, int H,
                            bool gate_logits, cudaStream_t s);
// One decoding step from the fused projection rows [B, ld] = [q | k | v | gate logits] (mixer_step.cu).
struct MixerStep {
  const __nv_bfloat16* qkvg;
  long long ld;
  int H;
  const float *cos, *sin;  // fp32 [table_rows, D], or null: no rotation
  long long table_rows;
  const long long* pos;    // position on the device, or null: pos_host
  long long pos_host;
  const float* state_in;   // fp32 [B, H, D, D]
  float* state_out;        // may be state_in
  __nv_bfloat16* out;      // [B, H * D]
  const __nv_bfloat16* x;  // delta rule with beta_w: the projection's input rows [B, dim]
  long long ldx;
  const __nv_bfloat16* beta_w;  // [H, dim], or null: write strength 1
  int dim;
};
void launch_mixer_step(const MixerStep& p, int B, int D, bool delta, cudaStream_t s);
// Write strengths of the delta rule (write_strength.cu): beta [rows, H] = sigmoid(x w^T), x rows of `dim` with pitch ldx, w [H, dim].
constexpr int STRENGTH_MAX_HEADS = 16;
void launch_strength_fwd(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, float* beta, int rows, int dim, int H,
                         cudaStream_t s);
// dx [rows, dim] and partial [strength_bwd_parts(rows, dim)][H * dim], whose sum over blocks is the gradient of w.
int strength_bwd_parts(int rows, int dim);
void launch_strength_bwd(const float* dbeta, const float* beta, const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w,
                         __nv_bfloat16* dx, float* partial, int rows, int dim, int H, cudaStream_t s);
// Gated DeltaNet token recurrence over T tokens (T = 1: one decode step) for B*H heads of dimension D (64 or 128):
// state [BH,D,D] fp32 in place; beta: null (1), fp32 [B*T,H] (beta_mode 1) or fp32 [B*T,H*D] (beta_mode 2).
void launch_gdn_recurrent(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta,
                          int beta_mode, float* state, const GlaMat& O, int B, int T, int H, int D, bool gate_logits,
                          float scale, cudaStream_t s);

// The same, sixteen tokens per round; `workspace`: fp32 [gdn_block_workspace_floats(...)], 16-byte aligned, 0 floats where the token
// recurrence is the faster one. q, k, v, g rows must start on 8-byte boundaries. `status`: device word, 0 or what a wait that ran out left.
long long gdn_block_workspace_floats(int B, int T, int H, int D);
void launch_gdn_blocks(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta, int beta_mode,
                       float* state, const GlaMat& O, int B, int T, int H, int D, bool gate_logits, float scale, float* workspace,
                       int* status, cudaStream_t s);

// ---- Gated DeltaNet, chunk-parallel training path (gdn_chunk_kernels.cu) ----
struct GdnDims {
  int B, T, H, D;    // D = 64 or 128 (keys and values)
  bool gate_logits;
};
// Per-chunk tensors produced by the forward pass and kept for the backward pass. nchunks = B * H * ceil(T / 64).
struct GdnScratch {
  __nv_bfloat16* U0;      // [nchunks, 64, D]   T (beta V)
  __nv_bfloat16* W;       // [nchunks, 64, D]   T (beta Kbar)
  __nv_bfloat16* Tm;      // [nchunks, 64, 64]  (I + L)^-1
  __nv_bfloat16* Kend;    // [nchunks, 64, D]   k e^{b_C - b}
  float* decay;           // [nchunks, D]       e^{b_C}
  float* Lraw;            // [nchunks, 64, 64]  strict decayed key-key scores (null: not kept)
  __nv_bfloat16* U;       // [nchunks, 64, D]   effective values
  __nv_bfloat16* states;  // [nchunks, D, D]    state before each chunk
  float* fin;             // [B * H, D, D]      state after the last token
};
struct GdnBwdScratch {
  float* G1;              // [nchunks, 64, D]
  float* H1;              // [nchunks, D, D]
  __nv_bfloat16* dU;      // [nchunks, 64, D]
  __nv_bfloat16* dSend;   // [nchunks, D, D]    gradient of the state after each chunk
  float* dS0;             // [B * H, D, D]      gradient of the initial state
  float* dq1;             // [nchunks, 64, D]
  float* dkw1;            // [nchunks, 64, D]
  float* dkr1;            // [nchunks, 64, D]
  __nv_bfloat16* dW;      // [nchunks, 64, D]
  __nv_bfloat16* dLraw;   // [nchunks, 64, 64]
  float* dbeta;           // [B * T, H] (null without beta)
  float* dgl_local;       // [B * T, H * D]     in-chunk part of the gate gradient
  float* chunk_tot;       // [B * H * D / 64, ceil(T / 64), 64] chunk totals (the layout gla_dg_finalize reads with H * D / 64 heads)
};
// out = scale * GatedDeltaNet(q, k, v, g, beta); beta fp32 [B*T, H] or null; init fp32 [B*H, D, D] or null.
void launch_gdn_chunk_fwd(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta,
                          const float* init, const GlaMat& O, const GdnScratch& w, const GdnDims& d, float scale,
                          int* status, cudaStream_t s);
// Writes dq, dk, dv and fills dbeta, dS0, dgl_local, chunk_tot; the gate gradient is completed by
// launch_gla_dg_finalize with H * D / 64 heads. dfin: gradient of the final state (fp32 [B*H, D, D]) or null.
void launch_gdn_chunk_bwd(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaMat& dO,
                          const float* beta, const float* dfin, const GlaMat& dQ, const GlaMat& dK, const GlaMat& dV,
                          const GdnScratch& w, const GdnBwdScratch& x, const GdnDims& d, float scale, int* status,
                          cudaStream_t s);

}  // namespace tb
