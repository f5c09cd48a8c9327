// Gated linear attention over fewer than 64 tokens (a short prompt, a chat's next turn, the ragged end of a sequence), forward
// and backward, all of it fp32 on the bf16 inputs:
//
//   S_t = diag(e^{g_t}) S_{t-1} + k_t v_t^T        o_t = S_t^T q_t
//   dS_t = q_t do_t^T + diag(e^{g_{t+1}}) dS_{t+1}    dq_t = S_t do_t    dk_t = dS_t v_t    dv_t = dS_t^T k_t
//   d log decay_t = sum_{u >= t} (q_u dq_u - k_u dk_u) + rowsum(dS_T * S_T)
//
// These tokens were a chain of about sixty element-wise launches around three fp32 products (1.0 ms a layer, nearly all of
// it host time). The tokens are walked one by one with the state in registers: a chunk on the tensor cores would round
// states and weighted keys to bf16, which this path never did. Sums over keys (o, dv) want all key rows of a
// value column in one CTA, sums over values (dq, dk) all value columns of a key row, so there are two splits of a head: 32
// columns or 32 rows per CTA, eight threads per column or row. Bound by latency, about 0.4 us a token: 37 tokens of 12 heads of 128 take 16 us
// (the layer 1086 -> 247 us), the last 9 tokens of three rows and 16 heads 10 us forward and 22 us backward.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "gla.cuh"
#include "gla_tiles.cuh"

namespace tb {

namespace {

constexpr int WIDE = 32, TT = 16, THREADS = 256;  // rows or columns of a CTA; tokens staged at a time

struct TailArgs {
  const __nv_bfloat16 *q, *k, *v, *g, *dout;  // first column of head 0, row 0
  long long q_ld, k_ld, v_ld, g_ld, do_ld;
  __nv_bfloat16 *out, *dq, *dk, *dv, *dg;
  long long out_ld, dq_ld, dk_ld, dv_ld, dg_ld;
  const float* state0;  // [B, H, D, D] before the first token, or null: zero
  float* state1;        // after the last token
  const float* dstate1;  // gradient of the state after the last token, or null
  const float* end1;    // rowsum(dstate1 * state1) [B, H, D], or null
  float* dstate0;
  float* end0;          // rowsum(dstate0 * state0)
  int H, rows, t0, n;   // rows per sequence; first token and number of tokens
  float floor;          // least log decay of a token
  int logits;
};

__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float raw_decay(float x, int logits) {
  return logits ? fminf(x, 0.f) - log1pf(__expf(-fabsf(x))) : (x > 0.f ? 0.f : x);
}
// Selections, not fmaxf: a gate that is not a number stays one, as in the PyTorch statements of these tokens.
__device__ __forceinline__ float at_least(float decay, float floor) { return decay < floor ? floor : decay; }

// Tokens [t, t + m) of `width` columns into dst[token][width] as fp32, optionally as decays e^{max(g, floor)}.
__device__ __forceinline__ void stage(const __nv_bfloat16* src, long long ld, int m, int width, float* dst) {
  for (int i = threadIdx.x; i < m * (width / 8); i += THREADS) {
    const int t = i / (width / 8), c = (i % (width / 8)) * 8;
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(src + t * ld + c), f);
    st8(dst + t * width + c, f);
  }
}
__device__ __forceinline__ void stage_decay(const __nv_bfloat16* src, long long ld, int m, int width, float* dst, float floor,
                                            int logits) {
  for (int i = threadIdx.x; i < m * (width / 8); i += THREADS) {
    const int t = i / (width / 8), c = (i % (width / 8)) * 8;
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(src + t * ld + c), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __expf(at_least(raw_decay(f[j], logits), floor));
    st8(dst + t * width + c, f);
  }
}

// The eight threads of a column (row) hold its elements in runs of four: element i of thread s is (i / 4) * 32 + s * 4 + i % 4,
// so that their 16-byte reads of a staged vector fall on different banks.
__device__ __forceinline__ int element(int i, int s) { return (i >> 2) * 32 + s * 4 + (i & 3); }

template <int N>
__device__ __forceinline__ void read_run(const float* vec, int s, float (&f)[N]) {
#pragma unroll
  for (int i = 0; i < N / 4; ++i) {
    const float4 x = *reinterpret_cast<const float4*>(vec + i * 32 + s * 4);
    f[4 * i] = x.x; f[4 * i + 1] = x.y; f[4 * i + 2] = x.z; f[4 * i + 3] = x.w;
  }
}

__device__ __forceinline__ void flush(const float* vals, int m, __nv_bfloat16* dst, long long ld) {  // vals [m][32]
  for (int i = threadIdx.x; i < m * 4; i += THREADS) {
    float f[8];
    ld8(vals + (i >> 2) * WIDE + (i & 3) * 8, f);
    *reinterpret_cast<uint4*>(dst + (i >> 2) * ld + (i & 3) * 8) = pack8(f);
  }
}

// 32 value columns of a head. REV: dv (walks backwards from dstate1); otherwise outputs and the final state.
template <int D, bool REV>
__global__ void __launch_bounds__(THREADS) gla_tail_values_kernel(const TailArgs p) {
  constexpr int RP = D / 8;
  __shared__ __align__(16) float sk[TT * D], sq[TT * D], se[TT * D], sv[TT * WIDE], so[TT * WIDE];
  const int c0 = (blockIdx.x % (D / WIDE)) * WIDE, h = blockIdx.y, b = blockIdx.x / (D / WIDE);
  const int col = threadIdx.x >> 3, s = threadIdx.x & 7;
  const long long row0 = (long long)b * p.rows + p.t0, sat = ((long long)b * p.H + h) * D * D + c0 + col;
  const float* init = REV ? p.dstate1 : p.state0;
  float S[RP];
#pragma unroll
  for (int i = 0; i < RP; ++i) S[i] = init != nullptr ? init[sat + (long long)element(i, s) * D] : 0.f;
  const int tiles = (p.n + TT - 1) / TT;
  for (int w = 0; w < tiles; ++w) {
    const int tile = REV ? tiles - 1 - w : w, ta = tile * TT, m = min(TT, p.n - ta);
    const long long r = row0 + ta;
    __syncthreads();
    stage(p.q + r * p.q_ld + h * D, p.q_ld, m, D, sq);
    stage(p.k + r * p.k_ld + h * D, p.k_ld, m, D, sk);
    stage_decay(p.g + r * p.g_ld + h * D, p.g_ld, m, D, se, p.floor, p.logits);
    if (REV) stage(p.dout + r * p.do_ld + h * D + c0, p.do_ld, m, WIDE, sv);
    else stage(p.v + r * p.v_ld + h * D + c0, p.v_ld, m, WIDE, sv);
    __syncthreads();
    for (int u = 0; u < m; ++u) {
      const int t = REV ? m - 1 - u : u;
      const float x = sv[t * WIDE + col];
      float q[RP], k[RP], e[RP], acc = 0.f;
      read_run<RP>(sq + t * D, s, q);
      read_run<RP>(sk + t * D, s, k);
      read_run<RP>(se + t * D, s, e);
#pragma unroll
      for (int i = 0; i < RP; ++i) {
        if (REV) {
          S[i] += q[i] * x;
          acc += k[i] * S[i];
          S[i] *= e[i];
        } else {
          S[i] = e[i] * S[i] + k[i] * x;
          acc += q[i] * S[i];
        }
      }
      acc = group_sum(acc);
      if (s == 0) so[t * WIDE + col] = acc;
    }
    __syncthreads();
    if (REV) flush(so, m, p.dv + r * p.dv_ld + h * D + c0, p.dv_ld);
    else flush(so, m, p.out + r * p.out_ld + h * D + c0, p.out_ld);
  }
  if (!REV) {
#pragma unroll
    for (int i = 0; i < RP; ++i) p.state1[sat + (long long)element(i, s) * D] = S[i];
  }
}

// 32 key rows of a head: a walk forwards for dq, one backwards for dk, the gate gradients and the gradient of the first state.
template <int D>
__global__ void __launch_bounds__(THREADS) gla_tail_keys_bwd_kernel(const TailArgs p) {
  constexpr int RP = D / 8;
  __shared__ __align__(16) float sv[TT * D], sd[TT * D], sk[TT * WIDE], sq[TT * WIDE], se[TT * WIDE], sx[TT * WIDE], sy[TT * WIDE];
  __shared__ float qdq[64 * WIDE];
  const int r0 = (blockIdx.x % (D / WIDE)) * WIDE, h = blockIdx.y, b = blockIdx.x / (D / WIDE);
  const int kr = threadIdx.x >> 3, s = threadIdx.x & 7;
  const long long row0 = (long long)b * p.rows + p.t0, hat = ((long long)b * p.H + h) * D + r0 + kr, sat = hat * D;
  const int tiles = (p.n + TT - 1) / TT, hc = h * D + r0;
  float S[RP];
#pragma unroll
  for (int i = 0; i < RP; ++i) S[i] = p.state0 != nullptr ? p.state0[sat + element(i, s)] : 0.f;
  for (int tile = 0; tile < tiles; ++tile) {
    const int ta = tile * TT, m = min(TT, p.n - ta);
    const long long r = row0 + ta;
    __syncthreads();
    stage(p.v + r * p.v_ld + h * D, p.v_ld, m, D, sv);
    stage(p.dout + r * p.do_ld + h * D, p.do_ld, m, D, sd);
    stage(p.q + r * p.q_ld + hc, p.q_ld, m, WIDE, sq);
    stage(p.k + r * p.k_ld + hc, p.k_ld, m, WIDE, sk);
    stage_decay(p.g + r * p.g_ld + hc, p.g_ld, m, WIDE, se, p.floor, p.logits);
    __syncthreads();
    for (int t = 0; t < m; ++t) {
      const float e = se[t * WIDE + kr], k = sk[t * WIDE + kr];
      float v[RP], d[RP], acc = 0.f;
      read_run<RP>(sv + t * D, s, v);
      read_run<RP>(sd + t * D, s, d);
#pragma unroll
      for (int i = 0; i < RP; ++i) {
        S[i] = e * S[i] + k * v[i];
        acc += S[i] * d[i];
      }
      acc = group_sum(acc);
      if (s == 0) {
        sx[t * WIDE + kr] = acc;
        qdq[(ta + t) * WIDE + kr] = sq[t * WIDE + kr] * acc;
      }
    }
    __syncthreads();
    flush(sx, m, p.dq + r * p.dq_ld + hc, p.dq_ld);
  }
  float suffix = p.end1 != nullptr ? p.end1[hat] : 0.f;
#pragma unroll
  for (int i = 0; i < RP; ++i) S[i] = p.dstate1 != nullptr ? p.dstate1[sat + element(i, s)] : 0.f;
  for (int tile = tiles - 1; tile >= 0; --tile) {
    const int ta = tile * TT, m = min(TT, p.n - ta);
    const long long r = row0 + ta;
    __syncthreads();
    stage(p.v + r * p.v_ld + h * D, p.v_ld, m, D, sv);
    stage(p.dout + r * p.do_ld + h * D, p.do_ld, m, D, sd);
    stage(p.q + r * p.q_ld + hc, p.q_ld, m, WIDE, sq);
    stage(p.k + r * p.k_ld + hc, p.k_ld, m, WIDE, sk);
    stage(p.g + r * p.g_ld + hc, p.g_ld, m, WIDE, se);  // gates as they are: their derivative is wanted too
    __syncthreads();
    for (int t = m - 1; t >= 0; --t) {
      const float q = sq[t * WIDE + kr], k = sk[t * WIDE + kr], x = se[t * WIDE + kr];
      const float decay = raw_decay(x, p.logits), e = __expf(at_least(decay, p.floor));
      float v[RP], d[RP], acc = 0.f;
      read_run<RP>(sv + t * D, s, v);
      read_run<RP>(sd + t * D, s, d);
#pragma unroll
      for (int i = 0; i < RP; ++i) {
        S[i] += q * d[i];
        acc += S[i] * v[i];
        S[i] *= e;
      }
      acc = group_sum(acc);
      if (s == 0) {
        suffix += qdq[(ta + t) * WIDE + kr] - k * acc;
        float slope = 0.f;
        if (p.logits) slope = decay < p.floor ? 0.f : 1.f / (1.f + __expf(x));
        else slope = (x <= 0.f && x >= p.floor) ? 1.f : 0.f;
        sx[t * WIDE + kr] = acc;
        sy[t * WIDE + kr] = suffix * slope;
      }
    }
    __syncthreads();
    flush(sx, m, p.dk + r * p.dk_ld + hc, p.dk_ld);
    flush(sy, m, p.dg + r * p.dg_ld + hc, p.dg_ld);
  }
#pragma unroll
  for (int i = 0; i < RP; ++i) p.dstate0[sat + element(i, s)] = S[i];
  if (s == 0) p.end0[hat] = suffix;
}

const __nv_bfloat16* at(const GlaMat& m) { return reinterpret_cast<const __nv_bfloat16*>(m.ptr) + m.col0; }
__nv_bfloat16* at_out(const GlaMat& m) { return reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(m.ptr)) + m.col0; }

TailArgs tail_args(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaTail& t) {
  for (const GlaMat* m : {&Q, &K, &V, &G})
    if (m->col0 % 8 != 0) throw std::runtime_error("gla tail: columns must start on 16-byte boundaries");
  if (t.n < 1 || t.n >= 64 || t.t0 < 0 || t.t0 + t.n > t.rows) throw std::runtime_error("gla tail: 1 to 63 tokens of a sequence");
  if (t.D != 64 && t.D != 128) throw std::runtime_error("gla tail: head dimension must be 64 or 128");
  TailArgs a{};
  a.q = at(Q), a.k = at(K), a.v = at(V), a.g = at(G);
  a.q_ld = Q.ld, a.k_ld = K.ld, a.v_ld = V.ld, a.g_ld = G.ld;
  a.H = t.H, a.rows = t.rows, a.t0 = t.t0, a.n = t.n;
  a.floor = t.floor, a.logits = t.gate_logits ? 1 : 0;
  return a;
}
void launched(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + " launch failed: " + cudaGetErrorString(e));
}

}  // namespace

void launch_gla_tail_fwd(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaMat& O, const float* state0,
                         float* state1, const GlaTail& t, cudaStream_t s) {
  if (t.B <= 0 || t.H <= 0) return;
  TailArgs a = tail_args(Q, K, V, G, t);
  a.out = at_out(O), a.out_ld = O.ld;
  a.state0 = state0, a.state1 = state1;
  const dim3 grid((unsigned)t.B * (t.D / WIDE), t.H);  // sequences along x: the other two dimensions end at 65535
  if (t.D == 64) gla_tail_values_kernel<64, false><<<grid, THREADS, 0, s>>>(a);
  else gla_tail_values_kernel<128, false><<<grid, THREADS, 0, s>>>(a);
  launched("gla_tail_fwd");
}

void launch_gla_tail_bwd(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaMat& dO, const GlaMat& dQ,
                         const GlaMat& dK, const GlaMat& dV, const GlaMat& dG, const float* state0, const float* dstate1,
                         const float* end1, float* dstate0, float* end0, const GlaTail& t, cudaStream_t s) {
  if (t.B <= 0 || t.H <= 0) return;
  TailArgs a = tail_args(Q, K, V, G, t);
  a.dout = at(dO), a.do_ld = dO.ld;
  a.dq = at_out(dQ), a.dk = at_out(dK), a.dv = at_out(dV), a.dg = at_out(dG);
  a.dq_ld = dQ.ld, a.dk_ld = dK.ld, a.dv_ld = dV.ld, a.dg_ld = dG.ld;
  a.state0 = state0, a.dstate1 = dstate1, a.end1 = end1, a.dstate0 = dstate0, a.end0 = end0;
  const dim3 grid((unsigned)t.B * (t.D / WIDE), t.H);  // sequences along x: the other two dimensions end at 65535
  if (t.D == 64) {
    gla_tail_keys_bwd_kernel<64><<<grid, THREADS, 0, s>>>(a);
    gla_tail_values_kernel<64, true><<<grid, THREADS, 0, s>>>(a);
  } else {
    gla_tail_keys_bwd_kernel<128><<<grid, THREADS, 0, s>>>(a);
    gla_tail_values_kernel<128, true><<<grid, THREADS, 0, s>>>(a);
  }
  launched("gla_tail_bwd");
}

}  // namespace tb
