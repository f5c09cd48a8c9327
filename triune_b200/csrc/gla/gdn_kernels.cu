// Gated DeltaNet, exact token recurrence in one kernel (inference / prefill / decode; no gradient).
//
//   v_pred = S_{t-1}^T k_t            u_t = v_t - v_pred
//   S_t    = diag(exp(g_t)) S_{t-1} + (beta_t * k_t) u_t^T          (g <= 0 per key dimension; beta per token and
//   o_t    = scale * S_t^T q_t                                        head, per key dimension, or absent = 1)
//
// One CTA per (batch, head). The dk x dv state lives in registers for the whole sequence: thread (part, c) owns
// rows [part*RP, part*RP + RP) of column c, so the two contractions of a token (k^T S and q^T S) are RP fused
// multiply-adds per thread plus a sum of the NPART partials through shared memory. Tokens are staged in blocks of 16
// through a double-buffered shared-memory ring with 16-byte loads, so global latency is paid once per block and
// overlaps the arithmetic of the previous block. A delta rule couples all key dimensions of a head (k^T S), so unlike
// plain GLA it cannot be split into 64-wide slices; the kernel is templated on the head dimension instead.
//
// Replaces the reference's per-token Python loop (triune/kernels/fast_gla.py:781-836) and its single-token decode.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <stdexcept>
#include <string>

#include "../common/per_device.h"
#include "../common/ptx.cuh"
#include "gla.cuh"

namespace tb {

namespace {


__device__ __forceinline__ float gdn_log_decay(float x, bool logits) {
  const float g = logits ? (fminf(x, 0.f) - log1pf(__expf(-fabsf(x)))) : fminf(x, 0.f);
  return fmaxf(g, GLA_MIN_LOG_DECAY);
}

// D: head dimension (keys and values). THREADS = D * NPART. GDN_TB: tokens per staged block.
template <int D, int NPART, int GDN_TB>
__global__ void __launch_bounds__(D* NPART) gdn_recurrent_kernel(
    const __nv_bfloat16* __restrict__ q, long long q_ld, int qcol, const __nv_bfloat16* __restrict__ k, long long k_ld,
    int kcol, const __nv_bfloat16* __restrict__ v, long long v_ld, int vcol, const __nv_bfloat16* __restrict__ g,
    long long g_ld, int gcol, const float* __restrict__ beta, int beta_mode /*0 none, 1 [B*T,H], 2 [B*T,H*D]*/,
    float* __restrict__ state /*[B*H, D, D] in/out*/, __nv_bfloat16* __restrict__ out, long long o_ld, int ocol, int T,
    int H, int logits, float scale) {
  constexpr int RP = D / NPART;          // state rows per thread
  constexpr int VEC = D / 8;             // 16-byte vectors per token and tensor
  __shared__ __align__(16) __nv_bfloat16 sIn[2][GDN_TB][4][D];  // q, k, v, g of a token block
  __shared__ float sBeta[2][GDN_TB][D];                         // beta per key dimension (mode 2) or [.][0] (mode 1)
  __shared__ float sK[D], sQ[D], sDec[D];                       // current token: beta*k, q, exp(g) in fp32
  __shared__ float sKraw[D];
  __shared__ float sPart[2][NPART][D];

  const int tid = threadIdx.x, c = tid % D, part = tid / D;
  const int bh = blockIdx.x, h = bh % H, b = bh / H;
  const long long row0 = (long long)b * T;

  float S[RP];
  {
    const float* sp = state + ((long long)bh * D + part * RP) * D + c;
#pragma unroll
    for (int r = 0; r < RP; ++r) S[r] = sp[(long long)r * D];
  }

  auto stage = [&](int blk, int buf) {
    const int t0 = blk * GDN_TB;
    for (int i = tid; i < GDN_TB * 4 * VEC; i += D * NPART) {
      const int tt = i / (4 * VEC), rem = i % (4 * VEC), which = rem / VEC, vec = rem % VEC;
      const int t = t0 + tt;
      if (t < T) {
        const __nv_bfloat16* src = which == 0   ? q + (row0 + t) * q_ld + qcol
                                   : which == 1 ? k + (row0 + t) * k_ld + kcol
                                   : which == 2 ? v + (row0 + t) * v_ld + vcol
                                                : g + (row0 + t) * g_ld + gcol;
        // asynchronous 16-byte copy: the block lands while the previous one is being computed
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&sIn[buf][tt][which][vec * 8])),
                     "l"(src + h * D + vec * 8)
                     : "memory");
      } else {
        *reinterpret_cast<uint4*>(&sIn[buf][tt][which][vec * 8]) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (beta_mode == 2) {
      for (int i = tid; i < GDN_TB * D; i += D * NPART) {
        const int tt = i / D, d = i % D, t = t0 + tt;
        sBeta[buf][tt][d] = t < T ? beta[((row0 + t) * H + h) * D + d] : 0.f;
      }
    } else if (beta_mode == 1) {
      if (tid < GDN_TB) sBeta[buf][tid][0] = (t0 + tid) < T ? beta[(row0 + t0 + tid) * H + h] : 0.f;
    }
  };

  const int nblk = (T + GDN_TB - 1) / GDN_TB;
  stage(0, 0);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int blk = 0; blk < nblk; ++blk) {
    const int buf = blk & 1;
    if (blk + 1 < nblk) stage(blk + 1, buf ^ 1);  // lands in the other buffer while this block is computed
    const int tcount = min(GDN_TB, T - blk * GDN_TB);
    for (int tt = 0; tt < tcount; ++tt) {
      // token operands in fp32: one thread per key dimension
      if (tid < D) {
        const float kk = __bfloat162float(sIn[buf][tt][1][tid]);
        const float bt = beta_mode == 0 ? 1.f : (beta_mode == 1 ? sBeta[buf][tt][0] : sBeta[buf][tt][tid]);
        sKraw[tid] = kk;
        sK[tid] = bt * kk;
        sQ[tid] = __bfloat162float(sIn[buf][tt][0][tid]);
        sDec[tid] = __expf(gdn_log_decay(__bfloat162float(sIn[buf][tt][3][tid]), logits != 0));
      }
      __syncthreads();
      float acc = 0.f;
#pragma unroll
      for (int r = 0; r < RP; ++r) acc += sKraw[part * RP + r] * S[r];
      sPart[0][part][c] = acc;
      __syncthreads();
      float vp = 0.f;
#pragma unroll
      for (int pp = 0; pp < NPART; ++pp) vp += sPart[0][pp][c];
      const float u = __bfloat162float(sIn[buf][tt][2][c]) - vp;
      float oacc = 0.f;
#pragma unroll
      for (int r = 0; r < RP; ++r) {
        const int d = part * RP + r;
        S[r] = sDec[d] * S[r] + sK[d] * u;
        oacc += sQ[d] * S[r];
      }
      sPart[1][part][c] = oacc;
      __syncthreads();
      if (part == 0) {
        float o = 0.f;
#pragma unroll
        for (int pp = 0; pp < NPART; ++pp) o += sPart[1][pp][c];
        out[(row0 + blk * GDN_TB + tt) * o_ld + ocol + h * D + c] = __float2bfloat16(o * scale);
      }
      // the next token's operand pass rewrites sK.. only after every thread passed the barrier above, and sPart[0] is
      // rewritten only after the next operand barrier: no further barrier needed here
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // block boundary: the staged next block is complete and this buffer may be overwritten
  }
  {
    float* sp = state + ((long long)bh * D + part * RP) * D + c;
#pragma unroll
    for (int r = 0; r < RP; ++r) sp[(long long)r * D] = S[r];
  }
}

// ------------------------------------------------------------------------------------------------
// The same recurrence, sixteen tokens at a time, for prompts.
//
// One token at a time the recurrence is a chain: a contraction over all key rows, its sum across threads, then the update
// that the next token's contraction waits for (2100 clocks a token in the kernel above). Sixteen tokens share ONE such round:
// with P_j = product of the decays up to and including token j of the block, S the state before it and L strictly lower,
//   x_j  = v_j - (k_j P_{j-1})^T S            L_ji = sum_d k_j (beta k)_i dec_{i+1..j-1}
//   u    = T x, T = (1 + L)^-1                A_ji = sum_d q_j (beta k)_i dec_{i+1..j}
//   o_j  = (q_j P_j)^T S + sum_{i<=j} A_ji u_i
//   S   <- P_15 S + sum_j (beta k_j dec_{j+1..15}) u_j^T
// Exponents are <= 0 as in the token form. What does not depend on the state (the scaled vectors, T and A) is formed once per
// head by gdn_block_prep in fp32, four warps per block of tokens, and left as a record. Value columns never mix, so the
// walk runs on B * H * D / 16 CTAs of 16 columns whose four warps share the key rows.
//
// The products of the walk are warp-level matrix instructions on tf32 numbers with fp32 sums, each operand as the sum of two:
// x = hi + lo keeps 22 to 24 bits, hi hi + hi lo + lo hi leaves 2^-23 of a product. The instruction cuts its sums off towards zero, so
// nothing that lasts is summed up in it: the state, the value minus what the state holds for it, and the 1 in T are added outside, in fp32, and
// the later eight tokens of a block, of which a short memory consists, reach the state by fp32 multiply-adds. Relative error of the state
// against 64 bits after 8192 tokens, 16 heads of 128, gate logits around 0, 2, 4, 8, 10, 14: eight tokens a round in fp32 multiply-adds 9.0e-8,
// 1.4e-7, 5.8e-7, 1.4e-6, 3.0e-6, 6.4e-6; here 7.4e-8, 1.4e-7, 2.0e-7, 4.1e-7, 1.1e-6, 6.8e-7; all in the instruction 1.4e-7, 1.9e-7, 4.3e-7,
// 1.1e-5, 1.6e-5, 9.9e-6 (926 instead of 987 us). After 2048 tokens, token by token: 7.0e-8, 1.1e-7, 5.5e-7, 1.3e-6, 8.1e-7, 5.8e-6.
// The state is held transposed: the fragment that the update leaves it in is the operand that the next round's contraction takes it from,
// the order of key rows within an instruction being free. Rows of a record are padded so that its fragments are read without bank conflicts.
//
// The launch that walks a segment of tokens also forms the next one's records, in CTAs behind its own. A block's outputs wait for the next
// round's barrier, so that there is one barrier a round. Bound by the issue slots of one warp per scheduler (69 matrix
// instructions of 12 clocks and some 800 others a round of 128-wide heads; eight warps a CTA repeat more than they hide: a ninth slower).
// Whole calls, eight tokens a round in fp32 multiply-adds -> here: one sequence of 8192 tokens, 16 heads of 128, 1229 -> 987 us
// (9010 token by token); 6 heads of 64 1034 -> 546; four sequences of 16384, 6 heads of 64 2162 -> 1136; 4 x 512, 16 heads of 128 279 -> 231;
// see gdn_in_blocks for the sizes that take it.
// ------------------------------------------------------------------------------------------------
constexpr int GB = 16;  // tokens per block
template <int D>
struct GdnRec {  // floats of a record: k P and q P [32][PK] | (beta k) dec [16][PE] | T - 1 [16][PT] | A [16][PT] | P_15 [D] | v bf16 [D][24]
  static constexpr int PK = D + 8, PE = D + 4, PT = 24, PV = 12;
  static constexpr int E = 2 * GB * PK, TRI = E + GB * PE, A = TRI + GB * PT, P = A + GB * PT, COMMON = P + D, FLOATS = COMMON + D * PV;
  static_assert(COMMON % 4 == 0 && PV % 4 == 0, "records are copied in 16-byte words");
};

// e^gdn_log_decay: a sigmoid where the gates are logits. Near 1, where errors add up over a long memory, it is formed from its distance to 1,
// so that only the last subtraction rounds.
__device__ __forceinline__ float gdn_decay(float x, bool logits) {
  if (!logits) return __expf(gdn_log_decay(x, false));
  const float e = __expf(-fabsf(x)), small = __fdividef(e, 1.f + e);
  return fmaxf(x > 0.f ? 1.f - small : small, GLA_MIN_DECAY);
}

// Sum of v[l] over the lanes, in lane l.
__device__ __forceinline__ float reduce_scatter32(float (&v)[32], int lane) {
  int n = 16;
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1, n >>= 1) {
    const bool up = (lane & s) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
  return v[0];
}

template <int N>
__device__ __forceinline__ void load_bf16_row(const __nv_bfloat16* p, uint32_t (&w)[N / 2]) {
  if constexpr (N == 4) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    w[0] = x.x;
    w[1] = x.y;
  } else {
    w[0] = *reinterpret_cast<const uint32_t*>(p);
  }
}
template <int N>
__device__ __forceinline__ void unpack_bf16(const uint32_t (&w)[N / 2], float (&f)[N]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

template <int N>
__device__ __forceinline__ void store_rec(float* p, const float (&f)[N]) {
  if constexpr (N == 4)
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  else
    *reinterpret_cast<float2*>(p) = make_float2(f[0], f[1]);
}
template <int N>
__device__ __forceinline__ void load_rec(const float* p, float (&f)[N]) {
  if constexpr (N == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
  } else {
    const float2 v = *reinterpret_cast<const float2*>(p);
    f[0] = v.x, f[1] = v.y;
  }
}

template <int D>
struct GdnPrepShared {
  float dec[GB][D];
  __nv_bfloat16 k[GB][D], q[GB][D];
  uint32_t v[D][GdnRec<D>::PV];  // pairs of tokens
  float L[GB][GB + 1], beta[GB];
};

struct GdnBlockArgs {
  const __nv_bfloat16 *q, *k, *v, *g;
  long long q_ld, k_ld, v_ld, g_ld, o_ld;
  int qcol, kcol, vcol, gcol, ocol;
  const float* beta;
  int beta_mode;
  float* state;
  __nv_bfloat16* out;
  int T, H, logits;
  float scale;
  int* status;
};

// Record `index` of [B * H, ceil(nt / GB)] for tokens [t0, t0 + nt) of every sequence, by a CTA of four warps. A warp carries the vectors
// of two tokens forward at a time, so that the later tokens' rows are read and unpacked half as often, and takes an early and a late pair.
template <int D>
__device__ __forceinline__ void gdn_block_prep(const GdnBlockArgs& a, GdnPrepShared<D>& sh, float* rec, int t0, int nt, int index) {
  const __nv_bfloat16 *q = a.q, *k = a.k, *v = a.v, *g = a.g;
  const long long q_ld = a.q_ld, k_ld = a.k_ld, v_ld = a.v_ld, g_ld = a.g_ld;
  const int qcol = a.qcol, kcol = a.kcol, vcol = a.vcol, gcol = a.gcol, beta_mode = a.beta_mode, T = a.T, H = a.H, logits = a.logits;
  const float* beta = a.beta;
  constexpr int N = D / 32;
  using R = GdnRec<D>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = (nt + GB - 1) / GB, bh = index / nb, blk = index % nb, h = bh % H;
  const long long row0 = (long long)(bh / H) * T + t0 + blk * GB;
  const int left = nt - blk * GB;
  float* out = rec + (long long)index * R::FLOATS;
#pragma unroll
  for (int i = tid; i < GB * (D / 4); i += 128) {  // eight bytes at a time: rows start on 8-byte boundaries
    const int j = i / (D / 4), c = (i % (D / 4)) * 4;
    const bool ok = j < left;
    const long long r = row0 + j;
    const uint2 zero = make_uint2(0u, 0u);
    *reinterpret_cast<uint2*>(&sh.k[j][c]) = ok ? *reinterpret_cast<const uint2*>(k + r * k_ld + kcol + h * D + c) : zero;
    *reinterpret_cast<uint2*>(&sh.q[j][c]) = ok ? *reinterpret_cast<const uint2*>(q + r * q_ld + qcol + h * D + c) : zero;
    const uint2 gw = ok ? *reinterpret_cast<const uint2*>(g + r * g_ld + gcol + h * D + c) : zero;
    const float x[4] = {__uint_as_float(gw.x << 16), __uint_as_float(gw.x & 0xffff0000u), __uint_as_float(gw.y << 16), __uint_as_float(gw.y & 0xffff0000u)};
    float f[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) f[n] = ok ? gdn_decay(x[n], logits != 0) : 1.f;
    *reinterpret_cast<float4*>(&sh.dec[j][c]) = make_float4(f[0], f[1], f[2], f[3]);
    const uint2 vw = ok ? *reinterpret_cast<const uint2*>(v + r * v_ld + vcol + h * D + c) : zero;
    unsigned short* vt = reinterpret_cast<unsigned short*>(sh.v[c]) + j;
    vt[0] = (unsigned short)vw.x, vt[2 * R::PV] = (unsigned short)(vw.x >> 16);
    vt[4 * R::PV] = (unsigned short)vw.y, vt[6 * R::PV] = (unsigned short)(vw.y >> 16);
  }
  if (tid < GB) sh.beta[tid] = (tid < left && beta_mode == 1) ? beta[(row0 + tid) * H + h] : 1.f;
  __syncthreads();
  for (int i = tid; i < D * 2; i += 128)  // sixteen values of a column: two 16-byte words
    *reinterpret_cast<uint4*>(out + R::COMMON + (i >> 1) * R::PV + (i & 1) * 4) = *reinterpret_cast<const uint4*>(&sh.v[i >> 1][(i & 1) * 4]);
  if (tid < D) {  // k_j P_{j-1}, q_j P_j; tokens past the end write nothing and leave the state as it is
    double p = 1.;  // products of numbers a few units below 1 all round to the same side in fp32
#pragma unroll
    for (int j = 0; j < GB; ++j) {
      out[j * R::PK + tid] = __bfloat162float(sh.k[j][tid]) * (float)p;
      p *= sh.dec[j][tid];
      out[(GB + j) * R::PK + tid] = __bfloat162float(sh.q[j][tid]) * (float)p;
    }
    out[R::P + tid] = (float)p;
  }
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const int i = half == 0 ? 2 * warp : GB - 2 - 2 * warp;  // w: (beta k)_i and (beta k)_{i+1} carried forward through the later decays
    float w[2][N], sums[2][2 * GB];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int n = 0; n < N; ++n)
        w[e][n] = __bfloat162float(sh.k[i + e][lane * N + n]) *
                  ((beta_mode == 2 && i + e < left) ? beta[(row0 + i + e) * H * D + h * D + lane * N + n] : sh.beta[i + e]);
#pragma unroll
      for (int j = 0; j < 2 * GB; ++j) sums[e][j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < GB; ++j) {
      if (j >= i) {  // the same for all lanes
        uint32_t kw[N / 2], qw[N / 2];
        float kf[N], qf[N], dec[N];
        load_bf16_row<N>(&sh.k[j][lane * N], kw);
        load_bf16_row<N>(&sh.q[j][lane * N], qw);
        unpack_bf16<N>(kw, kf);
        unpack_bf16<N>(qw, qf);
        load_rec<N>(&sh.dec[j][lane * N], dec);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (j > i + e) {
#pragma unroll
            for (int n = 0; n < N; ++n) {
              sums[e][j] += kf[n] * w[e][n];
              w[e][n] *= dec[n];
            }
          }
          if (j >= i + e) {
#pragma unroll
            for (int n = 0; n < N; ++n) sums[e][GB + j] += qf[n] * w[e][n];
          }
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      store_rec<N>(out + R::E + (i + e) * R::PE + lane * N, w[e]);
      const float v = reduce_scatter32(sums[e], lane);  // lanes 0..15: L[j = lane][i + e] (zero for i + e >= j), 16..31: A[j][i + e]
      if (lane < GB) sh.L[lane][i + e] = v;
      else out[R::A + (lane - GB) * R::PT + i + e] = v;
    }
  }
  __syncthreads();
  if (tid < GB) {  // column `tid` of (1 + L)^-1 - 1
    float t[GB];
#pragma unroll
    for (int i = 0; i < GB; ++i) {
      t[i] = i == tid ? 1.f : 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) t[i] -= sh.L[i][m] * t[m];
      out[R::TRI + i * R::PT + tid] = i == tid ? t[i] - 1.f : t[i];
    }
  }
}

constexpr int GDN_COLS = 16;  // value columns per CTA
constexpr int GDN_STAGES = 3;

struct Split {
  uint32_t hi, lo;
};
__device__ __forceinline__ Split split_tf32(float x) {
  Split s;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(s.hi) : "f"(x));
  s.lo = __float_as_uint(x - __uint_as_float(s.hi));
  return s;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// An accumulator tile (16 value columns x 8) as the operand of the next product: its columns 2 t and 2 t + 1 are k = t and t + 4.
__device__ __forceinline__ void operand(const float (&c)[4], Split (&v)[4]) {
  v[0] = split_tf32(c[0]), v[1] = split_tf32(c[2]), v[2] = split_tf32(c[1]), v[3] = split_tf32(c[3]);
}
// An instruction cuts off what is below the last bit of its largest term, always towards zero. So the small products of a sum are added up by
// themselves, the large ones in as few instructions as there are, and what has been summed up before is added in fp32.
struct Sum {
  float large[4], small[4];
  __device__ __forceinline__ Sum() {
#pragma unroll
    for (int i = 0; i < 4; ++i) large[i] = small[i] = 0.f;
  }
  __device__ __forceinline__ void multiply(const Split (&a)[4], float b0, float b1) {
    const Split x = split_tf32(b0), y = split_tf32(b1);
    mma_tf32(small, a[0].lo, a[1].lo, a[2].lo, a[3].lo, x.hi, y.hi);
    mma_tf32(small, a[0].hi, a[1].hi, a[2].hi, a[3].hi, x.lo, y.lo);
    mma_tf32(large, a[0].hi, a[1].hi, a[2].hi, a[3].hi, x.hi, y.hi);
  }
  __device__ __forceinline__ float operator[](int i) const { return large[i] + small[i]; }
};

template <int D>
struct GdnWalkShared {
  float stage[GDN_STAGES][GdnRec<D>::COMMON + GDN_COLS * GdnRec<D>::PV];
  float4 red[2][2][4][2][32];  // partial sums of the four warps, of alternating blocks: k P rows, q P rows
  uint64_t full[GDN_STAGES];
  int odd;                  // first token of a block at which something is no number
};

// One CTA's columns. A lane (g, t) = (lane / 4, lane % 4) of warp w holds the state of columns g, g + 8 and key rows w D / 4 + 8 n + 2 t + {0, 1}.
template <int D>
struct GdnWalk {
  static constexpr int NT = D / 32;  // tiles of eight key rows of a warp
  using R = GdnRec<D>;
  const GdnBlockArgs& a;
  GdnWalkShared<D>& sh;
  const float* const rec;
  const int nt, tid, lane, warp, g, t, bh, h, c0, nb;
  const long long row0;
  float S[NT][4];

  __device__ __forceinline__ GdnWalk(const GdnBlockArgs& a_, GdnWalkShared<D>& sh_, const float* rec_, int t0, int nt_)
      : a(a_), sh(sh_), rec(rec_), nt(nt_), tid(threadIdx.x), lane(threadIdx.x & 31), warp(threadIdx.x >> 5), g(lane >> 2), t(lane & 3), bh(blockIdx.x / (D / GDN_COLS)),
        h(bh % a_.H), c0((blockIdx.x % (D / GDN_COLS)) * GDN_COLS), nb((nt_ + GB - 1) / GB), row0((long long)(bh / a_.H) * a_.T + t0) {}

  __device__ __forceinline__ float* state_at(int n, int i) const {  // of S[n][i]
    return a.state + ((long long)bh * D + warp * (D / 4) + n * 8 + 2 * t + (i & 1)) * D + c0 + g + (i >> 1) * 8;
  }
  __device__ __forceinline__ void load_state() {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) S[n][i] = *state_at(n, i);
  }
  __device__ __forceinline__ void store_state() const {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) *state_at(n, i) = S[n][i];
  }
  __device__ __forceinline__ void start() {
    if (tid == 0) {
      for (int i = 0; i < GDN_STAGES; ++i) mbar_init(&sh.full[i], 1);
      mbar_fence_init();
    }
    __syncthreads();
  }
  // A block's record without the other CTAs' columns, by thread 0.
  __device__ __forceinline__ void fetch(int blk) {
    if (tid == 0 && blk < nb) {
      const float* from = rec + ((long long)bh * nb + blk) * R::FLOATS;
      float* to = sh.stage[blk % GDN_STAGES];
      uint64_t* bar = &sh.full[blk % GDN_STAGES];
      constexpr uint32_t common = R::COMMON * 4, columns = GDN_COLS * R::PV * 4;
      mbar_expect_tx(bar, common + columns);
      copy(to, from, common, bar);
      copy(to + R::COMMON, from + R::COMMON + c0 * R::PV, columns, bar);
    }
  }
  __device__ __forceinline__ static void copy(float* to, const float* from, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(to)), "l"(from), "r"(bytes),
                 "r"(smem_u32(bar))
                 : "memory");
  }
  // False where it never arrived. `nth`: how many records this stage held before this one.
  __device__ __forceinline__ bool landed(int blk, int nth) { return mbar_wait(&sh.full[blk % GDN_STAGES], nth & 1); }
  // Values of tokens 8 e + 2 t, 8 e + 2 t + 1 of columns g, then of g + 8.
  __device__ __forceinline__ void values(const float* r, int e, float (&f)[4]) const {
    const uint32_t lo = __float_as_uint(r[R::COMMON + g * R::PV + 4 * e + t]), hi = __float_as_uint(r[R::COMMON + (g + 8) * R::PV + 4 * e + t]);
    f[0] = __uint_as_float(lo << 16), f[1] = __uint_as_float(lo & 0xffff0000u);
    f[2] = __uint_as_float(hi << 16), f[3] = __uint_as_float(hi & 0xffff0000u);
  }

  __device__ __forceinline__ void leave(int buf, int part, const Sum& f, const Sum& s) const {
    sh.red[buf][part][warp][0][lane] = make_float4(f[0], f[1], f[2], f[3]);
    sh.red[buf][part][warp][1][lane] = make_float4(s[0], s[1], s[2], s[3]);
  }
  __device__ __forceinline__ void total(int buf, int part, int e, float (&s)[4]) const {
    s[0] = s[1] = s[2] = s[3] = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float4 f = sh.red[buf][part][w][e][lane];
      s[0] += f.x, s[1] += f.y, s[2] += f.z, s[3] += f.w;
    }
  }
  __device__ __forceinline__ bool put(const float (&o)[4], int blk, int e, int limit) const {  // outputs of tokens 8 e + 2 t + {0, 1}
    const int tok = 8 * e + 2 * t, left = min(limit, nt - blk * GB);
    __nv_bfloat16* to = a.out + (row0 + blk * GB + tok) * a.o_ld + (a.ocol + h * D + c0 + g);
    if (tok < left) to[0] = __float2bfloat16(o[0] * a.scale), to[8] = __float2bfloat16(o[2] * a.scale);
    if (tok + 1 < left) to[a.o_ld] = __float2bfloat16(o[1] * a.scale), to[a.o_ld + 8] = __float2bfloat16(o[3] * a.scale);
    return (tok < left && !(fmaxf(fabsf(o[0]), fabsf(o[2])) < INFINITY && o[0] == o[0] && o[2] == o[2])) ||
           (tok + 1 < left && !(fmaxf(fabsf(o[1]), fabsf(o[3])) < INFINITY && o[1] == o[1] && o[3] == o[3]));
  }

  // u of tokens 8 to 15, of columns g and g + 8
  __device__ __forceinline__ void gather(const float (&u1)[4], float (&v)[8][2]) const {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) v[2 * n + (i & 1)][i >> 1] = __shfl_sync(0xffffffffu, u1[i], (lane & ~3) | n);
  }
  // S of eight key rows <- P_15 S + sum_j (beta k_j dec_{j+1..15}) u_j^T. The later eight tokens, of which a short memory consists, in fp32.
  __device__ __forceinline__ void advance(const float* r, int n, const Split (&u0)[4], const float (&v)[8][2]) {
    const int d = warp * (D / 4) + 8 * n;
    const float2 p = *reinterpret_cast<const float2*>(r + R::P + d + 2 * t);
    const float* e = r + R::E + 2 * t * R::PE + d + g;
    Sum early;
    early.multiply(u0, e[0], e[R::PE]);
    float add[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) add[i] = early[i];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 w = *reinterpret_cast<const float2*>(r + R::E + (8 + j) * R::PE + d + 2 * t);
      add[0] = __fmaf_rn(w.x, v[j][0], add[0]), add[1] = __fmaf_rn(w.y, v[j][0], add[1]);
      add[2] = __fmaf_rn(w.x, v[j][1], add[2]), add[3] = __fmaf_rn(w.y, v[j][1], add[3]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) S[n][i] = __fmaf_rn(S[n][i], (i & 1) ? p.y : p.x, add[i]);
  }
  // o plus what the tokens of the block itself add to outputs of eight of them: `a0`, `a1` their rows of A
  __device__ __forceinline__ void add_block(float (&o)[4], int e, const Split (&u0)[4], const Split (&u1)[4], float2 a0, float2 a1) const {
    Sum sum;
    sum.multiply(u0, a0.x, a0.y);
    if (e == 1) sum.multiply(u1, a1.x, a1.y);
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] += sum[i];
  }

  // A block's round, its record in `r`: outputs of its tokens before `limit`, and the state after all of them. Tokens from
  // `limit` on count as nothing (LIMIT), as they are behind a token that is no number. True where an output is no number.
  template <bool LIMIT>
  __device__ __forceinline__ bool round(const float* r, int blk, int limit) {
    Sum acc[4];  // [16 columns] x [k P of tokens 0-7, 8-15 | q P of tokens 0-7, 8-15], of this warp's key rows
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      Split s[4];
      operand(S[n], s);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 b = *reinterpret_cast<const float2*>(r + (8 * j + g) * R::PK + warp * (D / 4) + 8 * n + 2 * t);
        acc[j].multiply(s, b.x, b.y);
      }
    }
    const int buf = blk & 1;
    leave(buf, 0, acc[0], acc[1]);
    leave(buf, 1, acc[2], acc[3]);
    __syncthreads();  // and every warp is done with the block before
    float x[2][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float f[4];
      values(r, e, f);
      total(buf, 0, e, x[e]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[e][i] = f[i] - x[e][i];
        if (LIMIT && 8 * e + 2 * t + (i & 1) >= limit) x[e][i] = 0.f;
      }
    }
    float u[2][4];
    {
      Split x0[4], x1[4];
      operand(x[0], x0);
      operand(x[1], x1);
      const float* tri = r + R::TRI + 2 * t;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        Sum sum;
        const float2 b0 = *reinterpret_cast<const float2*>(tri + (8 * e + g) * R::PT);
        sum.multiply(x0, b0.x, b0.y);
        if (e == 1) {
          const float2 b1 = *reinterpret_cast<const float2*>(tri + (8 + g) * R::PT + 8);
          sum.multiply(x1, b1.x, b1.y);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) u[e][i] = LIMIT && 8 * e + 2 * t + (i & 1) >= limit ? 0.f : x[e][i] + sum[i];
      }
    }
    Split u0[4], u1[4];
    operand(u[0], u0);
    operand(u[1], u1);
    float after[8][2];
    gather(u[1], after);
#pragma unroll
    for (int n = 0; n < NT; ++n) advance(r, n, u0, after);
    bool odd = false;
    if (warp < 2) {  // outputs of tokens 8 warp + ...
      float o[4];
      total(buf, 1, warp, o);
      const float* tri = r + R::A + (8 * warp + g) * R::PT + 2 * t;
      add_block(o, warp, u0, u1, *reinterpret_cast<const float2*>(tri), *reinterpret_cast<const float2*>(tri + 8));
      odd = put(o, blk, warp, limit);
    }
    return odd;
  }

  __device__ __forceinline__ bool state_odd() const {
    bool odd = false;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) odd |= !(fabsf(S[n][i]) < INFINITY);
    return odd;
  }

  // How a walk ended, for all threads: fine; with an output or the state no number, or with a record that came late: to be walked again; with
  // a record that still had not landed, so that its stage may not be used for anything else.
  enum End { FINE, AGAIN, LOST };

  // The whole segment. The state in memory is as it was. The rounds
  // are those of round(), in another order: a block's outputs wait for the next round's barrier, so that there is one barrier a
  // round, and what they need from the state is multiplied while the triangle's short chain runs.
  __device__ __forceinline__ End walk() {
    start();
    fetch(0);
    fetch(1);
    int issued = min(nb, 2);  // records on their way or there, as thread 0 counts them
    load_state();
    bool odd = false, late = !landed(0, 0);
    int at = 0, lap = 0;      // stage of the block, records that it held before
    Split u0[4], u1[4];       // of the block before
    float2 a0, a1;            // its row of A
    a0 = a1 = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) u0[i] = u1[i] = Split{0u, 0u};
    auto outputs = [&](int blk) {  // of a block whose sums all warps have left
      const int e = warp & 1;
      if ((warp >> 1) == (blk & 1)) {
        float o[4];
        total(blk & 1, 1, e, o);
        add_block(o, e, u0, u1, a0, a1);
        odd |= put(o, blk, e, GB);
      }
    };
    for (int blk = 0; blk < nb; ++blk) {
      const float* r = sh.stage[at];
      const int buf = blk & 1;
      Split s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) operand(S[n], s[n]);
      Sum kp[2];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 b = *reinterpret_cast<const float2*>(r + (8 * j + g) * R::PK + warp * (D / 4) + 8 * n + 2 * t);
          kp[j].multiply(s[n], b.x, b.y);
        }
      leave(buf, 0, kp[0], kp[1]);
      __syncthreads();  // all warps' sums; the record of the block before has been read
      if (!late && blk + 2 < nb) fetch(blk + 2), issued = blk + 3;  // in its place
      if (blk > 0) outputs(blk - 1);
      float x[2][4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float f[4];
        values(r, e, f);
        total(buf, 0, e, x[e]);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[e][i] = f[i] - x[e][i];
      }
      float u[2][4];
      Sum qp[2];
      {
        Split x0[4], x1[4];
        operand(x[0], x0);
        operand(x[1], x1);
        const float* tri = r + R::TRI + g * R::PT + 2 * t;
        const float2 b0 = *reinterpret_cast<const float2*>(tri), b1 = *reinterpret_cast<const float2*>(tri + 8 * R::PT),
                     b2 = *reinterpret_cast<const float2*>(tri + 8 * R::PT + 8);
        Sum sum[2];
        sum[0].multiply(x0, b0.x, b0.y);
        sum[1].multiply(x0, b1.x, b1.y);
        sum[1].multiply(x1, b2.x, b2.y);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) u[e][i] = x[e][i] + sum[e][i];
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 b = *reinterpret_cast<const float2*>(r + (GB + 8 * j + g) * R::PK + warp * (D / 4) + 8 * n + 2 * t);
          qp[j].multiply(s[n], b.x, b.y);
        }
      leave(buf, 1, qp[0], qp[1]);
      operand(u[0], u0);
      operand(u[1], u1);
      a0 = *reinterpret_cast<const float2*>(r + R::A + (8 * (warp & 1) + g) * R::PT + 2 * t);
      a1 = *reinterpret_cast<const float2*>(r + R::A + (8 * (warp & 1) + g) * R::PT + 2 * t + 8);
      float after[8][2];
      gather(u[1], after);
#pragma unroll
      for (int n = 0; n < NT; ++n) advance(r, n, u0, after);
      if (++at == GDN_STAGES) at = 0, ++lap;
      if (blk + 1 < nb && !late) late = !landed(blk + 1, lap);  // what did not arrive is read as it is, and walked again
    }
    __syncthreads();
    if (nb > 0) outputs(nb - 1);
    if (!__syncthreads_or(odd || late || state_odd())) return FINE;
    // nothing else goes into a stage, and nothing leaves, while a copy into it is in flight
    bool lost = false;
    if (tid == 0 && late)
      for (int b = max(0, issued - GDN_STAGES); b < issued; ++b) lost |= !landed(b, b / GDN_STAGES);
    return __syncthreads_or(lost) ? LOST : AGAIN;
  }

  // The same where something is no number. A later token of a block enters an earlier one's sums times a zero of a triangle, which
  // is nothing unless it is infinite or no number, and an operand of two parts does not carry an infinity. So: rounds up to the block at
  // which something turns up, of that block the tokens before it, and then token by token as the recurrence says.
  __device__ void walk_again() {
    load_state();
    for (int blk = 0; blk < nb; ++blk) {
      __syncthreads();
      if (tid == 0) sh.odd = GB;
      float* r = sh.stage[0];
      const float* src = rec + ((long long)bh * nb + blk) * R::FLOATS;
      for (int i = tid; i < R::COMMON + GDN_COLS * R::PV; i += 128) r[i] = src[i < R::COMMON ? i : i + c0 * R::PV];
      __syncthreads();
      // the first token with a part that is no number
      int first = GB;
      for (int i = tid; i < GB * D; i += 128) {
        const int tok = i / D, d = i % D;
        const bool bad = !(fabsf(r[tok * R::PK + d]) < INFINITY) || !(fabsf(r[(GB + tok) * R::PK + d]) < INFINITY) ||
                         !(fabsf(r[R::E + tok * R::PE + d]) < INFINITY);
        if (bad) first = min(first, tok);
      }
      for (int i = tid; i < GB * GB; i += 128) {
        const int tok = i / GB, m = i % GB;
        if (!(fabsf(r[R::TRI + tok * R::PT + m]) < INFINITY) || !(fabsf(r[R::A + tok * R::PT + m]) < INFINITY)) first = min(first, tok);
      }
      for (int i = tid; i < D; i += 128)
        if (!(fabsf(r[R::P + i]) < INFINITY)) first = min(first, GB - 1);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float f[4];
        values(r, e, f);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (!(fabsf(f[i]) < INFINITY)) first = min(first, 8 * e + 2 * t + (i & 1));
      }
      if (first < GB) atomicMin(&sh.odd, first);
      __syncthreads();
      int limit = sh.odd;
      float kept[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) kept[n][i] = S[n][i];
      bool stop = limit < GB;
      if (stop) {
        // vectors of the tokens from `limit` on must not meet the zeros either
        for (int i = tid; i < GB * D; i += 128) {
          const int tok = i / D, d = i % D;
          if (tok >= limit) r[tok * R::PK + d] = r[(GB + tok) * R::PK + d] = r[R::E + tok * R::PE + d] = 0.f;
        }
        for (int i = tid; i < GB * GB; i += 128) {
          const int tok = i / GB, m = i % GB;
          if (tok >= limit || m >= limit) r[R::TRI + tok * R::PT + m] = r[R::A + tok * R::PT + m] = 0.f;
        }
        __syncthreads();
        if (__syncthreads_or(round<true>(r, blk, limit))) limit = 0;  // too large for a sum already
      } else {
        stop = __syncthreads_or(round<false>(r, blk, GB) || state_odd());
      }
      if (stop) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) S[n][i] = kept[n][i];
        tokens(blk * GB, blk * GB + (limit < GB ? limit : 0));  // what overflows is as the token kernel has it
        return;
      }
    }
    store_state();
  }

  // Token by token from `from` on; outputs from token `first` on. The state goes through shared memory: thread (p, c) has D / 8 rows of column c.
  __device__ void tokens(int from, int first) {
    constexpr int RP = D / 8;
    __syncthreads();
    float* Sm = sh.stage[0];                    // [D][16]
    float *kr = Sm + D * GDN_COLS, *kb = kr + D, *qr = kb + D, *dec = qr + D;
    float* part = dec + D;                      // [2][8][16]
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) Sm[(warp * (D / 4) + n * 8 + 2 * t + (i & 1)) * GDN_COLS + g + (i >> 1) * 8] = S[n][i];
    __syncthreads();
    const int c = tid % GDN_COLS, p = tid / GDN_COLS;
    float st[RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) st[i] = Sm[(p * RP + i) * GDN_COLS + c];
    for (int tok = from; tok < nt; ++tok) {
      const long long row = row0 + tok;
      __syncthreads();
      for (int d = tid; d < D; d += 128) {
        const float kk = __bfloat162float(a.k[row * a.k_ld + a.kcol + h * D + d]);
        const float b = a.beta_mode == 0 ? 1.f : a.beta_mode == 1 ? a.beta[row * a.H + h] : a.beta[(row * a.H + h) * D + d];
        kr[d] = kk;
        kb[d] = b * kk;
        qr[d] = __bfloat162float(a.q[row * a.q_ld + a.qcol + h * D + d]);
        dec[d] = __expf(gdn_log_decay(__bfloat162float(a.g[row * a.g_ld + a.gcol + h * D + d]), a.logits != 0));
      }
      __syncthreads();
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < RP; ++i) acc += kr[p * RP + i] * st[i];
      part[p * GDN_COLS + c] = acc;
      __syncthreads();
      float u = __bfloat162float(a.v[row * a.v_ld + a.vcol + h * D + c0 + c]), o = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) u -= part[i * GDN_COLS + c];
#pragma unroll
      for (int i = 0; i < RP; ++i) {
        st[i] = dec[p * RP + i] * st[i] + kb[p * RP + i] * u;
        o += qr[p * RP + i] * st[i];
      }
      part[(8 + p) * GDN_COLS + c] = o;
      __syncthreads();
      if (p == 0 && tok >= first) {
        o = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) o += part[(8 + i) * GDN_COLS + c];
        a.out[row * a.o_ld + a.ocol + h * D + c0 + c] = __float2bfloat16(o * a.scale);
      }
    }
#pragma unroll
    for (int i = 0; i < RP; ++i) a.state[((long long)bh * D + p * RP + i) * D + c0 + c] = st[i];
  }
};

// In a function of its own, so that its registers are not the common walk's.
template <int D>
__device__ __noinline__ void gdn_walk_again(const GdnBlockArgs& a, GdnWalkShared<D>& sh, const float* rec, int t0, int nt) {
  GdnWalk<D> w(a, sh, rec, t0, nt);
  w.walk_again();
}

// The first `walks` CTAs walk tokens [t0, t0 + nt) by the records in `rec`; the others form those of the tokens after them, of which there
// are `next_nt`, in `next_rec`, on the SMs and issue slots that the walk leaves free.
template <int D>
__global__ void __launch_bounds__(128) gdn_block_kernel(const __grid_constant__ GdnBlockArgs a, int walks, const float* rec, int t0, int nt,
                                                        float* next_rec, int next_nt) {
  extern __shared__ __align__(16) uint8_t block_smem[];
  if ((int)blockIdx.x >= walks) {
    if (walks == 0 && blockIdx.x == 0 && threadIdx.x == 0) *a.status = ST_OK;  // the first launch, which walks nothing
    gdn_block_prep<D>(a, *reinterpret_cast<GdnPrepShared<D>*>(block_smem), next_rec, t0 + nt, next_nt, (int)blockIdx.x - walks);
    return;
  }
  GdnWalkShared<D>& sh = *reinterpret_cast<GdnWalkShared<D>*>(block_smem);
  GdnWalk<D> w(a, sh, rec, t0, nt);
  const typename GdnWalk<D>::End end = w.walk();
  if (end == GdnWalk<D>::FINE) w.store_state();
  else if (end == GdnWalk<D>::AGAIN) gdn_walk_again<D>(a, sh, rec, t0, nt);
  else if (threadIdx.x == 0) *a.status = ST_TIMEOUT_FULL;
}

template <int D>
void run_blocks(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta, int beta_mode, float* state,
                const GlaMat& O, int B, int T, int H, bool logits, float scale, float* rec, int* status, int seg, cudaStream_t s) {
  auto p = [](const GlaMat& m) { return reinterpret_cast<const __nv_bfloat16*>(m.ptr); };
  constexpr int walk_smem = (int)sizeof(GdnWalkShared<D>), prep_smem = (int)sizeof(GdnPrepShared<D>);
  static PerDeviceOnce once;
  if (once.first_use()) {
    const cudaError_t e = cudaFuncSetAttribute(gdn_block_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, walk_smem);
    if (e != cudaSuccess) throw std::runtime_error(std::string("gdn_blocks attribute: ") + cudaGetErrorString(e));
  }
  const GdnBlockArgs a{p(Q), p(K), p(V), p(G), Q.ld, K.ld, V.ld, G.ld, O.ld, Q.col0, K.col0, V.col0, G.col0, O.col0, beta, beta_mode, state,
                       reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(O.ptr)), T, H, logits ? 1 : 0, scale, status};
  auto tokens = [&](int t0) { return T - t0 < seg ? T - t0 : seg; };
  auto records = [&](int nt) { return B * H * ((nt + GB - 1) / GB); };
  float* half[2] = {rec, rec + (long long)records(tokens(0)) * GdnRec<D>::FLOATS};
  gdn_block_kernel<D><<<records(tokens(0)), 128, prep_smem, s>>>(a, 0, nullptr, 0, 0, half[0], tokens(0));
  for (int t0 = 0, i = 0; t0 < T; t0 += seg, ++i) {
    const int nt = tokens(t0), after = t0 + nt < T ? tokens(t0 + nt) : 0, walks = B * H * (D / GDN_COLS);
    gdn_block_kernel<D><<<walks + records(after), 128, walk_smem, s>>>(a, walks, half[i & 1], t0, nt, half[~i & 1], after);
  }
}

constexpr int rec_floats(int D) { return D == 64 ? GdnRec<64>::FLOATS : GdnRec<128>::FLOATS; }

// Tokens per segment: whole blocks whose records (36 KB for heads of 128, 20 KB for 64) fill at most 40 MB, so that with the next segment's
// they are read back from the 126 MB L2, but at least 128 tokens, so that the launch of a segment stays small beside its walk (256 heads of
// 128, 512 tokens: 702 us, and 806 with 64). Above 147 heads of 128 or 262 of 64 the second rule holds and records come from
// memory in part: 512 heads of 128 have 146 MB a segment, 291 MB with the next one's.
int segment_tokens(int BH, int D) {
  const long long blocks = (40ll << 20) / ((long long)BH * rec_floats(D) * 4);
  return (int)(blocks < 8 ? 8 : blocks) * GB;
}

}  // namespace

// Sixteen tokens a round win where the recurrence is a chain that the chip waits for: the walk's work grows with the heads, the token
// kernel's time hardly does until its CTAs fill the SMs, and a round costs the same for one token as for sixteen. Token kernel -> blocks, us:
// heads of 64: 16 heads, 8 tokens 7.1 -> 8.0, 12 tokens 9.5 -> 8.3, 512 tokens 315 -> 39; 128 heads, 17 tokens 13 -> 15, 24 tokens 17 -> 15; 256
// heads, 24 tokens 20 -> 21, 32 tokens 26 -> 22; 384 heads, 32 tokens 30 -> 31, 130 tokens 115 -> 116, 512 tokens 449 -> 420; 512 heads, 32
// tokens 36 -> 36, 130 tokens 137 -> 150, 512 tokens 533 -> 534.
// Heads of 128: 16 heads, 4 tokens 7.4 -> 9.8, 8 tokens 11.5 -> 10.7; 64 heads, 8 tokens 11.7 -> 14.4, 12 tokens 16.1 -> 15.5; 128 heads, 24
// tokens 28.7 -> 29.6, 32 tokens 38 -> 30; 512 heads, 24 tokens 85 -> 93, 32 tokens 111 -> 100, 512 tokens 1676 -> 1433. More than 512 heads
// would take more than 291 MB of records.
static bool gdn_in_blocks(long long heads, int T, int D) {
  if (D != 64 && D != 128) return false;
  const int least = D == 128 && heads <= 16 ? 8 : heads <= 64 ? 12 : heads <= 128 ? (D == 128 ? 26 : 24) : 32;
  return heads <= (D == 128 ? 512 : 384) && T >= least;
}

long long gdn_block_workspace_floats(int B, int T, int H, int D) {
  if (!gdn_in_blocks((long long)B * H, T, D)) return 0;
  const int seg = segment_tokens(B * H, D), nt = T < seg ? T : seg;
  return (long long)B * H * ((nt + GB - 1) / GB) * rec_floats(D) * (T > seg ? 2 : 1);
}

void launch_gdn_blocks(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta, int beta_mode,
                       float* state, const GlaMat& O, int B, int T, int H, int D, bool logits, float scale, float* workspace,
                       int* status, cudaStream_t s) {
  if (B <= 0 || T <= 0) return;
  const int seg = segment_tokens(B * H, D);
  if (D == 64)
    run_blocks<64>(Q, K, V, G, beta, beta_mode, state, O, B, T, H, logits, scale, workspace, status, seg, s);
  else if (D == 128)
    run_blocks<128>(Q, K, V, G, beta, beta_mode, state, O, B, T, H, logits, scale, workspace, status, seg, s);
  else
    throw std::runtime_error("gdn_blocks: head dimension must be 64 or 128");
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("gdn_blocks launch failed: ") + cudaGetErrorString(e));
}

void launch_gdn_recurrent(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta,
                          int beta_mode, float* state, const GlaMat& O, int B, int T, int H, int D, bool logits,
                          float scale, cudaStream_t s) {
  if (B <= 0 || T <= 0) return;
  auto p = [](const GlaMat& m) { return reinterpret_cast<const __nv_bfloat16*>(m.ptr); };
  auto po = reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(O.ptr));
  if (D == 64)
    gdn_recurrent_kernel<64, 4, 16><<<B * H, 256, 0, s>>>(p(Q), Q.ld, Q.col0, p(K), K.ld, K.col0, p(V), V.ld, V.col0, p(G),
                                                      G.ld, G.col0, beta, beta_mode, state, po, O.ld, O.col0, T, H,
                                                      logits ? 1 : 0, scale);
  else if (D == 128)
    gdn_recurrent_kernel<128, 4, 8><<<B * H, 512, 0, s>>>(p(Q), Q.ld, Q.col0, p(K), K.ld, K.col0, p(V), V.ld, V.col0, p(G),
                                                       G.ld, G.col0, beta, beta_mode, state, po, O.ld, O.col0, T, H,
                                                       logits ? 1 : 0, scale);
  else
    throw std::runtime_error("gdn_recurrent: head dimension must be 64 or 128");
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("gdn_recurrent launch failed: ") + cudaGetErrorString(e));
}

}  // namespace tb
