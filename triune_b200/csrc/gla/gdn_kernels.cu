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
// The same recurrence, eight tokens at a time, for prompts.
//
// One token at a time the recurrence is a chain: a contraction over all key rows, its sum across threads, then the update
// that the next token's contraction waits for (2100 clocks a token in the kernel above). Eight tokens share ONE such round:
// with P_j = product of the decays up to and including token j of the block and S the state before it,
//   x_j  = v_j - (k_j P_{j-1})^T S                                     eight contractions with the same S
//   u_j  = x_j - sum_{i<j} L_ji u_i      L_ji = sum_d k_j (beta k)_i dec_{i+1..j-1}
//   o_j  = (q_j P_j)^T S + sum_{i<=j} A_ji u_i    A_ji = sum_d q_j (beta k)_i dec_{i+1..j}
//   S   <- P_7 S + sum_j (beta k_j dec_{j+1..7}) u_j^T
// Everything is fp32 with exponents <= 0, as in the token form. What does not depend on the state (the scaled vectors and
// the small triangles) is formed once per head by gdn_block_prep_kernel, one warp per block of tokens, instead of by every
// group of value columns; it leaves records of 25 D + 128 floats. Value columns never mix, so the walk runs on
// B * H * D / 16 CTAs of 16 columns: a half warp holds two columns, 16 lanes x D / 16 rows each, and sums the 32
// partial results of a block (2 columns x 8 tokens x {k, q}) with one 30-exchange reduce-scatter that leaves two of them
// in each lane. Products run in packed f32x2 over row pairs. Bound by the latency of that chain (issue slots 37 % used at
// one warp per scheduler), not by memory (DRAM 3 %). Measured, 16 heads of 128, 8192 tokens: one sequence 9010 -> 1155 us
// (four tokens a round: 1853 us), four sequences 9056 -> 3460 us; 6 heads of 64: 5007 -> 896 us. Short prompts and many heads stay
// with the token kernel, see gdn_in_blocks.
// ------------------------------------------------------------------------------------------------
constexpr int GB = 8;  // tokens per block
constexpr int GDN_TRI = 2 * GB * GB;
template <int D>
constexpr int gdn_rec_floats() { return (1 + 3 * GB) * D + GDN_TRI; }  // P_7 | k P | q P | (beta k) dec | L | A

// Reduce-scatter of N values over the sixteen lanes of a half warp: lane l gets the sums of values l * N / 16 + [0, N / 16).
template <int N>
__device__ __forceinline__ void reduce_scatter16(float (&v)[N], int lane) {
  int n = N / 2;
#pragma unroll
  for (int s = 8; s >= 1; s >>= 1, n >>= 1) {
    const bool up = (lane & s) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
}

template <int N>
__device__ __forceinline__ void load_bf16_row(const __nv_bfloat16* p, bool ok, float (&f)[N]) {
  uint32_t w[N / 2];
  if constexpr (N == 4) {
    const uint2 x = ok ? *reinterpret_cast<const uint2*>(p) : make_uint2(0u, 0u);
    w[0] = x.x;
    w[1] = x.y;
  } else {
    w[0] = ok ? *reinterpret_cast<const uint32_t*>(p) : 0u;
  }
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

// Tokens [t0, t0 + nt) of every sequence -> records [B * H, ceil(nt / GB)]. One warp per record; D / 32 dims per lane.
template <int D>
__global__ void __launch_bounds__(128) gdn_block_prep_kernel(
    const __nv_bfloat16* __restrict__ q, long long q_ld, int qcol, const __nv_bfloat16* __restrict__ k, long long k_ld,
    int kcol, const __nv_bfloat16* __restrict__ g, long long g_ld, int gcol, const float* __restrict__ beta, int beta_mode,
    float* __restrict__ rec, int T, int t0, int nt, int H, int logits, int nrec) {
  constexpr int N = D / 32, REC = gdn_rec_floats<D>();
  const int lane = threadIdx.x & 31, id = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (id >= nrec) return;
  const int nb = (nt + GB - 1) / GB, bh = id / nb, blk = id % nb, h = bh % H;
  const long long row0 = (long long)(bh / H) * T + t0 + blk * GB;
  const int left = nt - blk * GB, d0 = h * D + lane * N;
  float qv[GB][N], kv[GB][N], dec[GB][N], bt[GB][N];
#pragma unroll
  for (int j = 0; j < GB; ++j) {
    const bool ok = j < left;
    const long long r = row0 + j;
    load_bf16_row<N>(q + r * q_ld + qcol + d0, ok, qv[j]);
    load_bf16_row<N>(k + r * k_ld + kcol + d0, ok, kv[j]);
    load_bf16_row<N>(g + r * g_ld + gcol + d0, ok, dec[j]);
    const float b1 = (ok && beta_mode == 1) ? beta[r * H + h] : 1.f;
#pragma unroll
    for (int i = 0; i < N; ++i) bt[j][i] = (ok && beta_mode == 2) ? beta[r * H * D + d0 + i] : b1;
  }
  float* out = rec + (long long)id * REC + lane * N;
  float p[N], f[N];
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = 1.f;
#pragma unroll
  for (int j = 0; j < GB; ++j) {  // k_j P_{j-1}, q_j P_j; tokens past the end write nothing and leave the state as it is
#pragma unroll
    for (int i = 0; i < N; ++i) {
      dec[j][i] = j < left ? __expf(gdn_log_decay(dec[j][i], logits != 0)) : 1.f;
      f[i] = kv[j][i] * p[i];
    }
    store_rec<N>(out + (1 + j) * D, f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      p[i] *= dec[j][i];
      f[i] = qv[j][i] * p[i];
    }
    store_rec<N>(out + (1 + GB + j) * D, f);
  }
  store_rec<N>(out, p);
  float* tri = rec + (long long)id * REC + (1 + 3 * GB) * D;
#pragma unroll
  for (int i = 0; i < GB; ++i) {  // w = (beta k)_i carried forward through the decays of the later tokens
    float w[N], sums[2 * GB];
#pragma unroll
    for (int j = 0; j < 2 * GB; ++j) sums[j] = 0.f;
#pragma unroll
    for (int n = 0; n < N; ++n) w[n] = bt[i][n] * kv[i][n];
#pragma unroll
    for (int j = i; j < GB; ++j) {
      if (j > i) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
          sums[j] += kv[j][n] * w[n];
          w[n] *= dec[j][n];
        }
      }
#pragma unroll
      for (int n = 0; n < N; ++n) sums[GB + j] += qv[j][n] * w[n];
    }
    store_rec<N>(out + (1 + 2 * GB + i) * D, w);
    reduce_scatter16(sums, lane);
    const float s = sums[0] + __shfl_xor_sync(0xffffffffu, sums[0], 16);
    if (lane < 16) tri[lane * GB + i] = s;  // lanes 0..7: L[j = lane][i] (zero for i >= j); lanes 8..15: A[j = lane - 8][i]
  }
}

constexpr int GDN_COLS = 16;  // value columns per CTA
constexpr int GDN_STAGES = 3;

// A later token of a block enters the sum of an earlier one's output times a zero of the triangle, which is nothing unless its value
// is infinite or no number. MASK leaves it out instead. Such a value stays in the state, whatever follows: without MASK, true is
// returned (to all threads) where the state ends up so, and the state in memory is as it was.
template <int D, bool MASK>
__device__ __forceinline__ bool gdn_walk(float (*stage)[gdn_rec_floats<D>()], const float* __restrict__ rec,
                                         const __nv_bfloat16* __restrict__ v, long long v_ld, int vcol, float* __restrict__ state,
                                         __nv_bfloat16* __restrict__ out, long long o_ld, int ocol, int T, int t0, int nt, int H,
                                         float scale) {
  constexpr int REC = gdn_rec_floats<D>(), NP = D / 32, NV = REC / 4;  // NP row pairs per lane
  const int tid = threadIdx.x, lane = tid & 31, l16 = lane & 15;
  const int bh = blockIdx.x / (D / GDN_COLS), h = bh % H;
  const int c0 = (blockIdx.x % (D / GDN_COLS)) * GDN_COLS + (tid >> 4) * 2;  // two columns per half warp
  const int nb = (nt + GB - 1) / GB;
  const long long row0 = (long long)(bh / H) * T + t0;
  const float* src = rec + (long long)bh * nb * REC;
  auto row = [&](int pr) { return (pr >> 1) * 64 + l16 * 4 + (pr & 1) * 2; };  // 16 lanes read 256 consecutive bytes

  uint64_t S[2][NP];
  float* sp = state + (long long)bh * D * D + c0;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const float2 x = *reinterpret_cast<const float2*>(sp + (long long)row(i) * D);
    const float2 y = *reinterpret_cast<const float2*>(sp + (long long)(row(i) + 1) * D);
    S[0][i] = pack_f2(x.x, y.x);
    S[1][i] = pack_f2(x.y, y.y);
  }
  auto fetch = [&](int blk) {
    if (blk < nb) {
      const float4* from = reinterpret_cast<const float4*>(src + (long long)blk * REC);
      float4* to = reinterpret_cast<float4*>(&stage[blk % GDN_STAGES][0]);
      for (int i = tid; i < NV; i += 128)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to + i)), "l"(from + i)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // lane l of a half warp ends up with the results of tokens j, j + 1 for {k, q}[l >> 3] and column (l >> 2) & 1
  const int j = (l16 & 3) * 2, col = (l16 >> 2) & 1;
  const bool reads = l16 >= 8;
  const unsigned short* vp = reinterpret_cast<const unsigned short*>(v) + vcol + h * D + c0 + col;
  uint32_t vraw[2], vnext[2];
  auto values = [&](int blk) {  // raw bits: converting here would wait for the load
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = blk * GB + j + e;
      vnext[e] = (!reads && t < nt) ? (uint32_t)vp[(row0 + t) * v_ld] : 0u;
    }
  };
  values(0);
  fetch(0);
  fetch(1);
  for (int blk = 0; blk < nb; ++blk) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // this block's record has landed for every thread, and the one before it has been read by every thread
    fetch(blk + 2);
    vraw[0] = vnext[0];
    vraw[1] = vnext[1];
    values(blk + 1);
    const float* r = &stage[blk % GDN_STAGES][0];
    float val[4 * GB];
#pragma unroll
    for (int w = 0; w < 2 * GB; ++w) {
      uint64_t a0, a1;
#pragma unroll
      for (int i = 0; i < NP; i += 2) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(r + (1 + w) * D + row(i));
        a0 = i == 0 ? mul2(x.x, S[0][0]) : fma2(x.x, S[0][i], a0);
        a1 = i == 0 ? mul2(x.x, S[1][0]) : fma2(x.x, S[1][i], a1);
        a0 = fma2(x.y, S[0][i + 1], a0);
        a1 = fma2(x.y, S[1][i + 1], a1);
      }
      float lo, hi;
      unpack_f2(a0, lo, hi);
      val[(w / GB) * 2 * GB + w % GB] = lo + hi;
      unpack_f2(a1, lo, hi);
      val[(w / GB) * 2 * GB + GB + w % GB] = lo + hi;
    }
    reduce_scatter16(val, lane);
    const float x0 = __uint_as_float(vraw[0] << 16) - val[0], x1 = __uint_as_float(vraw[1] << 16) - val[1];
    const float* tri = r + (1 + 3 * GB) * D;
    float u[2][GB];
#pragma unroll
    for (int i = 0; i < GB; ++i) {
#pragma unroll
      for (int c = 0; c < 2; ++c) u[c][i] = __shfl_sync(0xffffffffu, (i & 1) ? x1 : x0, (lane & 16) + c * 4 + i / 2);
    }
#pragma unroll
    for (int i = 1; i < GB; ++i) {
      float l[GB];
      *reinterpret_cast<float4*>(l) = *reinterpret_cast<const float4*>(tri + i * GB);
      if (i > 4) *reinterpret_cast<float4*>(l + 4) = *reinterpret_cast<const float4*>(tri + i * GB + 4);
#pragma unroll
      for (int m = 0; m < i; ++m) {
        u[0][i] -= l[m] * u[0][m];
        u[1][i] -= l[m] * u[1][m];
      }
    }
#pragma unroll
    for (int i = 0; i < NP; i += 2) {
      const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(r + row(i));
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        S[c][i] = mul2(S[c][i], p.x);
        S[c][i + 1] = mul2(S[c][i + 1], p.y);
      }
    }
#pragma unroll
    for (int w = 0; w < GB; ++w) {
      const uint64_t u0 = pack_f2(u[0][w], u[0][w]), u1 = pack_f2(u[1][w], u[1][w]);
#pragma unroll
      for (int i = 0; i < NP; i += 2) {
        const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(r + (1 + 2 * GB + w) * D + row(i));
        S[0][i] = fma2(e.x, u0, S[0][i]);
        S[0][i + 1] = fma2(e.y, u0, S[0][i + 1]);
        S[1][i] = fma2(e.x, u1, S[1][i]);
        S[1][i + 1] = fma2(e.y, u1, S[1][i + 1]);
      }
    }
    if (reads) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = blk * GB + j + e;
        if (t < nt) {
          const float* a = tri + GB * GB + (j + e) * GB;
          float o = val[e];
#pragma unroll
          for (int m = 0; m < GB; ++m)
            if (!MASK || m <= j + e) o += a[m] * (col ? u[1][m] : u[0][m]);
          out[(row0 + t) * o_ld + ocol + h * D + c0 + col] = __float2bfloat16(o * scale);
        }
      }
    }
  }
  if (!MASK) {
    bool odd = false;
#pragma unroll
    for (int i = 0; i < 2 * NP; ++i) {
      float a, b;
      unpack_f2(S[i & 1][i >> 1], a, b);
      odd |= !(fabsf(a) < INFINITY) || !(fabsf(b) < INFINITY);
    }
    if (__syncthreads_or(odd)) return true;
  }
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    float a, b, c, d;
    unpack_f2(S[0][i], a, b);
    unpack_f2(S[1][i], c, d);
    *reinterpret_cast<float2*>(sp + (long long)row(i) * D) = make_float2(a, c);
    *reinterpret_cast<float2*>(sp + (long long)(row(i) + 1) * D) = make_float2(b, d);
  }
  return false;
}

// The masked walk in a function of its own: 8192 tokens, 16 heads of 128 take 1031 us without it, 1064 with it, and 1107 with its
// selections in the common loop.
template <int D>
__device__ __noinline__ void gdn_walk_again(float (*stage)[gdn_rec_floats<D>()], const float* __restrict__ rec,
                                            const __nv_bfloat16* __restrict__ v, long long v_ld, int vcol, float* __restrict__ state,
                                            __nv_bfloat16* __restrict__ out, long long o_ld, int ocol, int T, int t0, int nt, int H,
                                            float scale) {
  gdn_walk<D, true>(stage, rec, v, v_ld, vcol, state, out, o_ld, ocol, T, t0, nt, H, scale);
}

template <int D>
__global__ void __launch_bounds__(128) gdn_block_walk_kernel(const float* __restrict__ rec, const __nv_bfloat16* __restrict__ v,
                                                             long long v_ld, int vcol, float* __restrict__ state,
                                                             __nv_bfloat16* __restrict__ out, long long o_ld, int ocol, int T,
                                                             int t0, int nt, int H, float scale) {
  __shared__ __align__(16) float stage[GDN_STAGES][gdn_rec_floats<D>()];
  if (gdn_walk<D, false>(stage, rec, v, v_ld, vcol, state, out, o_ld, ocol, T, t0, nt, H, scale))
    gdn_walk_again<D>(stage, rec, v, v_ld, vcol, state, out, o_ld, ocol, T, t0, nt, H, scale);
}

template <int D>
void run_blocks(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta, int beta_mode, float* state,
                const GlaMat& O, int B, int T, int H, bool logits, float scale, float* rec, int seg, cudaStream_t s) {
  auto p = [](const GlaMat& m) { return reinterpret_cast<const __nv_bfloat16*>(m.ptr); };
  for (int t0 = 0; t0 < T; t0 += seg) {
    const int nt = T - t0 < seg ? T - t0 : seg, nrec = B * H * ((nt + GB - 1) / GB);
    gdn_block_prep_kernel<D><<<(nrec + 3) / 4, 128, 0, s>>>(p(Q), Q.ld, Q.col0, p(K), K.ld, K.col0, p(G), G.ld, G.col0, beta,
                                                           beta_mode, rec, T, t0, nt, H, logits ? 1 : 0, nrec);
    gdn_block_walk_kernel<D><<<B * H * (D / GDN_COLS), 128, 0, s>>>(rec, p(V), V.ld, V.col0, state,
                                                                   reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(O.ptr)), O.ld,
                                                                   O.col0, T, t0, nt, H, scale);
  }
}

// Tokens per segment: whole blocks whose records fill at most 48 MB (they are read back from the 126 MB L2), at least 128
// tokens so that the two launches of a segment stay small beside its walk.
int segment_tokens(int BH, int D) {
  const long long per_block = (long long)BH * ((1 + 3 * GB) * D + GDN_TRI) * 4;
  const long long blocks = (48ll << 20) / per_block;
  return (int)(blocks < 16 ? 16 : blocks) * GB;
}

}  // namespace

// Eight tokens a round win where the recurrence is a chain that the chip waits for: the walk's work grows with the heads, the token
// kernel's time hardly does until its CTAs fill the SMs. Token kernel -> blocks, us: 16 heads of 64, 8 tokens 10 -> 10.5, 16 tokens 14 ->
// 12, 512 tokens 318 -> 71; 256 of 64, 16 tokens 17 -> 20, 32 tokens 30 -> 28; 512 of 64, 130 tokens 142 -> 157, 512 tokens 539 -> 530; 16 of
// 128, 8 tokens 14 -> 13; 128 of 128, 16 tokens 24 -> 32, 32 tokens 42 -> 41; 256 of 128, 130 tokens 223 -> 240, 512 tokens 849 -> 796;
// 1024 of 64, 512 tokens 963 -> 1019.
static bool gdn_in_blocks(long long heads, int T, int D) {
  if (D != 64 && D != 128) return false;
  if (T >= 512) return heads <= 512;
  const long long halves = heads * (D / 64);
  return T >= (D == 128 && heads <= 16 ? 8 : 12) && halves <= 448 && T * 8 >= halves;
}

long long gdn_block_workspace_floats(int B, int T, int H, int D) {
  if (!gdn_in_blocks((long long)B * H, T, D)) return 0;
  const int seg = segment_tokens(B * H, D), nt = T < seg ? T : seg;
  return (long long)B * H * ((nt + GB - 1) / GB) * ((1 + 3 * GB) * D + GDN_TRI);
}

void launch_gdn_blocks(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const float* beta, int beta_mode,
                       float* state, const GlaMat& O, int B, int T, int H, int D, bool logits, float scale, float* workspace,
                       cudaStream_t s) {
  if (B <= 0 || T <= 0) return;
  const int seg = segment_tokens(B * H, D);
  if (D == 64)
    run_blocks<64>(Q, K, V, G, beta, beta_mode, state, O, B, T, H, logits, scale, workspace, seg, s);
  else if (D == 128)
    run_blocks<128>(Q, K, V, G, beta, beta_mode, state, O, B, T, H, logits, scale, workspace, seg, s);
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
