// Chunked gated linear attention on tcgen05 tensor cores (head_dim 64 or 128, chunk 64).
//
// Recurrence (per batch, head): S_t = diag(exp(g_t)) S_{t-1} + k_t v_t^T, o_t = q_t^T S_t, with g <= 0 a
// per-key-dimension log decay. With b = cumsum(g) inside a chunk:
//   o_t = (q_t * e^{b_t})^T S_0 + sum_{s<=t} [ sum_d q_td k_sd e^{b_td - b_sd} ] v_s
//   S_C = diag(e^{b_C}) S_0 + sum_s (k_s * e^{b_C - b_s}) v_s^T
// The score term has a per-dimension weight, so it only factors into a matrix product around a reference
// row. Keys are referenced per 16-token sub-chunk j to r_j = b at the row before the sub-chunk:
//   K~[s]    = k_s * e^{r_j - b_s}      (s in sub-chunk j; exponent in [0, 80])
//   Q~(j)[t] = q_t * e^{b_t - r_j}      (t >= 16 j; exponent <= 0)
// and P[:, 16j:16j+16] = Q~(j) K~_j^T is one MMA (M=64, N=16, K=64) per sub-chunk.
//
// A head of 128 is NS = 2 slices of 64 key dimensions and of 64 value dimensions. The decay is diagonal, so the key slices
// only meet in P (a sum over slices, accumulated in TMEM) and in the sums over values; one CTA walks the key slices of a
// head's chunk with all value slices at hand. Before, the slices were laid out as four heads of 64 by copies, and outputs and
// gradients of the copies summed by further passes. Attention over 8 x 1024 tokens, 12 heads of 128: forward 640 -> 170 us (state
// contributions 54, scan 33, outputs 81), backward 1150 -> 340 us (state gradients 91, main kernel 215, gates 32).
//
// Replaces the reference's Triton chunk kernel and scan (triune/kernels/fast_gla.py:33-380, 569-689).
#include "gla.cuh"

#include <cuda.h>

#include <stdexcept>
#include <string>

#include "../common/per_device.h"
#include "../common/ptx.cuh"
#include "../common/tma_desc.h"
#include "gla_tiles.cuh"

namespace tb {

namespace {

constexpr int C = 64;             // chunk length (tokens)
constexpr int D = 64;             // key or value dimensions of one slice of a head
constexpr int GLA_THREADS = 128;
// Row pitch (floats) of the fp32 scratch matrices in shared memory (cumulative log decay, gate-gradient terms).
// Rows stay 16-byte aligned and consecutive rows start one 16-byte bank group apart, so float4 accesses with one
// row per lane are conflict-free (a pitch of 64 puts every row on the same banks: 16-way conflicts).
constexpr int BST = 68;
constexpr int BMAT_BYTES = C * BST * 4;

// Fills bmat[t][d] (fp32, 64x64) with the inclusive cumulative log decay of the gate tile, for a block of NTHR =
// 64 * P threads (P in {2,4,8}). Thread (part, d) scans its 64/P tokens of column d in registers (independent
// shared-memory reads, no round trip per token), publishes the part's total, and after ONE barrier adds the totals of
// the earlier parts while writing its rows. (The previous form scanned in place in shared memory: 64/P dependent
// load-add-store round trips twice, up to 2.5 K clocks in the 128-thread kernel.)
// `totals`: NTHR floats of scratch.
template <int NTHR>
__device__ __forceinline__ void build_cumsum(const uint8_t* g_tile, float* bmat, float* totals, bool logits) {
  constexpr int PARTS = NTHR / 64, LEN = C / PARTS;
  const int tid = threadIdx.x, d = tid & 63, part = tid >> 6;
  float c[LEN];
  float run = 0.f;
#pragma unroll
  for (int i = 0; i < LEN; ++i) {
    const int r = part * LEN + i;
    const __nv_bfloat16 x = *reinterpret_cast<const __nv_bfloat16*>(g_tile + sw_off(r, d >> 3) + (d & 7) * 2);
    run += log_decay(__bfloat162float(x), logits);
    c[i] = run;
  }
  totals[part * 64 + d] = run;
  __syncthreads();
  float base = 0.f;
  for (int pp = 0; pp < part; ++pp) base += totals[pp * 64 + d];
#pragma unroll
  for (int i = 0; i < LEN; ++i) bmat[(part * LEN + i) * BST + d] = base + c[i];
  __syncthreads();
}

struct Bars {
  uint64_t tma, tma_vs;
  uint64_t mma[3];
  uint32_t tmem_slot;
  int failed;
};

// ------------------------------------------------------------------------------------------------
// Phase 1 (and its backward twin): out[bh, c] = (X * e^{w})^T Y  (fp32, head size squared), w = b_last - b or b.
// One CTA per chunk and key slice: X scaled once for all value slices.
// ------------------------------------------------------------------------------------------------
template <int NS>
__global__ void __launch_bounds__(GLA_THREADS) gla_chunk_outer_kernel(const __grid_constant__ CUtensorMap tmX,
                                                                      const __grid_constant__ CUtensorMap tmY,
                                                                      const __grid_constant__ CUtensorMap tmG,
                                                                      int xcol, int ycol, int gcol, int mode,
                                                                      float* __restrict__ out_kv,
                                                                      float* __restrict__ out_decay, int NT, int H,
                                                                      int logits, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ float totals[GLA_THREADS];
  constexpr int HD = NS * D;
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sX = smem;
  uint8_t* sG = smem + TILE;
  uint8_t* sY = smem + 2 * TILE;  // NS tiles
  float* bmat = reinterpret_cast<float*>(smem + (2 + NS) * TILE);
  Bars* bars = reinterpret_cast<Bars*>(smem + (2 + NS) * TILE + BMAT_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cidx = blockIdx.x / NS, slice = blockIdx.x % NS;
  const int chunk = cidx % NT, bh = cidx / NT, h = bh % H, b = bh / H;

  if (tid == 0) {
    mbar_init(&bars->tma, 1);
    mbar_init(&bars->mma[0], 1);
    bars->failed = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_slot, NS * 64);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_slot;
  if (tid == 0) {
    mbar_expect_tx(&bars->tma, (2 + NS) * TILE);
    tma_load_3d(sX, &tmX, &bars->tma, xcol + h * HD + slice * D, chunk * C, b);
    tma_load_3d(sG, &tmG, &bars->tma, gcol + h * HD + slice * D, chunk * C, b);
#pragma unroll
    for (int j = 0; j < NS; ++j) tma_load_3d(sY + j * TILE, &tmY, &bars->tma, ycol + h * HD + j * D, chunk * C, b);
  }
  bool ok = mbar_wait(&bars->tma, 0);
  if (!ok) bars->failed = ST_TIMEOUT_FULL;
  __syncthreads();
  ok = bars->failed == 0;
  if (ok) {
    build_cumsum<GLA_THREADS>(sG, bmat, totals, logits != 0);
    for (int idx = tid; idx < 512; idx += blockDim.x) {
      const int row = idx >> 3, ch = idx & 7;
      uint4* px = reinterpret_cast<uint4*>(sX + sw_off(row, ch));
      float f[8], bt[8], bl[8];
      unpack8(*px, f);
      ld8(bmat + row * BST + ch * 8, bt);
      ld8(bmat + 63 * BST + ch * 8, bl);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] *= __expf(mode == 0 ? (bl[i] - bt[i]) : bt[i]);
      *px = pack8(f);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after_sync();
      constexpr uint32_t idesc = make_idesc(64, 64, 1, 1, 1, 1);
      const uint32_t ax = smem_u32(sX), ay = smem_u32(sY);
#pragma unroll
      for (int j = 0; j < NS; ++j) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem + 64 * j, desc_mn(ax, k), desc_mn(ay + j * TILE, k), idesc, k > 0);
      }
      umma_commit(&bars->mma[0]);
    }
    ok = mbar_wait(&bars->mma[0], 0);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after_sync();
      float* dst = out_kv + ((long long)cidx * HD + slice * D + (warp * 16 + (lane & 15))) * HD;
#pragma unroll
      for (int half = 0; half < 2 * NS; ++half) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem + ((uint32_t)(warp * 32) << 16) + half * 32, r);
        tmem_ld_wait();
        if (lane < 16) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(dst + half * 32 + i) =
                make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]),
                            __uint_as_float(r[i + 3]));
        }
      }
      if (mode == 0 && out_decay != nullptr && tid < D) out_decay[(long long)cidx * HD + slice * D + tid] = __expf(bmat[63 * BST + tid]);
    } else if (lane == 0) {
      bars->failed = ST_TIMEOUT_TMEM;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (bars->failed != 0 && tid == 0 && status != nullptr) atomicCAS(status, 0, bars->failed);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, NS * 64);
  }
}

// ------------------------------------------------------------------------------------------------
// Phase 2: inter-chunk scan, sequential over chunks, two neighbouring state elements a thread. Bound by memory: what a chunk adds does not
// depend on the state, so a batch of eight chunks is read while the one before is added up (one chunk read at a time, one
// element a thread -> here: 16 x 2048 tokens, 6 heads of 64, 15 -> 11 us; 4 x 16384 36 -> 30, 5.0 TB/s; 8 x 1024, 12 heads of 128, 37 ->
// 27; 8192, 16 heads of 128, 45 -> 33, 6.0 TB/s).
// ------------------------------------------------------------------------------------------------
constexpr int SCAN_BATCH = 8, SCAN_THREADS = 128;

template <int NS>
__global__ void __launch_bounds__(SCAN_THREADS) gla_scan_kernel(const float* __restrict__ kv, const float* __restrict__ decay,
                                                                const float* __restrict__ init, __nv_bfloat16* __restrict__ states,
                                                                float* __restrict__ final_state, int NT, int reverse) {
  constexpr int HD = NS * D, E = HD * HD, PER = E / (2 * SCAN_THREADS);
  const int bh = blockIdx.x / PER;
  const int e = ((blockIdx.x % PER) * SCAN_THREADS + threadIdx.x) * 2;  // elements e, e + 1 of the head's state
  const int dk = e / HD;
  const long long blk0 = (long long)bh * NT + (reverse ? NT - 1 : 0);
  const float* kp = kv + blk0 * E + e;
  const float* dp = decay + blk0 * HD + dk;
  __nv_bfloat16* sp = states + blk0 * E + e;
  const int step = reverse ? -1 : 1;
  // a caller's state may start on any number
  float2 s = init ? make_float2(init[(long long)bh * E + e], init[(long long)bh * E + e + 1]) : make_float2(0.f, 0.f);
  float2 add[2][SCAN_BATCH];
  float dec[2][SCAN_BATCH];
  auto read = [&](int first, float2 (&x)[SCAN_BATCH], float (&d)[SCAN_BATCH]) {
#pragma unroll
    for (int i = 0; i < SCAN_BATCH; ++i) {
      if (first + i < NT) {
        x[i] = *reinterpret_cast<const float2*>(kp + (long long)(first + i) * step * E);
        d[i] = dp[(first + i) * step * HD];
      }
    }
  };
  auto walk = [&](int first, const float2 (&x)[SCAN_BATCH], const float (&d)[SCAN_BATCH]) {
#pragma unroll
    for (int i = 0; i < SCAN_BATCH; ++i) {
      if (first + i < NT) {
        *reinterpret_cast<__nv_bfloat162*>(sp + (long long)(first + i) * step * E) = __floats2bfloat162_rn(s.x, s.y);
        s.x = d[i] * s.x + x[i].x;
        s.y = d[i] * s.y + x[i].y;
      }
    }
  };
  read(0, add[0], dec[0]);
  for (int c = 0; c < NT; c += 2 * SCAN_BATCH) {
    read(c + SCAN_BATCH, add[1], dec[1]);
    walk(c, add[0], dec[0]);
    read(c + 2 * SCAN_BATCH, add[0], dec[0]);
    walk(c + SCAN_BATCH, add[1], dec[1]);
  }
  if (final_state) final_state[(long long)bh * E + e] = s.x, final_state[(long long)bh * E + e + 1] = s.y;
}

// ------------------------------------------------------------------------------------------------
// Shared operand construction for phase 3 (forward) and the main backward kernel.
//   sQ -> sA[0..3]: Q~(j)[t] = q_t e^{b_t - r_j} for t >= 16 j (zero rows above), r_0 = 0, r_j = b[16j-1]
//   sK -> sKt:      K~[s]    = k_s e^{r_j(s) - b_s}
// ------------------------------------------------------------------------------------------------
// Factor tables of a chunk. With r_0 = 0 and r_j = b[16j-1] (the cumulative log decay just before sub-chunk j) and
// b_C = b[63]:
//   ftab[i][j][d] = e^{r_i - r_j}  for j <= i (<= 1; zero elsewhere)      gl[i][d] = e^{b_C - r_i}  (<= 1)
// Every exponential of the form e^{b_t - r_j} then costs one multiply on top of e^{b_t - r_i} (i = sub-chunk of t),
// which a thread computes once per element: the special-function unit was a quarter of the backward kernel's time.
constexpr int FTAB_FLOATS = 4 * 4 * D;
// The forward kernel only needs j < i (the diagonal is 1): row i (i - 1) / 2 + j.
constexpr int FTAB_LOWER_FLOATS = 6 * D;

__device__ __forceinline__ void build_factor_tables_lower(const float* bmat, float* ftab) {
  for (int idx = threadIdx.x; idx < FTAB_LOWER_FLOATS; idx += blockDim.x) {
    const int r = idx >> 6, d = idx & 63, i = r >= 3 ? 3 : (r >= 1 ? 2 : 1), j = r - i * (i - 1) / 2;
    const float rj = j == 0 ? 0.f : bmat[(16 * j - 1) * BST + d];
    ftab[idx] = __expf(bmat[(16 * i - 1) * BST + d] - rj);
  }
  __syncthreads();
}
constexpr int GL_FLOATS = 4 * D;

__device__ __forceinline__ void build_factor_tables(const float* bmat, float* ftab, float* gl) {
  for (int idx = threadIdx.x; idx < FTAB_FLOATS; idx += blockDim.x) {
    const int i = idx >> 8, j = (idx >> 6) & 3, d = idx & 63;
    float f = 0.f;
    if (j <= i) {
      const float ri = i == 0 ? 0.f : bmat[(16 * i - 1) * BST + d];
      const float rj = j == 0 ? 0.f : bmat[(16 * j - 1) * BST + d];
      f = j == i ? 1.f : __expf(ri - rj);
    }
    ftab[idx] = f;
  }
  if (gl != nullptr) {
    for (int idx = threadIdx.x; idx < GL_FLOATS; idx += blockDim.x) {
      const int i = idx >> 6, d = idx & 63;
      const float ri = i == 0 ? 0.f : bmat[(16 * i - 1) * BST + d];
      gl[idx] = __expf(bmat[63 * BST + d] - ri);
    }
  }
  __syncthreads();
}

// The four Q~ tiles; with ALL (and a whole factor table) their rows before the sub-chunk are written as zeros. A thread reads and writes the same place
// of every tile, so an output tile may be the q or k tile itself.
struct QTiles {
  uint8_t* t[4];
};
template <bool ALL>
__device__ __forceinline__ void build_score_operands(const uint8_t* sQ, const uint8_t* sK, const QTiles& sA, uint8_t* sKt,
                                                     uint8_t* sKe, const float* bmat, const float* ftab,
                                                     const float* gl) {
  for (int idx = threadIdx.x; idx < 512; idx += blockDim.x) {
    const int row = idx >> 3, ch = idx & 7;
    const uint32_t off = sw_off(row, ch);
    float q[8], k[8], bt[8], rj[8];
    unpack8(*reinterpret_cast<const uint4*>(sQ + off), q);
    unpack8(*reinterpret_cast<const uint4*>(sK + off), k);
    ld8(bmat + row * BST + ch * 8, bt);
    const int jrow = row >> 4;
    if (jrow == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) rj[i] = 0.f;
    } else {
      ld8(bmat + (16 * jrow - 1) * BST + ch * 8, rj);
    }
    float qe[8], o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) qe[i] = q[i] * __expf(bt[i] - rj[i]);  // q_t e^{b_t - r_jrow}
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j < jrow) {
        float f[8];
        ld8(ftab + (ALL ? jrow * 4 + j : jrow * (jrow - 1) / 2 + j) * D + ch * 8, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = qe[i] * f[i];
      } else if (j == jrow) {
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = qe[i];
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = 0.f;
      }
      if (ALL || j <= jrow) *reinterpret_cast<uint4*>(sA.t[j] + off) = pack8(o);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = k[i] * __expf(rj[i] - bt[i]);  // K~: k_s e^{r_j(s) - b_s}
    *reinterpret_cast<uint4*>(sKt + off) = pack8(o);
    if (sKe != nullptr) {  // K_end[s] = k_s e^{b_C - b_s} = K~[s] e^{b_C - r_j(s)}
      float g8[8];
      ld8(gl + jrow * D + ch * 8, g8);
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] *= g8[i];
      *reinterpret_cast<uint4*>(sKe + off) = pack8(o);
    }
  }
}

// Issue the score MMAs P[:, 16j:16j+16] = Q~(j) K~_j^T into TMEM columns [p_col, p_col+64).
__device__ __forceinline__ void issue_score_mmas(uint32_t tmem, uint32_t p_col, const QTiles& sA, uint32_t kt_addr, bool add) {
  constexpr uint32_t idesc = make_idesc(64, 16, 1, 1, 0, 0);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t a = smem_u32(sA.t[j]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      umma_bf16(tmem + p_col + 16 * j, desc_k(a, k), desc_k(kt_addr + j * 2048, k), idesc, k > 0 || add);
  }
}

// ------------------------------------------------------------------------------------------------
// Phase 3 forward: o = Q~(0) S_c + mask(P) V
// A CTA takes a chunk of a head and walks its key slices; the Q~ tiles replace the q and gate tiles, K~ the k tile, so that
// three CTAs (NS = 1: 75 KB each) or two (NS = 2: 108 KB) share an SM and one's loads hide behind the others' operand
// construction, which bounds the kernel (8192 tokens, 16 heads of 128: 96 us, 2.1 TB/s; a third CTA took 16 x 2048 tokens, 6 heads
// of 64 from 83 to 65 us, 4 x 16384 from 160 to 125, 2.4 TB/s). Rows of Q~(j) before sub-chunk j stay unwritten: they only
// reach scores that the mask discards.
// ------------------------------------------------------------------------------------------------
template <int NS>
struct FwdGeom {
  static constexpr int TILES = 5 + NS + NS * NS;  // Q K G | 2 more Q~ | V | S
  static constexpr int SMEM = TILES * TILE + BMAT_BYTES + FTAB_LOWER_FLOATS * 4 + 256;
  static constexpr int TMEM_COLS = NS == 1 ? 128 : 256;  // scores, outputs of each value slice
  static constexpr int CTAS = NS == 1 ? 3 : 2;           // per SM
};

constexpr int FWD_THREADS = 256;

template <int NS>
__global__ void __launch_bounds__(FWD_THREADS, FwdGeom<NS>::CTAS) gla_fwd_out_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                  const __grid_constant__ CUtensorMap tmK,
                                                                  const __grid_constant__ CUtensorMap tmV,
                                                                  const __grid_constant__ CUtensorMap tmG,
                                                                  const __grid_constant__ CUtensorMap tmS, int qcol,
                                                                  int kcol, int vcol, int gcol,
                                                                  __nv_bfloat16* __restrict__ out, long long out_ld,
                                                                  int ocol, int NT, int rows, int H, int logits, int* status) {
  extern __shared__ __align__(1024) uint8_t smem[];  // no static shared memory before it: the space is wanted whole
  constexpr int HD = NS * D;
  using G = FwdGeom<NS>;
  uint8_t* sQ = smem;
  uint8_t* sK = smem + TILE;
  uint8_t* sG = smem + 2 * TILE;
  uint8_t* sV = smem + 5 * TILE;                  // NS tiles
  uint8_t* sS = smem + (5 + NS) * TILE;           // NS x NS tiles (key slice, value slice)
  const QTiles sA{{sQ, sG, smem + 3 * TILE, smem + 4 * TILE}};
  uint8_t* sP = smem + 4 * TILE;                  // once the score products have read Q~(3)
  float* bmat = reinterpret_cast<float*>(smem + G::TILES * TILE);
  float* ftab = bmat + C * BST;
  Bars* bars = reinterpret_cast<Bars*>(smem + G::TILES * TILE + BMAT_BYTES + FTAB_LOWER_FLOATS * 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk = blockIdx.x % NT, bh = blockIdx.x / NT, h = bh % H, b = bh / H;

  if (tid == 0) {
    mbar_init(&bars->tma, 1);
    mbar_init(&bars->tma_vs, 1);
    mbar_init(&bars->mma[0], 1);
    mbar_init(&bars->mma[1], 1);
    bars->failed = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_slot, G::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_slot;
  auto load_slice = [&](int i) {
    mbar_expect_tx(&bars->tma, 3 * TILE);
    tma_load_3d(sG, &tmG, &bars->tma, gcol + h * HD + i * D, chunk * C, b);
    tma_load_3d(sQ, &tmQ, &bars->tma, qcol + h * HD + i * D, chunk * C, b);
    tma_load_3d(sK, &tmK, &bars->tma, kcol + h * HD + i * D, chunk * C, b);
  };
  if (tid == 0) {
    load_slice(0);
    mbar_expect_tx(&bars->tma_vs, (NS + NS * NS) * TILE);
#pragma unroll
    for (int i = 0; i < NS * NS; ++i)
      tma_load_3d(sS + i * TILE, &tmS, &bars->tma_vs, (i % NS) * D, blockIdx.x * HD + (i / NS) * D, 0);
#pragma unroll
    for (int j = 0; j < NS; ++j) tma_load_3d(sV + j * TILE, &tmV, &bars->tma_vs, vcol + h * HD + j * D, chunk * C, b);
  }
  // eight warps: TMEM lane quarter (warp & 3) x 32-column half (warp >> 2) of every 64-column accumulator
  const int quarter = warp & 3, c0 = (warp >> 2) * 32;
  const int row = quarter * 16 + (lane & 15);
  bool ok = true;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    if (i > 0 && tid == 0) load_slice(i);  // the products of slice i - 1 have read its tiles
    ok = mbar_wait(&bars->tma, i & 1);
    if (i == 0) ok = mbar_wait(&bars->tma_vs, 0) && ok;
    if (!ok) bars->failed = ST_TIMEOUT_FULL;
    __syncthreads();
    ok = bars->failed == 0;
    if (!ok) break;
    build_cumsum<FWD_THREADS>(sG, bmat, ftab, logits != 0);
    build_factor_tables_lower(bmat, ftab);
    build_score_operands<false>(sQ, sK, sA, sK, nullptr, bmat, ftab, nullptr);
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after_sync();
      issue_score_mmas(tmem, 0, sA, smem_u32(sK), i > 0);
      constexpr uint32_t id_qs = make_idesc(64, 64, 1, 1, 0, 1);
      const uint32_t a0 = smem_u32(sQ);
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const uint32_t ss = smem_u32(sS + (i * NS + j) * TILE);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem + 64 + 64 * j, desc_k(a0, k), desc_mn(ss, k), id_qs, k > 0 || i > 0);
      }
      umma_commit(&bars->mma[0]);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->mma[0], i & 1));
    if (!ok && lane == 0) bars->failed = ST_TIMEOUT_TMEM;
    if (i + 1 < NS) {
      __syncthreads();
      ok = bars->failed == 0;
      if (!ok) break;
    }
  }
  if (ok) {
    tc_fence_after_sync();
    float v[32];
    load_acc_cols<32>(tmem, c0, quarter, v);
    if (lane < 16) store_row_cols<32>(sP, row, c0, v, row);
    fence_proxy_async_smem();
    tc_fence_before_sync();
  }
  __syncthreads();
  ok = bars->failed == 0;
  if (ok) {
    if (tid == 0) {
      tc_fence_after_sync();
      constexpr uint32_t id_pv = make_idesc(64, 64, 1, 1, 0, 1);
      const uint32_t ap = smem_u32(sP), av = smem_u32(sV);
#pragma unroll
      for (int j = 0; j < NS; ++j) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem + 64 + 64 * j, desc_k(ap, k), desc_mn(av + j * TILE, k), id_pv, 1u);
      }
      umma_commit(&bars->mma[1]);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->mma[1], 0));
    if (ok) {
      tc_fence_after_sync();
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        float v[32];
        load_acc_cols<32>(tmem, 64 + 64 * j + c0, quarter, v);
        if (lane < 16) {
          __nv_bfloat16* dst = out + ((long long)b * rows + chunk * C + row) * out_ld + ocol + h * HD + j * D + c0;
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            float o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = v[ch * 8 + i];
            *reinterpret_cast<uint4*>(dst + ch * 8) = pack8(o);
          }
        }
      }
    } else if (lane == 0) {
      bars->failed = ST_TIMEOUT_TMEM;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (bars->failed != 0 && tid == 0 && status != nullptr) atomicCAS(status, 0, bars->failed);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, G::TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------
// Main backward kernel (per chunk): dq, dk, dv and the in-chunk part of the gate gradient.
//   dP = mask(dO V^T)
//   dv = P^T dO + K_end dS_end          K_end[s] = k_s e^{b_C - b_s}
//   dq = e^{b_t} (dO S_c^T) + sum_j e^{b_t - r_j} (dP_j K~_j)
//   dk = e^{b_C - b_s} (V dS_end^T) + e^{r_j(s) - b_s} (dP^T Q~(j(s)))
//   dg_t = sum_{tau >= t} (q dq - k dk)   (suffix over the whole sequence; chunk suffix added by dg_finalize)
// ------------------------------------------------------------------------------------------------
// A CTA is persistent over the chunks of all heads; per chunk it walks the key slices, each with all value slices, so the
// gradients of queries, keys and gates of a slice are complete where they are formed and dv gathers over the slices in TMEM.
// One slice of a 128-wide head needs 11 input tiles: q, k and gate tiles are double-buffered; the dO, V and state tiles are
// only when NS = 1 (227 KB); with NS = 2 their loads are issued as soon as the products that read them are done and hide
// behind the operand construction of the next slice. TMEM: P, then R2 | dP | dv | T_j, then U_j (R1 shares T_0's factor).
template <int NS>
struct BwdGeom {
  static constexpr int NB = NS == 1 ? 2 : 1;                                // buffers of the V/dO and S/dS tiles
  static constexpr int VS0 = 6, SS0 = VS0 + NB * 2 * NS, A0 = SS0 + NB * 2 * NS;  // first tiles: Q K G (x2) | V dO | S dS | operands
  static constexpr int TILES = A0 + 8;                                      // A0..3 Kt Kend P dP
  static constexpr int SMEM = TILES * TILE + 2 * BMAT_BYTES + (FTAB_FLOATS + GL_FLOATS) * 4 + 1024 + 256;
};

constexpr int BWD_THREADS = 512;

struct BwdBars {
  uint64_t q[2], v[2], s[2];  // input tiles: Q K G; V dO; S dS
  uint64_t mma[3];
  uint32_t tmem_slot;
  int failed;
};

template <int NS>
__global__ void __launch_bounds__(BWD_THREADS) gla_bwd_main_kernel(
    const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmG,
    const __grid_constant__ CUtensorMap tmdO, const __grid_constant__ CUtensorMap tmS,
    const __grid_constant__ CUtensorMap tmdS, int qcol, int kcol, int vcol, int gcol, int docol,
    __nv_bfloat16* __restrict__ dq, long long dq_ld, int dqcol, __nv_bfloat16* __restrict__ dk, long long dk_ld,
    int dkcol, __nv_bfloat16* __restrict__ dv, long long dv_ld, int dvcol, float* __restrict__ dgl_local,
    float* __restrict__ chunk_tot, int NT, int rows, int H, int logits, int nchunks, int* status, long long* dbg) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ float totals[BWD_THREADS];
  using G = BwdGeom<NS>;
  constexpr int HD = NS * D, NB = G::NB;
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  // optional phase timers (developer aid): thread 0 adds the clocks spent up to each mark to dbg[i]
  const bool timed = dbg != nullptr && threadIdx.x == 0;
  long long tmark = timed ? clock64() : 0;
  auto mark = [&](int i) {
    if (timed) {
      const long long now = clock64();
      atomicAdd(reinterpret_cast<unsigned long long*>(dbg + i), (unsigned long long)(now - tmark));
      tmark = now;
    }
  };
  const QTiles sA{{smem + G::A0 * TILE, smem + (G::A0 + 1) * TILE, smem + (G::A0 + 2) * TILE, smem + (G::A0 + 3) * TILE}};
  uint8_t* sKt = smem + (G::A0 + 4) * TILE;
  uint8_t* sKe = smem + (G::A0 + 5) * TILE;
  uint8_t* sP = smem + (G::A0 + 6) * TILE;
  uint8_t* sdP = smem + (G::A0 + 7) * TILE;
  float* bmat = reinterpret_cast<float*>(smem + G::TILES * TILE);
  float* dmat = bmat + C * BST;
  float* ftab = dmat + C * BST;
  float* gl = ftab + FTAB_FLOATS;
  BwdBars* bars = reinterpret_cast<BwdBars*>(smem + G::TILES * TILE + 2 * BMAT_BYTES + (FTAB_FLOATS + GL_FLOATS) * 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->q[i], 1);
      mbar_init(&bars->v[i], 1);
      mbar_init(&bars->s[i], 1);
    }
    for (int i = 0; i < 3; ++i) mbar_init(&bars->mma[i], 1);
    bars->failed = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_slot;
  mark(0);  // barrier init + TMEM allocation
  // Work item `it` of this CTA is key slice it % NS of its chunk number it / NS. Thread 0 issues every load and notes the parity
  // of the newest one per barrier: a loop that is left early waits (bounded) for the copies still in flight.
  const int items = (int)blockIdx.x < nchunks ? ((nchunks - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * NS : 0;
  uint32_t flight = 0, flight_par = 0;  // per barrier q0 q1 v0 v1 s0 s1: a load was issued; its parity
  auto issued = [&](int bar, uint32_t parity) {
    flight |= 1u << bar;
    flight_par = (flight_par & ~(1u << bar)) | (parity << bar);
  };
  auto place = [&](int it_, int& cidx_, int& h_, int& row_, int& b_) {
    cidx_ = blockIdx.x + (it_ / NS) * gridDim.x;
    const int bh_ = cidx_ / NT;
    h_ = bh_ % H, b_ = bh_ / H, row_ = (cidx_ % NT) * C;
  };
  auto issue_q = [&](int it_) {
    int cidx_, h_, row_, b_;
    place(it_, cidx_, h_, row_, b_);
    const int buf_ = it_ & 1, col_ = h_ * HD + (it_ % NS) * D;
    uint8_t* dst = smem + buf_ * 3 * TILE;
    uint64_t* bar = &bars->q[buf_];
    mbar_expect_tx(bar, 3 * TILE);
    tma_load_3d(dst, &tmQ, bar, qcol + col_, row_, b_);
    tma_load_3d(dst + TILE, &tmK, bar, kcol + col_, row_, b_);
    tma_load_3d(dst + 2 * TILE, &tmG, bar, gcol + col_, row_, b_);
    issued(buf_, (uint32_t)((it_ >> 1) & 1));
  };
  auto issue_v = [&](int it_) {  // of the chunk of item it_
    int cidx_, h_, row_, b_;
    place(it_, cidx_, h_, row_, b_);
    const int n_ = it_ / NS, buf_ = n_ % NB;
    uint8_t* dst = smem + (G::VS0 + buf_ * 2 * NS) * TILE;
    uint64_t* bar = &bars->v[buf_];
    mbar_expect_tx(bar, 2 * NS * TILE);
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      tma_load_3d(dst + j * TILE, &tmV, bar, vcol + h_ * HD + j * D, row_, b_);
      tma_load_3d(dst + (NS + j) * TILE, &tmdO, bar, docol + h_ * HD + j * D, row_, b_);
    }
    issued(2 + buf_, (uint32_t)((n_ / NB) & 1));
  };
  auto issue_s = [&](int it_) {
    int cidx_, h_, row_, b_;
    place(it_, cidx_, h_, row_, b_);
    const int buf_ = it_ % NB;
    uint8_t* dst = smem + (G::SS0 + buf_ * 2 * NS) * TILE;
    uint64_t* bar = &bars->s[buf_];
    mbar_expect_tx(bar, 2 * NS * TILE);
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      tma_load_3d(dst + j * TILE, &tmS, bar, j * D, cidx_ * HD + (it_ % NS) * D, 0);
      tma_load_3d(dst + (NS + j) * TILE, &tmdS, bar, j * D, cidx_ * HD + (it_ % NS) * D, 0);
    }
    issued(4 + buf_, (uint32_t)((it_ / NB) & 1));
  };
  if (tid == 0 && items > 0) {
    issue_q(0);
    issue_v(0);
    issue_s(0);
  }
  for (int it = 0; it < items; ++it) {
  const uint32_t par = (uint32_t)(it & 1);  // parity of the once-per-item MMA barriers
  const int slice = it % NS, nth = it / NS, vbuf = nth % NB, sbuf = it % NB;
  const bool first = slice == 0, last = slice == NS - 1;
  int cidx, h, row0, b;
  place(it, cidx, h, row0, b);
  const long long grow0 = (long long)b * rows + row0;  // first row of the chunk in the matrices
  uint8_t* sQ = smem + (it & 1) * 3 * TILE;
  uint8_t* sK = sQ + TILE;
  uint8_t* sG = sQ + 2 * TILE;
  uint8_t* sV = smem + (G::VS0 + vbuf * 2 * NS) * TILE;
  uint8_t* sdO = sV + NS * TILE;
  uint8_t* sS = smem + (G::SS0 + sbuf * 2 * NS) * TILE;
  uint8_t* sdS = sS + NS * TILE;
  if (tid == 0 && it + 1 < items) {
    fence_proxy_async_smem();  // the other buffer was last read through the generic proxy (previous item)
    issue_q(it + 1);
    if constexpr (NB == 2) {
      issue_v(it + 1);
      issue_s(it + 1);
    }
  }
  bool ok = mbar_wait(&bars->q[it & 1], (uint32_t)((it >> 1) & 1));
  if (!ok) bars->failed = ST_TIMEOUT_FULL;
  __syncthreads();
  mark(1);  // input tiles
  ok = bars->failed == 0;
  constexpr int CPW = 64 / (BWD_THREADS / 128);      // accumulator columns per warp (16 warps: 16)
  const int quarter = warp & 3, c0 = (warp >> 2) * CPW;  // TMEM lane quarter / first column of this warp
  const int row = quarter * 16 + (lane & 15);        // accumulator row owned by this thread when lane < 16
  if (ok) {
    build_cumsum<BWD_THREADS>(sG, bmat, totals, logits != 0);
    build_factor_tables(bmat, ftab, gl);
    build_score_operands<true>(sQ, sK, sA, sKt, sKe, bmat, ftab, gl);  // also K_end[s] = k_s e^{b_C - b_s}
    if (!mbar_wait(&bars->v[vbuf], (uint32_t)((nth / NB) & 1)) || !mbar_wait(&bars->s[sbuf], (uint32_t)((it / NB) & 1)))
      bars->failed = ST_TIMEOUT_FULL;
    fence_proxy_async_smem();
    __syncthreads();
    ok = bars->failed == 0;
  }
  mark(2);  // cumulative decay and operand tiles
  if (ok) {
    // ---- stage 1: P of this key slice (cols 0..63) and, once per chunk, dP = dO V^T (cols 64..127)
    if (tid == 0) {
      tc_fence_after_sync();
      issue_score_mmas(tmem, 0, sA, smem_u32(sKt), false);
      if (first) {
        constexpr uint32_t id = make_idesc(64, 64, 1, 1, 0, 0);
        const uint32_t a = smem_u32(sdO), bb = smem_u32(sV);
#pragma unroll
        for (int k = 0; k < 4 * NS; ++k)
          umma_bf16(tmem + 64, desc_k(a + (k >> 2) * TILE, k & 3), desc_k(bb + (k >> 2) * TILE, k & 3), id, k > 0);
      }
      umma_commit(&bars->mma[0]);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->mma[0], par));
    if (ok) {
      tc_fence_after_sync();
      float v[CPW];
      load_acc_cols<CPW>(tmem, 0 + c0, quarter, v);
      if (lane < 16) store_row_cols<CPW>(sP, row, c0, v, row);
      if (first) {
        load_acc_cols<CPW>(tmem, 64 + c0, quarter, v);
        if (lane < 16) store_row_cols<CPW>(sdP, row, c0, v, row);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
    } else if (lane == 0) {
      bars->failed = ST_TIMEOUT_TMEM;
    }
    __syncthreads();
    ok = bars->failed == 0;
  }
  mark(3);  // stage 1
  if (ok) {
    // ---- stage 2: dv (128 + 64 j, over the key slices), T_j = dP_j K~_j (256 + 64 j), R1 = dO S^T added to T_0
    if (tid == 0) {
      tc_fence_after_sync();
      constexpr uint32_t id_mm = make_idesc(64, 64, 1, 1, 1, 1);
      constexpr uint32_t id_kk = make_idesc(64, 64, 1, 1, 0, 0);
      constexpr uint32_t id_km = make_idesc(64, 64, 1, 1, 0, 1);
      const uint32_t aP = smem_u32(sP), adO = smem_u32(sdO), aKe = smem_u32(sKe), adS = smem_u32(sdS);
      const uint32_t aS = smem_u32(sS), adP = smem_u32(sdP), aKt = smem_u32(sKt);
#pragma unroll
      for (int j = 0; j < NS; ++j) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tmem + 128 + 64 * j, desc_mn(aP, k), desc_mn(adO + j * TILE, k), id_mm, k > 0 || !first);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem + 128 + 64 * j, desc_k(aKe, k), desc_mn(adS + j * TILE, k), id_km, 1u);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        umma_bf16(tmem + 256 + 64 * j, desc_k(adP, j), desc_mn(aKt, j), id_km, 0u);
#pragma unroll
      for (int k = 0; k < 4 * NS; ++k)
        umma_bf16(tmem + 256, desc_k(adO + (k >> 2) * TILE, k & 3), desc_k(aS + (k >> 2) * TILE, k & 3), id_kk, 1u);
      umma_commit(&bars->mma[1]);
    }
    // e^{b_t - r_i} for this thread's row (i = its sub-chunk) and columns: the only exponentials of this stage; the
    // shared-memory reads and the special-function work overlap the MMAs
    const int jrow = row >> 4;
    float e0[CPW];
    {
      float bt[CPW], rj[CPW];
      ld_row<CPW>(bmat + row * BST + c0, bt);
      if (jrow == 0) {
#pragma unroll
        for (int d = 0; d < CPW; ++d) rj[d] = 0.f;
      } else {
        ld_row<CPW>(bmat + (16 * jrow - 1) * BST + c0, rj);
      }
#pragma unroll
      for (int d = 0; d < CPW; ++d) e0[d] = __expf(bt[d] - rj[d]);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->mma[1], par));
    if (ok) {
      tc_fence_after_sync();
      float v[CPW];
      if (last) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          load_acc_cols<CPW>(tmem, 128 + 64 * j + c0, quarter, v);
          if (lane < 16) {
            __nv_bfloat16* dst = dv + (grow0 + row) * dv_ld + dvcol + h * HD + j * D + c0;
#pragma unroll
            for (int ch = 0; ch < CPW / 8; ++ch) {
              float o[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = v[ch * 8 + i];
              *reinterpret_cast<uint4*>(dst + ch * 8) = pack8(o);
            }
          }
        }
      }
      // dq = e^{b_t} R1 + sum_{j <= i} e^{b_t - r_j} T_j, with e^{b_t - r_j} = e0 * ftab[i][j] (r_0 = 0 covers R1)
      float acc[CPW];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        load_acc_cols<CPW>(tmem, 256 + 64 * j + c0, quarter, v);  // warp-collective: every lane executes the load
        if (j <= jrow) {
          float f[CPW];
          ld_row<CPW>(ftab + (jrow * 4 + j) * D + c0, f);
          if (j == 0) {
#pragma unroll
            for (int d = 0; d < CPW; ++d) acc[d] = v[d] * (e0[d] * f[d]);
          } else {
#pragma unroll
            for (int d = 0; d < CPW; ++d) acc[d] += v[d] * (e0[d] * f[d]);
          }
        }
      }
      if (lane < 16) {
        __nv_bfloat16* dst = dq + (grow0 + row) * dq_ld + dqcol + h * HD + slice * D + c0;
#pragma unroll
        for (int ch = 0; ch < CPW / 8; ++ch) {
          float o[8], q[8], qd[8];
          unpack8(*reinterpret_cast<const uint4*>(sQ + sw_off(row, c0 / 8 + ch)), q);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            o[i] = acc[ch * 8 + i];
            qd[i] = q[i] * o[i];
          }
          st8(dmat + row * BST + c0 + ch * 8, qd);
          *reinterpret_cast<uint4*>(dst + ch * 8) = pack8(o);
        }
      }
      tc_fence_before_sync();
    } else if (lane == 0) {
      bars->failed = ST_TIMEOUT_TMEM;
    }
    __syncthreads();
    ok = bars->failed == 0;
  }
  mark(4);  // stage 2
  if (ok) {
    // ---- stage 3: R2 = V dS^T (0..63, where P was), U_j = dP^T Q~(j) (256+64j)
    if (tid == 0) {
      tc_fence_after_sync();
      constexpr uint32_t id_kk = make_idesc(64, 64, 1, 1, 0, 0);
      constexpr uint32_t id_mm = make_idesc(64, 64, 1, 1, 1, 1);
      const uint32_t aV = smem_u32(sV), adS = smem_u32(sdS), adP = smem_u32(sdP);
#pragma unroll
      for (int k = 0; k < 4 * NS; ++k)
        umma_bf16(tmem, desc_k(aV + (k >> 2) * TILE, k & 3), desc_k(adS + (k >> 2) * TILE, k & 3), id_kk, k > 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t aA = smem_u32(sA.t[j]);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem + 256 + 64 * j, desc_mn(adP, k), desc_mn(aA, k), id_mm, k > 0);
      }
      umma_commit(&bars->mma[2]);
    }
    // dk = e^{b_C - b_s} R2 + e^{r_q - b_s} U_q with q the sub-chunk of s; e^{b_C - b_s} = e^{r_q - b_s} gl[q]
    float x0[CPW], gq[CPW];
    {
      float bt[CPW], br[CPW];
      ld_row<CPW>(bmat + row * BST + c0, bt);
      if (quarter > 0) {
        ld_row<CPW>(bmat + (16 * quarter - 1) * BST + c0, br);
      } else {
#pragma unroll
        for (int d = 0; d < CPW; ++d) br[d] = 0.f;
      }
#pragma unroll
      for (int d = 0; d < CPW; ++d) x0[d] = __expf(br[d] - bt[d]);
      ld_row<CPW>(gl + quarter * D + c0, gq);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->mma[2], par));
    if (ok) {
      tc_fence_after_sync();
      if constexpr (NB == 1) {  // the last products that read the V, dO, S and dS tiles are done
        if (tid == 0 && it + 1 < items) {
          issue_s(it + 1);
          if (last) issue_v(it + 1);
        }
      }
      float v[CPW], acc[CPW];
      load_acc_cols<CPW>(tmem, c0, quarter, v);
#pragma unroll
      for (int d = 0; d < CPW; ++d) acc[d] = v[d] * gq[d];
      load_acc_cols<CPW>(tmem, 256 + 64 * quarter + c0, quarter, v);  // rows of sub-chunk j = quarter live in accumulator j
#pragma unroll
      for (int d = 0; d < CPW; ++d) acc[d] = (acc[d] + v[d]) * x0[d];
      if (lane < 16) {
        __nv_bfloat16* dst = dk + (grow0 + row) * dk_ld + dkcol + h * HD + slice * D + c0;
#pragma unroll
        for (int ch = 0; ch < CPW / 8; ++ch) {
          float o[8], k[8], qd[8];
          unpack8(*reinterpret_cast<const uint4*>(sK + sw_off(row, c0 / 8 + ch)), k);
          ld8(dmat + row * BST + c0 + ch * 8, qd);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            o[i] = acc[ch * 8 + i];
            qd[i] -= k[i] * o[i];
          }
          st8(dmat + row * BST + c0 + ch * 8, qd);
          *reinterpret_cast<uint4*>(dst + ch * 8) = pack8(o);
        }
      }
    } else if (lane == 0) {
      bars->failed = ST_TIMEOUT_TMEM;
    }
    __syncthreads();
    ok = bars->failed == 0;
  }
  mark(5);  // stage 3
  if (ok) {
    // in-chunk suffix sum of (q dq - k dk) per key dimension: parts of PR rows in parallel, then the totals of the
    // later parts (left in their first rows) are added on the way out
    constexpr int NPARTS = BWD_THREADS / 64, PR = C / NPARTS;
    const int d = tid & 63, part = tid >> 6;
    float acc = 0.f;
    for (int t = PR * part + PR - 1; t >= PR * part; --t) {
      acc += dmat[t * BST + d];
      dmat[t * BST + d] = acc;
    }
    __syncthreads();
    float base = 0.f;
    for (int pp = part + 1; pp < NPARTS; ++pp) base += dmat[(PR * pp) * BST + d];
    float* dst = dgl_local + grow0 * (H * HD) + h * HD + slice * D + d;
    for (int t = PR * part; t < PR * part + PR; ++t) dst[(long long)t * (H * HD)] = dmat[t * BST + d] + base;
    if (part == 0) chunk_tot[((long long)((cidx / NT) * NS + slice) * NT + cidx % NT) * D + d] = dmat[d] + base;
  }
  mark(6);  // suffix sums
  if (timed) atomicAdd(reinterpret_cast<unsigned long long*>(dbg + 7), 1ull);
  // item boundary: every read of this item's tiles, scratch matrices and accumulators is done before the next
  // one rewrites them
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (bars->failed != 0) break;
  }  // item loop
  if (bars->failed != 0 && tid == 0) {
    uint64_t* all[6] = {&bars->q[0], &bars->q[1], &bars->v[0], &bars->v[1], &bars->s[0], &bars->s[1]};
    for (int i = 0; i < 6; ++i)
      if ((flight >> i) & 1u) (void)mbar_wait(all[i], (flight_par >> i) & 1u);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (bars->failed != 0 && tid == 0 && status != nullptr) atomicCAS(status, 0, bars->failed);
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// dg[t] = (local suffix + totals of later chunks) * d(log decay)/d(gate input). Heads are 64-wide slices here; rows past a sequence's end are left out. Bound by
// memory: eight columns a thread in 16-byte accesses, the later chunks' totals summed by four groups of threads (8 x 1024 tokens,
// 24 slices: 79 -> 32 us), the clamp's end compared with the logit instead of its logarithm formed (-> 24 us, 4.2 TB/s).
__global__ void __launch_bounds__(256) gla_dg_finalize_kernel(const float* __restrict__ dgl_local,
                                                              const float* __restrict__ chunk_tot,
                                                              const __nv_bfloat16* __restrict__ g, long long g_ld,
                                                              int gcol, __nv_bfloat16* __restrict__ dg, long long dg_ld,
                                                              int dgcol, int NT, int rows, int H, int logits,
                                                              const float* __restrict__ end_term) {
  __shared__ __align__(16) float carry[4][D];
  const int chunk = blockIdx.x % NT, bh = blockIdx.x / NT, h = bh % H, b = bh / H;
  const int tid = threadIdx.x;
  const long long row0 = (long long)b * rows + chunk * C;
  const int ch = (tid & 7) * 8, left = rows - chunk * C;  // rows of the sequence from row0 on
  // both rows of a thread are read ahead of the barrier
  uint4 gu[2];
  float loc[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if ((tid >> 3) + 32 * i >= left) continue;
    const long long r = row0 + (tid >> 3) + 32 * i;
    gu[i] = *reinterpret_cast<const uint4*>(g + r * g_ld + gcol + h * D + ch);
    ld8(dgl_local + r * (H * D) + h * D + ch, loc[i]);
  }
  {
    // end_term[bh][d] = sum_v dS_T[d][v] S_T[d][v]: the final state depends on every log decay of the sequence
    const int d = tid & 63, part = tid >> 6;
    float acc = (part == 0 && end_term != nullptr) ? end_term[(long long)bh * D + d] : 0.f;
#pragma unroll 4
    for (int c = chunk + 1 + part; c < NT; c += 4) acc += chunk_tot[((long long)bh * NT + c) * D + d];
    carry[part][d] = acc;
  }
  __syncthreads();
  float later[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) later[j] = (carry[0][ch + j] + carry[1][ch + j]) + (carry[2][ch + j] + carry[3][ch + j]);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if ((tid >> 3) + 32 * i >= left) continue;
    float x[8], o[8];
    unpack8(gu[i], x);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float deriv;
      if (logits) {
        // d logsigmoid = sigmoid(-x) where logsigmoid(x) is above the clamp, whose logit lies between the bf16 numbers -5 and -4.96875
        deriv = x[j] > GLA_MIN_LOGIT ? __fdividef(1.f, 1.f + __expf(x[j])) : 0.f;
      } else {
        deriv = (x[j] <= 0.f && x[j] >= GLA_MIN_LOG_DECAY) ? 1.f : 0.f;
      }
      o[j] = (loc[i][j] + later[j]) * deriv;
    }
    *reinterpret_cast<uint4*>(dg + (row0 + (tid >> 3) + 32 * i) * dg_ld + dgcol + h * D + ch) = pack8(o);
  }
}

// ------------------------------------------------------------------------------------------------
// Decode step: S <- diag(e^{g}) S + k v^T ; o = q^T S. One CTA per (batch, head), 64x64 state in fp32.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gla_decode_step_kernel(const __nv_bfloat16* __restrict__ q, long long q_ld, int qcol,
                                                              const __nv_bfloat16* __restrict__ k, long long k_ld, int kcol,
                                                              const __nv_bfloat16* __restrict__ v, long long v_ld, int vcol,
                                                              const __nv_bfloat16* __restrict__ g, long long g_ld, int gcol,
                                                              float* __restrict__ state, __nv_bfloat16* __restrict__ o,
                                                              long long o_ld, int ocol, int H, int logits) {
  __shared__ float sq[D], sk[D], sv[D], sd[D], part[4][D];
  const int bh = blockIdx.x, h = bh % H, b = bh / H;
  const int tid = threadIdx.x;
  if (tid < D) {
    sq[tid] = __bfloat162float(q[b * q_ld + qcol + h * D + tid]);
    sk[tid] = __bfloat162float(k[b * k_ld + kcol + h * D + tid]);
    sv[tid] = __bfloat162float(v[b * v_ld + vcol + h * D + tid]);
    sd[tid] = __expf(log_decay(__bfloat162float(g[b * g_ld + gcol + h * D + tid]), logits != 0));
  }
  __syncthreads();
  const int dv = tid & 63, quarter = tid >> 6;
  float* S = state + (long long)bh * D * D;
  float acc = 0.f;
#pragma unroll 4
  for (int i = quarter * 16; i < quarter * 16 + 16; ++i) {
    const float s = sd[i] * S[i * D + dv] + sk[i] * sv[dv];
    S[i * D + dv] = s;
    acc += sq[i] * s;
  }
  part[quarter][dv] = acc;
  __syncthreads();
  if (tid < D) o[b * o_ld + ocol + h * D + tid] = __float2bfloat16(part[0][tid] + part[1][tid] + part[2][tid] + part[3][tid]);
}

// {columns of the wide matrix, rows of one sequence, sequences}; boxes of 64 x 64
CUtensorMap tile_map(const GlaMat& m, long long rows, long long count) {
  return make_tmap_3d(m.ptr, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)m.ld, (uint64_t)rows, (uint64_t)count,
                      (uint64_t)m.ld * 2ull, (uint64_t)m.ld * 2ull * (uint64_t)rows, 64, 64);
}

void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + " launch failed: " + cudaGetErrorString(e));
}

template <typename K>
void set_smem(K kern, int bytes) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) throw std::runtime_error(std::string("cannot set shared memory size: ") + cudaGetErrorString(e));
}

void check_dims(const GlaDims& d) {
  if (d.T % C != 0 || d.T <= 0) throw std::runtime_error("gla kernels need T to be a positive multiple of 64");
  if (d.D != 64 && d.D != 128) throw std::runtime_error("gla kernels need head dimension 64 or 128");
  if (d.rows != 0 && d.rows < d.T) throw std::runtime_error("gla kernels: fewer rows than tokens");
}

int seq_rows(const GlaDims& d) { return d.rows != 0 ? d.rows : d.T; }

template <int NS>
void chunk_outer(int mode, const GlaMat& X, const GlaMat& Y, const GlaMat& G, float* out_kv, float* out_decay, const GlaDims& d,
                 int* status, cudaStream_t s) {
  const int rows = seq_rows(d);
  constexpr int SMEM = (2 + NS) * TILE + BMAT_BYTES + 1024 + 256;
  static PerDeviceOnce cfg;  // the attribute is per device
  if (cfg.first_use()) set_smem(gla_chunk_outer_kernel<NS>, SMEM);
  gla_chunk_outer_kernel<NS><<<d.B * d.H * (d.T / C) * NS, GLA_THREADS, SMEM, s>>>(
      tile_map(X, rows, d.B), tile_map(Y, rows, d.B), tile_map(G, rows, d.B), X.col0, Y.col0, G.col0, mode, out_kv, out_decay,
      d.T / C, d.H, d.gate_logits ? 1 : 0, status);
}

template <int NS>
void fwd_out(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const __nv_bfloat16* states, const GlaMat& O,
             const GlaDims& d, int* status, cudaStream_t s) {
  const int rows = seq_rows(d), grid = d.B * d.H * (d.T / C);
  const GlaMat S{states, NS * D, 0};
  static PerDeviceOnce cfg;  // the attribute is per device
  if (cfg.first_use()) set_smem(gla_fwd_out_kernel<NS>, FwdGeom<NS>::SMEM);
  gla_fwd_out_kernel<NS><<<grid, FWD_THREADS, FwdGeom<NS>::SMEM, s>>>(
      tile_map(Q, rows, d.B), tile_map(K, rows, d.B), tile_map(V, rows, d.B), tile_map(G, rows, d.B),
      tile_map(S, (long long)grid * NS * D, 1), Q.col0, K.col0, V.col0, G.col0,
      reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(O.ptr)), O.ld, O.col0, d.T / C, rows, d.H, d.gate_logits ? 1 : 0, status);
}

long long* g_gla_dbg = nullptr;

template <int NS>
void bwd_main(const GlaMat& Q, const GlaMat& K, const GlaMat& V, const GlaMat& G, const GlaMat& dO, const __nv_bfloat16* states,
              const __nv_bfloat16* dstates, const GlaMat& dQ, const GlaMat& dK, const GlaMat& dV, float* dgl_local, float* chunk_tot,
              const GlaDims& d, int* status, cudaStream_t s) {
  const int rows = seq_rows(d), nchunks = d.B * d.H * (d.T / C);
  const GlaMat S{states, NS * D, 0}, dS{dstates, NS * D, 0};
  const long long srows = (long long)nchunks * NS * D;
  static PerDeviceOnce cfg;  // the attribute is per device
  if (cfg.first_use()) set_smem(gla_bwd_main_kernel<NS>, BwdGeom<NS>::SMEM);
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    sms = n > 0 ? n : 148;
  }
  const int grid = nchunks < sms ? nchunks : sms;  // one persistent CTA per SM
  auto p = [](const GlaMat& m) { return reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(m.ptr)); };
  gla_bwd_main_kernel<NS><<<grid, BWD_THREADS, BwdGeom<NS>::SMEM, s>>>(
      tile_map(Q, rows, d.B), tile_map(K, rows, d.B), tile_map(V, rows, d.B), tile_map(G, rows, d.B), tile_map(dO, rows, d.B),
      tile_map(S, srows, 1), tile_map(dS, srows, 1), Q.col0, K.col0, V.col0, G.col0, dO.col0, p(dQ), dQ.ld, dQ.col0, p(dK), dK.ld,
      dK.col0, p(dV), dV.ld, dV.col0, dgl_local, chunk_tot, d.T / C, rows, d.H, d.gate_logits ? 1 : 0, nchunks, status, g_gla_dbg);
}

}  // namespace

void launch_gla_chunk_outer(int mode, GlaMat X, GlaMat Y, GlaMat G, float* out_kv, float* out_decay, GlaDims d,
                            int* status, cudaStream_t s) {
  check_dims(d);
  (d.D == 64 ? chunk_outer<1> : chunk_outer<2>)(mode, X, Y, G, out_kv, out_decay, d, status, s);
  check_launch("gla_chunk_outer");
}

void launch_gla_scan(const float* kv, const float* decay, const float* init, __nv_bfloat16* states, float* final_state,
                     int BH, int NT, int D_, bool reverse, cudaStream_t s) {
  if (D_ == 64)
    gla_scan_kernel<1><<<BH * (D * D / (2 * SCAN_THREADS)), SCAN_THREADS, 0, s>>>(kv, decay, init, states, final_state, NT, reverse ? 1 : 0);
  else
    gla_scan_kernel<2><<<BH * (4 * D * D / (2 * SCAN_THREADS)), SCAN_THREADS, 0, s>>>(kv, decay, init, states, final_state, NT, reverse ? 1 : 0);
  check_launch("gla_scan");
}

void launch_gla_fwd_out(GlaMat Q, GlaMat K, GlaMat V, GlaMat G, const __nv_bfloat16* states, GlaMat O, GlaDims d,
                        int* status, cudaStream_t s) {
  check_dims(d);
  (d.D == 64 ? fwd_out<1> : fwd_out<2>)(Q, K, V, G, states, O, d, status, s);
  check_launch("gla_fwd_out");
}

void gla_set_debug_buffer(long long* p) { g_gla_dbg = p; }

void launch_gla_bwd_main(GlaMat Q, GlaMat K, GlaMat V, GlaMat G, GlaMat dO, const __nv_bfloat16* states,
                         const __nv_bfloat16* dstates, GlaMat dQ, GlaMat dK, GlaMat dV, float* dgl_local,
                         float* chunk_tot, GlaDims d, int* status, cudaStream_t s) {
  check_dims(d);
  (d.D == 64 ? bwd_main<1> : bwd_main<2>)(Q, K, V, G, dO, states, dstates, dQ, dK, dV, dgl_local, chunk_tot, d, status, s);
  check_launch("gla_bwd_main");
}

void launch_gla_dg_finalize(const float* dgl_local, const float* chunk_tot, GlaMat G, GlaMat dG, GlaDims d,
                            cudaStream_t s, const float* end_term) {
  if (d.T % C != 0 || d.T <= 0) throw std::runtime_error("gla_dg_finalize: whole chunks of 64 tokens (of which `rows` are there)");
  const int slices = d.H * (d.D / 64), grid = d.B * slices * (d.T / C);
  gla_dg_finalize_kernel<<<grid, 256, 0, s>>>(dgl_local, chunk_tot, reinterpret_cast<const __nv_bfloat16*>(G.ptr), G.ld,
                                              G.col0, reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(dG.ptr)), dG.ld,
                                              dG.col0, d.T / C, seq_rows(d), slices, d.gate_logits ? 1 : 0, end_term);
  check_launch("gla_dg_finalize");
}

void launch_gla_decode_step(GlaMat Q, GlaMat K, GlaMat V, GlaMat G, float* state, GlaMat O, int B, int H,
                            bool gate_logits, cudaStream_t s) {
  auto p = [](const GlaMat& m) { return reinterpret_cast<const __nv_bfloat16*>(m.ptr); };
  gla_decode_step_kernel<<<B * H, 256, 0, s>>>(p(Q), Q.ld, Q.col0, p(K), K.ld, K.col0, p(V), V.ld, V.col0, p(G), G.ld,
                                               G.col0, state, reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(O.ptr)),
                                               O.ld, O.col0, H, gate_logits ? 1 : 0);
  check_launch("gla_decode_step");
}

}  // namespace tb
