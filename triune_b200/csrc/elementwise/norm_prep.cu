// Bandwidth-bound row kernels: RMSNorm (+ residual add) forward/backward and the GLA q/k feature
// map (ELU+1 -> L2 normalise -> half-split RoPE) forward/backward. A row of RMSNorm belongs to one warp (forward, many narrow
// rows) or to the warps of a block (other forwards, every backward), a (token, head) vector of the feature map to D / 8 lanes; all
// global traffic is in 16-byte accesses and every tensor is touched exactly once per pass.
//
// Reference semantics: triune/kernels/fast_rmsnorm.py:181-335 (norm, fused add-norm),
// triune/model/attention.py:14-80 and :509-531 (feature map + RoPE).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <stdexcept>
#include <string>

#include "../common/dependent_launch.cuh"
#include "../common/ptx.cuh"
#include "elementwise.cuh"

namespace tb {

namespace {

constexpr int NORM_PARTS = 148 * 2;  // blocks of the backward kernel: two per SM are resident

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void unpack_row8(const uint4& u, float (&f)[8]) {
  const uint32_t x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(x[i] << 16);
    f[2 * i + 1] = __uint_as_float(x[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack_row8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// Each lane holds up to MAXV 8-element vectors of its row (d <= 32*8*MAXV); MAXV is a template parameter so
// narrow models do not pay registers for wide ones.

template <bool HAS_RES, int MAXV>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ res,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          __nv_bfloat16* __restrict__ y,
                                                          __nv_bfloat16* __restrict__ sum_out,
                                                          float* __restrict__ rstd, int rows, int d, float eps) {
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nvec = d >> 3;
  for (long long row = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < rows;
       row += (long long)gridDim.x * warps_per_block) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * d);
    const uint4* rr = HAS_RES ? reinterpret_cast<const uint4*>(res + row * d) : nullptr;
    float vals[MAXV][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      const int v = lane + i * 32;
      if (v < nvec) {
        uint4 xv = xr[v];
        const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xv);
        if (HAS_RES) {
          uint4 rv = rr[v];
          const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rv);
          uint4 sv;
          uint32_t* s32 = reinterpret_cast<uint32_t*>(&sv);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 a = __bfloat1622float2(x2[j]), b = __bfloat1622float2(r2[j]);
            s32[j] = pack_bf16x2(a.x + b.x, a.y + b.y);
            float2 s = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&s32[j]));
            vals[i][2 * j] = s.x;
            vals[i][2 * j + 1] = s.y;
          }
          reinterpret_cast<uint4*>(sum_out + row * d)[v] = sv;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 a = __bfloat1622float2(x2[j]);
            vals[i][2 * j] = a.x;
            vals[i][2 * j + 1] = a.y;
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += vals[i][j] * vals[i][j];
      }
    }
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss / (float)d + eps);
    if (lane == 0 && rstd) rstd[row] = inv;
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      const int v = lane + i * 32;
      if (v < nvec) {
        uint4 wv = reinterpret_cast<const uint4*>(w)[v];
        const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
        uint4 ov;
        uint32_t* o32 = reinterpret_cast<uint32_t*>(&ov);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 wf = __bfloat1622float2(w2[j]);
          o32[j] = pack_bf16x2(vals[i][2 * j] * inv * wf.x, vals[i][2 * j + 1] * inv * wf.y);
        }
        reinterpret_cast<uint4*>(y + row * d)[v] = ov;
      }
    }
  }
}

// The same with a row spread over the warps of a block, eight columns a thread and R rows in flight, for wide rows (a warp that
// holds 1536 columns has little else in flight) and for few (decoding: one row is a chain of latencies, and a warp alone walks
// eight loads before it can sum). In a replayed graph, kernel above -> this one: 1 x 2048 4.5 -> 1.8 us, 1184 x 1024 3.3 -> 2.6,
// 8192 x 1536 12.3 -> 9.6 (with the residual 25.3 -> 18.2), 32768 x 2048 94 -> 46. Many rows of up to 1024 columns stay above
// (above, here): 8192 x 384 4.0, 4.2 us; 32768 x 512 8.2, 10.4; 8192 x 1024 5.3, 6.4; with the residual 4000 x 768 4.2, 5.8, 8192 x
// 1024 8.3, 9.3, but 2331 x 768 3.8, 3.3 and, out of L2, 16384 x 1024 25.4, 23.4: see rows_per_warp.
// `wpr` warps per row; the block's warps / wpr rows side by side.
template <bool HAS_RES, int R>
__global__ void __launch_bounds__(256) rmsnorm_fwd_wide_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                                                               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                               __nv_bfloat16* __restrict__ sum_out, float* __restrict__ rstd, int rows,
                                                               int d, float eps, int wpr) {
  __shared__ float red[2][8][R];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slots = (blockDim.x >> 5) / wpr;
  const int slot = warp / wpr, col = ((warp % wpr) * 32 + lane) * 8;
  const bool live = col < d;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  allow_dependents();
  wait_predecessors();  // launched over the end of the kernel before it
  const uint4 wv = live ? *reinterpret_cast<const uint4*>(w + col) : zero;
  int buf = 0;
  for (long long base = (long long)blockIdx.x * slots * R; base < rows; base += (long long)gridDim.x * slots * R, buf ^= 1) {
    const long long row0 = base + slot * R;
    uint4 xv[R];
    float ss[R];
#pragma unroll
    for (int i = 0; i < R; ++i) xv[i] = (live && row0 + i < rows) ? *reinterpret_cast<const uint4*>(x + (row0 + i) * d + col) : zero;
    if (HAS_RES) {
      uint4 rv[R];
#pragma unroll
      for (int i = 0; i < R; ++i) rv[i] = (live && row0 + i < rows) ? *reinterpret_cast<const uint4*>(res + (row0 + i) * d + col) : zero;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float a[8], b[8];
        unpack_row8(xv[i], a);
        unpack_row8(rv[i], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += b[j];
        xv[i] = pack_row8(a);
        if (live && row0 + i < rows) *reinterpret_cast<uint4*>(sum_out + (row0 + i) * d + col) = xv[i];
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float a[8];
      unpack_row8(xv[i], a);
      ss[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) ss[i] += a[j] * a[j];
      ss[i] = warp_sum(ss[i]);
    }
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) red[buf][warp][i] = ss[i];
    }
    __syncthreads();  // the other buffer's readers are past the barrier before this one
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float sum = 0.f;
      for (int p = 0; p < wpr; ++p) sum += red[buf][slot * wpr + p][i];
      const float inv = rsqrtf(sum / (float)d + eps);
      if (row0 + i < rows) {
        if (rstd && warp % wpr == 0 && lane == 0) rstd[row0 + i] = inv;
        if (live) {
          float a[8], wf[8];
          unpack_row8(xv[i], a);
          unpack_row8(wv, wf);
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] = a[j] * inv * wf[j];
          *reinterpret_cast<uint4*>(y + (row0 + i) * d + col) = pack_row8(a);
        }
      }
    }
  }
}

// dx = rstd * (w*dy - xhat * mean(w*dy*xhat)) [+ dres_in]; partial[block][d] = the block's sum over rows of dy * xhat.
// Eight columns a thread, a row spread over `wpr` warps, R rows in flight. One warp per row before, with the row, its gradient
// and the weight gradient's sums in 220 registers and one block per 64 rows, was bound by latency; so were the atomics at its
// end. With the sum over blocks, the residual's gradient and the conversion of dw, cold: 8192 x 2048 101 -> 46 us (2.9 TB/s),
// 8192 x 1536 81 -> 43, 16384 x 512 40 -> 32, 32768 x 384 47 -> 43; in a replayed graph 2331 x 2048 44 -> 11.6, 600 x 384 14.6 -> 5.9.
template <bool HAS_DRES, int R>
__global__ void __launch_bounds__(256, 2) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                             const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd,
                                                             const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                                                             float* __restrict__ partial, int rows, int d, int wpr) {
  __shared__ float red[2][8][R];
  __shared__ float cols[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slots = (blockDim.x >> 5) / wpr;
  const int slot = warp / wpr, col = ((warp % wpr) * 32 + lane) * 8;
  const bool live = col < d;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float wf[8], dw[8];
  unpack_row8(live ? *reinterpret_cast<const uint4*>(w + col) : zero, wf);
#pragma unroll
  for (int j = 0; j < 8; ++j) dw[j] = 0.f;
  int buf = 0;
  for (long long base = (long long)blockIdx.x * slots * R; base < rows; base += (long long)gridDim.x * slots * R, buf ^= 1) {
    const long long row0 = base + slot * R;
    uint4 xv[R], gv[R], rv[R];
    float inv[R], dot[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const bool in = row0 + i < rows;
      const long long at = (row0 + i) * d + col;
      inv[i] = in ? rstd[row0 + i] : 0.f;
      xv[i] = (live && in) ? *reinterpret_cast<const uint4*>(x + at) : zero;
      gv[i] = (live && in) ? *reinterpret_cast<const uint4*>(dy + at) : zero;
      if (HAS_DRES) rv[i] = (live && in) ? *reinterpret_cast<const uint4*>(dres + at) : zero;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float a[8], g[8];
      unpack_row8(xv[i], a);
      unpack_row8(gv[i], g);
      dot[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float gx = g[j] * (a[j] * inv[i]);
        dw[j] += gx;
        dot[i] += gx * wf[j];
      }
      dot[i] = warp_sum(dot[i]);
    }
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) red[buf][warp][i] = dot[i];
    }
    __syncthreads();  // the other buffer's readers are past the barrier before this one
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float sum = 0.f;
      for (int p = 0; p < wpr; ++p) sum += red[buf][slot * wpr + p][i];
      sum /= (float)d;
      if (live && row0 + i < rows) {
        float a[8], g[8];
        unpack_row8(xv[i], a);
        unpack_row8(gv[i], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = inv[i] * (g[j] * wf[j] - a[j] * inv[i] * sum);
        if (HAS_DRES) {
          float r[8];
          unpack_row8(rv[i], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] += r[j];
        }
        *reinterpret_cast<uint4*>(dx + (row0 + i) * d + col) = pack_row8(a);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) cols[warp][j * 32 + lane] = dw[j];
  __syncthreads();
  if (slot == 0 && live) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float sum = dw[j];
      for (int o = 1; o < slots; ++o) sum += cols[warp + o * wpr][j * 32 + lane];
      dw[j] = sum;
    }
    float4* out = reinterpret_cast<float4*>(partial + (long long)blockIdx.x * d + col);
    out[0] = make_float4(dw[0], dw[1], dw[2], dw[3]);
    out[1] = make_float4(dw[4], dw[5], dw[6], dw[7]);
  }
}

// Sums `parts` partial rows of N columns in a fixed order: 32 columns a block, eight groups of rows (one thread per column over all
// parts took 10 us for 296 x 384; now 2.5). Writes fp32 (added to what is there with `accumulate`) or bf16.
__global__ void __launch_bounds__(256) column_parts_kernel(const float* __restrict__ partial, int parts, int N, float* __restrict__ out,
                                                           __nv_bfloat16* __restrict__ out16, int accumulate) {
  __shared__ float red[8][33];
  const int group = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < N) {
#pragma unroll 8
    for (int p = group; p < parts; p += 8) s += partial[(long long)p * N + c];
  }
  red[group][lane] = s;
  __syncthreads();
  if (group == 0 && c < N) {
#pragma unroll
    for (int i = 1; i < 8; ++i) s += red[i][lane];
    if (out16 != nullptr) out16[c] = __float2bfloat16(s);
    else out[c] = accumulate ? out[c] + s : s;
  }
}

// ---------------------------------------------------------------- q/k feature map + RoPE
// in: rows of width in_ld holding q at column 0 and k at column k_col_offset (both [H, D]). One vector = one
// (token, head, q-or-k) row of D elements, handled by D/8 lanes with one 16-byte load each; the rotation
// partner of element i (i + D/2) lives in lane ^ (D/16). out: [tokens, 2, H, D] contiguous. cos/sin: rows of
// `tab_ld` floats of which D/2 are used, token t uses position (t % T) (tokens are laid out [B, T]); read in place and in 16-byte
// vectors. In the backward pass vectors are numbered in 32 bits: their division into token, head and side in 64 bits cost a seventh of
// the time (32768 tokens, 6 heads of 64, before -> after: 50 -> 40 us; 8192 tokens, 8 heads of 128: 36 -> 29).
template <int D>
struct PrepGeom {
  static constexpr int LPV = D / 8;        // lanes per vector
  static constexpr int VPW = 32 / LPV;     // vectors per warp
};

template <int LPV>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LPV / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]);
  u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]);
  u.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

__device__ __forceinline__ void table8(const float* t, long long at, float none, float (&f)[8]) {
  if (t == nullptr) {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = none;
    return;
  }
  const float4 a = *reinterpret_cast<const float4*>(t + at), b = *reinterpret_cast<const float4*>(t + at + 4);
  f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
}

// A warp takes one token: its lanes' rotary factors are read once for all heads, queries and keys, of which VPW vectors at a time pass
// through it, PREP_AHEAD steps of loads in flight. Few tokens are cut into `parts` of their vectors. Bound by instructions, then by
// memory; one vector after another with its token, head and factors looked up each time -> here: 32768 tokens, 6 heads of 64, 30 ->
// 25 us (4.1 TB/s); 8192, 12 of 128, 31 -> 21; 8192, 16 of 128, 49 -> 31; 65536, 6 of 64, 59 -> 49. The backward pass, with
// two rows and twice the registers a vector, is the slower for it (40 -> 51 us) and stays vector by vector.
constexpr int PREP_AHEAD = 4;

template <int D>
__global__ void __launch_bounds__(256) qk_prep_fwd_kernel(const __nv_bfloat16* __restrict__ in, long long in_ld,
                                                          int k_col_offset, __nv_bfloat16* __restrict__ out,
                                                          const float* __restrict__ cs, const float* __restrict__ sn, int tab_ld,
                                                          long long tokens, int T, int H, int parts) {
  constexpr int LPV = PrepGeom<D>::LPV, VPW = PrepGeom<D>::VPW;
  const int lane = threadIdx.x & 31, sub = lane % LPV, vin = lane / LPV, steps = (2 * H + VPW - 1) / VPW;
  const bool upper = sub >= LPV / 2;
  const int ci = (sub % (LPV / 2)) * 8;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < tokens * parts; item += warps) {
    const long long tok = parts == 1 ? item : item / parts;
    const int part = parts == 1 ? 0 : (int)(item - tok * parts);
    const int s0 = part * steps / parts, s1 = (part + 1) * steps / parts;
    const unsigned pos = (unsigned)tok % (unsigned)T;
    const __nv_bfloat16* src = in + tok * in_ld + sub * 8;
    __nv_bfloat16* dst = out + tok * 2 * H * D + sub * 8;
    float tc[8], ts[8];
    table8(cs, (long long)pos * tab_ld + ci, 1.f, tc);
    table8(sn, (long long)pos * tab_ld + ci, 0.f, ts);
    for (int s = s0; s < s1; s += PREP_AHEAD) {
      uint4 raw[PREP_AHEAD];
#pragma unroll
      for (int n = 0; n < PREP_AHEAD; ++n) {
        const int v = min((s + n) * VPW + vin, 2 * H - 1);  // queries' heads, then keys'
        if (s + n < s1) raw[n] = *reinterpret_cast<const uint4*>(src + (v < H ? v * D : k_col_offset + (v - H) * D));
      }
#pragma unroll
      for (int n = 0; n < PREP_AHEAD; ++n) {
        if (s + n >= s1) break;
        const int v = (s + n) * VPW + vin;
        float f[8];
        unpack_row8(raw[n], f);
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          f[i] = f[i] > 0.f ? f[i] + 1.f : __expf(f[i]);
          ss += f[i] * f[i];
        }
        ss = group_sum<LPV>(ss);
        const float inv = 1.0f / fmaxf(sqrtf(ss), 1e-6f);
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float mine = f[i] * inv;
          const float other = __shfl_xor_sync(0xffffffffu, mine, LPV / 2);
          const float c = tc[i], t = ts[i];
          o[i] = upper ? (mine * c + other * t) : (mine * c - other * t);
        }
        if (v < 2 * H) store8(dst + v * D, o);
      }
    }
  }
}

// Backward: recompute f and n from the raw input, undo the rotation on the incoming gradient, then
// d f = (dn - n (n . dn)) / |f| and d raw = d f * (raw > 0 ? 1 : f). Writes into d_in at the same
// column layout as `in` (q at 0, k at k_col_offset).
template <int D>
__global__ void __launch_bounds__(256) qk_prep_bwd_kernel(const __nv_bfloat16* __restrict__ in, long long in_ld,
                                                          int k_col_offset, const __nv_bfloat16* __restrict__ dout,
                                                          __nv_bfloat16* __restrict__ d_in, long long d_in_ld,
                                                          const float* __restrict__ cs, const float* __restrict__ sn, int tab_ld,
                                                          long long tokens, int T, int H) {
  constexpr int LPV = PrepGeom<D>::LPV, VPW = PrepGeom<D>::VPW;
  const int lane = threadIdx.x & 31, sub = lane % LPV, vin = lane / LPV;
  const long long total = tokens * 2 * H;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * VPW; base < total;
       base += warps * VPW) {
    const long long idx = base + vin;
    const bool live = idx < total;
    const unsigned cidx = (unsigned)(live ? idx : total - 1), pair = cidx / (unsigned)H, tok32 = pair >> 1;
    const int h = (int)(cidx - pair * (unsigned)H), which = (int)(pair & 1u);
    const long long tok = tok32;
    float raw[8], f[8], g[8], dn[8];
    load8(in + tok * in_ld + (which ? k_col_offset : 0) + h * D + sub * 8, raw);
    load8(dout + ((tok * 2 + which) * H + h) * D + sub * 8, g);
    float ss = 0.f;
    const bool upper = sub >= LPV / 2;
    const long long pos = tok32 % (unsigned)T;
    const int ci = (sub % (LPV / 2)) * 8;
    float tc[8], ts[8];
    table8(cs, pos * tab_ld + ci, 1.f, tc);
    table8(sn, pos * tab_ld + ci, 0.f, ts);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      f[i] = raw[i] > 0.f ? raw[i] + 1.f : __expf(raw[i]);
      ss += f[i] * f[i];
      const float other = __shfl_xor_sync(0xffffffffu, g[i], LPV / 2);
      const float c = tc[i], s = ts[i];
      // transpose of the rotation: lower half gets g*c + g_partner*s, upper half g*c - g_partner*s
      dn[i] = upper ? (g[i] * c - other * s) : (g[i] * c + other * s);
    }
    ss = group_sum<LPV>(ss);
    const float inv = 1.0f / fmaxf(sqrtf(ss), 1e-6f);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) dot += f[i] * inv * dn[i];
    dot = group_sum<LPV>(dot);
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float df = (dn[i] - f[i] * inv * dot) * inv;
      o[i] = df * (raw[i] > 0.f ? 1.f : f[i]);
    }
    if (live) store8(d_in + tok * d_in_ld + (which ? k_col_offset : 0) + h * D + sub * 8, o);
  }
}

// Parts that a token's vectors are cut into: enough warps for the chip (eight on each of 592 schedulers), a step at least for each.
inline int prep_parts(long long tokens, int H, int D) {
  const int steps = (2 * H + 256 / D - 1) / (256 / D);
  const long long want = (148ll * 32 + tokens - 1) / tokens;
  return (int)(want < 1 ? 1 : want > steps ? steps : want);
}

inline int row_grid(long long work_items, int per_block) {
  long long b = (work_items + per_block - 1) / per_block;
  const long long cap = 148ll * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}


// Warps per row and threads of a block of whole rows, rows in flight, blocks (at most `cap`) of the kernels that spread a row.
struct WideGeom {
  int wpr, threads, blocks;
  bool four;  // four rows in flight, where that leaves every SM two blocks; else one
};
WideGeom wide_geom(int rows, int d, int cap) {
  WideGeom g;
  g.wpr = (d + 255) / 256;
  const int slots = 8 / g.wpr;
  g.threads = slots * g.wpr * 32;
  g.four = rows >= 148 * 2 * slots * 4;
  const int per = slots * (g.four ? 4 : 1), need = (rows + per - 1) / per;
  g.blocks = need < cap ? need : cap;
  return g;
}

// Where a warp per row is the better forward kernel (figures above).
bool rows_per_warp(int rows, int d, bool residual) {
  if (d > 1024 || rows <= 148 * 8) return false;
  if (!residual || d <= 512) return true;
  return rows > 148 * 16 && (d <= 768 || rows <= 148 * 64);
}

template <bool HAS_RES>
void rmsnorm_fwd(const __nv_bfloat16* x, const __nv_bfloat16* res, const __nv_bfloat16* w, __nv_bfloat16* y, __nv_bfloat16* sum_out,
                 float* rstd, int rows, int d, float eps, cudaStream_t s) {
  if (rows_per_warp(rows, d, HAS_RES)) {
    const int grid = row_grid(rows, 8);
    if (d <= 512) rmsnorm_fwd_kernel<HAS_RES, 2><<<grid, 256, 0, s>>>(x, res, w, y, sum_out, rstd, rows, d, eps);
    else rmsnorm_fwd_kernel<HAS_RES, 4><<<grid, 256, 0, s>>>(x, res, w, y, sum_out, rstd, rows, d, eps);
    return;
  }
  const WideGeom g = wide_geom(rows, d, 148 * 8);
  const cudaError_t e = launch_dependent(g.four ? rmsnorm_fwd_wide_kernel<HAS_RES, 4> : rmsnorm_fwd_wide_kernel<HAS_RES, 1>, dim3(g.blocks),
                                         dim3(g.threads), s, x, res, w, y, sum_out, rstd, rows, d, eps, g.wpr);
  if (e != cudaSuccess) throw std::runtime_error(std::string("rmsnorm launch failed: ") + cudaGetErrorString(e));
}

template <bool HAS_DRES>
void rmsnorm_bwd(const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* dy, const float* rstd, const __nv_bfloat16* dres,
                 __nv_bfloat16* dx, float* partial, int rows, int d, cudaStream_t s) {
  const WideGeom g = wide_geom(rows, d, NORM_PARTS);
  if (g.four) rmsnorm_bwd_kernel<HAS_DRES, 4><<<g.blocks, g.threads, 0, s>>>(x, w, dy, rstd, dres, dx, partial, rows, d, g.wpr);
  else rmsnorm_bwd_kernel<HAS_DRES, 1><<<g.blocks, g.threads, 0, s>>>(x, w, dy, rstd, dres, dx, partial, rows, d, g.wpr);
}

}  // namespace

void launch_rmsnorm_fwd(const __nv_bfloat16* x, const __nv_bfloat16* res, const __nv_bfloat16* w, __nv_bfloat16* y,
                        __nv_bfloat16* sum_out, float* rstd, int rows, int d, float eps, cudaStream_t s) {
  if (rows == 0) return;
  if (res != nullptr) rmsnorm_fwd<true>(x, res, w, y, sum_out, rstd, rows, d, eps, s);
  else rmsnorm_fwd<false>(x, nullptr, w, y, nullptr, rstd, rows, d, eps, s);
}

void launch_column_parts(const float* partial, int parts, int N, const ColumnSum& out, cudaStream_t s) {
  column_parts_kernel<<<(N + 31) / 32, 256, 0, s>>>(partial, parts, N, out.out, out.out16, out.add ? 1 : 0);
}

int rmsnorm_bwd_parts(int rows, int d) { return wide_geom(rows, d, NORM_PARTS).blocks; }

void launch_rmsnorm_bwd(const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* dy, const float* rstd,
                        const __nv_bfloat16* dres, __nv_bfloat16* dx, float* partial, const ColumnSum& dw, int rows, int d,
                        cudaStream_t s) {
  if (rows > 0) {
    if (dres != nullptr) rmsnorm_bwd<true>(x, w, dy, rstd, dres, dx, partial, rows, d, s);
    else rmsnorm_bwd<false>(x, w, dy, rstd, nullptr, dx, partial, rows, d, s);
  }
  launch_column_parts(partial, rows > 0 ? rmsnorm_bwd_parts(rows, d) : 0, d, dw, s);
}

static void check_vectors(long long n) {  // 2^32 vectors of 64 are 550 GB
  if (n > 0xffffffffll) throw std::runtime_error("qk_prep: more than 2^32 vectors");
}

void launch_qk_prep_fwd(const __nv_bfloat16* in, long long in_ld, int k_col_offset, __nv_bfloat16* out, const float* cs,
                        const float* sn, int tab_ld, long long tokens, int T, int H, int D, cudaStream_t s) {
  if (tokens == 0) return;
  check_vectors(tokens * 2 * H);
  const int parts = prep_parts(tokens, H, D), grid = row_grid(tokens * parts, 8);
  if (D == 64)
    qk_prep_fwd_kernel<64><<<grid, 256, 0, s>>>(in, in_ld, k_col_offset, out, cs, sn, tab_ld, tokens, T, H, parts);
  else
    qk_prep_fwd_kernel<128><<<grid, 256, 0, s>>>(in, in_ld, k_col_offset, out, cs, sn, tab_ld, tokens, T, H, parts);
}

void launch_qk_prep_bwd(const __nv_bfloat16* in, long long in_ld, int k_col_offset, const __nv_bfloat16* dout,
                        __nv_bfloat16* d_in, long long d_in_ld, const float* cs, const float* sn, int tab_ld, long long tokens,
                        int T, int H, int D, cudaStream_t s) {
  if (tokens == 0) return;
  check_vectors(tokens * 2 * H);
  const int grid = row_grid(tokens * 2 * H, 8 * (256 / D));
  if (D == 64)
    qk_prep_bwd_kernel<64><<<grid, 256, 0, s>>>(in, in_ld, k_col_offset, dout, d_in, d_in_ld, cs, sn, tab_ld, tokens, T, H);
  else
    qk_prep_bwd_kernel<128><<<grid, 256, 0, s>>>(in, in_ld, k_col_offset, dout, d_in, d_in_ld, cs, sn, tab_ld, tokens, T, H);
}


// ------------------------------------------------------------------------------------------------
// Column sums of a bf16 matrix (bias gradients): out[n] (+)= sum_m x[m, n].
// Phase 1: a block owns a 256-column slab and every gridDim.y-th group of 8 rows; a warp reads 512 contiguous bytes
// of one row per step, a thread keeps 8 fp32 sums, the block's 8 warps are combined through shared memory and one
// partial row is written per block. Phase 2 adds the partial rows in a fixed order, so results are reproducible.
// ------------------------------------------------------------------------------------------------
namespace {

__global__ void __launch_bounds__(256) colsum_partial_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int M,
                                                             int N, float* __restrict__ partial) {
  __shared__ float red[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (col < N) {
#pragma unroll 4
    for (int m = blockIdx.y * 8 + warp; m < M; m += gridDim.y * 8) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + (long long)m * ld + col);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        acc[2 * i] += f.x;
        acc[2 * i + 1] += f.y;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[warp][lane * 8 + i] = acc[i];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < N) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
    partial[(long long)blockIdx.y * N + c] = s;
  }
}

}  // namespace

int colsum_parts(int M, int N) {
  const int slabs = (N + 255) / 256;
  int parts = (148 * 4 + slabs - 1) / slabs;
  const int max_parts = (M + 63) / 64;  // at least 8 rows per warp
  if (parts > max_parts) parts = max_parts;
  return parts < 1 ? 1 : parts;
}

void launch_colsum(const __nv_bfloat16* x, long long ld, int M, int N, float* partial, int parts,
                   const ColumnSum& out, cudaStream_t s) {
  dim3 grid((N + 255) / 256, parts);
  colsum_partial_kernel<<<grid, 256, 0, s>>>(x, ld, M, N, partial);
  launch_column_parts(partial, parts, N, out, s);
}

}  // namespace tb
