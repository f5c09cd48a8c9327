// One decoding step of a recurrent mixer (gated linear attention or the gated delta rule) from the fused projection row
// qkvg = [q | k | v | gate logits]: feature map, rotation, decay, write strength, state update and output in one launch.
//
//   q, k <- rope(normalize(elu + 1))     dec = exp(logsigmoid(gate))     beta = sigmoid(x . w_beta[h])  (delta rule, optional)
//   u = v, or v - S^T k                  S <- dec * S + (beta k) u^T     o = S^T q
//
// The step was ten to sixteen launches around a 4 us kernel (rotary rows gathered by index, feature map, 64-wide key and
// value slices expanded and summed again for 128-wide heads, the write strength's product, copies of the state), 35 us a layer;
// this kernel takes 3.0 us (16 heads of 128, one sequence). A CTA takes 32 value columns of one head (heads x D / 32
// CTAs, so that 16 heads read their 1 MB of state through 64 SMs); a thread holds D / 8 state rows of one column, read before
// anything else so that the latency of the state hides the feature map; sums across the eight row groups go through
// shared memory. Everything is fp32 from the projection row on. Bound by latency: two dependent reads and four barriers.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <stdexcept>
#include <string>

#include "../common/dependent_launch.cuh"
#include "mixer_math.cuh"

namespace tb {

namespace {

constexpr int MS_COLS = 32, MS_THREADS = 256, MS_PARTS = MS_THREADS / MS_COLS;

__device__ __forceinline__ float ms_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int D, bool DELTA>
__global__ void __launch_bounds__(MS_THREADS) mixer_step_kernel(const MixerStep p) {
  constexpr int RP = D / MS_PARTS, QW = D / 32;  // state rows per thread; warps per q or k vector
  __shared__ float feat[2][D], vec[2][D], dec[D], norm[MS_THREADS / 32], bsum[MS_THREADS / 32], part[2][MS_PARTS][MS_COLS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int GROUPS = D / MS_COLS;
  const int h = blockIdx.y, b = blockIdx.x / GROUPS, HD = p.H * D, c = (blockIdx.x % GROUPS) * MS_COLS + lane, r0 = warp * RP;
  const __nv_bfloat16* row = p.qkvg + (long long)b * p.ld + h * D;
  allow_dependents();
  wait_predecessors();

  float S[RP];
  const long long at = (((long long)b * p.H + h) * D + r0) * D + c;
#pragma unroll
  for (int r = 0; r < RP; ++r) S[r] = p.state_in[at + (long long)r * D];
  const float v = __bfloat162float(row[2 * HD + c]);
  float bdot = 0.f;
  if (DELTA && p.beta_w != nullptr) {
    const __nv_bfloat16 *x = p.x + (long long)b * p.ldx, *w = p.beta_w + (long long)h * p.dim;
    for (int i = tid * 8; i < p.dim; i += MS_THREADS * 8)
      bdot = mix_dot8(*reinterpret_cast<const uint4*>(x + i), *reinterpret_cast<const uint4*>(w + i), bdot);
    bdot = ms_warp_sum(bdot);
    if (lane == 0) bsum[warp] = bdot;
  }
  const int which = tid / D, d = tid % D;  // threads [0, D): q, [D, 2 D): k
  float f = 0.f;
  if (which < 2) {
    const float raw = __bfloat162float(row[which * HD + d]);
    f = mix_feature(raw);
    const float ss = ms_warp_sum(f * f);
    if (lane == 0) norm[warp] = ss;
    feat[which][d] = f;
  }
  for (int i = tid; i < D; i += MS_THREADS) {
    dec[i] = mix_decay(__bfloat162float(row[3 * HD + i]));
  }
  __syncthreads();
  if (which < 2) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < QW; ++i) ss += norm[which * QW + i];
    const float inv = mix_inverse_norm(ss);
    if (p.cos != nullptr) {
      const long long pos = p.pos != nullptr ? *p.pos : p.pos_host;
      const bool inside = pos >= 0 && pos < p.table_rows;  // past the table there is no rotation: NaN, never another row's
      const float cs = inside ? p.cos[pos * D + d] : NAN, sn = inside ? p.sin[pos * D + d] : NAN;
      f = mix_rotate(f, feat[which][d < D / 2 ? d + D / 2 : d - D / 2], cs, sn, d < D / 2);
    }
    vec[which][d] = f * inv;
  }
  __syncthreads();
  float u = v, beta = 1.f;
  if constexpr (DELTA) {
    float acc = 0.f;
#pragma unroll
    for (int r = 0; r < RP; ++r) acc = __fmaf_rn(vec[1][r0 + r], S[r], acc);
    part[0][warp][lane] = acc;
    if (p.beta_w != nullptr) {
      float z = 0.f;
#pragma unroll
      for (int i = 0; i < MS_THREADS / 32; ++i) z += bsum[i];
      beta = mix_strength(z);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MS_PARTS; ++i) u -= part[0][i][lane];
    u *= beta;
  }
  float acc = 0.f;
#pragma unroll
  for (int r = 0; r < RP; ++r) {
    S[r] = mix_state(S[r], dec[r0 + r], vec[1][r0 + r], u);
    acc = __fmaf_rn(vec[0][r0 + r], S[r], acc);
    p.state_out[at + (long long)r * D] = S[r];
  }
  part[1][warp][lane] = acc;
  __syncthreads();
  if (warp == 0) {
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < MS_PARTS; ++i) o += part[1][i][lane];
    p.out[(long long)b * HD + h * D + c] = __float2bfloat16(o);
  }
}

}  // namespace

void launch_mixer_step(const MixerStep& p, int B, int D, bool delta, cudaStream_t s) {
  if (B <= 0 || p.H <= 0) return;
  const dim3 grid((unsigned)B * (D / MS_COLS), p.H);  // sequences along x: the other two dimensions end at 65535
  void (*kernel)(const MixerStep) = nullptr;
  if (D == 64) kernel = delta ? mixer_step_kernel<64, true> : mixer_step_kernel<64, false>;
  else if (D == 128) kernel = delta ? mixer_step_kernel<128, true> : mixer_step_kernel<128, false>;
  else throw std::runtime_error("mixer_step: head dimension must be 64 or 128");
  const cudaError_t e = launch_dependent(kernel, grid, dim3(MS_THREADS), s, p);
  if (e != cudaSuccess) throw std::runtime_error(std::string("mixer_step launch failed: ") + cudaGetErrorString(e));
}

}  // namespace tb
