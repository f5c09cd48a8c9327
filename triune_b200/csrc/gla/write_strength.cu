// Write strengths of the delta rule, beta = sigmoid(x W^T) with x [rows, dim] and one row of W per head (up to 16), and their
// gradient. Both are passes over x; a library product of so few columns took 7 us forward and, split from the sigmoid and the
// conversions around it, nine launches in all (8192 x 1024, 8 heads: 13 us forward, 27 backward; 600 x 384: 6
// and 152, one 128 x 64 tile reducing over all rows). Now 5.7 and 29 us, 2.4 and 10 us.
//
// Forward: a CTA takes 16 rows, its eight warps slices of dim; rows and weights go from global memory straight into mma.sync
// fragments (the few heads are the narrow side), logits stay fp32. Backward: with dl = dbeta beta (1 - beta), one pass reads x
// once for dx = dl W and dW = dl^T x: a thread owns four columns, holds W and its sums for all heads, and walks the rows of its
// block; partial sums of the blocks are added in a fixed order afterwards.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "../common/ptx.cuh"
#include "gla.cuh"

namespace tb {

namespace {

constexpr int WARPS = 8, ROWS = 16, COLS = 512, STAGE = 32;  // columns and staged rows of a backward block

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: groups of eight heads. The order of k within a step of 32 is free as long as both fragments agree: a lane's eight
// contiguous values are the k pairs of two products.
template <int NT>
__global__ void __launch_bounds__(WARPS * 32) strength_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx,
                                                                  const __nv_bfloat16* __restrict__ w, float* __restrict__ beta, int rows,
                                                                  int dim, int H) {
  __shared__ float sums[WARPS][ROWS][NT * 8 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = blockIdx.x * ROWS, steps = (dim + 31) / 32;
  const bool in0 = r0 + g < rows, in1 = r0 + g + 8 < rows;
  const __nv_bfloat16* x0 = x + (long long)(r0 + g) * ldx + t * 8;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
#pragma unroll 4
  for (int s = warp; s < steps; s += WARPS) {
    const int k = s * 32;
    const bool in = k + t * 8 < dim;
    const uint4 a = (in0 && in) ? *reinterpret_cast<const uint4*>(x0 + k) : zero;
    const uint4 b = (in1 && in) ? *reinterpret_cast<const uint4*>(x0 + 8 * ldx + k) : zero;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int h = j * 8 + g;
      const uint4 v = (h < H && in) ? *reinterpret_cast<const uint4*>(w + (long long)h * dim + k + t * 8) : zero;
      mma16816(acc[j], a.x, b.x, a.y, b.y, v.x, v.y);
      mma16816(acc[j], a.z, b.z, a.w, b.w, v.z, v.w);
    }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    sums[warp][g][j * 8 + 2 * t] = acc[j][0];
    sums[warp][g][j * 8 + 2 * t + 1] = acc[j][1];
    sums[warp][g + 8][j * 8 + 2 * t] = acc[j][2];
    sums[warp][g + 8][j * 8 + 2 * t + 1] = acc[j][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ROWS * H; i += WARPS * 32) {
    const int r = i / H, h = i % H;
    if (r0 + r >= rows) break;
    float z = 0.f;
#pragma unroll
    for (int p = 0; p < WARPS; ++p) z += sums[p][r][h];
    beta[(long long)(r0 + r) * H + h] = 1.f / (1.f + __expf(-z));
  }
}

template <int HP>  // heads, rounded up to 8 or 16
__global__ void __launch_bounds__(COLS / 4) strength_bwd_kernel(const float* __restrict__ dbeta, const float* __restrict__ beta,
                                                                const __nv_bfloat16* __restrict__ x, long long ldx,
                                                                const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ dx,
                                                                float* __restrict__ partial, int rows, int dim, int H) {
  __shared__ __align__(16) float dl[STAGE][HP];
  const int col = blockIdx.y * COLS + threadIdx.x * 4;
  const bool live = col < dim;
  auto load4 = [](const __nv_bfloat16* p, float (&f)[4]) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    f[0] = __uint_as_float(u.x << 16), f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16), f[3] = __uint_as_float(u.y & 0xffff0000u);
  };
  float wv[HP][4], acc[HP][4];
#pragma unroll
  for (int h = 0; h < HP; ++h) {
#pragma unroll
    for (int j = 0; j < 4; ++j) wv[h][j] = acc[h][j] = 0.f;
    if (live && h < H) load4(w + (long long)h * dim + col, wv[h]);
  }
  for (int r0 = blockIdx.x * STAGE; r0 < rows; r0 += gridDim.x * STAGE) {
    __syncthreads();
    for (int i = threadIdx.x; i < STAGE * HP; i += COLS / 4) {
      const int r = r0 + i / HP, h = i % HP;
      float v = 0.f;
      if (r < rows && h < H) {
        const float be = beta[(long long)r * H + h];
        v = dbeta[(long long)r * H + h] * be * (1.f - be);
      }
      dl[i / HP][h] = v;
    }
    __syncthreads();
    if (!live) continue;
    const int m = min(STAGE, rows - r0);
#pragma unroll 2
    for (int r = 0; r < m; ++r) {
      float xv[4], o[4] = {0.f, 0.f, 0.f, 0.f};
      load4(x + (long long)(r0 + r) * ldx + col, xv);
#pragma unroll
      for (int h4 = 0; h4 < HP; h4 += 4) {
        const float4 d4 = *reinterpret_cast<const float4*>(&dl[r][h4]);
        const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[h4 + i][j] += d[i] * xv[j];
            o[j] += d[i] * wv[h4 + i][j];
          }
      }
      *reinterpret_cast<uint2*>(dx + (long long)(r0 + r) * dim + col) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
    }
  }
  if (!live) return;
#pragma unroll
  for (int h = 0; h < HP; ++h)
    if (h < H)
      *reinterpret_cast<float4*>(partial + ((long long)blockIdx.x * H + h) * dim + col) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
}

void check(const char* what, int dim, int H) {
  if (dim % 8 != 0 || H < 1 || H > STRENGTH_MAX_HEADS) throw std::runtime_error(std::string(what) + ": dim a multiple of 8, 1 to 16 heads");
}
void launched(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + " launch failed: " + cudaGetErrorString(e));
}

}  // namespace

void launch_strength_fwd(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, float* beta, int rows, int dim, int H,
                         cudaStream_t s) {
  check("strength_fwd", dim, H);
  if (rows == 0) return;
  const int grid = (rows + ROWS - 1) / ROWS;
  if (H <= 8) strength_fwd_kernel<1><<<grid, WARPS * 32, 0, s>>>(x, ldx, w, beta, rows, dim, H);
  else strength_fwd_kernel<2><<<grid, WARPS * 32, 0, s>>>(x, ldx, w, beta, rows, dim, H);
  launched("strength_fwd");
}

// Row blocks of the backward pass: two CTAs per SM over the column slabs, each with 32 rows at least.
int strength_bwd_parts(int rows, int dim) {
  const int slabs = (dim + COLS - 1) / COLS, most = 296 / slabs > 0 ? 296 / slabs : 1, need = (rows + STAGE - 1) / STAGE;
  return need < most ? need : most;
}

void launch_strength_bwd(const float* dbeta, const float* beta, const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w,
                         __nv_bfloat16* dx, float* partial, int rows, int dim, int H, cudaStream_t s) {
  check("strength_bwd", dim, H);
  if (rows == 0) return;
  const dim3 grid(strength_bwd_parts(rows, dim), (dim + COLS - 1) / COLS);
  if (H <= 8) strength_bwd_kernel<8><<<grid, COLS / 4, 0, s>>>(dbeta, beta, x, ldx, w, dx, partial, rows, dim, H);
  else strength_bwd_kernel<16><<<grid, COLS / 4, 0, s>>>(dbeta, beta, x, ldx, w, dx, partial, rows, dim, H);
  launched("strength_bwd");
}

}  // namespace tb
