// Products of a few rows (decoding: one token per sequence, short chat turns) with a K-major weight: C [M, N] = A [M, K] B [N, K]^T.
//
// Such a product is a stream over the weight: 2 N K bytes at a floor of memory bandwidth, with M <= 16 multiply-adds per
// weight. A 128-row tcgen05 tile has one CTA per 64 to 256 output columns, each with four to eight loads of the weight in
// flight (1 x 8192 x 2048: 24.8 us, five times the bytes' time). Here a warp owns 16 output columns over a slice of K: weights
// go from global memory straight into mma.sync A fragments (16 weight rows x 16), rows of A are the 8 columns of the B
// fragment, sums are fp32. The order of k within a 32-wide step is free as long as both fragments agree on it, so a lane's
// eight contiguous weights (one 16-byte load) are the k pairs {2 t, 2 t + 1, 2 t + 8, 2 t + 9} of two steps, and the four
// lanes of a row read a whole 128-byte line in two loads. The W warps of a CTA split K and their partial sums meet in
// shared memory; W is chosen so that about 16 warps per SM stream (16 KB in flight each SM at four loads a lane and more).
// Four steps of loads are kept in flight, and the kernel is launched over the end of the one before it (dependent_launch.cuh).
// Nothing is staged: a slice of A is read by one warp of the CTA only. Measured with the weight in DRAM (M = 1 to 8, before ->
// after): 8192 x 2048 20.2 -> 11.7 us, 2048 x 2048 18.6 -> 5.4, 2048 x 5632 39.0 -> 10.4, 32000 x 2048 36 -> 30, gated 5632 x
// 2048 23.2 -> 14.3; at 16 rows 20.1 -> 12.0, 18.5 -> 6.5, 39.0 -> 12.2, 34.6 -> 32.9, 23.3 -> 16.1.
#include <cuda_bf16.h>

#include <stdexcept>
#include <string>

#include "../common/dependent_launch.cuh"
#include "../common/ptx.cuh"
#include "tc_gemm.cuh"

namespace tb {

namespace {

constexpr int SK_ROWS = 16;  // weight rows per CTA (and per half of a gated CTA)

__device__ __forceinline__ void mma_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load_stream(const __nv_bfloat16* p, bool ok) {  // read once: do not keep it in L1
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (ok) asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// GLU: output column n pairs weight rows n (gate) and n + N (up). NT: groups of eight rows of A.
template <int W, int NT, bool GLU>
__global__ void __launch_bounds__(W * 32) skinny_kernel(const __nv_bfloat16* __restrict__ A, long long lda, const __nv_bfloat16* __restrict__ B,
                                                        long long ldb, __nv_bfloat16* __restrict__ C, long long ldc, int M, int N, int K,
                                                        float alpha, const __nv_bfloat16* __restrict__ bias, int gelu) {
  constexpr int PARTS = GLU ? 2 : 1;
  __shared__ float sums[W][PARTS][NT * 8][SK_ROWS + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * SK_ROWS;
  wait_predecessors();
  const int steps = (K + 63) / 64, s0 = (int)((long long)warp * steps / W), s1 = (int)((long long)(warp + 1) * steps / W);
  float acc[PARTS][NT][4];
#pragma unroll
  for (int p = 0; p < PARTS; ++p)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[p][j][i] = 0.f;
  const bool r0 = n0 + g < N, r1 = n0 + g + 8 < N;
  const __nv_bfloat16* w0 = B + (long long)(n0 + g) * ldb + t * 8;
#pragma unroll 4
  for (int s = s0; s < s1; ++s) {
    const int k = s * 64;
    const bool lo = k + t * 8 < K, hi = k + 32 + t * 8 < K;
    uint4 a[PARTS][4], b[NT][2];
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
      const __nv_bfloat16* w = w0 + (long long)p * N * ldb + k;
      a[p][0] = load_stream(w, r0 && lo);
      a[p][1] = load_stream(w + 8 * ldb, r1 && lo);
      a[p][2] = load_stream(w + 32, r0 && hi);
      a[p][3] = load_stream(w + 8 * ldb + 32, r1 && hi);
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int m = j * 8 + g;
      const __nv_bfloat16* x = A + (long long)m * lda + k + t * 8;
      b[j][0] = (m < M && lo) ? *reinterpret_cast<const uint4*>(x) : make_uint4(0u, 0u, 0u, 0u);
      b[j][1] = (m < M && hi) ? *reinterpret_cast<const uint4*>(x + 32) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int p = 0; p < PARTS; ++p)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          mma_16x8x16(acc[p][j], a[p][2 * h].x, a[p][2 * h + 1].x, a[p][2 * h].y, a[p][2 * h + 1].y, b[j][h].x, b[j][h].y);
          mma_16x8x16(acc[p][j], a[p][2 * h].z, a[p][2 * h + 1].z, a[p][2 * h].w, a[p][2 * h + 1].w, b[j][h].z, b[j][h].w);
        }
  }
  allow_dependents();  // the loads are in: the next kernel's blocks may come while sums meet and are written
#pragma unroll
  for (int p = 0; p < PARTS; ++p)
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      sums[warp][p][j * 8 + 2 * t][g] = acc[p][j][0];
      sums[warp][p][j * 8 + 2 * t + 1][g] = acc[p][j][1];
      sums[warp][p][j * 8 + 2 * t][g + 8] = acc[p][j][2];
      sums[warp][p][j * 8 + 2 * t + 1][g + 8] = acc[p][j][3];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < NT * 8 * SK_ROWS; i += W * 32) {
    const int m = i / SK_ROWS, n = i % SK_ROWS;
    if (m >= M || n0 + n >= N) continue;
    float v = 0.f, u = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      v += sums[w][0][m][n];
      if constexpr (GLU) u += sums[w][1][m][n];
    }
    if constexpr (GLU) {
      v = v * __fdividef(1.f, 1.f + __expf(-v)) * u;
    } else {
      v = fmaf(v, alpha, bias != nullptr ? __bfloat162float(bias[n0 + n]) : 0.f);
      if (gelu) v = gelu_tanh_f(v);
    }
    C[(long long)m * ldc + n0 + n] = __float2bfloat16(v);
  }
}

template <int W, int NT>
void run(const GemmArgs& a, int blocks, cudaStream_t s) {
  auto c = reinterpret_cast<__nv_bfloat16*>(a.C);
  const bool glu = (a.flags & GF_SWIGLU) != 0;
  const cudaError_t e = launch_dependent(glu ? skinny_kernel<W, NT, true> : skinny_kernel<W, NT, false>, dim3(blocks), dim3(W * 32), s, a.A, a.lda,
                                         a.B, a.ldb, c, a.ldc, a.M, a.N, a.K, glu ? 1.f : a.alpha, glu ? nullptr : a.bias,
                                         (a.flags & GF_GELU) != 0 ? 1 : 0);
  if (e != cudaSuccess) throw std::runtime_error(std::string("skinny_gemm launch failed: ") + cudaGetErrorString(e));
}

}  // namespace

bool launch_skinny_gemm(const GemmArgs& a, cudaStream_t s) {
  if (a.mode != GEMM_DENSE || a.batch > 1 || a.M > SKINNY_MAX_M || a.a_mn_major || a.b_mn_major || a.row_scale != nullptr ||
      a.aux_in != nullptr || a.aux_out != nullptr || (a.flags & ~(GF_GELU | GF_SWIGLU)) != 0)
    return false;
  if ((a.flags & GF_SWIGLU) && (a.glu_act != 0 || a.glu_bias != nullptr)) return false;
  // rows are read in 16-byte vectors
  if (a.K % 8 != 0 || ((reinterpret_cast<uintptr_t>(a.A) | reinterpret_cast<uintptr_t>(a.B)) & 15) != 0) return false;
  const int blocks = (a.N + SK_ROWS - 1) / SK_ROWS;
  const int warps = skinny_warps(a.N, a.K);
  if (a.M <= 8) {
    if (warps == 16) run<16, 1>(a, blocks, s);
    else if (warps == 8) run<8, 1>(a, blocks, s);
    else run<4, 1>(a, blocks, s);
  } else {
    if (warps == 16) run<16, 2>(a, blocks, s);
    else if (warps == 8) run<8, 2>(a, blocks, s);
    else run<4, 2>(a, blocks, s);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("skinny_gemm launch failed: ") + cudaGetErrorString(e));
  return true;
}

}  // namespace tb
