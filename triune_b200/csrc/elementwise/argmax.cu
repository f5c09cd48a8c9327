// Index of the largest value of each row of bf16 logits (a decoding step's choice of the next token), as torch.argmax orders them:
// NaN above everything, the first of equals, -0 equal to 0. One CTA per row, 16-byte loads; a value's order and its index travel as one
// 64-bit number whose maximum is taken. Bound by latency: 32000 logits take 5.3 us (a library reduction and a copy 10.7), a decoding
// step 277 instead of 284 us. Rows of up to 2048 values take 256 threads and those of up to 256 one warp: with 1024 threads each,
// 2048 rows of 256 took 9.9 us (the library 5.1), now 3.0; 2048 rows of 2000 11.2 (10.8), now 6.9.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "../common/dependent_launch.cuh"
#include "elementwise.cuh"

namespace tb {

namespace {

__device__ __forceinline__ uint32_t order16(uint32_t u) {  // bf16 bits -> a number in the order of the values
  if ((u & 0x7fffu) > 0x7f80u) return 0xffffu;
  if (u == 0x8000u) u = 0u;
  return (u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) argmax_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int V,
                                                              long long* __restrict__ out) {
  __shared__ unsigned long long red[THREADS / 32];
  wait_predecessors();
  const unsigned short* row = reinterpret_cast<const unsigned short*>(x + (long long)blockIdx.x * ld);
  uint32_t best = 0u, at = 0xffffffffu;  // indexes grow within a thread: only a larger value replaces the best
  auto take = [&](uint32_t bits, uint32_t i) {
    const uint32_t k = order16(bits);
    if (k > best || at == 0xffffffffu) best = k, at = i;
  };
  const int vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0 ? V / 8 : 0;
#pragma unroll 4
  for (int i = threadIdx.x; i < vec; i += THREADS) {
    const uint4 u = *reinterpret_cast<const uint4*>(row + i * 8);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      take(w[j] & 0xffffu, i * 8 + 2 * j);
      take(w[j] >> 16, i * 8 + 2 * j + 1);
    }
  }
  for (int i = vec * 8 + threadIdx.x; i < V; i += THREADS) take(row[i], i);
  unsigned long long v = at == 0xffffffffu ? 0ull : ((unsigned long long)best << 32) | (0xffffffffu - at);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < THREADS / 32 ? red[threadIdx.x] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
      v = w > v ? w : v;
    }
    if (threadIdx.x == 0) out[blockIdx.x] = (long long)(0xffffffffu - (uint32_t)v);
  }
}

}  // namespace

void launch_argmax_rows(const __nv_bfloat16* x, long long ld, int rows, int V, long long* out, cudaStream_t s) {
  if (rows <= 0) return;
  if (V <= 0) throw std::runtime_error("argmax_rows: empty rows");
  const int threads = V > 2048 ? 1024 : V > 256 ? 256 : 32;
  const cudaError_t e = launch_dependent(threads == 1024 ? argmax_rows_kernel<1024> : threads == 256 ? argmax_rows_kernel<256> : argmax_rows_kernel<32>,
                                         dim3(rows), dim3(threads), s, x, ld, V, out);
  if (e != cudaSuccess) throw std::runtime_error(std::string("argmax_rows launch failed: ") + cudaGetErrorString(e));
}

}  // namespace tb
