// One decoding step of a dense recurrent model (gated linear attention or the gated delta rule, SwiGLU or GELU feed-forward) in
// ONE launch: every layer, the head and the arg-max.
//
// A step reads every weight once, so its floor is their bytes at memory bandwidth (6 layers of 2048, 16 heads of 128: 0.8 GB, 124 us).
// As forty kernels it took 274 us: each starts with nothing in flight, ends in a wave that thins out, and none can read
// the next one's weights before its own input is there. Here one CTA per SM stays for the whole step. A producer thread walks the
// CTA's share of every weight of the model in order and copies it into a ring of shared memory (TMA, 16 KB a copy), as far ahead as
// the ring goes (180 KB a SM, 27 MB over the chip) and without regard to where the arithmetic is; consumer warps multiply what has
// arrived by the staged input rows (mma.sync, fp32 sums). Between phases CTAs hand one another words that carry the phase's number
// beside two values (see Poll): a reader polls the words themselves, and the weights of the phases to come keep arriving meanwhile. A
// counter and a barrier of the grid instead took 1.5 us more a phase.
//
// A block is sixteen weight rows (eight gate and eight up rows) over the whole reduction; blocks are dealt to CTAs in turn, each
// phase going on where the one before stopped, so that uneven phases even out over the ring. A reduction is cut into the
// slices that the product of few rows (skinny_gemm.cu) cuts it into; copies of one or more slices go to the warps in turn. Slice
// sums meet in shared memory and are added in that kernel's order, norms, mixer and roundings follow the kernels of a
// step in pieces as well: a token decoded here and one decoded there are the same numbers.
//
// No buffer is written while it may still be read: every phase but the mixer's reads its whole input, what a CTA hands over it
// hands over after its own reads, and the next writer of a buffer is four hand-overs later.
//
// A step in pieces -> here, us: one sequence, 6 layers of 2048 (GLA) 274 -> 189; 4 (delta rule) 306 -> 258; 8 354 -> 326; 4 x 768 153 ->
// 120; 1 x 1024 (delta rule) 177 -> 123; 8 x 1536 290 -> 273. Bound by the chain of a phase (input words from L2, norm, the last
// copies' matrix steps, sums: 3 to 8 us for 31 phases) and, at the head, by memory. Registers: 168 a thread with eight consumer warps (up
// to 4 bytes spilled), 96 with sixteen (24 to 124 bytes).
//
// The grid is launched cooperatively (its CTAs wait for one another) and takes every SM, so that two decoders on two streams take turns:
// requests of 16 and 19 ms by themselves took 34 and 35 ms side by side, one of 16 ms beside a stream of products of 8192^3 48 ms.
// Every wait has a time limit, after which the step sets the status word and a word that all waits look at, lets its copies land
// and returns; later steps return at once. The host reads the status once a request.
#include "dense_step.cuh"

#include <cstring>
#include <stdexcept>
#include <string>

#include "../common/per_device.h"
#include "../common/ptx.cuh"
#include "../common/tma_desc.h"
#include "../gemm/tc_gemm.cuh"
#include "../gla/mixer_math.cuh"

namespace tb {

namespace {

constexpr int BLOCK = 16;                // weight rows of a block: the rows of a matrix instruction
constexpr int UNIT = 64;                 // columns of a copy: 128-byte rows, swizzled
constexpr int UNIT_BYTES = BLOCK * UNIT * 2;
constexpr int MAX_UNITS = 96;            // of the ring
constexpr int ITEMS = 32;                // items in flight
constexpr int STRENGTH_THREADS = 256;    // of mixer_step_kernel, whose order of sums is kept
constexpr int MAX_GROUPS = 32;           // of 256 columns of a normed row

template <int CONSUMERS>
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(CONSUMERS) : "memory"); }
// The same, and whether any thread came with `bad`: all of them take the same way afterwards.
template <int CONSUMERS>
__device__ __forceinline__ bool consumer_barrier_any(bool bad) {
  uint32_t any;
  asm volatile(
      "{\n\t"
      ".reg .pred P, Q;\n\t"
      "setp.ne.u32 P, %1, 0;\n\t"
      "bar.red.or.pred Q, 1, %2, P;\n\t"
      "selp.u32 %0, 1, 0, Q;\n\t"
      "}\n"
      : "=r"(any)
      : "r"((uint32_t)bad), "n"(CONSUMERS)
      : "memory");
  return any != 0;
}

// The units of an item, one after the other, in one copy.
__device__ __forceinline__ void load_item(uint32_t dst, const void* map, uint64_t* bar, int row, int unit, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %3, %5}], [%2], %6;" ::"r"(dst),
      "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(unit), "l"(policy)
      : "memory");
}

// Sixteen weight rows times eight input rows.
__device__ __forceinline__ void mma_rows(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What CTAs hand to one another is a 64-bit word of two bf16 values (or one fp32) and the number of the phase that wrote it: a reader
// polls the word itself, so that a hand-over is one trip to L2 and back, without fences, counters or a second read.
struct Poll {
  unsigned int* sync;
  bool bad = false;
  // Called between two looks at a word that was not there yet; true when it is time to give up.
  __device__ __forceinline__ bool expired(unsigned int& looks, unsigned long long& t0) {
    if (bad) return true;
    if ((++looks & 255u) == 0) {
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > WAIT_LIMIT_NS || *reinterpret_cast<volatile unsigned int*>(sync) != 0u) bad = true;
    }
    return bad;
  }
};
// N words at once, those of `need` (bits); all loads of a look are in flight together.
template <int N>
__device__ __forceinline__ void read_words(const unsigned long long* const (&p)[N], uint32_t flag, uint32_t need, uint32_t (&value)[N], Poll& poll) {
  unsigned int looks = 0;
  unsigned long long t0 = 0, w[N];
  do {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (need >> i & 1) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w[i]) : "l"(p[i]) : "memory");
#pragma unroll
    for (int i = 0; i < N; ++i)
      if ((need >> i & 1) && (uint32_t)(w[i] >> 32) == flag) {
        value[i] = (uint32_t)w[i];
        need &= ~(1u << i);
      }
  } while (need != 0 && !poll.expired(looks, t0));
}
// Four consecutive words: eight bf16 values.
__device__ __forceinline__ uint4 read_row(const unsigned long long* p, uint32_t flag, Poll& poll) {
  unsigned int looks = 0;
  unsigned long long t0 = 0, a, b, c, d;
  for (;;) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(c), "=l"(d) : "l"(p + 2) : "memory");
    const bool there = (uint32_t)(a >> 32) == flag && (uint32_t)(b >> 32) == flag && (uint32_t)(c >> 32) == flag && (uint32_t)(d >> 32) == flag;
    if (there || poll.expired(looks, t0)) return make_uint4((uint32_t)a, (uint32_t)b, (uint32_t)c, (uint32_t)d);
  }
}
__device__ __forceinline__ void write_word(unsigned long long* p, uint32_t value, uint32_t flag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)flag << 32) | value) : "memory");
}
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float low_half(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float high_half(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ void unpack_words(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack_words(const float (&f)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ float sum_lanes(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }

__device__ __forceinline__ uint32_t value_order(float v) {  // as torch.argmax orders bf16 values: NaN above everything, -0 equal to 0
  uint32_t u = __bfloat16_as_ushort(__float2bfloat16(v));
  if ((u & 0x7fffu) > 0x7f80u) return 0xffffu;
  if (u == 0x8000u) u = 0u;
  return (u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u);
}

// The first block (or unit) of a phase that this CTA takes; every grid-th one after it is its own too.
__device__ __forceinline__ int own_first(int first) {
  const int c = (int)blockIdx.x - first;
  return c < 0 ? c + (int)gridDim.x : c;
}

// The sums of G slices of a block, each with its terms in the order of its columns: lane (g, t) has two weight rows and input rows
// 2 t, 2 t + 1. `w`: the first unit of 64 columns, `x`: this lane's input row at its first column, `width`: units of a slice.
// Weight rows are taken in the order 0 4 1 5 2 6 3 7: the two rows that eight lanes read at once are then swizzled apart.
template <int G>
__device__ __forceinline__ void multiply_slices(const uint8_t* w, const uint8_t* x, bool live, int width, float* sums, int mb, int lane) {
  const int g = lane >> 2, t = lane & 3, r = (g >> 1) | ((g & 1) << 2);
  w += r * 128 + ((t ^ r) * 16);
  x += t * 16;
  const int up = ((t ^ r) * 16) & 64 ? -64 : 64;  // the other half of the 128-byte row
  float acc[G][4];
#pragma unroll
  for (int j = 0; j < G; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
  const int wstep = width * UNIT_BYTES, xstep = width * (UNIT * 2);
#pragma unroll(2 / G)
  for (int s = 0; s < width; ++s, w += UNIT_BYTES, x += UNIT * 2) {
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const uint8_t *wj = w + j * wstep, *xj = x + j * xstep;
      const uint4 w0 = *reinterpret_cast<const uint4*>(wj), w1 = *reinterpret_cast<const uint4*>(wj + 1024);
      const uint4 w2 = *reinterpret_cast<const uint4*>(wj + up), w3 = *reinterpret_cast<const uint4*>(wj + up + 1024);
      uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
      if (live) x0 = *reinterpret_cast<const uint4*>(xj), x1 = *reinterpret_cast<const uint4*>(xj + 64);
      mma_rows(acc[j], w0.x, w1.x, w0.y, w1.y, x0.x, x0.y);
      mma_rows(acc[j], w0.z, w1.z, w0.w, w1.w, x0.z, x0.w);
      mma_rows(acc[j], w2.x, w3.x, w2.y, w3.y, x1.x, x1.y);
      mma_rows(acc[j], w2.z, w3.z, w2.w, w3.w, x1.z, x1.w);
    }
  }
#pragma unroll
  for (int j = 0; j < G; ++j) {
    float* to = sums + (j * mb + 2 * t) * BLOCK + r;
    if (2 * t < mb) to[0] = acc[j][0], to[8] = acc[j][2];
    if (2 * t + 1 < mb) to[BLOCK] = acc[j][1], to[BLOCK + 8] = acc[j][3];
  }
}

struct Shared {
  DensePhase phase[2];
  uint64_t full[ITEMS], empty[ITEMS];
  unsigned long long best[DENSE_STEP_MAX_ROWS];
  long long token[DENSE_STEP_MAX_ROWS];
  int item_at[ITEMS], item_units[ITEMS];  // of the items in flight: first unit of the ring; units taken, with those left out at its end
  float red[DENSE_STEP_MAX_ROWS][MAX_GROUPS], warp_sum[16];
  float feat[2][128], vec[2][128], dec[128], part[2][8][128];
  int failed, last;  // for the producer: the consumers have left; of all CTAs this one was done last
};
constexpr int PHASE_WORDS = sizeof(DensePhase) / 16;
static_assert(sizeof(DensePhase) % 16 == 0 && PHASE_WORDS <= 32, "a phase is copied in 16-byte words by one warp");

// D: head dimension. CG: value columns of a unit of the mixer (D * CG / 256 state elements a thread).
template <int D, int CG, int LOG_WARPS>
__global__ void __launch_bounds__((32 << LOG_WARPS) + 32, 1) dense_step_kernel(const DenseStep p) {
  constexpr int WARPS = 1 << LOG_WARPS, CONSUMERS = WARPS * 32;
  extern __shared__ uint8_t smem_raw[];
  __shared__ Shared sh;
  uint8_t* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // units, swizzled in 1024-byte tiles
  uint8_t* act = ring + p.units * UNIT_BYTES;                        // [B] input rows
  float* sums = reinterpret_cast<float*>(act + p.B * p.act_pitch);   // [slots][rows in use, a power of two][16]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int log_mb = p.B <= 1 ? 0 : p.B <= 2 ? 1 : p.B <= 4 ? 2 : 3, mb = 1 << log_mb;
  __nv_bfloat16* nws = reinterpret_cast<__nv_bfloat16*>(sums + p.slots * mb * BLOCK);  // norm weight [d]

  if (p.sync[0] != 0u) return;  // a step before this one did not finish
  if (tid == 0) {
    for (int i = 0; i < ITEMS; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 1);
    }
    sh.failed = 0;
    mbar_fence_init();
  }
  if (tid < DENSE_STEP_MAX_ROWS) sh.best[tid] = 0ull;
  if (tid < p.B) sh.token[tid] = p.token[tid];
  if (tid < PHASE_WORDS) reinterpret_cast<uint4*>(&sh.phase[0])[tid] = reinterpret_cast<const uint4*>(p.program)[tid];
  __syncthreads();
  volatile int* failed = &sh.failed;

  if (warp == WARPS) {
    // ---------------------------------------------------------------- producer: every weight of this CTA, in order
    if (lane != 0) return;
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    int unit = 0, free_units = p.units;
    uint32_t item = 0, oldest = 0;
    bool ok = true;
    for (int i = 0; i < p.phases && ok; ++i) {
      const DensePhase* ph = p.program + i;
      const int kind = ph->kind;
      if (kind == DP_MIX) continue;
      const int blocks = ph->blocks, block_rows = kind == DP_GATE_UP ? BLOCK / 2 : BLOCK, log_item = ph->log_item, wide = ph->wide;
      const int per_block = 1 << (ph->log_slices - log_item);
      const char* map = static_cast<const char*>(p.maps) + (size_t)i * 256;
      // a map may stand where an earlier plan had another
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map + 128) : "memory");
      uint32_t narrow = 0;  // the items that are one unit narrower
      for (int w = 0; w < per_block; ++w)
        if (ph->column[(w + 1) << log_item] - ph->column[w << log_item] < wide) narrow |= 1u << w;
      for (int blk = own_first(ph->first); blk < blocks && ok; blk += gridDim.x) {
        int c = 0;
        for (int w = 0; w < per_block; ++w) {
          const int less = (narrow >> w) & 1, n = wide - less;
          const bool wrap = unit + n > p.units;  // a copy is in one piece: what is left at the ring's end stays out
          const int skip = wrap ? p.units - unit : 0;
          while (ok && (free_units < n + skip || item - oldest == ITEMS)) {
            ok = mbar_wait(&sh.empty[oldest % ITEMS], (oldest / ITEMS) & 1) && *failed == 0;
            free_units += sh.item_units[oldest % ITEMS];
            ++oldest;
          }
          if (!ok) break;
          if (wrap) unit = 0;
          uint64_t* full = &sh.full[item % ITEMS];
          sh.item_units[item % ITEMS] = n + skip;
          sh.item_at[item % ITEMS] = unit;
          mbar_expect_tx(full, n * UNIT_BYTES);  // rows past the end read as zero, and count
          load_item(smem_u32(ring + unit * UNIT_BYTES), map + less * 128, full, blk * block_rows, c, policy);
          c += n;
          unit += n;
          free_units -= n + skip;
          ++item;
        }
      }
    }
    // nothing leaves while a copy into its shared memory is in flight
    for (; oldest != item; ++oldest) mbar_wait(&sh.full[oldest % ITEMS], (oldest / ITEMS) & 1);
    return;
  }

  // ------------------------------------------------------------------ consumers
  constexpr int MIXERS = D * CG <= 8192 ? 256 : CONSUMERS;                       // threads of a mixer unit
  constexpr int RPT = D * CG / MIXERS, EIGHTH = D / 8, SUBS = RPT / EIGHTH;  // state rows of a thread
  static_assert(RPT % EIGHTH == 0 && MIXERS <= CONSUMERS && MIXERS >= 2 * D, "units");
  constexpr int GROUPS = D / CG;
  const int g = lane >> 2;
  uint32_t item0 = 0;  // number of the phase's first item
  unsigned long long best = 0ull;
  const long long pos = *p.pos;
  const uint32_t flag0 = *p.epoch + 1;  // of phase 0; what a phase writes carries flag0 + its number
  Poll poll{p.sync};
  int code = 0;  // of this thread's wait that ran out
  const int units = p.B * p.H * GROUPS;
  const int en = tid & 7, eb = (tid >> 3) & (mb - 1), ej = tid >> (3 + log_mb), per_pass = CONSUMERS >> (3 + log_mb);  // epilogue: row pairs
  const int r0 = (tid / CG) * RPT, col = tid % CG, which = tid / D, dim = tid % D;                                      // mixer
  const int half_hd = p.hd / 2, half_d = p.d / 2;
  bool bad = false;
  auto mixer_barrier = [] { asm volatile("bar.sync 2, %0;" ::"n"(MIXERS) : "memory"); };

  for (int i = 0; i < p.phases; ++i) {
    const DensePhase& ph = sh.phase[i & 1];
    const int kind = ph.kind, k = ph.k;
    // ---- what does not depend on the phase before
    uint4 next = make_uint4(0u, 0u, 0u, 0u);
    if (tid < PHASE_WORDS && i + 1 < p.phases) next = reinterpret_cast<const uint4*>(p.program + i + 1)[tid];
    const bool normed = ph.norm != nullptr;
    const int mine_first = own_first(ph.first);
    const int head = kind == DP_PROJECT && mine_first < ph.strengths ? mine_first : -1;  // whose write strengths this CTA forms
    const int mine = kind == DP_MIX ? 0 : ph.blocks_each + (mine_first < ph.blocks_more ? 1 : 0);
    if (normed && (mine > 0 || head >= 0)) {  // only where the copies are waited for: two norms' weights never race for the same words
      const __nv_bfloat16* nw = ph.norm;
      for (int c = tid * 8; c < k; c += CONSUMERS * 8)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(nws + c)), "l"(nw + c) : "memory");
    }
    uint4 strength_w = make_uint4(0u, 0u, 0u, 0u);
    if (head >= 0 && tid < STRENGTH_THREADS && tid * 8 < k) strength_w = *reinterpret_cast<const uint4*>(ph.extra + (long long)head * k + tid * 8);
    float S[RPT], cs = 1.f, sn = 0.f;
    int unit = mine_first;
    float* const state = ph.state + (long long)r0 * D + col;
    auto state_at = [&](int u) { return state + (long long)(u / GROUPS) * D * D + (u % GROUPS) * CG; };
    if (kind == DP_MIX && tid < MIXERS) {
      if (unit < units) {
        const float* s = state_at(unit);
#pragma unroll
        for (int r = 0; r < RPT; ++r) S[r] = __ldcg(s + r * D);
      }
      if (ph.cos != nullptr && which < 2) {
        const bool inside = pos >= 0 && pos < ph.table_rows;  // past the table there is no rotation: NaN, never another row's
        cs = inside ? ph.cos[pos * D + dim] : NAN;
        sn = inside ? ph.sin[pos * D + dim] : NAN;
      }
    }
    const uint32_t flag = flag0 + (uint32_t)i;
    auto publish = [&] {  // the next phase's entry
      if (tid < PHASE_WORDS) reinterpret_cast<uint4*>(&sh.phase[(i + 1) & 1])[tid] = next;
    };
    bool published = false;
    if (kind == DP_MIX) {
      if (tid < MIXERS) {
      const bool delta = ph.delta != 0, rotate = ph.cos != nullptr, strengths = ph.strengths > 0;
      for (; unit < units; unit += gridDim.x) {
        const int bh = unit / GROUPS, h = bh % p.H, b = bh / p.H;
        const unsigned long long* row = p.qkvg + (long long)b * 4 * half_hd + h * (D / 2);
        const int c = (unit % GROUPS) * CG + col, gd = MIXERS - 1 - tid;
        const unsigned long long* const from[4] = {row + 2 * half_hd + (c >> 1), row + (which & 1) * half_hd + (dim >> 1),
                                                   row + 3 * half_hd + ((gd & (D - 1)) >> 1), p.beta + bh};
        uint32_t word[4] = {0u, 0u, 0u, 0u};
        read_words(from, flag - 1, 1u | (which < 2 ? 2u : 0u) | (gd < D ? 4u : 0u) | (strengths ? 8u : 0u), word, poll);
        const float v = (c & 1) ? high_half(word[0]) : low_half(word[0]), raw = (dim & 1) ? high_half(word[1]) : low_half(word[1]);
        const float logit = (gd & 1) ? high_half(word[2]) : low_half(word[2]), strength = __uint_as_float(word[3]);
        float f = 0.f;
        if (which < 2) {
          f = mix_feature(raw);
          const float ss = sum_lanes(f * f);
          if (lane == 0) sh.warp_sum[warp] = ss;
          sh.feat[which][dim] = f;
        }
        if (gd < D) sh.dec[gd] = mix_decay(logit);
        mixer_barrier();
        if (which < 2) {
          float ss = 0.f;
#pragma unroll
          for (int n = 0; n < D / 32; ++n) ss += sh.warp_sum[which * (D / 32) + n];
          if (rotate) f = mix_rotate(f, sh.feat[which][dim < D / 2 ? dim + D / 2 : dim - D / 2], cs, sn, dim < D / 2);
          sh.vec[which][dim] = f * mix_inverse_norm(ss);
        }
        mixer_barrier();
        float u = v;  // sums over key rows are formed from eighths of them
        if (delta) {
#pragma unroll
          for (int e = 0; e < SUBS; ++e) {
            float acc = 0.f;
#pragma unroll
            for (int r = e * EIGHTH; r < (e + 1) * EIGHTH; ++r) acc = __fmaf_rn(sh.vec[1][r0 + r], S[r], acc);
            sh.part[0][r0 / EIGHTH + e][col] = acc;
          }
          mixer_barrier();
#pragma unroll
          for (int n = 0; n < 8; ++n) u -= sh.part[0][n][col];
          if (strengths) u *= mix_strength(strength);
        }
        float* s = state_at(unit);
#pragma unroll
        for (int e = 0; e < SUBS; ++e) {
          float acc = 0.f;
#pragma unroll
          for (int r = e * EIGHTH; r < (e + 1) * EIGHTH; ++r) {
            S[r] = mix_state(S[r], sh.dec[r0 + r], sh.vec[1][r0 + r], u);
            acc = __fmaf_rn(sh.vec[0][r0 + r], S[r], acc);
            s[r * D] = S[r];
          }
          sh.part[1][r0 / EIGHTH + e][col] = acc;
        }
        const int after = unit + gridDim.x;
        if (after < units) {
          const float* from = state_at(after);
#pragma unroll
          for (int r = 0; r < RPT; ++r) S[r] = __ldcg(from + r * D);
        }
        mixer_barrier();
        if (tid < CG / 2) {
          float o0 = 0.f, o1 = 0.f;
#pragma unroll
          for (int n = 0; n < 8; ++n) o0 += sh.part[1][n][2 * tid], o1 += sh.part[1][n][2 * tid + 1];
          write_word(p.mixed + (long long)b * half_hd + (h * D + (unit % GROUPS) * CG) / 2 + tid, pack_pair(o0, o1), flag);
        }
      }
      }
    } else if (mine > 0 || head >= 0) {
      // ---- input rows into shared memory
      const int log_slices = ph.log_slices, log_item = ph.log_item, gated = kind == DP_GATE_UP ? 1 : 0;
      const unsigned long long* src =
          kind == DP_OUT ? p.mixed : kind == DP_DOWN ? p.hidden : gated || kind == DP_UP ? p.middle : p.stream;
      // what an output pair is added to: the embedding, the down projection of the layer before, or this layer's output projection
      auto residual = [&](int b, int r) {
        if (kind == DP_OUT && i == 2) return *reinterpret_cast<const uint32_t*>(p.embed + sh.token[b] * (long long)p.d + r);
        const unsigned long long* const from[1] = {(kind == DP_DOWN ? p.middle : p.stream) + (long long)b * half_d + r / 2};
        uint32_t word[1] = {0u};
        read_words(from, kind == DP_DOWN ? flag - 2 : flag - 3, 1u, word, poll);
        return word[0];
      };
      if (normed) {
        const int wpr = WARPS >> log_mb, b = warp >> (LOG_WARPS - log_mb), wr = warp & (wpr - 1), step = wpr * 256;
        if (b < p.B) {
          const __nv_bfloat16* row = p.embed + sh.token[b] * (long long)p.d;
          const unsigned long long* x = src + (long long)b * (k / 2);
          for (int w0 = wr * 256; w0 < k; w0 += step) {  // a sum for each 256 columns
            const int c = w0 + lane * 8;
            float ss = 0.f;
            if (c < k) {
              const uint4 v = i == 0 ? *reinterpret_cast<const uint4*>(row + c) : read_row(x + c / 2, flag - 1, poll);
              *reinterpret_cast<uint4*>(act + b * p.act_pitch + c * 2) = v;
              float f[8];
              unpack_words(v, f);
#pragma unroll
              for (int j = 0; j < 8; ++j) ss = __fmaf_rn(f[j], f[j], ss);
            }
            ss = sum_lanes(ss);
            if (lane == 0) sh.red[b][w0 >> 8] = ss;
          }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        consumer_barrier<CONSUMERS>();
        if (b < p.B) {
          float ss = 0.f;
          for (int n = 0; n * 256 < k; ++n) ss += sh.red[b][n];
          const float inv = rsqrtf(ss / (float)k + ph.eps);
#pragma unroll 2
          for (int w0 = wr * 256; w0 < k; w0 += step) {
            const int c = w0 + lane * 8;
            if (c < k) {
              uint4* at = reinterpret_cast<uint4*>(act + b * p.act_pitch + c * 2);
              float f[8], w[8];
              unpack_words(*at, f);
              unpack_words(*reinterpret_cast<const uint4*>(nws + c), w);
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = f[j] * inv * w[j];
              *at = pack_words(f);
            }
          }
        }
      } else {
        // every CTA begins elsewhere: all of them read the same rows at the same time
        const int vecs = k / 8, all = p.B * vecs;
        int b = 0, c = tid + ((int)((long long)blockIdx.x * all / gridDim.x) & ~3);
        for (int n = tid; n < all; n += CONSUMERS) {
          while (c >= vecs) {
            c -= vecs;
            if (++b == p.B) b = 0;
          }
          *reinterpret_cast<uint4*>(act + b * p.act_pitch + c * 16) = read_row(src + (long long)b * (k / 2) + c * 4, flag - 1, poll);
          c += CONSUMERS;
        }
      }
      consumer_barrier<CONSUMERS>();
      if (head >= 0) {
        if (tid < STRENGTH_THREADS) {  // as the mixer's own kernel forms it
          for (int b = 0; b < p.B; ++b) {
            float sum = 0.f;
            for (int c = tid * 8; c < k; c += STRENGTH_THREADS * 8) {
              const uint4 w = c < STRENGTH_THREADS * 8 ? strength_w : *reinterpret_cast<const uint4*>(ph.extra + (long long)head * k + c);
              sum = mix_dot8(*reinterpret_cast<const uint4*>(act + b * p.act_pitch + c * 2), w, sum);
            }
            sum = sum_lanes(sum);
            if (lane == 0) sh.red[b][warp] = sum;  // the norm's sums have been read
          }
        }
        consumer_barrier<CONSUMERS>();
        if (tid < p.B) {
          float z = 0.f;
#pragma unroll
          for (int n = 0; n < STRENGTH_THREADS / 32; ++n) z += sh.red[tid][n];
          write_word(p.beta + tid * p.H + head, __float_as_uint(z), flag);
        }
      }

      // ---- products, as many blocks at a time as the partial sums have room for
      const int log_items = log_slices - log_item;  // of a block
      const int per_round = p.slots >> log_slices, slices = 1 << log_slices;
      const uint8_t* a = act + g * p.act_pitch;
      const bool live = g < p.B;
      for (int done = 0; done < mine; done += per_round) {
        const int blocks = min(per_round, mine - done), items = blocks << log_items;
        for (int it = (int)((warp - item0) & (WARPS - 1)); it < items; it += WARPS) {
          const uint32_t item = item0 + it;
          const unsigned short* column = ph.column + ((it & ((1 << log_items) - 1)) << log_item);
          if (!poll.bad && !mbar_wait(&sh.full[item % ITEMS], (item / ITEMS) & 1)) poll.bad = true, code = ST_TIMEOUT_FULL;
          float* to = sums + ((it << log_item) << log_mb) * BLOCK;
          const uint8_t* w = ring + (sh.item_at[item % ITEMS] - column[0]) * UNIT_BYTES;
          for (int j = 0; j < 1 << log_item;) {
            const int c = column[j], width = column[j + 1] - c;
            if (j + 1 < 1 << log_item && column[j + 2] - column[j + 1] == width) {  // two chains of sums at a time
              multiply_slices<2>(w + c * UNIT_BYTES, a + c * (UNIT * 2), live, width, to + (j << log_mb) * BLOCK, mb, lane);
              j += 2;
            } else {
              multiply_slices<1>(w + c * UNIT_BYTES, a + c * (UNIT * 2), live, width, to + (j << log_mb) * BLOCK, mb, lane);
              ++j;
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.empty[item % ITEMS]);
        }
        item0 += items;
        if (done == 0) {
          publish();
          published = true;
          bad = consumer_barrier_any<CONSUMERS>(poll.bad);
          if (bad) break;
        } else {
          consumer_barrier<CONSUMERS>();
        }
        // ---- epilogue: two neighbouring outputs a thread
        for (int j = ej; j < blocks; j += per_pass) {
          const float* from = sums + (((j << log_slices) << log_mb) + eb) * BLOCK + 2 * en;
          const int stride = BLOCK << log_mb, rows = ph.rows, r = ((mine_first + (done + j) * (int)gridDim.x) * (BLOCK >> gated)) + 2 * en;
          if (eb >= p.B || r >= rows || (gated && en >= BLOCK / 4)) continue;
          uint32_t res = 0;
          if (kind == DP_OUT || kind == DP_DOWN) res = residual(eb, r);
          float2 v = make_float2(0.f, 0.f), up = v;  // of a gated block: rows 0 to 7 gate, 8 to 15 up
          const int up_rows = gated ? BLOCK / 2 : 0;
#pragma unroll 4
          for (int n = 0; n < slices; ++n) {
            const float2 f = *reinterpret_cast<const float2*>(from + n * stride), u = *reinterpret_cast<const float2*>(from + n * stride + up_rows);
            v.x += f.x, v.y += f.y, up.x += u.x, up.y += u.y;
          }
          const long long word = (long long)eb * (rows >> 1) + (r >> 1);
          auto biased = [&](float x, int n) { return __fadd_rn(x, ph.bias != nullptr ? __bfloat162float(ph.bias[n]) : 0.f); };
          if (kind == DP_PROJECT) {
            write_word(p.qkvg + word, pack_pair(v.x, v.y), flag);
          } else if (kind == DP_OUT) {
            write_word(p.middle + word, pack_pair(round_bf16(v.x * ph.scale) + low_half(res), round_bf16(v.y * ph.scale) + high_half(res)), flag);
          } else if (kind == DP_DOWN) {
            write_word(p.stream + word,
                       pack_pair(round_bf16(biased(v.x, r)) + low_half(res), round_bf16(biased(v.y, r + 1)) + high_half(res)), flag);
          } else if (kind == DP_HEAD) {
            auto take = [&](float x, int n) {
              const unsigned long long key = ((unsigned long long)value_order(x) << 32) | (0xffffffffu - (unsigned)n);
              best = key > best ? key : best;
            };
            take(v.x, r);
            if (r + 1 < rows) take(v.y, r + 1);
          } else if (gated) {
            write_word(p.hidden + word,
                       pack_pair(v.x * __fdividef(1.f, 1.f + __expf(-v.x)) * up.x, v.y * __fdividef(1.f, 1.f + __expf(-v.y)) * up.y), flag);
          } else {
            write_word(p.hidden + word, pack_pair(gelu_tanh_f(biased(v.x, r)), gelu_tanh_f(biased(v.y, r + 1))), flag);
          }
        }
        if (done + per_round < mine) consumer_barrier<CONSUMERS>();  // the sums are read before the next round writes them
      }
    }
    if (!published) {
      consumer_barrier<CONSUMERS>();  // the entry that is overwritten has been read
      publish();
      bad = consumer_barrier_any<CONSUMERS>(poll.bad);
    }
    if (bad) break;
  }

  // what residuals were waited for in the last phase that has any
  bad = consumer_barrier_any<CONSUMERS>(poll.bad);
  if (bad) {
    if (poll.bad) atomicCAS(p.status, 0, code != 0 ? code : ST_TIMEOUT_PEER);
    if (tid == 0) {
      *failed = 1;
      atomicOr(p.sync, 1u);
    }
    return;
  }
  // ------------------------------------------------------------------ the choice of the next token
  if (eb < p.B) atomicMax(&sh.best[eb], best);
  consumer_barrier<CONSUMERS>();
  if (tid < p.B) __stcg(p.best + blockIdx.x * DENSE_STEP_MAX_ROWS + tid, sh.best[tid]);
  consumer_barrier<CONSUMERS>();
  if (tid == 0) {
    __threadfence();
    sh.last = atomicAdd(p.sync + 1, 1u) == gridDim.x - 1;
    __threadfence();
  }
  consumer_barrier<CONSUMERS>();
  if (!sh.last) return;
  if (warp < p.B) {  // the last CTA: a warp per row
    unsigned long long v = 0ull;
    for (unsigned int c = lane; c < gridDim.x; c += 32) {
      const unsigned long long w = __ldcg(p.best + c * DENSE_STEP_MAX_ROWS + warp);
      v = w > v ? w : v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
      v = w > v ? w : v;
    }
    if (lane == 0) {
      p.out[warp * p.out_ld + *p.step] = sh.token[warp];
      p.token[warp] = (long long)(0xffffffffu - (uint32_t)v);
    }
  }
  consumer_barrier<CONSUMERS>();
  if (tid == 0) {
    *p.pos = pos + 1;
    *p.step += 1;
    *p.epoch += (unsigned)p.phases;
    p.sync[1] = 0u;
  }
}

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  return n;
}

template <int D, int CG, int LOG_WARPS>
void launch(const DenseStep& p, int grid, int smem, cudaStream_t s) {
  auto kernel = dense_step_kernel<D, CG, LOG_WARPS>;
  static PerDeviceOnce once;
  if (once.first_use()) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - (int)sizeof(Shared) - 1024);
    if (e != cudaSuccess) throw std::runtime_error(std::string("dense_step attribute: ") + cudaGetErrorString(e));
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((32 << LOG_WARPS) + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) throw std::runtime_error(std::string("dense_step launch failed: ") + cudaGetErrorString(e));
}

// Sixteen consumer warps from five sequences on: more loads of input rows in flight (8 sequences, 6 layers of 2048: 361 -> 337 us a step);
// with fewer sequences eight, whose registers hold everything (one: 194 against 205 us).
template <int D, int CG>
void launch_rows(const DenseStep& p, int grid, int smem, cudaStream_t s) {
  if (p.B > 4) launch<D, CG, 4>(p, grid, smem, s);
  else launch<D, CG, 3>(p, grid, smem, s);
}

}  // namespace

DenseStepGeom dense_step_geom(int B, int act_k, int d) {
  DenseStepGeom g{};
  const int mb = B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8;
  g.grid = sm_count();
  g.act_pitch = act_k * 2 + ((act_k * 2) % 128 == 64 ? 0 : 64);  // two rows of a quarter warp on different banks
  g.slots = mb <= 4 ? 64 : 48;
  const int most = 232448 - (int)sizeof(Shared) - 1024, fixed = B * g.act_pitch + g.slots * mb * BLOCK * 4 + d * 2 + 1024;
  const int units = (most - fixed) / UNIT_BYTES;
  g.units = g.grid <= 0 || d > MAX_GROUPS * 256 ? 0 : units < MAX_UNITS ? units : MAX_UNITS;
  g.smem = g.units * UNIT_BYTES + fixed;
  return g;
}

bool dense_step_cut(DensePhase& ph, const DenseStepGeom& geom) {
  const int slices = skinny_warps(ph.rows, ph.k), steps = ph.k / UNIT;
  auto log2 = [](int n) { int l = 0; while ((1 << l) < n) ++l; return l; };
  if (slices > geom.slots || ph.k % UNIT != 0 || slices > 16 || steps > 0xffff) return false;
  for (int w = 0; w <= slices; ++w) ph.column[w] = (unsigned short)(w * steps / slices);
  const int block_rows = ph.kind == DP_GATE_UP ? BLOCK / 2 : BLOCK;
  ph.blocks = (ph.rows + block_rows - 1) / block_rows;
  // an item is a slice, or as many as make 512 columns (256 where a CTA has one block and warps to spare) where slices are narrow; none
  // is empty. 512 columns are copies of 16 KB: a step of 6 layers of 2048 took 194 us with them, 230 with 8 KB (half the bytes of a
  // weight row at a time), 201 and 211 with 24 and 32 (few in flight)
  int n = 1;
  while (n < 4 && (steps < slices / n || 2 * n * steps <= (ph.blocks <= geom.grid ? 4 : 8) * slices)) n *= 2;
  int widest = 0, narrowest = steps;
  for (int w = 0; w < slices; w += n) {
    const int width = ph.column[w + n] - ph.column[w];
    widest = width > widest ? width : widest;
    narrowest = width < narrowest ? width : narrowest;
  }
  // copies are of two kinds; four are in flight at least, with what is left out at the ring's end
  if (narrowest <= 0 || narrowest < widest - 1 || widest * 5 > geom.units) return false;
  ph.wide = widest;
  ph.log_slices = log2(slices);
  ph.log_item = log2(n);
  ph.blocks_each = ph.blocks / geom.grid;
  ph.blocks_more = ph.blocks % geom.grid;
  return true;
}

void dense_step_maps(const DensePhase& ph, void* maps) {
  const bool gated = ph.kind == DP_GATE_UP;  // a block is eight gate rows and the eight up rows that go with them
  const uint64_t d[4] = {UNIT, (uint64_t)ph.rows, gated ? 2u : 1u, (uint64_t)ph.k / UNIT};
  const uint64_t stride[3] = {(uint64_t)ph.k * 2, (uint64_t)ph.k * 2 * (uint64_t)ph.rows, UNIT * 2};
  for (int i = 0; i < 2; ++i) {
    const uint32_t box[4] = {UNIT, (uint32_t)(gated ? BLOCK / 2 : BLOCK), gated ? 2u : 1u, (uint32_t)(ph.wide - i > 0 ? ph.wide - i : 1)};
    const CUtensorMap m = make_tmap_4d_box_bf16(ph.weight, d, stride, box);
    std::memcpy(static_cast<char*>(maps) + i * 128, &m, sizeof(m));
  }
}

// Columns of a mixer unit: as few as give every CTA at most one unit, so that all state reads of a phase are in flight at once, and
// whole heads where there are more than that. At least 32, so that an eighth of the key rows is one thread's.
static int unit_columns(int B, int H, int D, int grid) {
  int cg = 32;
  while (cg < D && (long long)B * H * (D / cg) > grid) cg *= 2;
  return cg;
}

int dense_step_units(int B, int H, int D, int grid) { return B * H * (D / unit_columns(B, H, D, grid)); }

void launch_dense_step(const DenseStep& p, int grid, int smem, int D, cudaStream_t s) {
  const int cg = unit_columns(p.B, p.H, D, grid);
  if (D == 128) {
    if (cg == 32) launch_rows<128, 32>(p, grid, smem, s);
    else if (cg == 64) launch_rows<128, 64>(p, grid, smem, s);
    else launch_rows<128, 128>(p, grid, smem, s);
  } else if (D == 64) {
    if (cg == 32) launch_rows<64, 32>(p, grid, smem, s);
    else launch_rows<64, 64>(p, grid, smem, s);
  } else {
    throw std::runtime_error("dense_step: head dimension must be 64 or 128");
  }
}

}  // namespace tb
