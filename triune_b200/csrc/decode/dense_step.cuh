// One decoding step of a dense recurrent model in one launch (dense_step.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace tb {

constexpr int DENSE_STEP_MAX_ROWS = 8;  // sequences: the columns of one matrix instruction

enum DensePhaseKind : int {
  DP_PROJECT = 0,  // qkvg and write-strength logits of the normed stream
  DP_MIX = 1,      // feature map, rotation, state update, mixer output
  DP_OUT = 2,      // stream after the mixer = stream + output projection
  DP_GATE_UP = 3,  // silu(gate) * up of the normed stream
  DP_UP = 4,       // gelu(product + bias) of the normed stream
  DP_DOWN = 5,     // stream after the feed-forward = stream + product (+ bias)
  DP_HEAD = 6,     // logits of the normed stream, their arg-max, the next token
};

// One entry of the step's program, in device memory.
struct alignas(16) DensePhase {
  const __nv_bfloat16* weight;  // [rows, k], rows contiguous; DP_GATE_UP: gate rows, then as many up rows
  const __nv_bfloat16* extra;   // DP_PROJECT: weight of the write strengths [heads, k], or null
  const __nv_bfloat16* norm;    // weight of the norm before the product [k], or null
  const __nv_bfloat16* bias;    // DP_UP, DP_DOWN: [rows], or null
  float* state;                 // DP_MIX: fp32 [B, H, D, D], updated in place
  const float *cos, *sin;       // DP_MIX: rotary tables [table_rows, D], or null
  long long table_rows;
  int kind, rows, k;
  int first;                    // CTA that takes block (or unit) 0; the others follow it in order
  int strengths, delta;         // heads with a write strength (DP_PROJECT, DP_MIX), delta rule (DP_MIX)
  float eps, scale;
  int log_slices, log_item;     // slices of the reduction, as the product of few rows cuts it, and those of one copy: powers of two
  int blocks, blocks_each, blocks_more;  // blocks of sixteen rows; per CTA, and how many CTAs have one more
  int wide;                     // units of 64 columns of the wider copies; the others have one less
  unsigned short column[18];    // first columns of the slices / 64, and the end
};

struct DenseStep {
  const DensePhase* program;
  const void* maps;  // CUtensorMap [phases][2]: a phase's wider and narrower copies
  int phases, B, d, H, hd;
  int act_pitch, units, slots;  // bytes between rows of the staged input, ring, partial sums
  const __nv_bfloat16* embed;                  // [vocab, d]
  long long *token, *out, *pos, *step;         // [B], [B, out_ld], [1], [1]
  long long out_ld;
  // hand-overs between CTAs, 64-bit words of two bf16 values and a flag: [B, d / 2], [B, d / 2], [B, 2 hd], [B, hd / 2], [B, feed-forward
  // width / 2], and the write strengths' logits, fp32 and a flag: [B, H]. All zero before the first launch.
  unsigned long long *stream, *middle, *qkvg, *mixed, *hidden, *beta;
  unsigned long long* best;                                // [grid, 8]
  unsigned int* sync;                                      // [2]: not 0: a step did not finish; CTAs done
  unsigned int* epoch;                                     // flags used so far
  int* status;
};

// CTAs of a step on this device, and its shared memory for `act_k` wide reductions; 0 units where it does not fit.
struct DenseStepGeom {
  int grid, act_pitch, units, slots, smem;
};
DenseStepGeom dense_step_geom(int B, int act_k, int d);
// Fills in how a phase's product is cut and dealt; false where the workspace has no room for it.
bool dense_step_cut(DensePhase& ph, const DenseStepGeom& geom);
// The two CUtensorMap of a phase's weight (128 bytes each) into `maps`.
void dense_step_maps(const DensePhase& ph, void* maps);
int dense_step_units(int B, int H, int D, int grid);      // units of a mixer phase
void launch_dense_step(const DenseStep& p, int grid, int smem, int D, cudaStream_t s);

}  // namespace tb
