// Host interface of the FP8 GEMMs inside the library: a launch computes up to MAX_GROUPS independent problems that share
// K and the 16-bit type (the two streams of a Qwen-Image block; a Wan block's projections of x and of the text context).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ksb {
namespace gemm {

constexpr int MAX_GROUPS = 4;

// out[m, n] = epi((A . W^T)[m, n] * sa[m] * sw[n] + bias[n]); epilogue: KSB_EPI_NONE / GELU_TANH / GATE_RESIDUAL
struct Problem {
  const void* a;       // e4m3 [M, K]
  const float* sa;     // [M]
  const void* w;       // e4m3 [N, K]
  const float* sw;     // [N]
  const void* bias;    // half [N] or null
  int64_t M, N;
  void* out;           // half [M, ldo]
  int64_t ldo;
  int epilogue;
  const void* resid;   // half [M, ldr]
  int64_t ldr;
  // gate row of output row m: gate + gate_stride * (gate_index ? gate_index[m] : rows_per_gate ? m / rows_per_gate : 0)
  const void* gate;
  int64_t gate_stride;
  int rows_per_gate;
  const int64_t* gate_index;
  int64_t gate_rows;  // with gate_index: the rows it may name (others take row 0)
  // Row sums of squares of the rounded outputs, or null: [sumsq_cols / 256][M], or with `fine` [sumsq_cols / 64][M], where
  // every form adds up a row's 64 columns in the same order (an RMSNorm behind the launch then does not depend on the form).
  float* tile_sumsq;
  int sumsq_cols;
  int fine;
  // Rows that the launch quantises itself (launch_quantises), in place of a and sa: half [M, x_ld], per token, or with x_static by
  // *x_scale (null: clamped only).  Neither x nor x_scale may overlap out.
  const void* x;
  int64_t x_ld;
  int x_static;
  const float* x_scale;
};

// Launches the problems.  `chained`: the launch follows another kernel of this library's own sequence on the stream, may
// start while that kernel drains, and may fetch weights (which no kernel of a sequence writes) before it has finished.  A launch
// that quantises its rows is the first of its sequence and has the caller's own kernels ahead, which may write weights: with
// `chained` it may start while they drain, but reads nothing before they have finished.
int run(const Problem* problems, int count, int64_t K, int dtype, bool chained, cudaStream_t st);

// Whether run takes this single problem's rows as halves and quantises them in the GEMM's own launch: a few rows, whose
// quantiser would be a launch of its own ahead of a GEMM that streams a weight.
bool launch_quantises(const Problem& p, int64_t K);

// Checks the fields of one problem (alignment, shapes); returns 0 or an error code with the text set.
int validate(const Problem& p, int64_t K, int dtype);

// The split-K form for launches too small to fill the GPU with whole tiles (fp8_gemm_split.cu).
struct SplitPlan {
  int bn;       // columns per tile: 64 or 128
  int splits;   // CTAs of a cluster that share a tile's K range
  int occupancy;  // CTAs per SM the shared-memory budget is cut for
  float us;     // estimated time
};
SplitPlan plan_split(const Problem* problems, int count, int64_t K, bool stats256);
int run_split(const Problem* problems, int count, int64_t K, int dtype, bool chained, cudaStream_t st, const SplitPlan& plan);
bool split_quantises(const Problem& p, int64_t K, const SplitPlan& plan);

}  // namespace gemm
}  // namespace ksb
