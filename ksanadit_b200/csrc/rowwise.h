// Host interface of the row-wise FP8 quantisers inside the library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ksb {
namespace rq {

enum Mode : int { PLAIN = 0, ADALN = 1, LN_AFFINE = 2, STATIC = 3 };
constexpr int MAX_SEGS = 4;

// Rows of one input with one kind of modulation.  Segments follow one another in the output.
struct Segment {
  const void* x;
  int64_t rows, ldx;
  // ADALN: the modulation row of row m is mod_stride * (mod_index ? mod_index[m] : rows_per_mod ? m / rows_per_mod : 0) elements
  // behind shift / scale; mod_index names one of mod_rows rows
  const void* shift;
  const void* scale;
  int64_t mod_stride;
  const int64_t* mod_index;
  int64_t mod_rows;
  int64_t rows_per_mod;
  int64_t row0;  // first output row (filled by run)
  int cta0, ctas;  // the CTAs that work on it (filled by run)
};

struct Params {
  Segment seg[MAX_SEGS];
  int segs;
  int64_t K;
  int round_product;  // ADALN: 0 = addcmul(shift, ln, 1+scale) (one rounding), 1 = ln * (1+scale) rounded, then + shift
  const float* w;     // LN_AFFINE
  const float* b;
  float eps;
  const float* scale_input;  // STATIC (may be null = clamp only)
  void* h_out;               // optional half copy of the transformed rows
  uint8_t* q;
  float* qscale;
  int* status;  // filled by run
};

int validate(const Params& p, int dtype);
int run(Mode mode, Params& p, int dtype, bool chained, cudaStream_t st);

// Bytes of a workspace that holds M quantised rows of K and their scales: [M][K] e4m3, then (at scale_offset) [M] fp32.
inline int64_t scale_offset(int64_t M, int64_t K) { return (M * K + 255) / 256 * 256; }
inline int64_t workspace_bytes(int64_t M, int64_t K) { return scale_offset(M, K) + (M * 4 + 255) / 256 * 256; }

}  // namespace rq
}  // namespace ksb
