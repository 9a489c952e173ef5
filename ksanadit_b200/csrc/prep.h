// Host interface of the attention pre-pass inside the library: the statistics and the quantisers of several operands (Q, K
// and V; of the self- and the cross-attention of a block; of several samples) run as one launch each.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ksb {
namespace prep {

constexpr int D = 128;
constexpr int MAX_JOBS = 12;
constexpr int MAX_STAT_CHUNKS = 64;

struct RopeGrid {
  const float2* table;  // [table_len][64] (cos, sin); pair p of a head uses axis f for p < nf, then h, then w
  int table_len, nf, nh;
  int F, Hh, Ww;
  int64_t pos0;  // global index of row 0 (sequence-parallel shard offset)
  int diag;      // 1: one running position drives all three axes (text tokens of the Qwen-Image block)
};

// RMSNorm (+ rotary embedding) applied to an operand as it is read.
struct NormSpec {
  const float* w;         // norm weight: [H * 128], or [128] with per_head
  int per_head;           // 1: over each head's 128 channels; 0: over all heads, from one of the two tables below
  const float* row_rstd;  // [L] 1 / rms per token
  const float* ssq;       // [ssq_tiles][ssq_stride] sums of squares per column tile of the producing GEMM
  int ssq_tiles;
  int64_t ssq_stride;
  float c, eps;           // 1 / rms = rsqrt(sum of the tiles / c + eps)
  RopeGrid rg;            // rg.table == nullptr: no rotation
  int per_frame;          // rg.Hh * rg.Ww, with the reciprocals the position decoding uses
  float inv_per_frame, inv_w;
};

enum Kind : int { QUANT_Q = 0, QUANT_K = 1, QUANT_V = 2 };  // one INT8 block of 128 tokens; two of 64; FP8 transposed

// An operand [L, H, 128] of half values with element strides ts (token) and hs (head).  With a norm, rows before `split`
// take ns[0], the others ns[1] (whose positions count from `split`); an operand with one norm has split = INT32_MAX, so that
// the rows past its end do not reach for ns[1] either.
struct Operand {
  const void* x;
  int64_t ts, hs;
  int L, H;
  int normed, split;
  NormSpec ns[2];
};

// Column sums (K) or absolute maxima (V) per chunk of tokens: part[chunk][H][128].
struct StatsJob {
  Operand op;
  void* normed_out;  // null, or where a normed operand goes, as [L][H][128]: its quantiser then needs no norm
  int is_max;
  int atomic_max;   // 1: part is [H][128], cleared by the caller, and receives the maximum over all chunks
  float* part;
  int chunks, chunk_tokens;
  int first;  // first CTA (filled by run_stats)
};

struct QuantJob {
  Operand op;
  int kind;
  float premul;       // 0: none
  const float* part;  // K: sums (mean = sum over chunks * inv_l) or null; V: maxima.  [chunks][H][128]
  int chunks;
  float inv_l;
  void* out;          // int8 [H][Lpad][128], or e4m3 [H][128][Lpad]
  float* scale;       // [H][Lpad / 128], [H][Lpad / 64] or [H][128]
  int first;          // first unit (filled by run_quant)
};

// Chunk count for L tokens and H heads, at most `most`: enough CTAs to fill the GPU twice, whole 128-token tiles.
int plan_chunks(int64_t L, int64_t H, int most);

int run_stats(StatsJob* jobs, int count, int dtype, bool chained, cudaStream_t st);
int run_quant(QuantJob* jobs, int count, int dtype, bool chained, cudaStream_t st);
// part[0] = sum over chunks * scale (is_max: maximum over chunks), in place, for `n` columns
int run_finish(float* part, int chunks, int64_t n, float scale, bool is_max, float* out, bool chained, cudaStream_t st);

// rstd[g][m] = rsqrt(sum over the tiles of column group g of sums[tile][m] / C + eps)
int run_rstd(const float* sums, int tiles_per_group, int groups, int M, int C, float eps, float* rstd, bool chained, cudaStream_t st);

int check_operand(const void* x, int dtype, int64_t L, int64_t H, int64_t Dh, int64_t ts, int64_t hs);
int make_rope_grid(RopeGrid& rg, const float* rope_table, int table_len, int nf, int nh, int F, int Hh, int Ww, int64_t pos0, int diag);
// Completes a norm whose w, tables and eps are set: adds the rotation and its position arithmetic.
int finish_norm(NormSpec& ns, int64_t L, const RopeGrid& rg);

inline int64_t pad128(int64_t L) { return (L + 127) / 128 * 128; }

}  // namespace prep
}  // namespace ksb
