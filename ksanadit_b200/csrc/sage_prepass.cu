// Attention pre-pass: K token-mean (smoothing vector), per-block INT8 quantisation of Q and K, per-(head, channel) FP8
// quantisation of V with the token axis made contiguous, optionally with the RMSNorm and the rotary embedding applied to Q
// and K as they are read.  Inputs are [L, H, 128] half tensors addressed by element strides, so they can be views into a
// fused QKV projection output.
//
// Algorithmic bytes per token and head (D = 128): Q or K quantiser 256 read + 128 written; K mean 256 read; V quantiser
// 2 x 256 read + 128 written.
//
// Two launches do all of it, each over a list of jobs (prep.h): the column statistics, then the quantisers.
#include "../../include/ksana_b200.h"
#include "common.cuh"
#include "host_utils.h"
#include "prep.h"

namespace ksb {
namespace prep {

// A 128-token tile of a head in a CTA: TL token lanes x 16 column groups of 8 channels, 128 / TL vectors per thread (tokens tl + TL * i).
constexpr int STATS_TL = 32;
constexpr int MEAN_CHUNK = 512;  // tokens per partial sum of the entry points that take a caller's scratch

template <bool V> struct Bool { static constexpr bool value = V; };

// x = q * d + r for 0 <= x < 2^24 (exact in fp32): the estimate from the reciprocal is within one of the quotient
__device__ __forceinline__ void divmod_small(int x, int d, float inv_d, int& q, int& r) {
  q = static_cast<int>(static_cast<float>(x) * inv_d);
  r = x - q * d;
  if (r < 0) { r += d; --q; } else if (r >= d) { r -= d; ++q; }
}

// (a, b) rotated by (cos, sin): the operation order both norm/RoPE kernels share, so that their results are the same bits.
// (Packed, the swapped and negated operands cost more moves than the packed instructions save.)
__device__ __forceinline__ float2 rope_pair(float a, float b, float2 cs) {
  return make_float2(__fmaf_rn(-b, cs.y, __fmul_rn(a, cs.x)), __fmaf_rn(b, cs.x, __fmul_rn(a, cs.y)));
}

// Grid coordinates of a thread's tokens: the 16 lanes that share a token would all decode the same position, so lane cg decodes
// the token of vector cg % (128 / TL) and the group exchanges the results (packed 10 bits per axis, or the one position of all
// axes; -1: the token is not rotated).
template <bool SEG, int TL> __device__ __forceinline__ int decode_position(const Operand& op, int l0) {
  const int cg = threadIdx.x & 15, tl = threadIdx.x >> 4;
  const int tok = l0 + tl + TL * (cg & (128 / TL - 1));
  const bool second = SEG && tok >= op.split;
  const NormSpec& ns = op.ns[second];
  if (!ns.rg.table) return -1;
  int cf, rem, ch, cw;
  divmod_small(static_cast<int>(ns.rg.pos0) + tok - (second ? op.split : 0), ns.per_frame, ns.inv_per_frame, cf, rem);
  divmod_small(rem, ns.rg.Ww, ns.inv_w, ch, cw);
  if (ns.rg.diag) return cf < ns.rg.F ? cf : -1;
  return cf < ns.rg.F ? (cf | (ch << 10) | (cw << 20)) : -1;
}

// Where a thread finds the (cos, sin) of its channel pairs p0 .. p0 + 3, two by two: which bits of the packed coordinates name the
// table row.  The same for every token, so a token costs two shifts and two 16-byte reads (picking the axes anew for every vector
// took 40 of the 250 instructions that a vector of 8 channels cost).
struct PairAxes {
  const float2* at;  // column p0 of the table
  int shift[2], next_shift[2], mask;
  __device__ __forceinline__ PairAxes(const Operand& op, bool second, int p0) {
    const RopeGrid& rg = op.ns[second].rg;
    at = (rg.table ? rg.table : op.ns[!second].rg.table) + p0;  // a segment that is not rotated reads what it does not use
    mask = rg.diag ? 0x3fffffff : 1023;
    auto bits = [&](int pair) { return rg.diag || pair < rg.nf ? 0 : (pair < rg.nf + rg.nh ? 10 : 20); };
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      shift[hf] = bits(p0 + 2 * hf);
      next_shift[hf] = bits(p0 + 2 * hf + 1);
    }
  }
  // the identity where not rotated, unless `all` says that no token of the warp needs it
  __device__ __forceinline__ void rotation(int coords, bool all, float2 (&rot)[4]) const {
    const int c = max(coords, 0);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const float4 t4 = *reinterpret_cast<const float4*>(at + ((c >> shift[hf]) & mask) * 64 + 2 * hf);
      rot[2 * hf] = make_float2(t4.x, t4.y);
      rot[2 * hf + 1] = make_float2(t4.z, t4.w);
      if (next_shift[hf] != shift[hf]) rot[2 * hf + 1] = at[((c >> next_shift[hf]) & mask) * 64 + 2 * hf + 1];  // the neighbour's axis differs
    }
    if (!all) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (coords < 0) rot[q] = make_float2(1.f, 0.f);
    }
  }
};

// 1 / rms over all heads of a tile's 128 tokens into shared memory, from the finished table or from the GEMM's sums of squares: TL / 8
// threads per token, the tiles in four shares.  A barrier must follow.  (With TL = 16 only a single operand comes with sums; without
// that branch the compiler makes a slower kernel of the one for single operands, with a table or a norm per head too: Q of 32760 x 40
// heads 174 -> 195 us.)
template <int TL> __device__ __forceinline__ void tile_rstd(const NormSpec& ns, int l0, int nvalid, float* s_rstd) {
  constexpr int PER = TL / 8, SHARES = 4 / PER, FEW = 6;
  if (ns.row_rstd) {
    const int t = threadIdx.x;
    if (t < 128) s_rstd[t] = t < nvalid ? ns.row_rstd[l0 + t] : 0.f;
    return;
  }
  const int t = threadIdx.x / PER, sub = threadIdx.x % PER;
  float s[SHARES];
#pragma unroll
  for (int k = 0; k < SHARES; ++k) s[k] = 0.f;
  if (t < nvalid) {
    const float* q = ns.ssq + l0 + t;
    if (SHARES > 1) {
      for (int i = sub * SHARES; i < ns.ssq_tiles; i += 4) {
#pragma unroll
        for (int k = 0; k < SHARES; ++k)
          if (i + k < ns.ssq_tiles) s[k] += ns.ssq[(i + k) * ns.ssq_stride + l0 + t];
      }
    } else if (ns.ssq_tiles <= 4 * FEW) {
      // all at once: the pre-pass of a block of 1560 x 12 heads 18.2 -> 17.3 us, 6000 x 12 60 -> 55 (40 heads are better off with the loop)
      float v[FEW];
#pragma unroll
      for (int k = 0; k < FEW; ++k) v[k] = sub + 4 * k < ns.ssq_tiles ? q[(sub + 4 * k) * ns.ssq_stride] : 0.f;
#pragma unroll
      for (int k = 0; k < FEW; ++k) s[0] += v[k];
    } else {
      for (int i = sub; i < ns.ssq_tiles; i += 4) s[0] += q[i * ns.ssq_stride];
    }
  }
  float r = s[0];
  if (SHARES == 2) r += s[SHARES - 1];
  if (PER == 4) r += __shfl_xor_sync(0xffffffffu, r, 1);
  r += __shfl_xor_sync(0xffffffffu, r, PER / 2);
  if (sub == 0) s_rstd[t] = rsqrtf(r / ns.c + ns.eps);
}

__device__ __forceinline__ void norm_weights(const NormSpec& ns, int h, int c, float2 (&w2)[4]) {
  const float* wp = ns.w + (ns.per_head ? 0 : h * D) + c;
  const float4 w0 = *reinterpret_cast<const float4*>(wp), w1 = *reinterpret_cast<const float4*>(wp + 4);
  w2[0] = make_float2(w0.x, w0.y); w2[1] = make_float2(w0.z, w0.w); w2[2] = make_float2(w1.x, w1.y); w2[3] = make_float2(w1.z, w1.w);
}

// RMSNorm and rotation of one 8-channel vector with the rounding points of the in-place kernel (norm output rounded to
// half, rotation in fp32, rounded to half).
template <typename T, bool PER_HEAD, bool ROPE>
__device__ __forceinline__ uint4 normalise(const uint4& raw, float r, float eps, const float2 (&w2)[4], const float2 (&rot)[4]) {
  uint32_t wd[4] = {raw.x, raw.y, raw.z, raw.w};
  float2 f[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) f[q] = HalfOps<T>::unpack2(wd[q]);
  if (PER_HEAD) {
    float hsum = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      hsum = __fmaf_rn(f[q].x, f[q].x, hsum);
      hsum = __fmaf_rn(f[q].y, f[q].y, hsum);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) hsum += __shfl_xor_sync(0xffffffffu, hsum, o);  // the 16 lanes of a token; every lane takes part
    r = rsqrtf(hsum / (float)D + eps);
  }
  const float2 r2 = make_float2(r, r);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    wd[q] = HalfOps<T>::pack2(__fmul2_rn(__fmul2_rn(f[q], r2), w2[q]));
    if (ROPE) {
      const float2 y = HalfOps<T>::unpack2(wd[q]);
      wd[q] = HalfOps<T>::pack2(rope_pair(y.x, y.y, rot[q]));  // the identity leaves y as it is
    }
  }
  return make_uint4(wd[0], wd[1], wd[2], wd[3]);
}

// The vectors of a thread in tile (l0, head h), normalised: f(i, y) for every i with y as packed halves, rows at or past nvalid
// included.  A norm over all heads has one segment; the per-head norm may change in the middle of a tile (SEG).
template <typename T, int TL, bool PER_HEAD, bool ROPE, bool SEG, typename F>
__device__ __forceinline__ void each_normalised(const Operand& op, int h, int l0, const uint4 (&raw)[128 / TL], const float* s_rstd, F&& f) {
  constexpr int VECS = 128 / TL;
  const int cg = threadIdx.x & 15, tl = threadIdx.x >> 4, lane = threadIdx.x & 31;
  float2 w2[4];
  bool second = SEG && l0 >= op.split;
  norm_weights(op.ns[second], h, cg * 8, w2);
  float eps = op.ns[second].eps;
  const int packed = ROPE ? decode_position<SEG, TL>(op, l0) : -1;
  const bool all_rotated = ROPE && __all_sync(0xffffffffu, packed >= 0);
  PairAxes axes(op, second, cg * 4);
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    if (SEG && (l0 + tl + TL * i >= op.split) != second) {  // only in the tile that holds the end of the first segment
      second = true;
      norm_weights(op.ns[1], h, cg * 8, w2);
      eps = op.ns[1].eps;
      if (ROPE) axes = PairAxes(op, true, cg * 4);
    }
    float2 rot[4];
    if (ROPE) axes.rotation(__shfl_sync(0xffffffffu, packed, (lane & 16) | i), all_rotated, rot);
    f(i, normalise<T, PER_HEAD, ROPE>(raw[i], PER_HEAD ? 0.f : s_rstd[tl + TL * i], eps, w2, rot));
  }
}

// Runs f<PER_HEAD, ROPE> for the operand's norm.
template <typename F> __device__ __forceinline__ void with_norm(const Operand& op, F&& f) {
  const bool rotates = op.ns[0].rg.table != nullptr || op.ns[1].rg.table != nullptr;
  if (op.ns[0].per_head) {
    if (rotates) f(Bool<true>{}, Bool<true>{}); else f(Bool<true>{}, Bool<false>{});
  } else {
    if (rotates) f(Bool<false>{}, Bool<true>{}); else f(Bool<false>{}, Bool<false>{});
  }
}

// The job a CTA works on.  A launch of one normed operand with one segment has kernels of its own (ONE; see quant_kernel for which
// operands): its fields then are at fixed places of the constant bank, not loads at an index behind one another in the loop over a
// tile.  75600 x 40 heads with a rotation, us,
// indexed / fixed: Q 426 / 406 (now 388), K 474 / 455 (now 434), K mean 312 / 293; with a norm per head 470 / 435, 519 / 476, 371 / 292.  (Fewer
// forms of norm in one kernel, or one norm per pass over a tile, did not help the indexed form: 64 registers spill.)
template <typename P> __device__ __forceinline__ int my_job(const P& p) {
  int ji = 0;
  while (ji + 1 < p.count && static_cast<int>(blockIdx.x) >= p.j[ji + 1].first) ++ji;
  return ji;
}

// ---------------------------------------------------------------------------------- column statistics
struct StatsParams {
  StatsJob j[MAX_JOBS];
  int count;
};

// One CTA = one (job, chunk of tokens, head).
template <typename T, bool NORM, bool ONE>
__global__ void __launch_bounds__(16 * STATS_TL, 2) stats_kernel(const __grid_constant__ StatsParams p) {
  __shared__ float red[32][D + 1];
  __shared__ float s_rstd[2][128];
  const StatsJob& job = p.j[ONE ? 0 : my_job(p)];
  const Operand& op = job.op;
  const int u = blockIdx.x - job.first, chunk = u / op.H, h = u - chunk * op.H;
  const int cg = threadIdx.x & 15, tl = threadIdx.x >> 4, c = cg * 8;
  const T* x = static_cast<const T*>(op.x) + static_cast<int64_t>(h) * op.hs + c;
  const int t0 = chunk * job.chunk_tokens, t1 = min(op.L, t0 + job.chunk_tokens);
  pdl_wait();
  pdl_release();
  float2 acc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
  auto load_tile = [&](int l0, int nvalid, uint4 (&raw)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = tl + 32 * i;
      raw[i] = t < nvalid ? *reinterpret_cast<const uint4*>(x + static_cast<int64_t>(l0 + t) * op.ts) : make_uint4(0, 0, 0, 0);
    }
  };
  if (NORM && op.normed) {
    with_norm(op, [&](auto per_head, auto rope) {
      constexpr bool PH = decltype(per_head)::value;
      int par = 0;
      for (int l0 = t0; l0 < t1; l0 += 128, par ^= 1) {
        const int nvalid = min(128, t1 - l0);
        uint4 raw[4];
        load_tile(l0, nvalid, raw);
        if (!PH) {
          tile_rstd<STATS_TL>(op.ns[0], l0, nvalid, s_rstd[par]);
          __syncthreads();
        }
        each_normalised<T, STATS_TL, PH, decltype(rope)::value, PH && !ONE>(op, h, l0, raw, s_rstd[par], [&](int i, const uint4& y) {
          if (tl + 32 * i < nvalid) {
            if (!ONE && job.normed_out) *reinterpret_cast<uint4*>(static_cast<T*>(job.normed_out) + (static_cast<int64_t>(l0 + tl + 32 * i) * op.H + h) * D + c) = y;
            const uint32_t wd[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = __fadd2_rn(acc[q], HalfOps<T>::unpack2(wd[q]));
          }
        });
      }
    });
  } else {
    auto sweep = [&](auto is_max) {
      for (int l0 = t0; l0 < t1; l0 += 128) {
        uint4 raw[4];
        load_tile(l0, t1 - l0, raw);  // rows past the end hold zeros: neutral in both reductions
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t wd[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 f = HalfOps<T>::unpack2(wd[q]);
            acc[q] = decltype(is_max)::value ? make_float2(fmaxf(acc[q].x, fabsf(f.x)), fmaxf(acc[q].y, fabsf(f.y))) : __fadd2_rn(acc[q], f);
          }
        }
      }
    };
    if (job.is_max) sweep(Bool<true>{}); else sweep(Bool<false>{});
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    red[tl][c + 2 * q] = acc[q].x;
    red[tl][c + 2 * q + 1] = acc[q].y;
  }
  __syncthreads();
  if (threadIdx.x < D) {
    float r = red[0][threadIdx.x];
#pragma unroll
    for (int j = 1; j < 32; ++j) r = job.is_max ? fmaxf(r, red[j][threadIdx.x]) : r + red[j][threadIdx.x];
    if (job.atomic_max) atomicMax(reinterpret_cast<int*>(job.part) + h * D + threadIdx.x, __float_as_int(r));  // non-negative floats order like their bits
    else job.part[(static_cast<int64_t>(chunk) * op.H + h) * D + threadIdx.x] = r;
  }
}

// 32 columns per CTA, the chunks over 16 warps: a single thread per column would wait for up to 64 loads one after another
constexpr int FINISH_GROUPS = 16;
__global__ void __launch_bounds__(32 * FINISH_GROUPS) finish_kernel(const float* part, int chunks, int n, float scale, int is_max, float* out) {
  __shared__ float red[FINISH_GROUPS][32];
  pdl_wait();
  pdl_release();
  const int g = threadIdx.x >> 5, i = blockIdx.x * 32 + (threadIdx.x & 31);
  float s = 0.f;
  if (i < n) {
    for (int c = g; c < chunks; c += FINISH_GROUPS) {
      const float v = part[static_cast<int64_t>(c) * n + i];
      s = is_max ? fmaxf(s, v) : s + v;
    }
  }
  red[g][threadIdx.x & 31] = s;
  __syncthreads();
  if (g == 0 && i < n) {
#pragma unroll
    for (int k = 1; k < FINISH_GROUPS; ++k) s = is_max ? fmaxf(s, red[k][threadIdx.x]) : s + red[k][threadIdx.x];
    out[i] = s * scale;
  }
}

// ---------------------------------------------------------------------------------- quantisers
struct QuantParams {
  QuantJob j[MAX_JOBS];
  int count;
};

struct QuantShared {
  float rstd[128];
  float part[4][D];
  float red[2][16];
  uint32_t vtile[D][32];  // [d][token / 4]
};

// The sums (or maxima) of a head over the chunks, in four shares per column, when there is more than one chunk.
template <int TL> __device__ __forceinline__ void gather_parts(const QuantJob& job, int h, bool is_max, QuantShared& sh) {
  constexpr int SHARES = 32 / TL;  // per thread
  const int col = threadIdx.x & (D - 1), g = threadIdx.x >> 7;
  float s[SHARES];
#pragma unroll
  for (int q = 0; q < SHARES; ++q) s[q] = 0.f;
  for (int k = g * SHARES; k < job.chunks; k += 4) {
#pragma unroll
    for (int q = 0; q < SHARES; ++q) {
      if (k + q >= job.chunks) break;
      const float v = job.part[(static_cast<int64_t>(k + q) * job.op.H + h) * D + col];
      s[q] = is_max ? fmaxf(s[q], v) : s[q] + v;
    }
  }
#pragma unroll
  for (int q = 0; q < SHARES; ++q) sh.part[g * SHARES + q][col] = s[q];
}

// 4 consecutive tokens of 8 channels per thread and turn, one 32-bit word per channel into a [channel][token] tile whose 16-byte
// groups are XOR-swizzled by the channel group (word writes and 128-bit row reads are almost conflict free).
template <typename T, int TL>
__device__ __forceinline__ void v_unit(const QuantJob& job, int tile, int h, QuantShared& sh) {
  constexpr int TURNS = 32 / TL, THREADS = 16 * TL;
  const Operand& op = job.op;
  const int tid = threadIdx.x, cg = tid & 15, tl = tid >> 4, c = cg * 8, l0 = tile * 128;
  const int64_t Lpad = static_cast<int64_t>((op.L + 127) >> 7) << 7;
  const T* x = static_cast<const T*>(op.x) + static_cast<int64_t>(l0 + tl * 4) * op.ts + static_cast<int64_t>(h) * op.hs + c;
  uint4 raw[TURNS][4];
#pragma unroll
  for (int n = 0; n < TURNS; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      raw[n][i] = l0 + (tl + n * TL) * 4 + i < op.L ? *reinterpret_cast<const uint4*>(x + (n * TL * 4 + i) * op.ts) : make_uint4(0, 0, 0, 0);
  if (job.chunks > 1) gather_parts<TL>(job, h, true, sh);
  __syncthreads();
  if (tid < D) {  // the maxima give way to the multipliers
    const float a = job.chunks > 1 ? fmaxf(fmaxf(sh.part[0][tid], sh.part[1][tid]), fmaxf(sh.part[2][tid], sh.part[3][tid])) : job.part[h * D + tid];
    sh.part[0][tid] = (a > 0.f) ? __fdiv_rn(448.f, a) : 1.f;
    if (tile == 0) job.scale[h * D + tid] = (a > 0.f) ? __fdiv_rn(a, 448.f) : 1.f;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float ia = sh.part[0][c + 2 * q], ib = sh.part[0][c + 2 * q + 1];
#pragma unroll
    for (int n = 0; n < TURNS; ++n) {
      float2 f[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) f[i] = HalfOps<T>::unpack2(reinterpret_cast<const uint32_t*>(&raw[n][i])[q]);
      const int sw = (tl + n * TL) ^ ((cg & 7) << 2);
      sh.vtile[c + 2 * q][sw] = cvt_e4m3x4(__fmul_rn(f[0].x, ia), __fmul_rn(f[1].x, ia), __fmul_rn(f[2].x, ia), __fmul_rn(f[3].x, ia));
      sh.vtile[c + 2 * q + 1][sw] = cvt_e4m3x4(__fmul_rn(f[0].y, ib), __fmul_rn(f[1].y, ib), __fmul_rn(f[2].y, ib), __fmul_rn(f[3].y, ib));
    }
  }
  __syncthreads();
  uint8_t* vt = static_cast<uint8_t*>(job.out) + static_cast<int64_t>(h) * D * Lpad + l0;
#pragma unroll
  for (int i = 0; i < D * 8 / THREADS; ++i) {  // 128 rows (d) x 128 bytes: 8 x 16-byte stores per row
    const int j = tid + i * THREADS, d = j >> 3, k = j & 7;
    *reinterpret_cast<uint4*>(vt + d * Lpad + k * 16) = *reinterpret_cast<const uint4*>(&sh.vtile[d][(k ^ ((d >> 3) & 7)) << 2]);
  }
}

// The quantiser proper, on a tile whose vectors are in registers (packed halves): `value` applies the mean or the softmax
// scale.  TWO: blocks of 64 tokens (the first and the second half of the vectors), else one block of 128.
template <typename T, int TL, bool TWO, typename Value>
__device__ __forceinline__ void write_int8(const QuantJob& job, int tile, int h, int nvalid, const uint4 (&raw)[128 / TL], float am0, float am1, QuantShared& sh,
                                           Value&& value) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cg = tid & 15, tl = tid >> 4;
  const int64_t tiles = (job.op.L + 127) >> 7;
  am0 = warp_max(am0);
  if (TWO) am1 = warp_max(am1);
  if (lane == 0) {
    sh.red[0][warp] = am0;
    if (TWO) sh.red[1][warp] = am1;
  }
  __syncthreads();
  float inv[2];
#pragma unroll
  for (int b = 0; b < (TWO ? 2 : 1); ++b) {
    const float4* rp = reinterpret_cast<const float4*>(sh.red[b]);
    float a = 0.f;
#pragma unroll
    for (int i = 0; i < TL / 8; ++i) {
      const float4 v = rp[i];
      a = fmaxf(fmaxf(a, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    }
    inv[b] = (a > 0.f) ? __fdiv_rn(127.f, a) : 1.f;
    if (tid == 0) job.scale[(TWO ? 2 : 1) * (h * tiles + tile) + b] = (a > 0.f) ? __fdiv_rn(a, 127.f) : 1.f;
  }
  int8_t* o = static_cast<int8_t*>(job.out) + ((h * tiles + tile) * 128 + tl) * D + cg * 8;
#pragma unroll
  for (int i = 0; i < 128 / TL; ++i) {
    const uint32_t wd[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
    const float iv = inv[TWO ? i / (64 / TL) : 0];
    // round-half-even to an integer without a conversion instruction: adding 1.5 * 2^23 leaves the two's complement
    // integer in the low mantissa bits (|x * inv| <= 127 * (1 + 2^-23) by construction, so the clamp to +-127 can never
    // bind); the low bytes of four sums are gathered with byte permutes.  The sums are scalar on purpose: the product must be
    // rounded before the addition (a packed multiply followed by a packed add was observed to round like one fused operation,
    // which breaks ties such as 63.5 the other way).
    uint32_t t[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 v = __fmul2_rn(value(HalfOps<T>::unpack2(wd[q]), q), make_float2(iv, iv));
      t[2 * q] = __float_as_uint(__fadd_rn(v.x, 12582912.f));
      t[2 * q + 1] = __float_as_uint(__fadd_rn(v.y, 12582912.f));
    }
    uint32_t w[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      w[g] = __byte_perm(__byte_perm(t[4 * g], t[4 * g + 1], 0x0040), __byte_perm(t[4 * g + 2], t[4 * g + 3], 0x0040), 0x5410);
      if (tl + TL * i >= nvalid) w[g] = 0;  // padding rows quantise to 0 whatever the mean
    }
    *reinterpret_cast<uint2*>(o + TL * i * D) = make_uint2(w[0], w[1]);
  }
}

// Q (one block of 128 tokens, times the softmax scale) or K (two of 64, minus the mean); GENERIC: either, with or without
// mean and scale (centred before scaled).
template <typename T, int TL, bool TWO, bool GENERIC, bool NORM, bool ONE>
__device__ __forceinline__ void int8_unit(const QuantJob& job, int tile, int h, QuantShared& sh) {
  const Operand& op = job.op;
  const int cg = threadIdx.x & 15, tl = threadIdx.x >> 4, c = cg * 8, l0 = tile * 128;
  const int nvalid = min(128, op.L - l0);
  const T* x = static_cast<const T*>(op.x) + static_cast<int64_t>(l0 + tl) * op.ts + static_cast<int64_t>(h) * op.hs + c;
  constexpr int VECS = 128 / TL;
  uint4 raw[VECS];
#pragma unroll
  for (int i = 0; i < VECS; ++i) raw[i] = tl + TL * i < nvalid ? *reinterpret_cast<const uint4*>(x + TL * i * op.ts) : make_uint4(0, 0, 0, 0);
  const bool normed = NORM && op.normed;
  const bool rstd = normed && !op.ns[0].per_head;
  const bool centred = GENERIC ? job.part != nullptr : TWO, scaled = GENERIC ? job.premul != 0.f : !TWO;
  const bool parts = centred && job.chunks > 1;
  if (rstd) tile_rstd<TL>(op.ns[0], l0, nvalid, sh.rstd);
  if (parts) gather_parts<TL>(job, h, false, sh);
  if (rstd || parts) __syncthreads();
  float2 nmu[4];  // minus the mean: x - mu and x + (-mu) are the same number
  if (centred) {
    float m[8];
    if (parts) {
#pragma unroll
      for (int e = 0; e < 8; ++e) m[e] = (sh.part[0][c + e] + sh.part[1][c + e]) + (sh.part[2][c + e] + sh.part[3][c + e]);
    } else {
      *reinterpret_cast<float4*>(m) = *reinterpret_cast<const float4*>(job.part + h * D + c);
      *reinterpret_cast<float4*>(m + 4) = *reinterpret_cast<const float4*>(job.part + h * D + c + 4);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) nmu[q] = make_float2(-(m[2 * q] * job.inv_l), -(m[2 * q + 1] * job.inv_l));
  }
  const float2 pm2 = make_float2(job.premul, job.premul);
  auto value = [&](float2 v, int q) -> float2 {
    if (centred) v = __fadd2_rn(v, nmu[q]);
    if (scaled) v = __fmul2_rn(v, pm2);
    return v;
  };
  float am[2] = {0.f, 0.f};
  auto take = [&](int i) {
    if (tl + TL * i < nvalid) {
      float& a = am[TWO ? i / (VECS / 2) : 0];
      const uint32_t wd[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 v = value(HalfOps<T>::unpack2(wd[q]), q);
        a = fmax3(a, fabsf(v.x), fabsf(v.y));
      }
    }
  };
  if constexpr (NORM) {
    if (normed) {
      with_norm(op, [&](auto per_head, auto rope) {
        constexpr bool PH = decltype(per_head)::value;
        each_normalised<T, TL, PH, decltype(rope)::value, PH && !ONE>(op, h, l0, raw, sh.rstd, [&](int i, const uint4& y) {
          raw[i] = y;
          take(i);
        });
      });
    }
  }
  if (!normed) {
#pragma unroll
    for (int i = 0; i < VECS; ++i) take(i);
  }
  write_int8<T, TL, TWO>(job, tile, h, nvalid, raw, am[0], am[1], sh, value);
}

// One CTA = one unit: a (128-token tile, head) of a job, heads fastest, held in registers between the absmax reduction and
// the quantisation.  These single-shot CTAs hide their load latency by their number.  Instructions bound them (13.7 a value
// without a norm, 30.7 with one per head and a rotation, before the figures below), a third of them the same for every thread:
// TL = 16 halves those and takes twice as long per CTA, so it is for launches of many waves, and not for norms per head, whose
// eight vectors spill, nor where a unit adds up its rows' squares itself (few threads, many loads one after another: 40 heads, fp16, Q of
// 6000 tokens 39 / 50, the whole pre-pass of 3000 103 / 113).  us in the chain of kernels, TL 32 / 16: 32760 x 40 heads, Q 121 / 106; 7145 x 24 heads
// fp16, Q, K and V 59 / 53; 2 x 32760 x 12 heads, normed Q 92 / 74; 1560 x 12 heads, normed Q 5.8 / 7.9; 1101 x 24 heads, norm per head,
// 12.7 / 20.7.
// A single normed operand with a rotation (ONE) takes TL = 16 from one unit per SM on, with two CTAs per SM: 128 registers, 4 bytes spilt.
// 75600 x 40 heads, Q 418 / 388, K 459 / 434; below one unit per SM a CTA's own time is the launch's: K with a norm per head, 500 x 12
// heads 6.8 / 8.2, 200 x 40 6.9 / 8.3.  Without a rotation there is less to share, and the kernel of several operands is the faster one:
// Q of 32760 x 40 heads 119 against 149 as ONE of TL = 16, 152 of 32; 1000 x 40 heads 9.7 against 10.8.  (A launch of one operand alone
// takes TL = 16 from four units per SM on, 12000 x 12 heads 16.6 / 14.5, without a norm from two: Q of 3000 x 40 heads 12.4 / 10.2.)
// A persistent form with a cp.async ring and the rotation kept in registers across the heads (128 registers, one CTA per SM)
// took a third longer on every operand.
template <typename T, int TL, bool NORM, bool GENERIC, bool ONE>
__global__ void __launch_bounds__(16 * TL, TL == 32 || ONE ? 2 : NORM ? 3 : 4) quant_kernel(const __grid_constant__ QuantParams p) {
  __shared__ __align__(16) QuantShared sh;
  const QuantJob& job = p.j[ONE ? 0 : my_job(p)];
  const int u = blockIdx.x - job.first, tile = u / job.op.H, h = u - tile * job.op.H;
  pdl_wait();
  pdl_release();
  if (job.kind == QUANT_V) {
    v_unit<T, TL>(job, tile, h, sh);
  } else if (job.kind == QUANT_Q) {
    int8_unit<T, TL, false, GENERIC, NORM, ONE>(job, tile, h, sh);
  } else {
    int8_unit<T, TL, true, GENERIC, NORM, ONE>(job, tile, h, sh);
  }
}

// ---------------------------------------------------------------------------------- RMSNorm (+ RoPE) in place
// RMSNorm over all C = H*128 channels (or over each head's 128) with an fp32 weight, optionally followed by
// the 3-axis rotary embedding, applied in place to a [L, C] half view (row stride ld).  A row is owned by
// the 4 warps of a CTA (one 128-bit vector of 8 channels per thread and step), read once, held in registers
// in packed form across the sum-of-squares reduction, and written once; many CTAs share an SM.
// Rounding points follow the eager sequence: norm output rounded to half, rotation computed in fp32
// (the eager path uses fp64) and rounded to half.
constexpr int NR_THREADS = 128;
constexpr int NR_MAX_VEC = 8;  // C <= 128 * 8 * 8 = 8192

struct PeerTables {
  float* p[KSB_MAX_PEERS];
};

// rstd[which][rank * M + m] = rsqrt(sum over the tiles of `which` of tile_sumsq[tile][m] / C + eps), written into
// every peer's table (plain peer stores).
__global__ void rstd_scatter_kernel(const float* __restrict__ tile_sumsq, int tiles_per_which, int M, int C, float eps,
                                    PeerTables peers, int n_peers, int rank) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * M) return;
  const int which = i / M, m = i - which * M;
  float s = 0.f;
  for (int t = 0; t < tiles_per_which; ++t) s += tile_sumsq[(int64_t)(which * tiles_per_which + t) * M + m];
  const float r = rsqrtf(s / (float)C + eps);
  const int64_t L_all = (int64_t)n_peers * M;
  for (int d = 0; d < n_peers; ++d) peers.p[d][which * L_all + (int64_t)rank * M + m] = r;
}

template <typename T, bool ROPE, bool PER_HEAD, int NV>
__global__ void __launch_bounds__(NR_THREADS, NV <= 5 ? 6 : 4) rmsnorm_rope_kernel(T* __restrict__ x, int64_t L, int C, int64_t ld,
                                                                     const float* __restrict__ w, float eps, RopeGrid rg,
                                                                     const float* __restrict__ row_rstd) {
  __shared__ float red[2][NR_THREADS / 32];
  const int nvec = C / 8;
  int par = 0;
  for (int64_t l = blockIdx.x; l < L; l += gridDim.x, par ^= 1) {
    T* row = x + l * ld;
    uint4 cur[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int j = threadIdx.x + i * NR_THREADS;
      cur[i] = (j < nvec) ? *reinterpret_cast<const uint4*>(row + j * 8) : make_uint4(0, 0, 0, 0);
    }
    float rstd_v[NV];
    if (PER_HEAD) {
      // each head's 128 channels = 16 consecutive 8-channel vectors = 16 consecutive lanes
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const T* t = reinterpret_cast<const T*>(&cur[i]);
        float hs = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float f = HalfOps<T>::to_f(t[e]);
          hs = __fmaf_rn(f, f, hs);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) hs += __shfl_xor_sync(0xffffffffu, hs, o);
        rstd_v[i] = rsqrtf(hs / (float)D + eps);
      }
    } else if (row_rstd) {
      const float r = row_rstd[l];
#pragma unroll
      for (int i = 0; i < NV; ++i) rstd_v[i] = r;
    } else {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const T* t = reinterpret_cast<const T*>(&cur[i]);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float f = HalfOps<T>::to_f(t[e]);
          ss += f * f;
        }
      }
      ss = warp_sum(ss);
      if ((threadIdx.x & 31) == 0) red[par][threadIdx.x >> 5] = ss;
      __syncthreads();
      const float r = rsqrtf((red[par][0] + red[par][1] + red[par][2] + red[par][3]) / (float)C + eps);
#pragma unroll
      for (int i = 0; i < NV; ++i) rstd_v[i] = r;
    }
    int cf = 0, ch = 0, cw = 0;
    bool rotate = false;
    if (ROPE) {
      const int64_t pos = rg.pos0 + l;
      const int64_t per_frame = (int64_t)rg.Hh * rg.Ww;
      if (pos < (int64_t)rg.F * per_frame) {
        rotate = true;
        cf = (int)(pos / per_frame);
        const int rem = (int)(pos - (int64_t)cf * per_frame);
        ch = rem / rg.Ww;
        cw = rem - ch * rg.Ww;
        if (rg.diag) ch = cw = cf;
      }
    }
    // A thread's vectors are 1024 channels (8 heads) apart, so they all cover the same four rotation pairs of
    // their heads: the (cos, sin) entries -- and a per-head weight -- are fetched once per row, not per vector.
    static_assert((NR_THREADS * 8) % D == 0, "a thread's vectors must fall on the same channels of their heads");
    const int p0 = ((threadIdx.x * 8) & (D - 1)) >> 1;
    float2 rot[4];
    if (ROPE && rotate) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int pr = p0 + q;
        const int coord = pr < rg.nf ? cf : (pr < rg.nf + rg.nh ? ch : cw);
        rot[q] = rg.table[(int64_t)coord * 64 + pr];
      }
    }
    float wh[8];
    if (PER_HEAD) {
      const float4 w0 = *reinterpret_cast<const float4*>(w + 2 * p0), w1 = *reinterpret_cast<const float4*>(w + 2 * p0 + 4);
      wh[0] = w0.x; wh[1] = w0.y; wh[2] = w0.z; wh[3] = w0.w; wh[4] = w1.x; wh[5] = w1.y; wh[6] = w1.z; wh[7] = w1.w;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int j = threadIdx.x + i * NR_THREADS;
      if (j < nvec) {
        const T* t = reinterpret_cast<const T*>(&cur[i]);
        float wv[8];
        if (PER_HEAD) {
#pragma unroll
          for (int e = 0; e < 8; ++e) wv[e] = wh[e];
        } else {
          const float4 w0 = *reinterpret_cast<const float4*>(w + j * 8), w1 = *reinterpret_cast<const float4*>(w + j * 8 + 4);
          wv[0] = w0.x; wv[1] = w0.y; wv[2] = w0.z; wv[3] = w0.w; wv[4] = w1.x; wv[5] = w1.y; wv[6] = w1.z; wv[7] = w1.w;
        }
        float y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = HalfOps<T>::to_f(HalfOps<T>::from_f(HalfOps<T>::to_f(t[e]) * rstd_v[i] * wv[e]));
        if (ROPE && rotate) {
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float2 yr = rope_pair(y[e], y[e + 1], rot[e >> 1]);
            y[e] = yr.x;
            y[e + 1] = yr.y;
          }
        }
        uint4 o;
        T* ot = reinterpret_cast<T*>(&o);
#pragma unroll
        for (int e = 0; e < 8; ++e) ot[e] = HalfOps<T>::from_f(y[e]);
        *reinterpret_cast<uint4*>(row + j * 8) = o;
      }
    }
  }
}

// rstd[g][m] = rsqrt(sum over the tiles of column group g of tile_sumsq[tile][m] / C + eps)
__global__ void rstd_finish_kernel(const float* __restrict__ tile_sumsq, int tiles_per_group, int groups, int M, int C, float eps,
                                   float* __restrict__ rstd) {
  pdl_wait();
  pdl_release();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= groups * M) return;
  const int g = i / M, m = i - g * M;
  float s = 0.f;
  for (int t = 0; t < tiles_per_group; ++t) s += tile_sumsq[(int64_t)(g * tiles_per_group + t) * M + m];
  rstd[i] = rsqrtf(s / (float)C + eps);
}

// ---------------------------------------------------------------------------------- built-in scratch
// Scratch of the allocation-free V quantiser entry point: per-(head, channel) absmax words.  It lives in
// the library image, so every GPU that loads the library holds these 256 KB until the process exits.
constexpr int64_t NOALLOC_MAX_HD = 65536;  // heads * 128 <= 65536, i.e. at most 512 heads
static __device__ __align__(256) float g_v_amax_scratch[NOALLOC_MAX_HD];

// In host code the array's name is only a handle: the device address has to be asked for, once per device,
// with that device current.  Returns nullptr (with the error text set) if the runtime refuses.
static float* v_amax_scratch_address() {
  static float* cached[64] = {nullptr};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    fail(KSB_ERR_CUDA, "cudaGetDevice failed or device index out of range: %s", cudaGetErrorString(e));
    return nullptr;
  }
  if (!cached[dev]) {
    float* ptr = nullptr;
    e = cudaGetSymbolAddress((void**)&ptr, g_v_amax_scratch);
    if (e != cudaSuccess || ptr == nullptr) {
      fail(KSB_ERR_CUDA, "cudaGetSymbolAddress(built-in scratch) failed: %s", cudaGetErrorString(e));
      return nullptr;
    }
    cached[dev] = ptr;
  }
  return cached[dev];
}

int check_operand(const void* x, int dtype, int64_t L, int64_t H, int64_t Dh, int64_t ts, int64_t hs) {
  if (dtype != KSB_BF16 && dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  if (Dh != D) return fail(KSB_ERR_UNSUPPORTED, "head size %lld is not supported (only 128)", (long long)Dh);
  if (L <= 0 || L > INT32_MAX - 128 || H <= 0 || H > 65535 || L * H > (int64_t)INT32_MAX * 64) return fail(KSB_ERR_INVALID, "bad shape L=%lld H=%lld", (long long)L, (long long)H);
  if (!x || !aligned16(x) || ts % 8 != 0 || hs % 8 != 0) return fail(KSB_ERR_INVALID, "input must be 16-byte aligned with strides multiple of 8 elements");
  return 0;
}

// Fills a RopeGrid from the C-ABI arguments (rope_table == nullptr: no rotation).
int make_rope_grid(RopeGrid& rg, const float* rope_table, int table_len, int nf, int nh, int F, int Hh, int Ww, int64_t pos0, int diag) {
  rg = RopeGrid{};
  if (!rope_table) return 0;
  if (nf < 0 || nh < 0 || nf + nh > 64 || F <= 0 || Hh <= 0 || Ww <= 0) return fail(KSB_ERR_INVALID, "bad rope grid");
  if (F > table_len || (!diag && (Hh > table_len || Ww > table_len))) return fail(KSB_ERR_INVALID, "rope table too short for the grid");
  if (diag && (Hh != 1 || Ww != 1)) return fail(KSB_ERR_INVALID, "diag positions need a grid of (F, 1, 1)");
  if (!aligned16(rope_table)) return fail(KSB_ERR_INVALID, "rope table must be 16-byte aligned");
  rg.table = reinterpret_cast<const float2*>(rope_table); rg.table_len = table_len; rg.nf = nf; rg.nh = nh;
  rg.F = F; rg.Hh = Hh; rg.Ww = Ww; rg.pos0 = pos0; rg.diag = diag ? 1 : 0;
  return 0;
}

int finish_norm(NormSpec& ns, int64_t L, const RopeGrid& rg) {
  if (!ns.w || !aligned16(ns.w)) return fail(KSB_ERR_INVALID, "norm weight null or unaligned");
  if (!ns.per_head && !ns.row_rstd && !ns.ssq) return fail(KSB_ERR_INVALID, "a norm over all heads needs the row_rstd table");
  ns.rg = rg;
  if (rg.table) {
    if (!rg.diag && (rg.F > 1024 || rg.Hh > 1024 || rg.Ww > 1024)) return fail(KSB_ERR_UNSUPPORTED, "rope grids reach 1024 positions per axis");
    if (rg.pos0 < 0 || rg.pos0 + L > (1 << 24)) return fail(KSB_ERR_INVALID, "token positions must stay below 2^24");
    ns.per_frame = rg.Hh * rg.Ww;
    ns.inv_per_frame = 1.0f / (float)ns.per_frame;
    ns.inv_w = 1.0f / (float)rg.Ww;
  }
  return 0;
}

int plan_chunks(int64_t L, int64_t H, int most) {
  const int64_t tiles = (L + 127) / 128;
  int64_t n = (8 * (int64_t)sm_count() + H - 1) / H;  // four waves of two CTAs per SM: the last one costs little
  if (n > tiles) n = tiles;
  if (n > most) n = most;
  if (n < 1) n = 1;
  const int64_t per = (tiles + n - 1) / n;
  return (int)((tiles + per - 1) / per);
}

template <typename Job> static bool one_normed(const Job* jobs, int count) { return count == 1 && jobs[0].op.normed && jobs[0].op.split == INT32_MAX; }

int run_stats(StatsJob* jobs, int count, int dtype, bool chained, cudaStream_t st) {
  if (count < 1 || count > MAX_JOBS) return fail(KSB_ERR_INVALID, "1..%d statistics jobs per launch", MAX_JOBS);
  StatsParams p;
  p.count = count;
  int ctas = 0;
  bool norm = false;
  for (int i = 0; i < count; ++i) {
    StatsJob& j = jobs[i];
    const int64_t tiles = (j.op.L + 127) / 128;
    j.chunk_tokens = (int)((tiles + j.chunks - 1) / j.chunks) * 128;
    j.first = ctas;
    ctas += j.chunks * j.op.H;
    norm = norm || j.op.normed;
    p.j[i] = j;
  }
  auto pick = [&](auto t) -> const void* {
    using T = decltype(t);
    if (one_normed(jobs, count)) return (const void*)stats_kernel<T, true, true>;
    return norm ? (const void*)stats_kernel<T, true, false> : (const void*)stats_kernel<T, false, false>;
  };
  const void* fn = dtype == KSB_BF16 ? pick(__nv_bfloat16{}) : pick(__half{});
  return launch_kernel("column statistics", fn, dim3((unsigned)ctas), dim3(16 * STATS_TL), 0, st, 1, chained, p);
}

int run_finish(float* part, int chunks, int64_t n, float scale, bool is_max, float* out, bool chained, cudaStream_t st) {
  const float* in = part;
  const int n32 = (int)n, max32 = is_max ? 1 : 0;
  return launch_kernel("column statistics (finish)", (const void*)finish_kernel, dim3((unsigned)((n + 31) / 32)), dim3(32 * FINISH_GROUPS), 0, st, 1, chained, in, chunks, n32, scale, max32, out);
}

int run_quant(QuantJob* jobs, int count, int dtype, bool chained, cudaStream_t st) {
  if (count < 1 || count > MAX_JOBS) return fail(KSB_ERR_INVALID, "1..%d quantiser jobs per launch", MAX_JOBS);
  QuantParams p;
  p.count = count;
  int64_t units = 0;
  bool norm = false, generic = false, per_head = false, sums = false;
  for (int i = 0; i < count; ++i) {
    QuantJob& j = jobs[i];
    j.first = (int)units;
    units += ((j.op.L + 127) / 128) * (int64_t)j.op.H;
    norm = norm || j.op.normed;
    per_head = per_head || (j.op.normed && j.op.ns[0].per_head);
    sums = sums || (j.op.normed && j.op.ns[0].ssq && !j.op.ns[0].row_rstd);
    generic = generic || (j.kind == QUANT_Q && (j.part || j.premul == 0.f)) || (j.kind == QUANT_K && (!j.part || j.premul != 0.f));
    p.j[i] = j;
  }
  if (units > INT32_MAX) return fail(KSB_ERR_INVALID, "problem too large");
  const bool rope = jobs[0].op.ns[0].rg.table != nullptr;
  const bool one = !generic && one_normed(jobs, count) && (rope || per_head);
  const bool many = !generic && (one ? rope && units > (int64_t)sm_count() : !sums && !per_head && units >= (count > 1 ? 8 : norm ? 4 : 2) * (int64_t)sm_count());  // see quant_kernel
  auto pick = [&](auto t) -> const void* {
    using T = decltype(t);
    if (generic) return norm ? (const void*)quant_kernel<T, 32, true, true, false> : (const void*)quant_kernel<T, 32, false, true, false>;
    if (one) return many ? (const void*)quant_kernel<T, 16, true, false, true> : (const void*)quant_kernel<T, 32, true, false, true>;
    if (many) return norm ? (const void*)quant_kernel<T, 16, true, false, false> : (const void*)quant_kernel<T, 16, false, false, false>;
    return norm ? (const void*)quant_kernel<T, 32, true, false, false> : (const void*)quant_kernel<T, 32, false, false, false>;
  };
  const void* fn = dtype == KSB_BF16 ? pick(__nv_bfloat16{}) : pick(__half{});
  return launch_kernel("operand quantisers", fn, dim3((unsigned)units), dim3(many ? 256 : 512), 0, st, 1, chained, p);
}

int run_rstd(const float* sums, int tiles_per_group, int groups, int M, int C, float eps, float* rstd, bool chained, cudaStream_t st) {
  const int n = groups * M;
  return launch_kernel("rstd from tile sums", (const void*)rstd_finish_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, 1, chained, sums, tiles_per_group,
                       groups, M, C, eps, rstd);
}

// The Operand of the entry points that take one segment and a finished 1 / rms table.
static int plain_operand(Operand& op, const void* x, int64_t L, int64_t H, int64_t ts, int64_t hs) {
  op = Operand{};
  op.x = x; op.ts = ts; op.hs = hs; op.L = (int)L; op.H = (int)H; op.split = INT32_MAX;
  return 0;
}
static int normed_operand(Operand& op, const void* x, int64_t L, int64_t H, int64_t ts, int64_t hs, const float* norm_w, int per_head,
                          const float* row_rstd, float eps, const RopeGrid& rg) {
  plain_operand(op, x, L, H, ts, hs);
  op.normed = 1;
  NormSpec& ns = op.ns[0];
  ns.w = norm_w; ns.per_head = per_head ? 1 : 0; ns.row_rstd = per_head ? nullptr : row_rstd; ns.eps = eps; ns.c = (float)(H * D);
  return finish_norm(ns, L, rg);
}

// Sums over whole-call chunks of MEAN_CHUNK tokens at most, into the caller's scratch, then the mean.
static int column_mean(const Operand& op, int dtype, float* partial, float* mean, cudaStream_t st) {
  StatsJob j{};
  j.op = op; j.part = partial;
  const int64_t room = (op.L + MEAN_CHUNK - 1) / MEAN_CHUNK;
  j.chunks = plan_chunks(op.L, op.H, room < MAX_STAT_CHUNKS ? (int)room : MAX_STAT_CHUNKS);
  if (int rc = run_stats(&j, 1, dtype, false, st)) return rc;
  return run_finish(partial, j.chunks, (int64_t)op.H * D, 1.0f / (float)op.L, false, mean, true, st);
}

}  // namespace prep
}  // namespace ksb

using namespace ksb;

extern "C" {

int64_t ksb_sage_kmean_scratch_floats(int64_t L, int64_t H, int64_t D) {
  return ((L + prep::MEAN_CHUNK - 1) / prep::MEAN_CHUNK) * H * D;
}

int ksb_sage_kmean(const void* k, int dtype, int64_t L, int64_t H, int64_t D, int64_t token_stride, int64_t head_stride,
                   float* partial, float* km, ksb_stream_t stream) {
  if (int rc = prep::check_operand(k, dtype, L, H, D, token_stride, head_stride)) return rc;
  if (!partial || !km) return fail(KSB_ERR_INVALID, "null pointer");
  prep::Operand op;
  prep::plain_operand(op, k, L, H, token_stride, head_stride);
  return prep::column_mean(op, dtype, partial, km, static_cast<cudaStream_t>(stream));
}

int64_t ksb_rmsnorm_rope_scratch_floats(int64_t L, int64_t C) {
  return ((L + prep::MEAN_CHUNK - 1) / prep::MEAN_CHUNK) * C;
}

int ksb_rowsumsq_to_rstd_scatter(const float* tile_sumsq, int64_t M, int64_t C, float eps, float* const* peer_rstd,
                                 int n_peers, int rank, ksb_stream_t stream) {
  if (!tile_sumsq || !peer_rstd || M <= 0 || C <= 0 || C % 256 != 0) return fail(KSB_ERR_INVALID, "bad arguments");
  if (n_peers < 1 || n_peers > KSB_MAX_PEERS || rank < 0 || rank >= n_peers) return fail(KSB_ERR_INVALID, "bad peer count / rank");
  prep::PeerTables pt{};
  for (int i = 0; i < n_peers; ++i) {
    if (!peer_rstd[i]) return fail(KSB_ERR_INVALID, "peer table %d is null", i);
    pt.p[i] = peer_rstd[i];
  }
  const int n = (int)(2 * M);
  prep::rstd_scatter_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(tile_sumsq, (int)(C / 256), (int)M, (int)C, eps, pt, n_peers, rank);
  return check_launch("rstd scatter");
}

int ksb_rmsnorm_rope_inplace(void* x, int dtype, int64_t L, int64_t C, int64_t ld, const float* w, int per_head,
                             const float* row_rstd, float eps, const float* rope_table, int table_len, int nf, int nh, int F, int Hh, int Ww, int64_t pos0,
                             int diag, float* colsum_partial, float* colmean, ksb_stream_t stream) {
  if (dtype != KSB_BF16 && dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  if (L <= 0 || C <= 0 || C % 128 != 0 || C > prep::NR_THREADS * 8 * prep::NR_MAX_VEC) return fail(KSB_ERR_INVALID, "C=%lld must be a multiple of 128 and <= 8192", (long long)C);
  if (!x || !w || !aligned16(x) || !aligned16(w) || ld < C || ld % 8 != 0) return fail(KSB_ERR_INVALID, "x/w null, unaligned or bad row stride");
  if ((colsum_partial == nullptr) != (colmean == nullptr)) return fail(KSB_ERR_INVALID, "colsum_partial and colmean go together");
  if (row_rstd && per_head) return fail(KSB_ERR_INVALID, "row_rstd and per_head exclude each other");
  prep::RopeGrid rg{};
  if (int rc = prep::make_rope_grid(rg, rope_table, table_len, nf, nh, F, Hh, Ww, pos0, diag)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t cap = (int64_t)sm_count() * 16;
  const int blocks = (int)(L < cap ? L : cap);
  const bool wide = C > prep::NR_THREADS * 8 * 4;  // more than 4 vectors per thread
#define KSB_LAUNCH_NR(T, R, P, NV) prep::rmsnorm_rope_kernel<T, R, P, NV><<<blocks, prep::NR_THREADS, 0, st>>>(static_cast<T*>(x), L, (int)C, ld, w, eps, rg, row_rstd)
  const bool five = C > prep::NR_THREADS * 8 * 4 && C <= prep::NR_THREADS * 8 * 5;  // e.g. 5120: five vectors per thread, six CTAs per SM
#define KSB_LAUNCH_NR3(T, R, P) do { if (five) KSB_LAUNCH_NR(T, R, P, 5); else if (wide) KSB_LAUNCH_NR(T, R, P, 8); else KSB_LAUNCH_NR(T, R, P, 4); } while (0)
#define KSB_LAUNCH_NR2(T)                                                          \
  do {                                                                             \
    if (rope_table) { if (per_head) KSB_LAUNCH_NR3(T, true, true); else KSB_LAUNCH_NR3(T, true, false); } \
    else { if (per_head) KSB_LAUNCH_NR3(T, false, true); else KSB_LAUNCH_NR3(T, false, false); }           \
  } while (0)
  if (dtype == KSB_BF16) KSB_LAUNCH_NR2(__nv_bfloat16); else KSB_LAUNCH_NR2(__half);
#undef KSB_LAUNCH_NR2
#undef KSB_LAUNCH_NR3
#undef KSB_LAUNCH_NR
  if (int rc = check_launch("rmsnorm/rope")) return rc;
  if (colmean) {
    // per-channel mean of the values just written (the K smoothing vector), over x seen as [L, C/128, 128]
    prep::Operand op;
    prep::plain_operand(op, x, L, C / 128, ld, 128);
    return prep::column_mean(op, dtype, colsum_partial, colmean, st);
  }
  return 0;
}

static int quant_int8_job(const prep::Operand& op, int dtype, int block, float premul, const float* mean, void* out, float* scale, cudaStream_t st) {
  if (block != 128 && block != 64) return fail(KSB_ERR_INVALID, "block must be 128 or 64");
  if (!out || !scale || !aligned16(out)) return fail(KSB_ERR_INVALID, "null or unaligned output");
  prep::QuantJob j{};
  j.op = op; j.kind = block == 128 ? prep::QUANT_Q : prep::QUANT_K; j.premul = premul;
  j.part = mean; j.chunks = 1; j.inv_l = 1.f;
  j.out = out; j.scale = scale;
  return prep::run_quant(&j, 1, dtype, false, st);
}

int ksb_sage_quant_int8(const void* x, int dtype, int64_t L, int64_t H, int64_t D, int64_t token_stride, int64_t head_stride,
                        int block, float premul, const float* mean, void* out, float* scale, ksb_stream_t stream) {
  if (int rc = prep::check_operand(x, dtype, L, H, D, token_stride, head_stride)) return rc;
  prep::Operand op;
  prep::plain_operand(op, x, L, H, token_stride, head_stride);
  return quant_int8_job(op, dtype, block, premul, mean, out, scale, static_cast<cudaStream_t>(stream));
}

int ksb_rowsumsq_to_rstd(const float* tile_sumsq, int64_t M, int64_t C, int groups, float eps, float* rstd, ksb_stream_t stream) {
  if (!tile_sumsq || !rstd || M <= 0 || C <= 0 || C % 256 != 0 || groups < 1 || groups * M > INT32_MAX) return fail(KSB_ERR_INVALID, "bad arguments");
  return prep::run_rstd(tile_sumsq, (int)(C / 256), groups, (int)M, (int)C, eps, rstd, false, static_cast<cudaStream_t>(stream));
}

int ksb_sage_kmean_normed(const void* k, int dtype, int64_t L, int64_t H, int64_t D, int64_t token_stride, int64_t head_stride,
                          const float* norm_w, int per_head, const float* row_rstd, float eps, const float* rope_table, int table_len,
                          int nf, int nh, int F, int Hh, int Ww, int64_t pos0, int diag, float* partial, float* km, ksb_stream_t stream) {
  if (int rc = prep::check_operand(k, dtype, L, H, D, token_stride, head_stride)) return rc;
  if (!partial || !km) return fail(KSB_ERR_INVALID, "null pointer");
  prep::RopeGrid rg;
  if (int rc = prep::make_rope_grid(rg, rope_table, table_len, nf, nh, F, Hh, Ww, pos0, diag)) return rc;
  prep::Operand op;
  if (int rc = prep::normed_operand(op, k, L, H, token_stride, head_stride, norm_w, per_head, row_rstd, eps, rg)) return rc;
  return prep::column_mean(op, dtype, partial, km, static_cast<cudaStream_t>(stream));
}

int ksb_sage_quant_int8_normed(const void* x, int dtype, int64_t L, int64_t H, int64_t D, int64_t token_stride, int64_t head_stride,
                               int block, float premul, const float* mean, const float* norm_w, int per_head, const float* row_rstd,
                               float eps, const float* rope_table, int table_len, int nf, int nh, int F, int Hh, int Ww, int64_t pos0,
                               int diag, void* out, float* scale, ksb_stream_t stream) {
  if (int rc = prep::check_operand(x, dtype, L, H, D, token_stride, head_stride)) return rc;
  prep::RopeGrid rg;
  if (int rc = prep::make_rope_grid(rg, rope_table, table_len, nf, nh, F, Hh, Ww, pos0, diag)) return rc;
  prep::Operand op;
  if (int rc = prep::normed_operand(op, x, L, H, token_stride, head_stride, norm_w, per_head, row_rstd, eps, rg)) return rc;
  return quant_int8_job(op, dtype, block, premul, mean, out, scale, static_cast<cudaStream_t>(stream));
}

int ksb_sage_quant_v_fp8(const void* v, int dtype, int64_t L, int64_t H, int64_t D, int64_t token_stride, int64_t head_stride,
                         float* amax, void* vt, float* vs, ksb_stream_t stream) {
  if (int rc = prep::check_operand(v, dtype, L, H, D, token_stride, head_stride)) return rc;
  if (!amax || !vt || !vs || !aligned16(vt)) return fail(KSB_ERR_INVALID, "null or unaligned output");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(amax, 0, sizeof(float) * H * D, st) != cudaSuccess) return fail(KSB_ERR_CUDA, "memset failed");
  prep::StatsJob s{};
  prep::plain_operand(s.op, v, L, H, token_stride, head_stride);
  s.is_max = 1; s.atomic_max = 1; s.part = amax;
  s.chunks = prep::plan_chunks(L, H, prep::MAX_STAT_CHUNKS);
  if (int rc = prep::run_stats(&s, 1, dtype, false, st)) return rc;
  prep::QuantJob j{};
  j.op = s.op; j.kind = prep::QUANT_V; j.part = amax; j.chunks = 1; j.out = vt; j.scale = vs;
  return prep::run_quant(&j, 1, dtype, true, st);
}

int ksb_sage_quant_v_fp8_noalloc(const void* v, int dtype, int64_t L, int64_t H, int64_t D, int64_t token_stride,
                                 int64_t head_stride, void* vt, float* vs, ksb_stream_t stream) {
  if (int rc = prep::check_operand(v, dtype, L, H, D, token_stride, head_stride)) return rc;
  if (H * D > prep::NOALLOC_MAX_HD)
    return fail(KSB_ERR_INVALID, "ksb_sage_quant_v_fp8_noalloc: heads * head_size = %lld exceeds the built-in scratch of %lld words; "
                "use ksb_sage_quant_v_fp8 with caller-provided scratch", (long long)(H * D), (long long)prep::NOALLOC_MAX_HD);
  float* amax = prep::v_amax_scratch_address();  // first call on a device resolves the address
  if (!amax) return KSB_ERR_CUDA;
  // same two passes as ksb_sage_quant_v_fp8; the absmax words are cleared first because the array keeps
  // whatever the previous call left in it
  return ksb_sage_quant_v_fp8(v, dtype, L, H, D, token_stride, head_stride, amax, vt, vs, stream);
}

}  // extern "C"
