// Row kernels: per-token FP8 (e4m3) activation quantiser, alone or fused behind
// LayerNorm + adaLN modulate / affine LayerNorm.  A row is owned by 1, 2, 4 or 8 warps (by its width), read
// once from HBM with 2 x 128-bit loads per 16 elements, held in registers across the reductions, and
// written once (16 e4m3 bytes per 128-bit store); a CTA of 4 warps keeps up to 4 rows in flight (of 8: one) and
// several CTAs share an SM.  Algorithmic bytes per row: 2K (read) + K (write) + 4 (scale).
//
// Rounding points follow the eager PyTorch sequence this replaces, so the FP8 bytes match it bit for
// bit: s = amax/448 (fp32 divide), inv = half(1/s), q = e4m3(half(x * inv)).
#include <algorithm>

#include "../../include/ksana_b200.h"
#include "common.cuh"
#include "host_utils.h"
#include "rowwise.h"

namespace ksb {
namespace rq {

constexpr int CHUNK = 16;      // elements per thread-chunk: two 128-bit loads, one 128-bit e4m3 store
template <int WPR> constexpr int THREADS = WPR == 8 ? 256 : 128;  // a row is owned by WPR = 1, 2, 4 or 8 warps
// NC chunks per thread: K <= wpr * 32 * 16 * NC

// The segment a CTA works on.
__device__ __forceinline__ const Segment& my_segment(const Params& p) {
  int i = 0;
  while (i + 1 < p.segs && static_cast<int>(blockIdx.x) >= p.seg[i + 1].cta0) ++i;
  return p.seg[i];
}
__device__ __forceinline__ int64_t mod_offset(const Params& p, const Segment& g, int64_t row) {
  if (!g.mod_index) return g.mod_stride * (row / g.rows_per_mod);
  const int64_t index = g.mod_index[row], m = checked_row(index, g.mod_rows);
  if (m != index) report_input(p.status, KSB_ERR_BAD_INDEX);
  return g.mod_stride * m;
}
__device__ __forceinline__ bool broadcast(const Segment& g) { return !g.mod_index && g.rows_per_mod == 0; }

template <typename T> __device__ __forceinline__ float round_half(float v) { return HalfOps<T>::to_f(HalfOps<T>::from_f(v)); }

// Reduction over the WPR warps that own one row.  `red` is [2][8] floats per CTA, double-buffered by `par`.
template <int WPR, bool IS_MAX> __device__ __forceinline__ float row_reduce(float v, float* red, int par, int warp) {
  v = IS_MAX ? warp_max(v) : warp_sum(v);
  if (WPR == 1) return v;
  if ((threadIdx.x & 31) == 0) red[par * 8 + warp] = v;
  __syncthreads();
  const int g0 = (warp / WPR) * WPR;
  float r = red[par * 8 + g0];
#pragma unroll
  for (int i = 1; i < WPR; ++i) r = IS_MAX ? fmaxf(r, red[par * 8 + g0 + i]) : r + red[par * 8 + g0 + i];
  return r;
}

// Pairs of halves in one word: conversions to and from fp32 (one instruction per pair), and half arithmetic that gives the bits
// of the fp32 form.  A product of two halves is exact in fp32, and for a sum fp32 has the 2 p + 2 bits that make rounding
// twice the same as rounding once (p = 8 or 11).
template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
  typedef __nv_bfloat162 H2;
  static __device__ __forceinline__ uint32_t pack(float2 v) { return word(__floats2bfloat162_rn(v.x, v.y)); }
  static __device__ __forceinline__ float2 unpack(uint32_t u) { return __bfloat1622float2(h2(u)); }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) { return word(__hmul2_rn(h2(a), h2(b))); }
  static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) { return word(__hadd2_rn(h2(a), h2(b))); }
  static __device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t x) { return word(__hmax2(h2(a), __habs2(h2(x)))); }
  static __device__ __forceinline__ uint32_t e4m3x4(uint32_t a, uint32_t b) {
    const float2 x = unpack(a), y = unpack(b);
    return cvt_e4m3x4(x.x, x.y, y.x, y.y);
  }
  static __device__ __forceinline__ H2 h2(uint32_t u) { return *reinterpret_cast<H2*>(&u); }
  static __device__ __forceinline__ uint32_t word(H2 h) { return *reinterpret_cast<uint32_t*>(&h); }
};
template <> struct Pair<__half> {
  typedef __half2 H2;
  static __device__ __forceinline__ uint32_t pack(float2 v) { return word(__floats2half2_rn(v.x, v.y)); }
  static __device__ __forceinline__ float2 unpack(uint32_t u) { return __half22float2(h2(u)); }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) { return word(__hmul2_rn(h2(a), h2(b))); }
  static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) { return word(__hadd2_rn(h2(a), h2(b))); }
  static __device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t x) { return word(__hmax2(h2(a), __habs2(h2(x)))); }
  static __device__ __forceinline__ uint32_t e4m3x4(uint32_t a, uint32_t b) {
    const float2 x = unpack(a), y = unpack(b);
    return cvt_e4m3x4(x.x, x.y, y.x, y.y);
  }
  static __device__ __forceinline__ H2 h2(uint32_t u) { return *reinterpret_cast<H2*>(&u); }
  static __device__ __forceinline__ uint32_t word(H2 h) { return *reinterpret_cast<uint32_t*>(&h); }
};
// Pair arithmetic, written as two scalar instructions: the packed fp32x2 forms were measured here and bring
// nothing (same instruction count and time; the values do not sit in aligned register pairs) and make the
// affine-LayerNorm variant spill.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }

// How an adaLN launch modulates: one row for all, from shared memory, or (ROWS) anything, row by row where it has to be; the
// product fused into an fp32 fma (FMA) or rounded first (ROUND).  A constant, so that a launch's code is only its own form.
enum Modulation : int { FMA = 0, ROUND = 1, ROWS_FMA = 2, ROWS_ROUND = 3 };

// CTAs per SM that the registers of a row's NC chunks per thread leave room for.  Modulation read row by row waits for more of
// memory: there six CTAs with a few spilled words beat five (18000 x 5120 141 -> 133 us, rounded 138 -> 125).
constexpr int row_occupancy(int mode, int wpr, int nc, int mod) {
  if (mode == PLAIN || mode == STATIC) return nc <= 4 ? 8 : nc <= 6 ? 6 : 5;
  if (wpr == 8) return 2;
  return nc > 3 ? 4 : mod >= ROWS_FMA ? 6 : 5;
}

// NC chunks of 16 elements per thread.  PLAIN and STATIC keep the row in its packed half form; the LayerNorm variants unpack it
// once to fp32, keep that through the statistics and the modulation, and pack the result, from which absmax and quantiser
// work.  They are bound by instruction issue before HBM, most of it conversions: so whatever half arithmetic gives the same
// bits stays packed, and with a staged modulation five CTAs per SM without spills beat six with.  Measured: adaLN 75600 x 5120
// 343 us, with a rounded product 309; 65520 x 1536 80 and 71; 75600 x 13824 1016 and 862 (eight warps per row; 2200 with four,
// which had to unpack the row again in every pass); affine norm 75600 x 5120 326 (issue slots 68 % busy, ALU 50 %).  PLAIN is
// at the memory's rate: 75600 x 13824 455 us, 6.9 TB/s.  Rounding points are those of the eager sequence.
template <typename T, int MODE, int WPR, int NC, int MOD>
__global__ void __launch_bounds__(THREADS<WPR>, row_occupancy(MODE, WPR, NC, MOD)) rowwise_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float red[3][2][8];
  typedef Pair<T> P;
  constexpr bool NORM = MODE == ADALN || MODE == LN_AFFINE;
  constexpr bool FP32_STAGED = WPR < 8;  // wide rows leave no room for modulation vectors as fp32
  constexpr int RPC = THREADS<WPR> / 32 / WPR;  // rows per CTA per iteration
  constexpr int GT = WPR * 32;          // threads per row
  const int warp = threadIdx.x >> 5;
  const int rg = warp / WPR;            // row slot of this warp
  const int t = threadIdx.x - rg * GT;  // thread index inside the row group
  const int nchunks = static_cast<int>(p.K / CHUNK);
  const Segment& g = my_segment(p);
  const T* x = static_cast<const T*>(g.x);
  const bool staged = MODE == LN_AFFINE || (MODE == ADALN && (MOD == FMA || MOD == ROUND || broadcast(g)));
  constexpr bool round_product = MOD == ROUND || MOD == ROWS_ROUND;
  if (MODE != LN_AFFINE) {  // an affine norm's vectors are weights: they are staged before the rows they wait for
    pdl_wait();
    pdl_release();
  }
  // Staged vectors (adaLN: 1 + scale rounded to half, and shift; affine LN: weight and bias) are kept as units of 4 elements in
  // unit-major order (unit u of chunk ch at index u * nchunks + ch): consecutive threads own consecutive chunks and read
  // consecutive units, no bank conflicts.  Where they enter an fp32 fma they are kept as fp32, else (round_product) as halves.
  float4* s_mul = reinterpret_cast<float4*>(smem);  // [4][nchunks]
  float4* s_add = s_mul + 4 * nchunks;
  uint2* h_mul = reinterpret_cast<uint2*>(smem);    // [4][nchunks]
  uint2* h_add = h_mul + 4 * nchunks;
  const float2 one = make_float2(1.f, 1.f);
  if (NORM && staged) {
    for (int i = threadIdx.x; i < 4 * nchunks; i += THREADS<WPR>) {
      const int ch = i >> 2, u = i & 3, dst = u * nchunks + ch;
      if (MODE == ADALN) {
        const uint2 cw = *reinterpret_cast<const uint2*>(static_cast<const T*>(g.scale) + ch * CHUNK + u * 4);
        const uint2 sw = *reinterpret_cast<const uint2*>(static_cast<const T*>(g.shift) + ch * CHUNK + u * 4);
        const uint2 m = make_uint2(P::pack(add2(one, P::unpack(cw.x))), P::pack(add2(one, P::unpack(cw.y))));  // (1 + scale) in half
        if (round_product || !FP32_STAGED) {
          h_mul[dst] = m;
          h_add[dst] = sw;
        } else {
          const float2 m0 = P::unpack(m.x), m1 = P::unpack(m.y), a0 = P::unpack(sw.x), a1 = P::unpack(sw.y);
          s_mul[dst] = make_float4(m0.x, m0.y, m1.x, m1.y);
          s_add[dst] = make_float4(a0.x, a0.y, a1.x, a1.y);
        }
      } else {
        s_mul[dst] = *reinterpret_cast<const float4*>(p.w + ch * CHUNK + u * 4);
        s_add[dst] = p.b ? *reinterpret_cast<const float4*>(p.b + ch * CHUNK + u * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    __syncthreads();
  }
  if (MODE == LN_AFFINE) {
    pdl_wait();
    pdl_release();
  }
  int par = 0;
  for (int64_t base = static_cast<int64_t>(static_cast<int>(blockIdx.x) - g.cta0) * RPC; base < g.rows; base += static_cast<int64_t>(g.ctas) * RPC, par ^= 1) {
    const int64_t row = base + rg, orow = g.row0 + row;
    const bool live = row < g.rows;
    uint32_t pw[NC][8];  // the row (transformed by the norm) as pairs of halves: what is quantised
    const T* xr = x + row * g.ldx;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int ch = t + c * GT;
      uint4 a = make_uint4(0, 0, 0, 0), b = make_uint4(0, 0, 0, 0);
      if (live && ch < nchunks) {
        a = *reinterpret_cast<const uint4*>(xr + ch * CHUNK);
        b = *reinterpret_cast<const uint4*>(xr + ch * CHUNK + 8);
      }
      pw[c][0] = a.x; pw[c][1] = a.y; pw[c][2] = a.z; pw[c][3] = a.w;
      pw[c][4] = b.x; pw[c][5] = b.y; pw[c][6] = b.z; pw[c][7] = b.w;
    }
    // Behind the row's loads, which do not need it; its vectors are on their way to L1 while the statistics are taken (waiting for them
    // in the last pass: 18000 x 5120 133 -> 123 us, 7145 x 3072 34.8 -> 33.2, 1101 x 3072 6.33 -> 6.20).
    const int64_t mod = (MODE == ADALN && !staged && live) ? mod_offset(p, g, row) : 0;
    if (MODE == ADALN && !staged && live) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int ch = t + c * GT;
        if (ch < nchunks) {
          asm volatile("prefetch.global.L1 [%0];" ::"l"(static_cast<const T*>(g.scale) + mod + ch * CHUNK));
          asm volatile("prefetch.global.L1 [%0];" ::"l"(static_cast<const T*>(g.shift) + mod + ch * CHUNK));
        }
      }
    }
    if constexpr (NORM) {
      float f[NC][16];
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 v = P::unpack(pw[c][i]);
          f[c][2 * i] = v.x;
          f[c][2 * i + 1] = v.y;
          acc = add2(acc, v);
        }
      const float mean = row_reduce<WPR, false>(acc.x + acc.y, &red[0][0][0], par, warp) / static_cast<float>(p.K);
      const float2 nm2 = make_float2(-mean, -mean);
      acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (t + c * GT < nchunks) {
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float2 d = add2(make_float2(f[c][i], f[c][i + 1]), nm2);
            acc = fma2(d, d, acc);
          }
        }
      }
      const float var = row_reduce<WPR, false>(acc.x + acc.y, &red[1][0][0], par, warp) / static_cast<float>(p.K);
      const float rstd = rsqrtf(var + p.eps);
      const float2 r2 = make_float2(rstd, rstd);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int ch = t + c * GT;
        if (live && ch < nchunks) {
          uint4 rs = make_uint4(0, 0, 0, 0), ra = rs;  // per-row modulation: scale and shift of units u, u + 1
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float2 ln[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) ln[j] = mul2(add2(make_float2(f[c][4 * u + 2 * j], f[c][4 * u + 2 * j + 1]), nm2), r2);
            uint32_t* w = pw[c] + 2 * u;
            if (MODE == LN_AFFINE) {
              const float4 mu = s_mul[u * nchunks + ch], ad = s_add[u * nchunks + ch];
              w[0] = P::pack(fma2(ln[0], make_float2(mu.x, mu.y), make_float2(ad.x, ad.y)));
              w[1] = P::pack(fma2(ln[1], make_float2(mu.z, mu.w), make_float2(ad.z, ad.w)));
            } else {
              const uint32_t l0 = P::pack(ln[0]), l1 = P::pack(ln[1]);  // F.layer_norm output in half
              uint2 m, a;
              if (staged && !round_product && FP32_STAGED) {
                const float4 mu = s_mul[u * nchunks + ch], ad = s_add[u * nchunks + ch];
                w[0] = P::pack(fma2(P::unpack(l0), make_float2(mu.x, mu.y), make_float2(ad.x, ad.y)));
                w[1] = P::pack(fma2(P::unpack(l1), make_float2(mu.z, mu.w), make_float2(ad.z, ad.w)));
                continue;
              }
              if (staged) {
                m = h_mul[u * nchunks + ch];
                a = h_add[u * nchunks + ch];
              } else {  // per-row modulation
                if (u % 2 == 0) {
                  rs = *reinterpret_cast<const uint4*>(static_cast<const T*>(g.scale) + mod + ch * CHUNK + u * 4);
                  ra = *reinterpret_cast<const uint4*>(static_cast<const T*>(g.shift) + mod + ch * CHUNK + u * 4);
                }
                const uint32_t one_h = P::pack(one);
                a = u % 2 == 0 ? make_uint2(ra.x, ra.y) : make_uint2(ra.z, ra.w);
                m = u % 2 == 0 ? make_uint2(P::add(one_h, rs.x), P::add(one_h, rs.y)) : make_uint2(P::add(one_h, rs.z), P::add(one_h, rs.w));  // (1 + scale) in half
              }
              if (round_product) {
                w[0] = P::add(P::mul(l0, m.x), a.x);
                w[1] = P::add(P::mul(l1, m.y), a.y);
              } else {
                w[0] = P::pack(fma2(P::unpack(l0), P::unpack(m.x), P::unpack(a.x)));
                w[1] = P::pack(fma2(P::unpack(l1), P::unpack(m.y), P::unpack(a.y)));
              }
            }
          }
          if (p.h_out) {
            T* ho = static_cast<T*>(p.h_out) + orow * p.K + ch * CHUNK;
            *reinterpret_cast<uint4*>(ho) = make_uint4(pw[c][0], pw[c][1], pw[c][2], pw[c][3]);
            *reinterpret_cast<uint4*>(ho + 8) = make_uint4(pw[c][4], pw[c][5], pw[c][6], pw[c][7]);
          }
        }
      }
    }
    float inv_h;  // multiplier already rounded to half precision
    float row_scale;
    if (MODE == STATIC) {
      if (p.scale_input) {
        row_scale = *p.scale_input;
        inv_h = round_half<T>(__frcp_rn(row_scale));
      } else {
        row_scale = 1.f;
        inv_h = 1.f;
      }
    } else {
      uint32_t m0 = 0, m1 = 0;  // a row's tail beyond K is zero
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          m0 = P::max_abs(m0, pw[c][i]);
          m1 = P::max_abs(m1, pw[c][i + 1]);
        }
      const float2 a0 = P::unpack(m0), a1 = P::unpack(m1);
      const float am = row_reduce<WPR, true>(fmaxf(fmaxf(a0.x, a0.y), fmaxf(a1.x, a1.y)), &red[2][0][0], par, warp);
      row_scale = (am > 0.f) ? __fdiv_rn(am, 448.f) : 1.f;
      inv_h = round_half<T>(__frcp_rn(row_scale));
    }
    if (live) {
      if (t == 0) p.qscale[orow] = row_scale;
      uint8_t* qr = p.q + orow * p.K;
      const uint32_t i2 = P::pack(make_float2(inv_h, inv_h));
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int ch = t + c * GT;
        if (ch < nchunks) {
          uint32_t o[4];  // the product is formed in half precision, then rounded to e4m3
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = P::e4m3x4(P::mul(pw[c][2 * i], i2), P::mul(pw[c][2 * i + 1], i2));
          *reinterpret_cast<uint4*>(qr + ch * CHUNK) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
  }
}

template <typename T, int MODE, int WPR, int NC, int MOD> static int launch_mod(Params& p, size_t smem, bool chained, cudaStream_t st) {
  const void* fn = (const void*)rowwise_kernel<T, MODE, WPR, NC, MOD>;
  int occupancy = row_occupancy(MODE, WPR, NC, MOD);
  static DeviceOnce limit;
  if (smem > 47 * 1024)  // with the static part, 48 KB is the limit without asking
    if (int rc = limit.raise_smem(fn, 2 * 16384 * (int)sizeof(float))) return rc;  // what the widest row stages
  // As many CTAs as are resident at once (227 KB of shared memory per SM, 1 KB of it per CTA the system's), in proportion to
  // the segments' rows: a part wave at the end would cost up to a tenth (65 520 rows: 2.7 waves before)
  if (smem > 0) occupancy = std::min<int>(occupancy, (int)(227 * 1024 / (smem + 1280)));
  int64_t cap = static_cast<int64_t>(sm_count()) * std::max(occupancy, 1);
  constexpr int RPC = THREADS<WPR> / 32 / WPR;
  int64_t M = 0;
  for (int i = 0; i < p.segs; ++i) M += p.seg[i].rows;
  // Quantisers without a norm stage nothing and run at the memory's rate, where SMs differ: from eight rows' turns per CTA on,
  // eight waves of CTAs even that out (us, one wave / eight: 75600 x 5120 183 / 170, 75600 x 13824 502 / 455, 65520 x 1536
  // 49.1 / 45.4; below, more CTAs cost: 7145 x 3072, three turns, 7.03 / 7.13)
  if ((MODE == PLAIN || MODE == STATIC) && M > 8 * cap * RPC) cap *= 8;
  int grid = 0;
  for (int i = 0; i < p.segs; ++i) {
    Segment& g = p.seg[i];
    const int64_t want = (g.rows + RPC - 1) / RPC, share = std::max<int64_t>(1, cap * g.rows / M);
    g.cta0 = grid;
    g.ctas = (int)std::min(want, share);
    grid += g.ctas;
  }
  return launch_kernel("rowwise quantiser", fn, dim3((unsigned)grid), dim3(THREADS<WPR>), smem, st, 1, chained, p);
}

template <typename T, int MODE, int WPR, int NC> static int launch_as(Params& p, bool chained, cudaStream_t st) {
  if constexpr (MODE == ADALN) {
    bool one_row = true, staged = false;
    for (int i = 0; i < p.segs; ++i) {
      const bool single = !p.seg[i].mod_index && p.seg[i].rows_per_mod == 0;
      one_row = one_row && single;
      staged = staged || single;
    }
    const size_t smem = staged ? 2 * p.K * (p.round_product || WPR == 8 ? sizeof(T) : sizeof(float)) : 0;
    if (!one_row) return p.round_product ? launch_mod<T, MODE, WPR, NC, ROWS_ROUND>(p, smem, chained, st) : launch_mod<T, MODE, WPR, NC, ROWS_FMA>(p, smem, chained, st);
    if (p.round_product) return launch_mod<T, MODE, WPR, NC, ROUND>(p, smem, chained, st);
    return launch_mod<T, MODE, WPR, NC, FMA>(p, smem, chained, st);
  } else {
    return launch_mod<T, MODE, WPR, NC, FMA>(p, MODE == LN_AFFINE ? 2 * p.K * sizeof(float) : 0, chained, st);
  }
}

template <typename T, int MODE> static int launch_t(Params& p, bool chained, cudaStream_t st) {
  constexpr bool NORM = MODE == ADALN || MODE == LN_AFFINE;
  int64_t M = 0;
  for (int i = 0; i < p.segs; ++i) {
    p.seg[i].row0 = M;
    M += p.seg[i].rows;
  }
  // narrow rows: 1 or 2 warps per row; wide rows: four, and eight where a norm keeps the row as fp32 (eight chunks of a thread
  // would take 128 registers for it)
  const int wpr = p.K <= 2048 ? 1 : p.K <= 4096 ? 2 : NORM && p.K > 8192 ? 8 : 4;
  const int64_t per_thread = (p.K + wpr * 32 * CHUNK - 1) / (wpr * 32 * CHUNK);  // chunks
  if (wpr == 1) return per_thread <= 3 ? launch_as<T, MODE, 1, 3>(p, chained, st) : launch_as<T, MODE, 1, 4>(p, chained, st);
  if (wpr == 2) return per_thread <= 3 ? launch_as<T, MODE, 2, 3>(p, chained, st) : launch_as<T, MODE, 2, 4>(p, chained, st);
  if constexpr (NORM) {
    if (wpr == 8) return per_thread <= 3 ? launch_as<T, MODE, 8, 3>(p, chained, st) : launch_as<T, MODE, 8, 4>(p, chained, st);
  }
  if (per_thread <= 3) return launch_as<T, MODE, 4, 3>(p, chained, st);
  if (per_thread <= 4) return launch_as<T, MODE, 4, 4>(p, chained, st);
  if constexpr (!NORM) return per_thread <= 6 ? launch_as<T, MODE, 4, 6>(p, chained, st) : launch_as<T, MODE, 4, 8>(p, chained, st);
  return fail(KSB_ERR_UNSUPPORTED, "row too wide");
}

int run(Mode mode, Params& p, int dtype, bool chained, cudaStream_t st) {
  int n = 0;  // empty segments drop out
  for (int i = 0; i < p.segs; ++i)
    if (p.seg[i].rows > 0) p.seg[n++] = p.seg[i];
  p.segs = n;
  if (n == 0) return 0;
  p.status = status_words();
  const bool bf = dtype == KSB_BF16;
  switch (mode) {
    case PLAIN: return bf ? launch_t<__nv_bfloat16, PLAIN>(p, chained, st) : launch_t<__half, PLAIN>(p, chained, st);
    case ADALN: return bf ? launch_t<__nv_bfloat16, ADALN>(p, chained, st) : launch_t<__half, ADALN>(p, chained, st);
    case LN_AFFINE: return bf ? launch_t<__nv_bfloat16, LN_AFFINE>(p, chained, st) : launch_t<__half, LN_AFFINE>(p, chained, st);
    default: return bf ? launch_t<__nv_bfloat16, STATIC>(p, chained, st) : launch_t<__half, STATIC>(p, chained, st);
  }
}

int validate(const Params& p, int dtype) {
  if (dtype != KSB_BF16 && dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  for (int i = 0; i < p.segs; ++i) {
    const Segment& g = p.seg[i];
    if (g.rows < 0 || p.K <= 0) return fail(KSB_ERR_INVALID, "bad shape M=%lld K=%lld", (long long)g.rows, (long long)p.K);
    if (p.K % CHUNK != 0 || p.K > (int64_t)16384)
      return fail(KSB_ERR_INVALID, "K=%lld must be a multiple of 16 and <= 16384", (long long)p.K);
    if (g.ldx < p.K || g.ldx % 8 != 0) return fail(KSB_ERR_INVALID, "ldx=%lld must be >= K and a multiple of 8", (long long)g.ldx);
    if (g.rows > 0 && (!g.x || !p.q || !p.qscale)) return fail(KSB_ERR_INVALID, "null pointer");
    if (!aligned16(g.x) || !aligned16(p.q) || (p.h_out && !aligned16(p.h_out)))
      return fail(KSB_ERR_INVALID, "pointers must be 16-byte aligned");
    if (g.shift || g.scale)
      if (!g.shift || !g.scale || !aligned16(g.shift) || !aligned16(g.scale) || g.mod_stride % 8 != 0) return fail(KSB_ERR_INVALID, "shift/scale null or unaligned");
  }
  return 0;
}

}  // namespace rq
}  // namespace ksb

using namespace ksb;

extern "C" {

int ksb_quant_fp8_rowwise(const void* x, int dtype, int64_t M, int64_t K, int64_t ldx, void* q, float* scale,
                          ksb_stream_t stream) {
  rq::Params p{};
  p.segs = 1; p.seg[0].x = x; p.seg[0].rows = M; p.seg[0].ldx = ldx; p.K = K; p.q = static_cast<uint8_t*>(q); p.qscale = scale;
  if (int rc = rq::validate(p, dtype)) return rc;
  return rq::run(rq::PLAIN, p, dtype, false, static_cast<cudaStream_t>(stream));
}

int ksb_quant_fp8_static(const void* x, int dtype, int64_t M, int64_t K, int64_t ldx, const float* scale_input,
                         void* q, float* scale_out, ksb_stream_t stream) {
  rq::Params p{};
  p.segs = 1; p.seg[0].x = x; p.seg[0].rows = M; p.seg[0].ldx = ldx; p.K = K; p.q = static_cast<uint8_t*>(q); p.qscale = scale_out;
  p.scale_input = scale_input;
  if (int rc = rq::validate(p, dtype)) return rc;
  return rq::run(rq::STATIC, p, dtype, false, static_cast<cudaStream_t>(stream));
}

int ksb_adaln_quant_fp8(const void* x, int dtype, int64_t M, int64_t K, int64_t ldx, const void* shift,
                        const void* scale, int64_t mod_rows, int round_product, float eps, void* h_out, void* q,
                        float* qscale, ksb_stream_t stream) {
  rq::Params p{};
  rq::Segment& g = p.seg[0];
  p.segs = 1; g.x = x; g.rows = M; g.ldx = ldx; g.shift = shift; g.scale = scale; g.mod_stride = K; g.rows_per_mod = mod_rows == 1 ? 0 : 1;
  p.round_product = round_product ? 1 : 0; p.K = K; p.eps = eps;
  p.h_out = h_out; p.q = static_cast<uint8_t*>(q); p.qscale = qscale;
  if (int rc = rq::validate(p, dtype)) return rc;
  if (!shift || !scale) return fail(KSB_ERR_INVALID, "shift/scale null or unaligned");
  if (mod_rows != 1 && mod_rows != M) return fail(KSB_ERR_INVALID, "mod_rows must be 1 or M");
  return rq::run(rq::ADALN, p, dtype, false, static_cast<cudaStream_t>(stream));
}

int ksb_layernorm_quant_fp8(const void* x, int dtype, int64_t M, int64_t K, int64_t ldx, const float* w,
                            const float* b, float eps, void* h_out, void* q, float* qscale, ksb_stream_t stream) {
  rq::Params p{};
  p.segs = 1; p.seg[0].x = x; p.seg[0].rows = M; p.seg[0].ldx = ldx; p.K = K; p.w = w; p.b = b; p.eps = eps;
  p.h_out = h_out; p.q = static_cast<uint8_t*>(q); p.qscale = qscale;
  if (int rc = rq::validate(p, dtype)) return rc;
  if (!w || !aligned16(w) || (b && !aligned16(b))) return fail(KSB_ERR_INVALID, "weight / bias null or not 16-byte aligned");
  return rq::run(rq::LN_AFFINE, p, dtype, false, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
