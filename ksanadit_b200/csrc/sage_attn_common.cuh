// Pieces shared by the two attention kernels (one Q block per CTA with tile lists; two Q blocks per CTA, dense):
// tile geometry, launch parameters, and the per-row softmax arithmetic.
#pragma once
#include "../../include/ksana_b200.h"
#include "common.cuh"

namespace ksb {
namespace attn {

constexpr int BQ = 128, BKV = 128, D = 128;
constexpr int UMMA_K = 32;
constexpr int KST = 2, VST = 2;
constexpr int TILE_BYTES = 128 * 128;
constexpr int THREADS = 256;
constexpr int TMEM_COLS = 256;  // S: columns 0..127 (s32), O: columns 128..255 (f32)
constexpr int KERNEL_ID = 2;
constexpr float S_MAGIC = 12582912.0f;  // 1.5 * 2^23 = 0x4B400000: one ulp is 1 on [2^23, 2^24)
constexpr float REF_SLACK = 3.5f;  // a row's reference point moves only when its maximum exceeds it by more than this
constexpr float P_SHIFT = 5.0f;  // P carries a static factor 2^5 into e4m3: at most 2^(5 + REF_SLACK) = 362 is ever rounded
constexpr int PST = 2;  // P buffers: P of tile g goes to buffer g & 1, so it never waits for the previous P.V
constexpr int NUM_BARS = 16;
// Q | P x PST | K x KST | V x VST | barriers.  The dynamic shared memory window itself must be 1024-byte aligned
// (checked at kernel start): with two CTAs per SM there is no room for alignment slack.
constexpr int NUM_TILES = 1 + PST + KST + VST;
constexpr int CONST_BYTES = 768;  // two 384-byte blocks of repeated 16-byte chunks: A and B of the accumulator pre-load MMA
constexpr int SMEM_BYTES = NUM_TILES * TILE_BYTES + CONST_BYTES + 8 * NUM_BARS + 64;

struct Params {
  const float* qs;
  const float* ks;
  const float* vs;
  int H, Lq, Lk, nq, nkv;
  const int32_t* offsets;
  const int32_t* entries;
  const int32_t* order;  // optional permutation of the Q blocks of a head (longest list first)
  void* out;
  int64_t out_ts, out_hs, out_bs;
  int heads_per_batch;  // heads h / heads_per_batch of the launch belong to one sample (its output starts out_bs further on)
  int bulk_out;  // the output goes through its tensor map (two-block kernel)
  int* status;
  // optional fused exchange: output row l goes to peers[l / rows_per_peer], row l % rows_per_peer
  void* peers[KSB_MAX_PEERS];
  int n_peers;
  int rows_per_peer;
};

// Offset of head h's first output row.
__device__ __forceinline__ int64_t head_offset(const Params& p, int h) {
  const int b = h / p.heads_per_batch;
  return b * p.out_bs + static_cast<int64_t>(h - b * p.heads_per_batch) * p.out_hs;
}

struct Work {
  int h, qt, n;
  const int32_t* ents;
};

__device__ __forceinline__ Work get_work(const Params& p, int idx) {
  Work w;
  w.h = idx / p.nq;
  w.qt = idx - w.h * p.nq;
  if (p.order) w.qt = p.order[w.qt];
  if (p.offsets) {
    const int a = p.offsets[w.qt], b = p.offsets[w.qt + 1];
    w.n = b - a;
    w.ents = p.entries + a;
  } else {
    w.n = p.nkv;
    w.ents = nullptr;
  }
  return w;
}
__device__ __forceinline__ int entry_at(const Work& w, int j) { return w.ents ? w.ents[j] : (j * 4 + 3); }


// Max over 64 scores (as floats) held in two 32-register chunks: four independent chains, each step
// folding two new values with a three-input max.
__device__ __forceinline__ float tree_max64(const uint32_t (&a)[32], const uint32_t (&b)[32]) {
  float m0 = fmaxf(__uint_as_float(a[0]), __uint_as_float(a[1])), m1 = fmaxf(__uint_as_float(a[2]), __uint_as_float(a[3]));
  float m2 = fmaxf(__uint_as_float(b[0]), __uint_as_float(b[1])), m3 = fmaxf(__uint_as_float(b[2]), __uint_as_float(b[3]));
#pragma unroll
  for (int i = 4; i < 32; i += 4) {
    m0 = fmax3(m0, __uint_as_float(a[i]), __uint_as_float(a[i + 1]));
    m1 = fmax3(m1, __uint_as_float(a[i + 2]), __uint_as_float(a[i + 3]));
    m2 = fmax3(m2, __uint_as_float(b[i]), __uint_as_float(b[i + 1]));
    m3 = fmax3(m3, __uint_as_float(b[i + 2]), __uint_as_float(b[i + 3]));
  }
  return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
}

// P = exp2(f * sc + c) for one 32-score chunk (f = 12582912 + S as fp32) -> 8 words of packed e4m3; the
// exact (unrounded) values are added into four independent packed accumulators.  A masked score holds -inf
// and yields 0 (or 2^-126, which rounds to 0 and vanishes in the row sum).
__device__ __forceinline__ void exp_chunk(const uint32_t (&s)[32], float sc, float c, uint32_t* pk, float2 (&acc)[4]) {
  const float2 sc2 = make_float2(sc, sc), c2 = make_float2(c, c);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float2 x01 = __ffma2_rn(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), sc2, c2);
    const float2 x23 = __ffma2_rn(make_float2(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])), sc2, c2);
    const float2 e01 = make_float2(fast_exp2(x01.x), fast_exp2(x01.y));
    const float2 e23 = make_float2(fast_exp2(x23.x), fast_exp2(x23.y));
    acc[(i >> 2) & 3] = __fadd2_rn(acc[(i >> 2) & 3], e01);
    acc[((i >> 2) + 2) & 3] = __fadd2_rn(acc[((i >> 2) + 2) & 3], e23);
    pk[i >> 2] = cvt_e4m3x4(e01.x, e01.y, e23.x, e23.y);
  }
}


// Where output row `qrow` of head h goes.
template <typename T> __device__ __forceinline__ T* out_row(const Params& p, int h, int qrow) {
  if (p.n_peers > 0) {
    const int dest = min(qrow / p.rows_per_peer, p.n_peers - 1);  // rows past Lq are never stored
    return static_cast<T*>(p.peers[dest]) + static_cast<int64_t>(qrow - dest * p.rows_per_peer) * p.out_ts + static_cast<int64_t>(h) * p.out_hs;
  }
  return static_cast<T*>(p.out) + static_cast<int64_t>(qrow) * p.out_ts + head_offset(p, h);
}

// Normalises one Q block's O (tensor memory `o`, a row per thread; the block's last P.V is done) and stores it: warp `qrt` of
// the block handles rows 32 qrt .. 32 qrt + 31, `vs4` are the V scales of columns 4 lane .. 4 lane + 3.
// The rows pass through the warp's own part of the two P buffers at `stage` (columns 0..63 in the first, 64..127 in the second,
// 16-byte units swizzled by row), so that 16 lanes write the 256 bytes of a row.  The V scales wait in the second part until
// it is needed.  Read from global memory column by column, and with a store per lane and 16 bytes that touched 32 cache lines,
// the epilogue took 8000 cycles, as long as three score tiles; now 3500 (32760 x 512, 40 heads: 451 -> 330 us).
//
// `map`: the output as a tensor map, or null: the two parts then leave as bulk stores that lane 0 issues and that read them while the
// warp goes on (it waits for them before the next P is written there).
template <typename T>
__device__ __forceinline__ void store_block(const Params& p, int h, int qt, int qrt, uint32_t o, float inv_l, uint32_t stage, const float4& vs4, const CUtensorMap* map = nullptr) {
  uint32_t lane;  // read again here: what is derived from it then does not sit in registers through the main loop
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  const uint32_t st0 = stage + qrt * 32 * 128, st1 = st0 + TILE_BYTES;
  const uint32_t row = lane * 128, sw = (lane & 7) << 4;  // rows of a warp start at a multiple of 8
  const float2 inv2 = make_float2(inv_l, inv_l);
  st_shared_v4(st1 + lane * 16, make_uint4(__float_as_uint(vs4.x), __float_as_uint(vs4.y), __float_as_uint(vs4.z), __float_as_uint(vs4.w)));
  __syncwarp();
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t r[2][32];
    tmem_ld32(o + 64 * half, r[0]);
    tmem_ld32(o + 64 * half + 32, r[1]);
    uint4 v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = ld_shared_v4(st1 + 256 * half + 16 * i);
    tmem_wait_ld();
    __syncwarp();  // second half: every lane has its scales before their place is written
    const uint32_t dst = (half ? st1 : st0) + row;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t* a = &r[u >> 2][8 * (u & 3) + 4 * i];
        const uint4 s = v[2 * u + i];
        w[2 * i] = HalfOps<T>::pack2(__fmul2_rn(__fmul2_rn(make_float2(__uint_as_float(a[0]), __uint_as_float(a[1])), inv2), make_float2(__uint_as_float(s.x), __uint_as_float(s.y))));
        w[2 * i + 1] = HalfOps<T>::pack2(__fmul2_rn(__fmul2_rn(make_float2(__uint_as_float(a[2]), __uint_as_float(a[3])), inv2), make_float2(__uint_as_float(s.z), __uint_as_float(s.w))));
      }
      st_shared_v4(dst + ((u << 4) ^ sw), make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
  if (map) {
    fence_proxy_async_smem();
    __syncwarp();
    const int row0 = qt * BQ + qrt * 32;
    if (lane == 0 && row0 < p.Lq) {
      const int sample = h / p.heads_per_batch, head = h - sample * p.heads_per_batch;
      tma_store_4d(map, st0, 0, row0, head, sample);
      tma_store_4d(map, st1, 64, row0, head, sample);
      bulk_commit();
    }
    return;
  }
  __syncwarp();
  const uint32_t unit = lane & 15, sub = lane >> 4;
  const uint32_t src = (unit & 8 ? st1 : st0) + sub * 128, u4 = (unit & 7) << 4;
  const int qrow = qt * BQ + qrt * 32 + static_cast<int>(sub);
  if (p.n_peers > 0) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      const uint4 x = ld_shared_v4(src + i * 256 + (u4 ^ (((2 * i + sub) & 7) << 4)));
      if (qrow + 2 * i < p.Lq) *reinterpret_cast<uint4*>(out_row<T>(p, h, qrow + 2 * i) + unit * 8) = x;
    }
  } else {
    T* dst = out_row<T>(p, h, qrow) + unit * 8;
    const int64_t step = 2 * p.out_ts;
#pragma unroll 1
    for (int i = 0; i < 16; i += 4) {
      uint4 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = ld_shared_v4(src + (i + k) * 256 + (u4 ^ (((2 * (i + k) + sub) & 7) << 4)));
#pragma unroll
      for (int k = 0; k < 4; ++k, dst += step)
        if (qrow + 2 * (i + k) < p.Lq) *reinterpret_cast<uint4*>(dst) = x[k];
    }
  }
  __syncwarp();  // the next block's P goes to the same place
}

// The V scales store_block takes; the table need not be 16-byte aligned.
__device__ __forceinline__ float4 lane_v_scales(const Params& p, int h, int lane) {
  const float* s = p.vs + h * D + 4 * lane;
  if ((reinterpret_cast<uintptr_t>(p.vs) & 15) == 0) return __ldg(reinterpret_cast<const float4*>(s));
  return make_float4(__ldg(s), __ldg(s + 1), __ldg(s + 2), __ldg(s + 3));
}

}  // namespace attn
}  // namespace ksb
