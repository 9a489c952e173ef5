// Dense Sage-style attention with TWO 128-row Q blocks of a head per CTA, one CTA per SM.
//
// Same arithmetic, tile shapes and per-block pipeline as sage_attn_kernel (see sage_attn.cu), but the two Q blocks
// that used to run as two independent CTAs on an SM now live in one CTA and share every K and V^T tile: the tile is
// fetched from L2 and written to shared memory once for 256 query rows instead of once per 128.  Under the 1 kW cap
// that traffic decides the clock: with it halved the kernel holds the maximum SM clock where the one-block kernel
// settles ~6 % lower.
//
// Warp roles (384 threads):
//   warp 0        TMA producer: both Q blocks once per work item, then K and V^T tiles through 4-deep rings
//   warps 1, 2    MMA issuer of half 0 / half 1 (one thread each): S = Q.K^T of tile j+1 queued before P.V of tile j;
//                 a ring stage is free when both issuers' MMAs on it have completed (barrier count 2)
//   warp 3        idle (donates registers)
//   warps 4..7    softmax of half 0, warps 8..11 of half 1: one row per thread, as in the one-block kernel
// Tensor memory (512 columns): half h has S at 256 h, O at 256 h + 128.  The halves are independent pipelines; only
// the producer and the ring barriers are shared, so one half's softmax still overlaps the other half's MMAs.
// Where that gains (takes_turns) the halves take turns (TURNS): a softmax warp starts a tile's exponentials when the other half's warp on its
// scheduler is three quarters through its own.  One half's output stage, hand-offs, waits and row maxima then lie under the other's
// exponentials.  That needs exponentials that one warp issues at close to the unit's rate: a row takes 1240 cycles alone in exp_row's
// order (1024 is the unit's bound) and 1360 - 1400 in the compiler's, so the halves used to be better off in step beyond four tiles.
// An odd last block pair has one live half; the other half's issuer keeps the rings moving by arriving in place of
// its MMAs.
// Tile lists (block-sparse masks) are given per PAIR of Q blocks: the union of the two blocks' lists, each entry =
// KV tile * 16 + keep bits of block 2i (bits 0-1: tokens 0-63 / 64-127 of the tile) + keep bits of block 2i+1 (bits
// 2-3).  Both halves walk the whole union; a half masks the 64-token halves it does not keep (a tile it does not keep
// at all costs it a fully masked pass: P = 0), so pairing pays only where the two lists nearly coincide; the host
// side decides (ops.py) and otherwise sends tile lists to the one-block kernel.
#include "sage_attn_common.cuh"
#include "host_utils.h"

namespace ksb {
namespace attn {
namespace dual {

#ifndef KSB_ATTN_DUAL_RING
#define KSB_ATTN_DUAL_RING 4
#endif
constexpr int RST = KSB_ATTN_DUAL_RING;  // K and V ring depth
constexpr int THREADS2 = 384;
constexpr int TMEM_COLS2 = 512;
constexpr int KERNEL_ID2 = 3;
constexpr int NUM_BARS2 = 40;
// Q x 2 | P x 2 halves x 2 buffers | K x RST | V x RST | constants | barriers
constexpr int NUM_TILES2 = 2 + 4 + 2 * RST;
constexpr int SMEM_BYTES2 = 1024 + NUM_TILES2 * TILE_BYTES + CONST_BYTES + 8 * NUM_BARS2 + 64;
// Registers of a softmax thread, by what the schedule ptxas makes of them takes: without turns 200 / 216 / 224 give 442 / 431 / 465 us
// (7145 x 24 heads) and 4280 / 4210 / 4490 (32760 x 12 heads); with turns 160 / 168 / 184 / 200 give 308 / 294 / 295 / 296 (32760 x 512,
// 40 heads) and 27.8 / 26.7 / 26.7 / 26.7 (1560 x 12 heads); tile lists of pairs 200 / 216: 8064 x 12 heads 170.3 / 168.1, 32256 x 12 heads
// 1574 / 1556, 7145 x 24 heads, all tiles, 524 / 519.
constexpr int PRODUCER_REGS = 56;
template <bool TURNS> constexpr int SOFTMAX_REGS = TURNS ? 168 : 216;
// Whether the halves take turns (see the softmax warps); without / with turns, us: 32760 queries x 128 keys, 40 heads 169 / 141, 512 keys
// 323 / 294; 32760 x 640, 12 heads 123 / 113; 1101 x 24 heads 22.6 / 20.8; 1560 x 12 28.7 / 26.7; 16384 x 4096 keys, 12 heads 306 / 299;
// 7145 x 24 432 / 429; 12288 x 12 576 / 572.  What they save of a pair lies at its ends, so it shrinks with the KV: nothing is left of it
// above 96 tiles, nor, above 24, in launches of more than 540 tiles of pairs per SM, which run at the power cap from there on (8500 x 40
// heads 1029 / 1038, 11600 x 40 1825 / 1854, 70000 x 5000 keys, 12 heads 1461 / 1468, x 9000 2517 / 2567; but x 2000 614 / 599).  One Q
// block per head has nothing to take turns with, and exp_row's order is the slower one then (100 queries x 1024 keys, 24 heads 14.7 /
// 15.2, 4000 keys 42.6 / 45.2), but for the few tiles that cost the same either way.
__host__ __device__ constexpr bool takes_turns(int64_t heads, int nq, int nkv, int sms) {
  if (nkv <= 4) return true;
  return nq > 1 && (nkv <= 24 || (nkv <= 96 && heads * ((nq + 1) / 2) * nkv <= 540 * (int64_t)sms));
}

struct PairWork {
  int h, pr, n;
  const int32_t* ents;
};
// LISTS = false is the dense kernel: every pair walks all KV tiles and the list code compiles away.
template <bool LISTS>
__device__ __forceinline__ PairWork get_pair(const Params& p, int idx, int npairs) {
  PairWork w;
  w.h = idx / npairs;
  w.pr = idx - w.h * npairs;
  if (LISTS && p.order) w.pr = p.order[w.pr];
  if (LISTS && p.offsets) {
    const int a = p.offsets[w.pr];
    w.n = p.offsets[w.pr + 1] - a;
    w.ents = p.entries + a;
  } else {
    w.n = p.nkv;
    w.ents = nullptr;
  }
  return w;
}
template <bool LISTS>
__device__ __forceinline__ int pair_entry(const PairWork& w, int j) { return (LISTS && w.ents) ? w.ents[j] : (j * 16 + 15); }

// The arithmetic of exp_chunk for a whole row of 128 scores, P stored as it is formed, with the steps spelled out in the order they
// are to issue: the special-function unit is fed eight scores ahead of the sums, conversions and stores that read its results, so
// that one warp keeps it busy by itself while the other half's warp is between tiles.  Volatile, or the compiler puts the
// conversions of a row behind one another.  Same bits as exp_chunk.  `next_half` runs three quarters through.
__device__ __forceinline__ float2 ordered_fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm volatile("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
               : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 ordered_add2(float2 a, float2 b) {
  float2 r;
  asm volatile("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
               : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float ordered_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t ordered_e4m3x4(float2 a, float2 b) {
  uint32_t r;
  asm volatile("{\n\t.reg .b16 l, h;\n\tcvt.rn.satfinite.e4m3x2.f32 l, %2, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 h, %4, %3;\n\tmov.b32 %0, {l, h};\n\t}"
               : "=r"(r) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
template <typename F>
__device__ __forceinline__ void exp_row(const uint32_t (&s)[4][32], float sc0, float sc1, float c0, float c1, uint32_t prow, int row, float2 (&acc)[4], F&& next_half) {
  constexpr int PAIRS = 64, EXP_AHEAD = 4, ARG_AHEAD = 8;  // in pairs of scores; 2 / 4 and 8 / 12 measure the same
  float2 x[PAIRS], e[PAIRS];
  uint32_t pk[PAIRS / 2];
  auto arg = [&](int k) {
    const float sc = k < PAIRS / 2 ? sc0 : sc1, c = k < PAIRS / 2 ? c0 : c1;
    x[k] = ordered_fma2(make_float2(__uint_as_float(s[k >> 4][2 * (k & 15)]), __uint_as_float(s[k >> 4][2 * (k & 15) + 1])), make_float2(sc, sc), make_float2(c, c));
  };
  auto exps = [&](int k) { e[k] = make_float2(ordered_exp2(x[k].x), 0.f); e[k].y = ordered_exp2(x[k].y); };
#pragma unroll
  for (int k = 0; k < ARG_AHEAD; ++k) arg(k);
#pragma unroll
  for (int k = 0; k < EXP_AHEAD; ++k) exps(k);
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) {
    if (k + ARG_AHEAD < PAIRS) arg(k + ARG_AHEAD);
    if (k + EXP_AHEAD < PAIRS) exps(k + EXP_AHEAD);
    const int a = ((k >> 1) + 2 * (k & 1)) & 3;  // exp_chunk's order of sums
    acc[a] = ordered_add2(acc[a], e[k]);
    if (k & 1) pk[k >> 1] = ordered_e4m3x4(e[k - 1], e[k]);
    if ((k & 7) == 7) {
      const int c = k >> 3;
      st_shared_v4(prow + ((c ^ (row & 7)) << 4), make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]));
    }
    if (k == PAIRS * 3 / 4 - 1) next_half();
  }
}

template <typename T, bool LISTS, bool TURNS, bool BULK>  // BULK: output by bulk stores
__global__ void __launch_bounds__(THREADS2, 1)
sage_attn_dual_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t q_smem = base, p_smem = base + 2 * TILE_BYTES;
  const uint32_t k_smem = base + 6 * TILE_BYTES, v_smem = k_smem + RST * TILE_BYTES;
  const uint32_t const_smem = v_smem + RST * TILE_BYTES;
  const uint32_t bars = const_smem + CONST_BYTES;
  const uint32_t q_full = bars, q_empty = bars + 8, k_full = bars + 16, k_empty = k_full + 8 * RST, v_full = k_empty + 8 * RST,
                 v_empty = v_full + 8 * RST;
  const uint32_t half_bars = v_empty + 8 * RST;  // per half: s_full, s_empty, p_full x 2, p_empty x 2 (48 bytes)
  const uint32_t turn0 = half_bars + 96;         // TURNS: per softmax warp quarter, half 0's turn and half 1's
  const uint32_t tmem_slot = bars + 8 * NUM_BARS2 + 16;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(gen + NUM_TILES2 * TILE_BYTES + CONST_BYTES + 8 * NUM_BARS2 + 16);
  static_assert(2 + 4 * RST + 12 + 8 <= NUM_BARS2, "barrier block too small");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int npairs = (p.nq + 1) >> 1;
  const int total = p.H * npairs;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);  // both issuers are done with their Q block
    for (int s = 0; s < RST; ++s) {
      mbar_init(k_full + 8 * s, 1);
      mbar_init(k_empty + 8 * s, 2);  // both halves' MMAs on the stage have completed
      mbar_init(v_full + 8 * s, 1);
      mbar_init(v_empty + 8 * s, 2);
    }
    for (int h = 0; h < 2; ++h) {
      const uint32_t hb = half_bars + 48 * h;
      mbar_init(hb, 1);      // s_full
      mbar_init(hb + 8, 4);  // s_empty: one arrival per softmax warp
      for (int b = 0; b < 2; ++b) {
        mbar_init(hb + 16 + 8 * b, 4);  // p_full
        mbar_init(hb + 32 + 8 * b, 1);  // p_empty
      }
    }
    if (TURNS)
      for (int i = 0; i < 8; ++i) mbar_init(turn0 + 8 * i, 1);
    fence_barrier_init();
  }
  if (threadIdx.x < CONST_BYTES / 4) {
    // operands of the accumulator pre-load MMA (see sage_attn.cu)
    const uint32_t word = (threadIdx.x & 3) ? 0u : (threadIdx.x < CONST_BYTES / 8 ? 0x3F80u : 0x4AC0u);
    reinterpret_cast<uint32_t*>(gen + NUM_TILES2 * TILE_BYTES)[threadIdx.x] = word;
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS2);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_release();
  const uint32_t tmem_base = *tmem_slot_gen;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- TMA producer
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
      uint32_t wi = 0, it = 0;
      bool ok = true;
      for (int idx = blockIdx.x; idx < total && ok; idx += gridDim.x) {
        const PairWork w = get_pair<LISTS>(p, idx, npairs);
        if (w.n == 0) continue;
        const int h = w.h, qt0 = w.pr * 2;
        const bool two = qt0 + 1 < p.nq;
        if (!mbar_wait(q_empty, (wi & 1) ^ 1, p.status, (KERNEL_ID2 << 16) | 1)) { ok = false; break; }
        mbar_arrive_expect_tx(q_full, (two ? 2 : 1) * TILE_BYTES);
        tma_load_2d(q_smem, &tmap_q, q_full, 0, (h * p.nq + qt0) * BQ);
        if (two) tma_load_2d(q_smem + TILE_BYTES, &tmap_q, q_full, 0, (h * p.nq + qt0 + 1) * BQ);
        for (int j = 0; j < w.n; ++j, ++it) {
          const int t = pair_entry<LISTS>(w, j) >> 4;
          const uint32_t s = it % RST, ph = (it / RST) & 1;
          if (!mbar_wait(k_empty + 8 * s, ph ^ 1, p.status, (KERNEL_ID2 << 16) | 2)) { ok = false; break; }
          mbar_arrive_expect_tx(k_full + 8 * s, TILE_BYTES);
          tma_load_2d(k_smem + s * TILE_BYTES, &tmap_k, k_full + 8 * s, 0, (h * p.nkv + t) * BKV);
          if (!mbar_wait(v_empty + 8 * s, ph ^ 1, p.status, (KERNEL_ID2 << 16) | 3)) { ok = false; break; }
          mbar_arrive_expect_tx(v_full + 8 * s, TILE_BYTES);
          tma_load_2d(v_smem + s * TILE_BYTES, &tmap_v, v_full + 8 * s, t * BKV, h * D);
        }
        ++wi;
      }
    } else if ((warp == 1 || warp == 2) && lane == 0) {
      // ---------------------------------------------------------------- MMA issuer of one half
      const int hf = warp - 1;
      const uint32_t hb = half_bars + 48 * hf;
      const uint32_t s_full = hb, s_empty = hb + 8, p_full = hb + 16, p_empty = hb + 32;
      const uint32_t tmem_s = tmem_base + 256 * hf, tmem_o = tmem_s + 128;
      constexpr uint32_t idesc_qk = IDESC_S8_S32(BQ, BKV);
      constexpr uint32_t idesc_pv = IDESC_F8_E4M3_F32(BQ, D);
      constexpr uint32_t idesc_pre = IDESC_BF16_F32(BQ, BKV);
      const uint64_t dq = make_kmajor_sw128_desc(q_smem + hf * TILE_BYTES);
      const uint64_t dca = make_noswizzle_desc(const_smem, 16, 16);
      const uint64_t dcb = make_noswizzle_desc(const_smem + CONST_BYTES / 2, 16, 16);
      uint32_t wi = 0, itk = 0, itv = 0, g = 0;
      bool ok = true;
      auto issue_qk = [&](uint32_t gg) -> bool {
        const uint32_t s = itk % RST, ph = (itk / RST) & 1;
        if (!mbar_wait(k_full + 8 * s, ph, p.status, (KERNEL_ID2 << 16) | 4)) return false;
        if (!mbar_wait(s_empty, gg & 1, p.status, (KERNEL_ID2 << 16) | 5)) return false;  // S read by the softmax warps (completion #gg)
        tc_fence_after();
        const uint64_t dk = make_kmajor_sw128_desc(k_smem + s * TILE_BYTES);
        mma_bf16_ss(tmem_s, dca, dcb, idesc_pre, 0);  // every accumulator = 12582912.0f
#pragma unroll
        for (int kk = 0; kk < D / UMMA_K; ++kk) mma_i8_ss(tmem_s, dq + 2 * kk, dk + 2 * kk, idesc_qk, 1);
        mma_commit(s_full);
        mma_commit(k_empty + 8 * s);
        ++itk;
        return true;
      };
      for (int idx = blockIdx.x; idx < total && ok; idx += gridDim.x) {
        const PairWork w = get_pair<LISTS>(p, idx, npairs);
        if (w.n == 0) continue;
        const int nt = w.n, qt = w.pr * 2 + hf;
        if (!mbar_wait(q_full, wi & 1, p.status, (KERNEL_ID2 << 16) | 6)) { ok = false; break; }
        if (qt >= p.nq) {
          // no block for this half: hand every stage back as soon as it has been filled
          mbar_arrive(q_empty);
          for (int j = 0; j < nt && ok; ++j, ++itk, ++itv) {
            const uint32_t s = itk % RST, ph = (itk / RST) & 1;
            if (!mbar_wait(k_full + 8 * s, ph, p.status, (KERNEL_ID2 << 16) | 4)) { ok = false; break; }
            mbar_arrive(k_empty + 8 * s);
            if (!mbar_wait(v_full + 8 * s, ph, p.status, (KERNEL_ID2 << 16) | 7)) { ok = false; break; }
            mbar_arrive(v_empty + 8 * s);
          }
          ++wi;
          continue;
        }
        if (!issue_qk(g)) { ok = false; break; }
        for (int j = 0; j < nt; ++j) {
          if (j + 1 < nt) {
            if (!issue_qk(g + 1)) { ok = false; break; }
          } else {
            mma_commit(q_empty);  // every S = Q.K^T of this block has been issued
          }
          const uint32_t s = itv % RST, ph = (itv / RST) & 1;
          if (!mbar_wait(v_full + 8 * s, ph, p.status, (KERNEL_ID2 << 16) | 7)) { ok = false; break; }
          const uint32_t pb = g & 1, pph = (g >> 1) & 1;
          if (!mbar_wait(p_full + 8 * pb, pph, p.status, (KERNEL_ID2 << 16) | 8)) { ok = false; break; }
          const uint64_t dp = make_kmajor_sw128_desc(p_smem + (2 * hf + pb) * TILE_BYTES);
          tc_fence_after();
          const uint64_t dv = make_kmajor_sw128_desc(v_smem + s * TILE_BYTES);
#pragma unroll
          for (int kk = 0; kk < BKV / UMMA_K; ++kk) mma_f8_ss(tmem_o, dp + 2 * kk, dv + 2 * kk, idesc_pv, (j | kk) != 0);
          mma_commit(p_empty + 8 * pb);
          mma_commit(v_empty + 8 * s);
          ++itv;
          ++g;
        }
        ++wi;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SOFTMAX_REGS<TURNS>));
    // ------------------------------------------------------------------ softmax warps (one row per thread)
    const int hf = (warp - 4) >> 2;
    const int qrt = warp & 3;
    const int row = qrt * 32 + lane;
    const uint32_t hb = half_bars + 48 * hf;
    const uint32_t s_full = hb, s_empty = hb + 8, p_full = hb + 16, p_empty = hb + 32;
    const uint32_t tmem_s = tmem_base + 256 * hf, tmem_o = tmem_s + 128;
    const uint32_t lane_sel = static_cast<uint32_t>(qrt * 32) << 16;
    const int nk64 = p.nkv * 2;
    uint32_t g = 0, turn = 0;  // tiles, and turns taken
    bool ok = true;
    // the score accumulator is free for the first S = Q.K^T (completion #0 of s_empty)
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(s_empty);
    for (int idx = blockIdx.x; idx < total && ok; idx += gridDim.x) {
      const PairWork w = get_pair<LISTS>(p, idx, npairs);
      const int h = w.h, qt = w.pr * 2 + hf;
      if (qt >= p.nq) continue;
      const int qrow = qt * BQ + row;
      if (w.n == 0) {  // both blocks of the pair have empty lists: zeros
        if (qrow < p.Lq) {
          T* orow = out_row<T>(p, h, qrow);
#pragma unroll
          for (int c = 0; c < D; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
      const bool both = w.pr * 2 + 1 < p.nq;  // an odd last block is on its own
      const float qsc = p.qs[h * p.nq + qt];
      float m_ref = -INFINITY, l = 0.f;
      // per-tile metadata (list entry and the two K-block scales) is fetched one tile ahead
      int e_next = pair_entry<LISTS>(w, 0);
      float ks0_next = p.ks[h * nk64 + 2 * (e_next >> 4)], ks1_next = p.ks[h * nk64 + 2 * (e_next >> 4) + 1];
      for (int j = 0; j < w.n; ++j) {
        const int e = e_next;
        const float sc0 = qsc * ks0_next, sc1 = qsc * ks1_next;
        if (j + 1 < w.n) {
          e_next = pair_entry<LISTS>(w, j + 1);
          ks0_next = p.ks[h * nk64 + 2 * (e_next >> 4)];
          ks1_next = p.ks[h * nk64 + 2 * (e_next >> 4) + 1];
        }
        const int t = LISTS ? (e >> 4) : j, halves = LISTS ? ((e >> (2 * hf)) & 3) : 3;
        const int valid = min(BKV, p.Lk - t * BKV);
        const bool full = (halves == 3) && (valid == BKV);
        if (!mbar_wait_warp(s_full, g & 1, p.status, (KERNEL_ID2 << 16) | 9)) { ok = false; break; }
        tc_fence_after();
        uint32_t s[4][32];
        tmem_ld32(tmem_s + lane_sel + 0, s[0]);
        tmem_ld32(tmem_s + lane_sel + 32, s[1]);
        tmem_ld32(tmem_s + lane_sel + 64, s[2]);
        tmem_ld32(tmem_s + lane_sel + 96, s[3]);
        tmem_wait_ld();
        // the scores are in registers: hand the accumulator back to the MMA issuer
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty);
        if (!full) {
          // masked columns (ragged tail or a 64-token half this block does not keep) become -inf: never the maximum, P = 0
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const int col = c * 32 + i;
              const bool keep = (col < valid) && ((halves >> (col >> 6)) & 1);
              if (!keep) s[c][i] = 0xff800000u;
            }
        }
        // exact: both operands of the subtraction are integers below 2^24
        const float m_tile = fmaxf((tree_max64(s[0], s[1]) - S_MAGIC) * sc0, (tree_max64(s[2], s[3]) - S_MAGIC) * sc1);
        const bool grow = m_tile > m_ref + REF_SLACK;  // also true for the first tile with a valid score (m_ref = -inf)
        const bool rescale = __any_sync(0xffffffffu, grow);
        float alpha = 1.f;
        if (rescale) {
          const float m_new = grow ? m_tile : m_ref;
          alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2(m_ref - m_new);
          l *= alpha;
          m_ref = m_new;
        }
        const float neg_m = (m_ref == -INFINITY) ? 0.f : (P_SHIFT - m_ref);
        uint32_t pk[32];
        float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const float c0 = fmaf(-S_MAGIC, sc0, neg_m), c1 = fmaf(-S_MAGIC, sc1, neg_m);
        // no wait for the P buffer: S_j was issued behind the P.V of tile j - 2, its last reader (see sage_attn.cu)
        const uint32_t pb = g & 1;
        // Stored by volatile asm: the compiler then keeps each chunk's exponentials with its stores instead of spreading the
        // live values of four chunks (32760 columns, dense: 1.54 -> 1.50 us per pair of tiles; with plain stores and the
        // same epilogue 1.69)
        const uint32_t prow = p_smem + (2 * hf + pb) * TILE_BYTES + row * 128;
        if (BULK && j == 0) {  // the last block's output has left the P buffers
          if (lane == 0) bulk_wait_source_read<0>();
          __syncwarp();
        }
        if (TURNS && both) {
          // the other half's warp on this scheduler is three quarters through its exponentials of the tile before
          if (!mbar_wait_warp(turn0 + 16 * qrt + 8 * hf, (turn & 1) ^ (hf ^ 1), p.status, (KERNEL_ID2 << 16) | 11)) { ok = false; break; }
          ++turn;
        }
        if constexpr (TURNS) {
          exp_row(s, sc0, sc1, c0, c1, prow, row, acc, [&] { if (both && lane == 0) mbar_arrive(turn0 + 16 * qrt + 8 * (hf ^ 1)); });
        } else {
#pragma unroll
          for (int hh = 0; hh < 4; ++hh) {
            exp_chunk(s[hh], hh < 2 ? sc0 : sc1, hh < 2 ? c0 : c1, pk + 8 * hh, acc);
#pragma unroll
            for (int c = 2 * hh; c < 2 * hh + 2; ++c)
              st_shared_v4(prow + ((c ^ (row & 7)) << 4), make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]));
          }
        }
        l += ((acc[0].x + acc[0].y) + (acc[1].x + acc[1].y)) + ((acc[2].x + acc[2].y) + (acc[3].x + acc[3].y));
        fence_proxy_async_smem();
        if (rescale && j > 0) {
          // O *= alpha; the previous tile's P.V (the other P buffer) must have finished writing O
          if (!mbar_wait_warp(p_empty + 8 * (pb ^ 1), ((g - 1) >> 1) & 1, p.status, (KERNEL_ID2 << 16) | 10)) { ok = false; break; }
          tc_fence_after();
          uint32_t o[4][32];
          tmem_ld32(tmem_o + lane_sel + 0, o[0]);
          tmem_ld32(tmem_o + lane_sel + 32, o[1]);
          tmem_ld32(tmem_o + lane_sel + 64, o[2]);
          tmem_ld32(tmem_o + lane_sel + 96, o[3]);
          tmem_wait_ld();
          const float2 a2 = make_float2(alpha, alpha);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 r = __fmul2_rn(make_float2(__uint_as_float(o[c][i]), __uint_as_float(o[c][i + 1])), a2);
              o[c][i] = __float_as_uint(r.x);
              o[c][i + 1] = __float_as_uint(r.y);
            }
            tmem_st32(tmem_o + lane_sel + 32 * c, o[c]);
          }
          tmem_wait_st();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + 8 * pb);
        ++g;
      }
      if (!ok) break;
      // ---- epilogue of the block: wait for the last P.V, normalise, store
      const float4 vs4 = lane_v_scales(p, h, lane);
      if (!mbar_wait_warp(p_empty + 8 * ((g - 1) & 1), ((g - 1) >> 1) & 1, p.status, (KERNEL_ID2 << 16) | 12)) { ok = false; break; }
      tc_fence_after();
      const float inv_l = (l > 0.f) ? (1.f / l) : 0.f;
      store_block<T>(p, h, qt, qrt, tmem_o + lane_sel, inv_l, p_smem + 2 * hf * TILE_BYTES, vs4, BULK ? &tmap_o : nullptr);
      tc_fence_before();
    }
    if (BULK && lane == 0) bulk_wait_all();
  }

  // ------------------------------------------------------------------ common exit
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS2);
  }
}

}  // namespace dual
}  // namespace attn
}  // namespace ksb

using namespace ksb;

namespace ksb {
namespace attn {
namespace dual {

template <typename T, bool LISTS, bool TURNS, bool BULK>
static int launch_as(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const Params& p, bool chained, cudaStream_t st) {
  const void* fn = reinterpret_cast<const void*>(sage_attn_dual_kernel<T, LISTS, TURNS, BULK>);
  // setmaxnreg.inc blocks until the CTA's register pool (registers at launch x threads) holds what it asks for:
  // refuse a build whose launch-time register count cannot cover the targets
  static int checked = 0;
  if (checked == 0) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return fail(KSB_ERR_CUDA, "cannot read the attention kernel's attributes");
    checked = (fa.numRegs * THREADS2 >= 128 * PRODUCER_REGS + 256 * SOFTMAX_REGS<TURNS>) ? 1 : -1;
  }
  if (checked < 0) return KSB_ERR_UNSUPPORTED;
  static DeviceOnce limit;
  if (int rc = limit.raise_smem(fn, SMEM_BYTES2)) return rc;
  const int64_t total = (int64_t)p.H * ((p.nq + 1) / 2);
  const int grid = (int)(total < sm_count() ? total : sm_count());
  return launch_kernel("sage attention (two Q blocks per CTA)", fn, dim3((unsigned)grid), dim3(THREADS2), SMEM_BYTES2, st, 1, chained, tq, tk, tv, to, p);
}

}  // namespace dual
}  // namespace attn
}  // namespace ksb

// Whether the two-block kernel is to store its output in bulk: such stores leave while the next pair begins.  us, without / with: 32760
// queries x 77 keys, 12 heads 52.3 / 49.2, 128 keys, 40 heads 140 / 130, 512 keys 295 / 287, 16384 x 2048 keys, 12 heads 159 / 157.5; lists of
// pairs 8064 x 12 168 / 156.  Over more keys the pair's store is a small part of it (7145 x 24 432 / 434, 12288 x 12 574 / 578), where each CTA
// has one pair its store is all that is left (1101 x 24 20.6 / 21.0, 1560 x 512 keys, 12 heads 13.3 / 13.8), and without turns the
// compiler's schedule of the main loop suffers (16384 x 8 761 / 889).
bool ksb_attn_dual_stores_in_bulk(const attn::Params& p) {
  constexpr int MOST_TILES = 16;
  return p.offsets || (p.nkv <= MOST_TILES && (int64_t)p.H * ((p.nq + 1) / 2) > sm_count());
}

// Launches the two-block kernel.  Returns KSB_ERR_UNSUPPORTED (without an error text) when the build cannot run it, so that
// the caller falls back to the one-block kernel.
int ksb_attn_launch_dual(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const attn::Params& p, int dtype,
                         bool chained, cudaStream_t st) {
  namespace d = attn::dual;
  const bool turns = d::takes_turns(p.H, p.nq, p.nkv, sm_count());
#define KSB_LAUNCH_AS(T, LISTS, TURNS, BULK) d::launch_as<T, LISTS, TURNS, BULK>(tq, tk, tv, to, p, chained, st)
#define KSB_LAUNCH_DUAL(T)                                                                                     \
  (p.offsets ? (p.bulk_out ? KSB_LAUNCH_AS(T, true, false, true) : KSB_LAUNCH_AS(T, true, false, false))      \
   : turns   ? (p.bulk_out ? KSB_LAUNCH_AS(T, false, true, true) : KSB_LAUNCH_AS(T, false, true, false))            \
             : KSB_LAUNCH_AS(T, false, false, false))
  return dtype == KSB_BF16 ? KSB_LAUNCH_DUAL(__nv_bfloat16) : KSB_LAUNCH_DUAL(__half);
#undef KSB_LAUNCH_DUAL
#undef KSB_LAUNCH_AS
}
