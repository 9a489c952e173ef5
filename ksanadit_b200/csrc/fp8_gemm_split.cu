// The FP8 GEMM for launches that whole 256-row tiles cannot spread over the GPU: a few rows (a modulation vector, a text
// prompt) or few tiles with a long K.
//
// Every CTA computes one 128 x TN tile over its share of K and leaves; the `splits` CTAs of a cluster share a tile's K
// range and add their fp32 accumulators through distributed shared memory, in the order of K, so results do not depend on
// timing.  A splits only from K >= 2048 on (at least eight k-steps per CTA), so that short sums keep the order of the
// persistent kernel and give its bits.
//   warp 0      TMA producer; the A box has no more rows than the problem (rounded up to 8): at one row a k-step reads
//               16 KB of W and 1 KB of A, and the rest of the ring holds more stages
//   warp 1      MMA issuer (one thread), M128 x TN x K32, one accumulator
//   warps 4..7  accumulator -> shared memory (fp32 rows, over the drained ring)
//   all warps   sum of the shares, scales, bias, GELU / gated residual, row sums of squares, coalesced 16-byte stores:
//               a row's columns are spread over the lanes, so one valid row keeps 16 lanes busy instead of one
//
// A launch of a few rows quantises them itself (QUANT): the row quantiser's launch, and the wait for it, is then left out.
//
// What bounds it: at few rows the weight's way from HBM (1 x 18432 x 3072 with its quantiser: 12.5 us with a cold weight, 13.4 in
// two launches, 21.3 as one wave of 256-row tiles behind a quantiser), at a few hundred rows launch, ring fill and the operands' way
// into shared memory (512 x 1536 x 1536: 8.5 us, 12.8 before).
#include "../../include/ksana_b200.h"
#include "common.cuh"
#include "gemm.h"
#include "gemm_math.cuh"
#include "host_utils.h"

namespace ksb {
namespace gemm {
namespace split {

constexpr int BM = 128, BK = 128, UMMA_K = 32;
constexpr int THREADS = 256;
constexpr int KERNEL_ID = 4;
constexpr int MAX_STAGES = 16;
constexpr int BAR_BYTES = 2 * MAX_STAGES * 8 + 16 + 16;
constexpr int ACC_PAD = 4;  // floats between the rows of the shared accumulator copy: 16-byte row stores stay conflict free
template <int TN> constexpr int acc_bytes() { return BM * (TN + ACC_PAD) * 4; }
// The MMA reads 128 rows of A from a stage's base whatever the box height: the window extends this far past the ring.
constexpr int A_SPAN = BM * BK;

constexpr int QUANT_ROWS = 8;  // rows a launch can quantise itself: one 8-row group of the operand layout

struct Group {
  CUtensorMap ta, tw;
  int M, N, tiles_m, tiles_n, tile0;
  int epilogue;
  const float* sa;
  const float* sw;
  const void* bias;
  void* out;
  int64_t ldo;
  const void* resid;
  int64_t ldr;
  const void* gate;
  int64_t gate_stride;
  const int64_t* gate_index;
  int64_t gate_rows;
  int rows_per_gate;  // 0: one gate row
  float* tile_sumsq;
  int sumsq_cols;
  int wide_columns;  // sw and bias may be read 16 bytes at a time
};

struct Params {
  Group g[MAX_GROUPS];
  int n_groups, K;
  int splits, stages;
  int a_rows;  // rows of the A box
  int early_w;  // W may be fetched before the previous kernel has finished (QUANT: never)
  // QUANT: the rows as halves (gemm.h)
  const void* x;
  int64_t x_ld;
  int x_static;
  const float* x_scale;
  int* status;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// Up to QUANT_ROWS rows of halves to e4m3, with the rounding points of the row quantisers (bytes and scales are theirs): k-steps
// k0 .. k1 - 1 into the operand layout at `dst` (1024 bytes per k-step: 8 rows of 128 bytes, 16-byte units XORed with the row),
// one scale per row to `scales`.  All threads of the CTA; the largest value of a row is found by 8, 4, 2 or 1 warps, every CTA
// for itself (a row is a few KB out of L2, and the weight's first stages are on their way meanwhile).
template <typename T>
__device__ __forceinline__ void quantise_rows(const Params& p, int rows, int k0, int k1, uint8_t* dst, float* scales, float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* x = static_cast<const T*>(p.x);
  const int nvec = p.K >> 3;  // 8 halves
  if (!p.x_static) {
    const int wpr = rows <= 1 ? 8 : rows <= 2 ? 4 : rows <= 4 ? 2 : 1;
    const int r = warp / wpr;
    float m = 0.f;
    if (r < rows) {
      const uint4* row = reinterpret_cast<const uint4*>(x + r * p.x_ld);
#pragma unroll 4
      for (int i = (warp - r * wpr) * 32 + lane; i < nvec; i += wpr * 32) {
        const uint4 v = row[i];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = HalfOps<T>::unpack2(w[q]);
          m = fmax3(m, fabsf(f.x), fabsf(f.y));
        }
      }
    }
    m = warp_max(m);
    if (lane == 0) red[warp] = m;
    __syncthreads();
    if (threadIdx.x < rows) {
      float a = 0.f;
      for (int i = 0; i < wpr; ++i) a = fmaxf(a, red[threadIdx.x * wpr + i]);
      scales[threadIdx.x] = a > 0.f ? __fdiv_rn(a, 448.f) : 1.f;
    }
  } else if (threadIdx.x < rows) {
    scales[threadIdx.x] = p.x_scale ? *p.x_scale : 1.f;
  }
  __syncthreads();
  const bool clamp_only = p.x_static && !p.x_scale;
  const int units = (k1 - k0) * 8;  // 16 values each
  for (int i = threadIdx.x; i < units * rows; i += THREADS) {
    const int r = i / units, u = i - r * units;
    const int64_t k = static_cast<int64_t>(k0) * BK + u * 16;
    uint32_t o[4] = {0, 0, 0, 0};
    if (k < p.K) {
      const float inv = clamp_only ? 1.f : HalfOps<T>::to_f(HalfOps<T>::from_f(__frcp_rn(scales[r])));
      const uint4* src = reinterpret_cast<const uint4*>(x + r * p.x_ld + k);
      const uint4 a = src[0], b = src[1];
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 lo = HalfOps<T>::unpack2(w[2 * q]), hi = HalfOps<T>::unpack2(w[2 * q + 1]);
        lo = HalfOps<T>::unpack2(HalfOps<T>::pack2(make_float2(__fmul_rn(lo.x, inv), __fmul_rn(lo.y, inv))));
        hi = HalfOps<T>::unpack2(HalfOps<T>::pack2(make_float2(__fmul_rn(hi.x, inv), __fmul_rn(hi.y, inv))));
        o[q] = cvt_e4m3x4(lo.x, lo.y, hi.x, hi.y);
      }
    }
    *reinterpret_cast<uint4*>(dst + (u >> 3) * 1024 + r * 128 + (((u & 7) ^ r) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  fence_proxy_async_smem();
}

template <typename T, int TN, int KB, bool QUANT>  // KB: k-steps per stage; QUANT: A is quantised here
__global__ void __launch_bounds__(THREADS, 2) fp8_gemm_split_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // [barriers, row scales: one 1024-byte block][QUANT: A][ring], A and ring later the accumulator copy
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t acc = base + 1024;
  float* acc_gen = reinterpret_cast<float*>(smem_raw + 1024);
  const uint32_t full0 = base, empty0 = base + 8 * MAX_STAGES, done = base + 16 * MAX_STAGES, tmem_slot = done + 16;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_raw + 16 * MAX_STAGES + 16);
  float* row_scale = reinterpret_cast<float*>(smem_raw + 512);
  static_assert(BAR_BYTES <= 512, "barrier block");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = p.splits;
  const uint32_t rank = splits > 1 ? cluster_ctarank() : 0u;
  int tile = blockIdx.x / splits;
  int gi = 0;
  while (gi + 1 < p.n_groups && tile >= p.g[gi + 1].tile0) ++gi;
  const Group& g = p.g[gi];
  tile -= g.tile0;
  const int tn = tile / g.tiles_m, tm = tile - tn * g.tiles_m;
  const int num_k = (p.K + BK - 1) / BK;
  const int k0 = static_cast<int>(rank) * num_k / splits, k1 = (static_cast<int>(rank) + 1) * num_k / splits;
  const uint32_t ring = QUANT ? acc + 1024u * static_cast<uint32_t>(k1 - k0) : acc;
  const uint32_t a_bytes = QUANT ? 0u : static_cast<uint32_t>(p.a_rows) * BK, step_bytes = a_bytes + TN * BK, stage_bytes = KB * step_bytes;
  const uint32_t stages = static_cast<uint32_t>(p.stages);
  if ((base & 1023u) != 0) {  // uniform over the grid
    if (threadIdx.x == 0) report_error(p.status, KSB_ERR_BAD_SMEM_ALIGNMENT, (KERNEL_ID << 16) | 99);
    return;
  }
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_gen;

  int early = 0;  // W stages on their way before the producer's loop
  const int n = (k1 - k0 + KB - 1) / KB;
  // a stage holds KB k-steps, step i at i * step_bytes: A (unless QUANT), then W; the last stage may hold fewer
  auto expect = [&](uint32_t s, int k) { mbar_arrive_expect_tx(full0 + 8 * s, static_cast<uint32_t>(min(KB, k1 - k)) * step_bytes); };
  auto load = [&](const CUtensorMap* map, uint32_t dst, uint32_t s, int k, int y) {
    for (int i = 0; i < KB; ++i)
      if (i == 0 || k + i < k1) tma_load_2d(dst + i * step_bytes, map, full0 + 8 * s, (k + i) * BK, y);
  };
  if (QUANT) {
    // first kernel of its call: the one ahead is the caller's and may be writing the weight, so W waits for it as x does
    if (threadIdx.x == 0) tma_prefetch_desc(&g.tw);
    __syncwarp();
    pdl_wait();
  }
  if (threadIdx.x == 0 && (QUANT || p.early_w)) {
    for (; early < static_cast<int>(stages) && early < n; ++early) {
      expect(early, k0 + early * KB);
      load(&g.tw, ring + early * stage_bytes + a_bytes, early, k0 + early * KB, tn * TN);
    }
  }
  if (QUANT) {
    __syncwarp();
    quantise_rows<T>(p, g.M, k0, k1, smem_raw + 1024, row_scale, row_scale + QUANT_ROWS);
    __syncthreads();
  }
  if (warp == 0) {
    if (lane == 0) {
      if (!QUANT) tma_prefetch_desc(&g.ta);
      pdl_wait();
      uint32_t s = 0, ph = 1;
      for (int it = 0; it < n; ++it) {
        const uint32_t dst = ring + s * stage_bytes;
        const int k = k0 + it * KB;
        if (it >= early) {
          if (!mbar_wait(empty0 + 8 * s, ph, p.status, (KERNEL_ID << 16) | 1)) break;
          expect(s, k);
          load(&g.tw, dst + a_bytes, s, k, tn * TN);
        }
        if (!QUANT) load(&g.ta, dst, s, k, tm * BM);
        if (++s == stages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = IDESC_F8_E4M3_F32(BM, TN);
      uint32_t s = 0, ph = 0;
      bool ok = true;
      for (int k = k0; k < k1; k += KB) {
        if (!mbar_wait(full0 + 8 * s, ph, p.status, (KERNEL_ID << 16) | 2)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int i = 0; i < KB; ++i) {
          if (i == 0 || k + i < k1) {
            const uint32_t sa = ring + s * stage_bytes + i * step_bytes;
            const uint64_t da = make_kmajor_sw128_desc(QUANT ? acc + 1024u * static_cast<uint32_t>(k + i - k0) : sa), db = make_kmajor_sw128_desc(sa + a_bytes);
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk) mma_f8_ss(tmem, da + 2 * kk, db + 2 * kk, idesc, (k + i > k0) || kk != 0);
          }
        }
        mma_commit(empty0 + 8 * s);
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      if (ok) mma_commit(done);
    }
  }
  __syncwarp();
  pdl_wait();
  pdl_release();
  // The parameters of this thread's eight columns (the same for all of its rows) are asked for ahead of the accumulator: behind it, a few
  // rows' launch waited for them as long as the memory takes (1 x 18432 x 3072 13.0 -> 12.5 us, 1 x 9216 x 1536 7.0 -> 6.4).  With more
  // than 32 rows (KB = 1) they go to L1 only: held in registers they cost 24 per thread, and a CTA then finds room beside the kernel
  // ahead later (512 x 1008 x 13824 27.2 us in registers, 21.3 so; 145 x 4608 x 13824 36.6 / 34.5; 33 x 1536 x 1536 7.9 / 8.1).
  constexpr int LPR = TN / 8;  // lanes per row
  static_assert(THREADS % LPR == 0, "a thread keeps its columns from row to row");
  constexpr bool AHEAD = KB == 2;
  const int c0 = static_cast<int>(threadIdx.x) % LPR * 8;
  float sw8[8];
  uint32_t b4[4];
  auto read_columns = [&](int n) {
    const T* bias = static_cast<const T*>(g.bias);
#pragma unroll
    for (int i = 0; i < 4; ++i) b4[i] = 0;
    if (g.wide_columns) {
      *reinterpret_cast<float4*>(sw8) = *reinterpret_cast<const float4*>(g.sw + n);
      *reinterpret_cast<float4*>(sw8 + 4) = *reinterpret_cast<const float4*>(g.sw + n + 4);
      if (bias) *reinterpret_cast<uint4*>(b4) = *reinterpret_cast<const uint4*>(bias + n);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) sw8[i] = g.sw[n + i];
      if (bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i) b4[i] = HalfOps<T>::pack2(make_float2(HalfOps<T>::to_f(bias[n + 2 * i]), HalfOps<T>::to_f(bias[n + 2 * i + 1])));
      }
    }
  };
  if (tn * TN + c0 < g.N) {
    if (AHEAD) {
      read_columns(tn * TN + c0);
    } else {
      auto prefetch = [](const void* x) { asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<uintptr_t>(x) & ~static_cast<uintptr_t>(15))); };
      prefetch(g.sw + tn * TN + c0);
      if (g.bias) prefetch(static_cast<const T*>(g.bias) + tn * TN + c0);
    }
  }
  // Every thread waits for the accumulator: all loads have arrived and all MMAs have read the ring by then.
  const bool ok = mbar_wait_warp(done, 0, p.status, (KERNEL_ID << 16) | 3);
  tc_fence_after();
  const int rows = min(BM, g.M - tm * BM);
  __syncthreads();
  if (warp >= 4 && ok) {
    const int q = warp & 3;
    if (q * 32 < rows) {
      float* dst = acc_gen + (q * 32 + lane) * (TN + ACC_PAD);
#pragma unroll
      for (int c0 = 0; c0 < TN; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(q * 32) << 16) + c0, r);
        tmem_wait_ld();
        if (q * 32 + lane < rows) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(dst + c0 + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
        }
      }
    }
  }
  tc_fence_before();
  if (splits > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TN);
  }

  // ------------------------------------------------------------------ sum of the shares and epilogue, 8 columns per lane
  const int vecs = rows * LPR;
  const bool want_ssq = g.tile_sumsq != nullptr && tn * TN < g.sumsq_cols;
  const int stride = THREADS * splits;
  for (int v0 = static_cast<int>(rank) * THREADS; v0 < vecs; v0 += stride) {
    const int v = v0 + threadIdx.x;
    const int r = v / LPR, c = AHEAD ? c0 : (v - r * LPR) * 8;
    const int row = tm * BM + r, n = tn * TN + c;
    const bool live = v < vecs && n < g.N;
    float ssq = 0.f;
    if (live) {
      const uint32_t off = static_cast<uint32_t>(r * (TN + ACC_PAD) + c) * 4;
      float a[8];
      {
        const float4 lo = *reinterpret_cast<const float4*>(reinterpret_cast<const uint8_t*>(acc_gen) + off);
        const float4 hi = *reinterpret_cast<const float4*>(reinterpret_cast<const uint8_t*>(acc_gen) + off + 16);
        a[0] = lo.x; a[1] = lo.y; a[2] = lo.z; a[3] = lo.w; a[4] = hi.x; a[5] = hi.y; a[6] = hi.z; a[7] = hi.w;
      }
      if (splits > 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = 0.f;
        for (int sidx = 0; sidx < splits; ++sidx) {  // in the order of K
          const uint32_t src = mapa_shared(acc + off, static_cast<uint32_t>(sidx));
          const float4 lo = ld_cluster_f4(src), hi = ld_cluster_f4(src + 16);
          a[0] += lo.x; a[1] += lo.y; a[2] += lo.z; a[3] += lo.w; a[4] += hi.x; a[5] += hi.y; a[6] += hi.z; a[7] += hi.w;
        }
      }
      const float sa = QUANT ? row_scale[r] : g.sa[row];
      if (!AHEAD) read_columns(n);
      float2 y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        y[i] = scale_pair(make_float2(a[2 * i], a[2 * i + 1]), sa, make_float2(sw8[2 * i], sw8[2 * i + 1]), HalfOps<T>::unpack2(b4[i]));
      if (g.epilogue == KSB_EPI_GELU_TANH) {
        gelu8<T>(y);
      } else if (g.epilogue == KSB_EPI_GATE_RESIDUAL) {
        const int64_t grow = g.gate_index ? checked_row(g.gate_index[row], g.gate_rows) : (g.rows_per_gate ? static_cast<int64_t>(row / g.rows_per_gate) : 0);
        const uint4 rw = *reinterpret_cast<const uint4*>(static_cast<const T*>(g.resid) + static_cast<int64_t>(row) * g.ldr + n);
        const uint4 gw = *reinterpret_cast<const uint4*>(static_cast<const T*>(g.gate) + grow * g.gate_stride + n);
        const uint32_t r4[4] = {rw.x, rw.y, rw.z, rw.w}, g4[4] = {gw.x, gw.y, gw.z, gw.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = gate_pair<T>(y[i], HalfOps<T>::unpack2(g4[i]), HalfOps<T>::unpack2(r4[i]));
      }
      const uint4 o = make_uint4(HalfOps<T>::pack2(y[0]), HalfOps<T>::pack2(y[1]), HalfOps<T>::pack2(y[2]), HalfOps<T>::pack2(y[3]));
      if (ok) *reinterpret_cast<uint4*>(static_cast<T*>(g.out) + static_cast<int64_t>(row) * g.ldo + n) = o;
      ssq = unit_squares<T>(o);
    }
    if (want_ssq) {  // uniform over the CTA: the eight lanes of 64 columns are neighbours
#pragma unroll
      for (int s = 1; s < 8; s <<= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, s);
      if (live && (c & 63) == 0) g.tile_sumsq[static_cast<int64_t>(n >> 6) * g.M + row] = ssq;
    }
  }
  if (splits > 1) cluster_sync_all();  // no CTA leaves while another reads its share
}

static int smem_for(int tn, int ring_bytes) {
  const int ring = ring_bytes + A_SPAN, acc = BM * (tn + ACC_PAD) * 4;
  return 1024 + (ring > acc ? ring : acc);
}

}  // namespace split

static int a_box_rows(const Problem* pr, int count) {
  int64_t most = 0;
  for (int i = 0; i < count; ++i) most = pr[i].M > most ? pr[i].M : most;
  return most >= split::BM ? split::BM : (int)((most + 7) / 8 * 8);
}

// The (columns, splits) with the least estimated time, in microseconds, from the measured parts of a launch: a k-step takes
// 0.19 (up to 32 rows; two steps per stage), 0.26 (64 columns) or 0.30 (128 columns), 1.6 times that where two CTAs share an
// SM; a launch 4.4 - 6 besides, a cluster's exchange 0.8 + 0.35 (few rows) or
// 1.2 + 0.7 per CTA; the weight's way from HBM (6 TB/s) bounds it below.
// Splits start at K = 2048.  Clusters of four or more do not fill every SM one CTA each (a few SMs of a partition are left
// over: 36 clusters of four ran as two waves), so close to that they take the smaller shared-memory budget.
SplitPlan plan_split(const Problem* pr, int count, int64_t K, bool stats256) {
  SplitPlan best{0, 0, 0, 0.f};
  if (stats256) return best;
  const int sms = sm_count();
  const double num_k = (double)((K + split::BK - 1) / split::BK);
  const int a_rows = a_box_rows(pr, count);
  double w_bytes = 0;
  for (int i = 0; i < count; ++i) w_bytes += (double)pr[i].N * (double)K;
  for (int tn : {128, 64}) {
    int64_t tiles = 0;
    for (int i = 0; i < count; ++i) tiles += ((pr[i].M + 127) / 128) * ((pr[i].N + tn - 1) / tn);
    for (int s : {1, 2, 4, 8}) {
      if (s > 1 && (K < 2048 || num_k / s < 8)) break;
      const int64_t ctas = tiles * s;
      if (ctas > 2 * sms) break;
      const double step = a_rows <= 32 ? 0.19 : (tn == 64 ? 0.26 : 0.30), base = a_rows <= 32 ? 4.4 : (tn == 64 ? 5.5 : 6.2);
      double t = base + num_k / s * step * (ctas > sms ? 1.6 : 1.0) + (s == 1 ? 0.0 : a_rows <= 32 ? 0.8 + 0.35 * s : 1.2 + 0.7 * s);
      const double hbm = 4.0 + w_bytes / 6.0e6;
      if (t < hbm) t = hbm;
      if (best.us == 0.f || t < 0.97 * best.us) best = SplitPlan{tn, s, ctas > (s >= 4 ? sms - 28 : sms) ? 2 : 1, (float)t};
    }
  }
  return best;
}

// Shared memory of a launch: k-steps per stage, stages that fit, bytes of the ring (and of A, where the launch quantises it).
struct SplitLayout {
  int kb, stages, ring_bytes;
};
static SplitLayout split_layout(int a_rows, int64_t K, const SplitPlan& plan, bool quantises) {
  // Two k-steps per stage halve the hand-offs (a step of few rows takes 190 ns instead of 220), but leave half the stages:
  // with 128 rows that costs more than it gives (128 x 9472 x 16384: 45.7 us against 40.4).
  const int kb = a_rows <= 32 ? 2 : 1;
  const int num_k = (int)((K + split::BK - 1) / split::BK), own = (num_k + plan.splits - 1) / plan.splits;
  const int a_bytes = quantises ? own * 1024 : 0;
  const int stage_bytes = kb * ((quantises ? 0 : a_rows) + plan.bn) * split::BK;
  const int budget = plan.occupancy == 2 ? 113 * 1024 : 227 * 1024;
  int stages = (budget - 1024 - split::A_SPAN - a_bytes) / stage_bytes;
  const int need = (own + kb - 1) / kb;
  if (stages > need) stages = need;
  if (stages > split::MAX_STAGES) stages = split::MAX_STAGES;
  return SplitLayout{kb, stages, a_bytes + stages * stage_bytes};
}

// Rows that fit one operand group, room for all their k-steps beside four stages of W, and few enough values that every CTA can
// quantise them while the first stages arrive; over a large weight an SM's CTAs follow one another and each does it again.
// Quantiser and GEMM one after the other / in one launch, weights cold, us (M x N x K):
// up to 10240 values: 1 x 1536 x 1536 6.9 / 5.5, 6 x 1536 x 1536 7.1 / 6.7, 6 x 8960 x 1536 8.1 / 7.9, 3 x 3072 x 3072 8.3 / 7.7,
// 2 x 5120 x 5120 10.6 / 10.6, 1 x 1536 x 8960 9.3 / 8.4; beyond: 8 x 8960 x 1536 8.0 / 8.2, 3 x 5120 x 5120 10.7 / 11.2,
// 8 x 2048 x 2048 7.7 / 8.2 (4 x 3072 x 3072 8.3 / 7.9);
// weights above 48 MiB, up to 6144 values: 1 x 18432 x 3072 13.4 / 12.5, 2 x 18432 x 3072 13.3 / 13.2, 1 x 13824 x 5120 15.8 / 15.9;
// beyond: 3 x 18432 x 3072 13.5 / 13.7, 5 x 18432 x 3072 13.5 / 14.5, 1 x 5120 x 13824 17.4 / 19.1.
bool split_quantises(const Problem& p, int64_t K, const SplitPlan& plan) {
  const int64_t most = p.N * K > (int64_t)48 << 20 ? 6144 : 10240;
  if (p.M > split::QUANT_ROWS || p.M * K > most || plan.bn == 0) return false;
  const SplitLayout l = split_layout(a_box_rows(&p, 1), K, plan, true);
  const int num_k = (int)((K + split::BK - 1) / split::BK), need = ((num_k + plan.splits - 1) / plan.splits + l.kb - 1) / l.kb;
  return l.stages >= (need < 4 ? need : 4);
}

template <typename T, int TN, int KB, bool QUANT>
static int launch_split(const split::Params& p, int grid, int smem, bool chained, cudaStream_t st) {
  auto kernel = split::fp8_gemm_split_kernel<T, TN, KB, QUANT>;
  static DeviceOnce smem_limit;
  if (int rc = smem_limit.raise_smem(reinterpret_cast<const void*>(kernel), 232448)) return rc;
  return launch_kernel("fp8 gemm (split K)", reinterpret_cast<const void*>(kernel), dim3((unsigned)grid), dim3(split::THREADS), smem, st, p.splits, chained, p);
}

int run_split(const Problem* pr, int count, int64_t K, int dtype, bool chained, cudaStream_t st, const SplitPlan& plan) {
  split::Params p{};
  p.n_groups = count; p.K = (int)K; p.splits = plan.splits; p.early_w = chained ? 1 : 0;
  p.a_rows = a_box_rows(pr, count);
  p.status = status_words();
  if (!p.status) return fail(KSB_ERR_CUDA, "status words unavailable");
  const bool quantises = pr[0].x != nullptr;
  if (quantises && (count != 1 || !split_quantises(pr[0], K, plan))) return fail(KSB_ERR_INVALID, "these rows have to be quantised beforehand");
  p.x = pr[0].x; p.x_ld = pr[0].x_ld; p.x_static = pr[0].x_static; p.x_scale = pr[0].x_scale;
  const SplitLayout layout = split_layout(p.a_rows, K, plan, quantises);
  p.stages = layout.stages;
  int tiles = 0;
  for (int i = 0; i < count; ++i) {
    const Problem& q = pr[i];
    split::Group& g = p.g[i];
    if (!quantises)
      if (int rc = encode_tmap_2d(&g.ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q.a, (uint64_t)K, (uint64_t)q.M, (uint64_t)K, split::BK, (uint32_t)p.a_rows)) return rc;
    if (int rc = encode_tmap_2d(&g.tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q.w, (uint64_t)K, (uint64_t)q.N, (uint64_t)K, split::BK, (uint32_t)plan.bn)) return rc;
    g.M = (int)q.M; g.N = (int)q.N;
    g.tiles_m = (int)((q.M + split::BM - 1) / split::BM); g.tiles_n = (int)((q.N + plan.bn - 1) / plan.bn);
    g.tile0 = tiles;
    tiles += g.tiles_m * g.tiles_n;
    g.epilogue = q.epilogue; g.sa = q.sa; g.sw = q.sw; g.bias = q.bias; g.out = q.out; g.ldo = q.ldo; g.resid = q.resid; g.ldr = q.ldr;
    g.gate = q.gate; g.gate_stride = q.gate_stride; g.gate_index = q.gate_index; g.gate_rows = q.gate_rows; g.rows_per_gate = q.rows_per_gate;
    g.tile_sumsq = q.tile_sumsq; g.sumsq_cols = q.sumsq_cols;
    g.wide_columns = aligned16(q.sw) && aligned16(q.bias);
  }
  const int smem = split::smem_for(plan.bn, layout.ring_bytes), grid = tiles * plan.splits;
#define KSB_LAUNCH_SPLIT(TN, KB, QUANT) \
  (dtype == KSB_BF16 ? launch_split<__nv_bfloat16, TN, KB, QUANT>(p, grid, smem, chained, st) : launch_split<__half, TN, KB, QUANT>(p, grid, smem, chained, st))
  if (quantises) return plan.bn == 64 ? KSB_LAUNCH_SPLIT(64, 2, true) : KSB_LAUNCH_SPLIT(128, 2, true);
  if (plan.bn == 64) return layout.kb == 2 ? KSB_LAUNCH_SPLIT(64, 2, false) : KSB_LAUNCH_SPLIT(64, 1, false);
  return layout.kb == 2 ? KSB_LAUNCH_SPLIT(128, 2, false) : KSB_LAUNCH_SPLIT(128, 1, false);
#undef KSB_LAUNCH_SPLIT
}

}  // namespace gemm
}  // namespace ksb
