// FP8 (e4m3) GEMM with per-token x per-output-channel scales on the Blackwell tensor cores.
//
//   out[m,n] = epi( (sum_k A[m,k] * W[n,k])_f32 * sa[m] * sw[n] + bias[n] )
//
// Persistent, warp-specialised kernel, one CTA per SM, over the tiles of up to four problems that share K (gemm.h):
//   warp 0      TMA producer: tiles of A and W per stage, 128-byte swizzle, STAGES-deep ring in shared memory, completion
//               on mbarriers
//   warp 1      MMA issuer: one thread issues tcgen05.mma (kind::f8f6f4) from shared-memory descriptors into a
//               tensor-memory accumulator; two accumulators alternate so the epilogue of tile i overlaps the main loop
//               of tile i+1
//   warps 2..17 epilogue: each takes 32 rows x 64 columns of a tile: tcgen05.ld, scales / bias / fused GELU-tanh or gated
//               residual, conversion to half, a piece of swizzled shared memory, one TMA store.  The residual arrives the
//               same way, in the piece its result overwrites, fetched one tile ahead.  (One thread per row with direct
//               16-byte accesses cost a cache tag per lane, 4096 cycles of the load/store unit per tile and operand:
//               more than a main loop of K = 1536.  65 520 x 1536 x 1536, gated: 248 -> 159 us; 65 520 x 8960 x 1536,
//               GELU: 1164 -> 810 us; 6889 x 9216 x 3072: 158 -> 145 us.)
//   warps 2..5  the scatter epilogue (fused Ulysses exchange) stages 128-byte row pieces in shared memory and sends each
//               with one bulk copy to the memory of the GPU that owns the head: NVLink carries 128-byte writes
// Tiles are visited in groups of `group_m` row-tiles (all column tiles of a group, row-tile fastest) so that
// CTAs running at the same time share operand tiles in L2.  The weight is streamed from HBM once per group,
// the group's activation rows stay in L2 while the group sweeps the columns: the host picks the group height so
// that those rows take about 32 MB (32 row-tiles at K = 5120, 16 at K = 13824).  Ragged M, N, K edges rely on TMA zero
// fill for loads and on clipped stores.
//
// Tensor-bound: 2*M*N*K flop per launch; minimal traffic M*K + N*K + 2*M*N bytes.
#include "../../include/ksana_b200.h"
#include "common.cuh"
#include "gemm.h"
#include "gemm_math.cuh"
#include "host_utils.h"

namespace ksb {
namespace gemm {

constexpr int BM = 128, BK = 128;  // BK in bytes == e4m3 elements
constexpr int BN = 256;            // columns per tile of the widest form (and of the scatter epilogue)
constexpr int UMMA_K = 32;
constexpr int A_BYTES = BM * BK;
constexpr int KERNEL_ID = 1;
// A piece: 32 rows x 64 columns of half = one epilogue warp's part of a tile, stored with one TMA instruction.
constexpr int PIECE_COLS = 64, PIECE_BYTES = 32 * PIECE_COLS * 2;
// Output staging of the scatter epilogue: one 128-byte row piece per epilogue thread, rows 144 bytes apart (the
// 16-byte skew keeps the 16-byte shared-memory stores of a quarter warp on distinct banks).
constexpr int SCATTER_COLS = 64, SCATTER_ROW_BYTES = SCATTER_COLS * 2 + 16, SCATTER_BYTES = 128 * SCATTER_ROW_BYTES;
// CTAS = 1: every CTA computes 128 x TN tiles on its own.  CTAS = 2: two CTAs of a cluster compute one 256 x TN tile
// with tcgen05.mma.cta_group::2 -- each holds its 128 rows of A and half of the rows of the W tile, so a stage of a
// 256-column tile is 32 KB instead of 48 KB per CTA (a third less operand traffic from L2 and into shared memory per
// flop).
// TN = 128, 192 and 224 are for launches whose 256-column tiles leave the last wave nearly empty (choose_form).
// SCATTER: four epilogue warps (one thread per accumulator row and all columns) and their bulk-copy staging.
template <int CTAS, int TN, bool SCATTER> struct Cfg {
  static constexpr int PARTS = (TN + PIECE_COLS - 1) / PIECE_COLS;  // of a row
  static constexpr bool NARROW = TN % PIECE_COLS != 0;  // the last part is half a piece
  static constexpr int EW = SCATTER ? 4 : 4 * PARTS;  // epilogue warps
  static constexpr int B_ROWS = TN / CTAS;
  static constexpr int B_BYTES = B_ROWS * BK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int OUT_BYTES = SCATTER ? SCATTER_BYTES : EW * PIECE_BYTES;
  static constexpr int STAGES = SCATTER ? (CTAS == 1 ? 4 : 6) : (CTAS == 1 ? 3 : (TN > 192 ? 5 : 6));
  static constexpr int THREADS = 64 + 32 * EW;
  static constexpr int ACC_COLS = TN > 128 ? 256 : 128;  // of tensor memory, per accumulator: what is allocated is a power of two
  static constexpr int TMEM_COLS = 2 * ACC_COLS;
  static constexpr int COLP_BYTES = TN * 10;  // sw, bias (fp32) and gate (half) per column
  static constexpr int NUM_BARS = 2 * STAGES + 4 + EW;
  static constexpr int BAR_BYTES = (NUM_BARS * 8 + 16 + 15) / 16 * 16;
  // [STAGES x (A | B)][output pieces / scatter staging][column parameters][barriers]; the window is 1024-byte aligned
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + OUT_BYTES + COLP_BYTES + BAR_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory");
};

// One problem of a launch, as the kernel reads it.
struct Group {
  CUtensorMap ta, tw, to, tr;  // A, W, output, residual
  CUtensorMap to_half, tr_half;  // the last two by half pieces, for tiles whose rows end in one
  int M, N, tiles_m, tiles_n, tile0;
  int epilogue;
  const float* sa;
  const float* sw;
  const void* bias;
  const void* gate;
  int64_t gate_stride;
  const int64_t* gate_index;
  int64_t gate_rows;
  int rows_per_gate;
  int gate_bcast;  // the gate is one row
  float* tile_sumsq;
  int sumsq_cols;  // tiles (with `fine`: pieces of 64 columns) that start below this column write their row sums of squares
  int fine;        // per 64 columns instead of per tile
};

struct Params {
  Group g[MAX_GROUPS];
  int n_groups, num_tiles, K;
  int group_m;  // row-tiles per rasterisation group
  int early_w;  // W may be fetched before the previous kernel has finished
  int* status;
  // KSB_EPI_SCATTER_HEADS (fused QKV projection + Ulysses exchange): the output row of local token m and
  // column n = which * C + head * 128 + d goes to peer head / heads_per_peer, into its [tokens_all, 3, heads_per_peer,
  // 128] buffer at token (rank * M + m); the sum of squares of every row of each 256-column tile is written to
  // tile_sumsq[tile_n][m] for the tiles of the Q and K thirds.
  void* peers[KSB_MAX_PEERS];
  int n_peers, rank, heads_per_peer, C;
};

__device__ __forceinline__ const Group& tile_coords(const Params& p, int tile, int& tm, int& tn) {
  int gi = 0;
  while (gi + 1 < p.n_groups && tile >= p.g[gi + 1].tile0) ++gi;
  const Group& g = p.g[gi];
  tile -= g.tile0;
  const int per_group = p.group_m * g.tiles_n;
  const int rg = tile / per_group;
  const int first_m = rg * p.group_m;
  const int rows = min(p.group_m, g.tiles_m - first_m);
  const int r = tile - rg * per_group;
  tm = first_m + r % rows;
  tn = r / rows;
  return g;
}

__device__ __forceinline__ void bulk_store_128(void* dst, uint32_t src_smem) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], 128;" ::"l"(dst), "r"(src_smem) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

template <typename T, int CTAS, int TN, bool SCATTER>
__global__ void __launch_bounds__(Cfg<CTAS, TN, SCATTER>::THREADS, 1) fp8_gemm_kernel(const __grid_constant__ Params p) {
  using C = Cfg<CTAS, TN, SCATTER>;
  constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES, EW = C::EW;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  uint8_t* gen = smem_raw;
  const uint32_t pieces = base + STAGES * STAGE_BYTES;
  uint8_t* colp_gen = gen + STAGES * STAGE_BYTES + C::OUT_BYTES;
  float* col_sw = reinterpret_cast<float*>(colp_gen);  // [TN] each
  float* col_bias = reinterpret_cast<float*>(colp_gen + TN * 4);
  T* col_gate = reinterpret_cast<T*>(colp_gen + TN * 8);
  const uint32_t bars = base + STAGES * STAGE_BYTES + C::OUT_BYTES + C::COLP_BYTES;
  const uint32_t full0 = bars, empty0 = full0 + 8 * STAGES, tfull0 = empty0 + 8 * STAGES, tempty0 = tfull0 + 16, resid0 = tempty0 + 16;
  const uint32_t tmem_slot = bars + C::NUM_BARS * 8;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(colp_gen + C::COLP_BYTES + C::NUM_BARS * 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A pair walks the 256-row tiles together; CTA `crank` of the pair owns rows crank * 128 .. + 127 of each.
  const uint32_t crank = CTAS == 2 ? cluster_ctarank() : 0u;
  const int worker = CTAS == 2 ? blockIdx.x >> 1 : blockIdx.x, workers = CTAS == 2 ? gridDim.x >> 1 : gridDim.x;
  const int num_tiles = p.num_tiles;
  const int num_k = (p.K + BK - 1) / BK;
  if ((base & 1023u) != 0) {  // uniform over the grid: the swizzled tiles need a 1024-byte aligned window
    if (threadIdx.x == 0) report_error(p.status, KSB_ERR_BAD_SMEM_ALIGNMENT, (KERNEL_ID << 16) | 99);
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);   // the producer's expect_tx arrival (of the even CTA in a pair) + the bytes of every load
      mbar_init(empty0 + 8 * s, 1);  // one commit (delivered to both CTAs of a pair)
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, EW * CTAS);  // one arrival per epilogue warp (of both CTAs, at the even CTA)
    }
    for (int r = 0; r < EW; ++r) mbar_init(resid0 + 8 * r, 1);  // residual piece of a warp
    fence_barrier_init();
  }
  if (warp == 1) {
    if (CTAS == 2) {
      tmem_alloc_pair(tmem_slot, C::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, C::TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();  // the partner's barriers exist before anything is signalled to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_gen;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      // both CTAs' loads of a stage are counted by the even CTA's barrier, whose MMA thread consumes them
      auto expect = [&](uint32_t s) {
        if (CTAS == 1) mbar_arrive_expect_tx(full0 + 8 * s, STAGE_BYTES);
        else if (crank == 0) mbar_arrive_expect_tx(full0 + 8 * s, 2 * STAGE_BYTES);
      };
      auto load = [&](const CUtensorMap* map, uint32_t dst, uint32_t s, int x, int y) {
        if (CTAS == 2) tma_load_2d_pair(dst, map, mapa_shared(full0 + 8 * s, 0), x, y);
        else tma_load_2d(dst, map, full0 + 8 * s, x, y);
      };
      uint32_t early = 0;  // stages whose W half is already on its way
      if (p.early_w && worker < num_tiles) {
        int tm, tn;
        const Group& g = tile_coords(p, worker, tm, tn);
        tma_prefetch_desc(&g.ta);
        for (; early < STAGES && early < static_cast<uint32_t>(num_k); ++early) {
          expect(early);
          load(&g.tw, base + early * STAGE_BYTES + A_BYTES, early, static_cast<int>(early) * BK, tn * TN + (int)crank * C::B_ROWS);
        }
      }
      pdl_wait();
      uint32_t it = 0;
      bool ok = true;
      for (int tile = worker; tile < num_tiles && ok; tile += workers) {
        int tm, tn;
        const Group& g = tile_coords(p, tile, tm, tn);
        for (int k = 0; k < num_k; ++k, ++it) {
          const uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
          const uint32_t sa = base + s * STAGE_BYTES;
          if (it >= early) {
            if (!mbar_wait(empty0 + 8 * s, ph ^ 1, p.status, (KERNEL_ID << 16) | 1)) { ok = false; break; }
            expect(s);
            load(&g.tw, sa + A_BYTES, s, k * BK, tn * TN + (int)crank * C::B_ROWS);
          }
          load(&g.ta, sa, s, k * BK, (tm * CTAS + (int)crank) * BM);
        }
        if (!SCATTER && ok && tile == worker && g.epilogue == KSB_EPI_GATE_RESIDUAL) {
          // The first tile's residual, behind all of its operands: asked for at the start, its 64 KB delay the second k-step by 1000
          // cycles.  (Later ones are fetched by the epilogue, one tile ahead.)
          for (int e = 0; e < EW; ++e) {
            const int row0 = (tm * CTAS + (int)crank) * BM + ((e + 2) & 3) * 32, col = tn * TN + (e >> 2) * PIECE_COLS;
            if (row0 >= g.M || col >= g.N) continue;
            const bool half = C::NARROW && (e >> 2) == C::PARTS - 1;
            mbar_arrive_expect_tx(resid0 + 8 * e, half ? PIECE_BYTES / 2 : PIECE_BYTES);
            tma_load_2d(pieces + static_cast<uint32_t>(e) * PIECE_BYTES, half ? &g.tr_half : &g.tr, resid0 + 8 * e, col, row0);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (in a pair: the even CTA's)
    if (lane == 0 && crank == 0) {
      constexpr uint32_t idesc = IDESC_F8_E4M3_F32(CTAS * BM, TN);
      uint32_t it = 0, tcount = 0;
      bool ok = true;
      for (int tile = worker; tile < num_tiles && ok; tile += workers, ++tcount) {
        const uint32_t acc = tcount & 1, aph = (tcount >> 1) & 1;
        if (!mbar_wait(tempty0 + 8 * acc, aph ^ 1, p.status, (KERNEL_ID << 16) | 2)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * C::ACC_COLS;
        for (int k = 0; k < num_k; ++k, ++it) {
          const uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
          if (!mbar_wait(full0 + 8 * s, ph, p.status, (KERNEL_ID << 16) | 3)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = base + s * STAGE_BYTES;
          const uint64_t da = make_kmajor_sw128_desc(sa), db = make_kmajor_sw128_desc(sa + A_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            if (CTAS == 2) mma_f8_ss_pair(d_tmem, da + 2 * kk, db + 2 * kk, idesc, (k | kk) != 0);
            else mma_f8_ss(d_tmem, da + 2 * kk, db + 2 * kk, idesc, (k | kk) != 0);
          }
          // frees the stage (in both CTAs) once these MMAs have read it
          if (CTAS == 2) mma_commit_pair(empty0 + 8 * s); else mma_commit(empty0 + 8 * s);
        }
        if (ok) {
          if (CTAS == 2) mma_commit_pair(tfull0 + 8 * acc); else mma_commit(tfull0 + 8 * acc);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2 .. 2 + EW - 1)
    if (!SCATTER && warp == 2 && lane < p.n_groups) {
      tma_prefetch_desc(&p.g[lane].to);
      if (p.g[lane].epilogue == KSB_EPI_GATE_RESIDUAL) tma_prefetch_desc(&p.g[lane].tr);
    }
    pdl_wait();
    pdl_release();
    const int q = warp & 3;  // tensor-memory lane quarter this warp may read
    const int ew = warp - 2;
    const int et = threadIdx.x - 64;
    constexpr int ET = EW * 32;  // epilogue threads
    uint32_t tcount = 0;
    bool failed = false;
    const uint32_t tempty_even = CTAS == 2 ? mapa_shared(tempty0, 0) : 0u;
    // this warp's piece of a tile (not SCATTER): columns col0 .. + 63 of its 32 rows
    const int part = ew >> 2, col0 = part * PIECE_COLS;
    const bool narrow = C::NARROW && part == C::PARTS - 1;  // half a piece: rows of 64 bytes, 64-byte swizzle
    const uint32_t my_piece = pieces + static_cast<uint32_t>(ew) * PIECE_BYTES, my_resid = resid0 + 8 * ew;
    uint8_t* piece_row = gen + STAGES * STAGE_BYTES + ew * PIECE_BYTES + lane * (narrow ? 64 : 128);
    const int swizzle = narrow ? (lane >> 1) & 3 : lane & 7;
    uint32_t resid_phase = 0;
    // What the epilogue needs from global memory is fetched one tile ahead: the columns' parameters and the row's scale
    // into registers, the residual into the pieces its results will overwrite.  Waiting for them in place cost two
    // thirds of a tile's time at K = 1536.
    int tm, tn, next_tm = 0, next_tn = 0;
    const Group* next_gp = nullptr;
    constexpr int CPT = TN > ET ? TN / ET : 1;  // columns per epilogue thread
    float c_sw[CPT], next_sa = 0.f;
    T c_bias[CPT], c_gate[CPT];
    const T zero = HalfOps<T>::from_f(0.f);
    auto fetch_columns = [&](int tile) {
      if (tile >= num_tiles) return;
      const Group& g = tile_coords(p, tile, next_tm, next_tn);
      next_gp = &g;
      if (CTAS == 2) next_tm = next_tm * 2 + (int)crank;  // this CTA's 128 rows of the 256-row tile
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        const int n = next_tn * TN + et + i * ET;
        const bool in = et + i * ET < TN && n < g.N;
        c_sw[i] = in ? g.sw[n] : 0.f;
        c_bias[i] = (in && g.bias) ? static_cast<const T*>(g.bias)[n] : zero;
        c_gate[i] = (in && g.gate_bcast) ? static_cast<const T*>(g.gate)[n] : zero;
      }
      const int row = next_tm * BM + q * 32 + lane;
      next_sa = row < g.M ? g.sa[row] : 0.f;
    };
    auto fetch_resid = [&](int tile) {
      if (SCATTER || tile >= num_tiles || lane != 0) return;
      const Group& g = *next_gp;
      if (g.epilogue != KSB_EPI_GATE_RESIDUAL) return;
      const int row0 = next_tm * BM + q * 32;
      const int col = next_tn * TN + col0;
      if (row0 >= g.M || col >= g.N) return;
      bulk_wait_source_read<0>();  // the piece has been stored
      mbar_arrive_expect_tx(my_resid, narrow ? PIECE_BYTES / 2 : PIECE_BYTES);
      tma_load_2d(my_piece, narrow ? &g.tr_half : &g.tr, my_resid, col, row0);
    };
    fetch_columns(worker);
    for (int tile = worker; tile < num_tiles; tile += workers, ++tcount) {
      tm = next_tm; tn = next_tn;
      const Group& g = *next_gp;
      const uint32_t acc = tcount & 1, aph = (tcount >> 1) & 1;
      // All epilogue warps leave together if any of their waits ran out (a warp must never be
      // left alone at the named barrier below); the same barrier protects the reuse of the column parameters.
      failed = named_bar_or(1, ET, failed);
      if (failed) break;
      // stage the per-column parameters of this tile
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        const int c = et + i * ET;
        if (c < TN) {
          col_sw[c] = c_sw[i];
          col_bias[c] = HalfOps<T>::to_f(c_bias[i]);
          if (g.gate_bcast) col_gate[c] = c_gate[i];
        }
      }
      const int row0 = tm * BM + q * 32, row = row0 + lane;
      const bool row_ok = row < g.M;
      const float sa = next_sa;
      asm volatile("bar.sync 1, %0;" ::"n"(ET) : "memory");
      fetch_columns(tile + workers);
      // Uniform over the tile; with `fine`, over the warp: tiles of 192 columns do not end where the table does, only pieces of 64 do.
      const bool want_ssq = g.tile_sumsq != nullptr && tn * TN + (g.fine ? col0 : 0) < g.sumsq_cols;
      const bool gated = g.epilogue == KSB_EPI_GATE_RESIDUAL;
      const bool valid = row0 < g.M && tn * TN + col0 < g.N;  // uniform over the warp
      if (!SCATTER) {  // ahead of the accumulator, which takes longer: 400 - 570 cycles less behind it
        if (!gated || !valid) {  // a residual's load has waited for this already; there is none past the problem's edge
          if (lane == 0) bulk_wait_source_read<0>();  // the piece's last store has read it
          __syncwarp();
        } else {
          if (mbar_wait_warp(my_resid, resid_phase, p.status, (KERNEL_ID << 16) | 5)) resid_phase ^= 1; else failed = true;
        }
      }
      if (!mbar_wait_warp(tfull0 + 8 * acc, aph, p.status, (KERNEL_ID << 16) | 4)) {
        failed = true;
        if (!SCATTER && want_ssq && !g.fine) {  // warps whose wait succeeded meet this one at the two barriers of the partial sums
          asm volatile("bar.sync 1, %0;" ::"n"(ET) : "memory");
          asm volatile("bar.sync 1, %0;" ::"n"(ET) : "memory");
        }
        continue;
      }
      tc_fence_after();
      const uint32_t t_row = tmem_base + acc * C::ACC_COLS + (static_cast<uint32_t>(q * 32) << 16);
      float ssq = 0.f;
      // 8 columns of this thread's row (four pairs), before the epilogue's own arithmetic
      auto scaled8 = [&](const uint32_t* r, int col, float2 (&y)[4]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 sw = *reinterpret_cast<const float4*>(col_sw + col + 4 * h), bi = *reinterpret_cast<const float4*>(col_bias + col + 4 * h);
          const uint32_t* a = r + 4 * h;
          y[2 * h] = scale_pair(make_float2(__uint_as_float(a[0]), __uint_as_float(a[1])), sa, make_float2(sw.x, sw.y), make_float2(bi.x, bi.y));
          y[2 * h + 1] = scale_pair(make_float2(__uint_as_float(a[2]), __uint_as_float(a[3])), sa, make_float2(sw.z, sw.w), make_float2(bi.z, bi.w));
        }
      };
      auto pack8 = [&](const float2 (&y)[4]) {
        return make_uint4(HalfOps<T>::pack2(y[0]), HalfOps<T>::pack2(y[1]), HalfOps<T>::pack2(y[2]), HalfOps<T>::pack2(y[3]));
      };
      if constexpr (SCATTER) {
        uint8_t* stage_row = gen + STAGES * STAGE_BYTES + et * SCATTER_ROW_BYTES;
#pragma unroll 1
        for (int c0 = 0; c0 < TN; c0 += 32) {
          uint32_t r[32];
          tmem_ld32(t_row + c0, r);
          tmem_wait_ld();
          if (row_ok) {
            // the staged row piece is rewritten every 64 columns: wait until the previous bulk copy has read it
            if ((c0 & 32) == 0) bulk_wait_source_read<0>();
#pragma unroll
            for (int v8 = 0; v8 < 4; ++v8) {
              float2 y[4];
              scaled8(r + v8 * 8, c0 + v8 * 8, y);
              const uint4 o = pack8(y);
              *reinterpret_cast<uint4*>(stage_row + ((c0 & 32) + v8 * 8) * 2) = o;
              if (want_ssq) ssq += unit_squares<T>(o);
            }
            if ((c0 & 32) != 0) {
              // 64 columns staged: they never straddle a head (128 columns) or a Q / K / V third (C % 256 == 0)
              const int n = tn * TN + c0 - 32;
              const int which = n / p.C, c = n - which * p.C;
              const int head = c >> 7, dest = head / p.heads_per_peer, hl = head - dest * p.heads_per_peer;
              T* dst = static_cast<T*>(p.peers[dest]) +
                       ((static_cast<int64_t>(p.rank) * g.M + row) * 3 + which) * (static_cast<int64_t>(p.heads_per_peer) * 128) + hl * 128 + (c & 127);
              fence_proxy_async_smem();
              bulk_store_128(dst, smem_u32(stage_row));
            }
          }
        }
        if (want_ssq && row_ok) g.tile_sumsq[static_cast<int64_t>(tn) * g.M + row] = ssq;
      } else {
        // the eight 16-byte units of the row, each through `f`(unit's pairs, its place in the piece, its first column)
        auto each8 = [&](auto&& f) {
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            if (hh == 1 && narrow) break;
            uint32_t r[32];
            tmem_ld32(t_row + col0 + hh * 32, r);
            tmem_wait_ld();
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int u = hh * 4 + v, col = col0 + u * 8;
              uint4* slot = reinterpret_cast<uint4*>(piece_row + ((u ^ swizzle) << 4));
              float2 y[4];
              scaled8(r + v * 8, col, y);
              f(y, slot, col);
              *slot = pack8(y);
            }
          }
        };
        if (g.epilogue == KSB_EPI_GELU_TANH) {
          each8([&](float2 (&y)[4], uint4*, int) { gelu8<T>(y); });
        } else if (gated) {
          const T* grow = nullptr;  // this row's own gate row
          if (!g.gate_bcast && row_ok)
            grow = static_cast<const T*>(g.gate) + (g.gate_index ? checked_row(g.gate_index[row], g.gate_rows) : static_cast<int64_t>(row / g.rows_per_gate)) * g.gate_stride + tn * TN;
          each8([&](float2 (&y)[4], uint4* slot, int col) {
            const uint4 rw = *slot;
            uint4 gw = make_uint4(0, 0, 0, 0);
            if (g.gate_bcast) gw = *reinterpret_cast<const uint4*>(col_gate + col);
            else if (grow && tn * TN + col < g.N) gw = *reinterpret_cast<const uint4*>(grow + col);
            const uint32_t r4[4] = {rw.x, rw.y, rw.z, rw.w}, g4[4] = {gw.x, gw.y, gw.z, gw.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = gate_pair<T>(y[i], HalfOps<T>::unpack2(g4[i]), HalfOps<T>::unpack2(r4[i]));
          });
        } else if (want_ssq) {
          float us[8];
          int un = 0;
          each8([&](float2 (&y)[4], uint4*, int) { us[un++] = unit_squares<T>(pack8(y)); });
          ssq = ((us[0] + us[1]) + (us[2] + us[3])) + ((us[4] + us[5]) + (us[6] + us[7]));
        } else {
          each8([](float2 (&)[4], uint4*, int) {});
        }
        // the accumulator is in registers or done with: hand it back before the store
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 2) mbar_arrive_cluster_relaxed(tempty_even + 8 * acc); else mbar_arrive(tempty0 + 8 * acc);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && valid) tma_store_2d(narrow ? &g.to_half : &g.to, my_piece, tn * TN + col0, row0);
        if (want_ssq && g.fine) {
          if (row_ok) g.tile_sumsq[static_cast<int64_t>((tn * TN + col0) / PIECE_COLS) * g.M + row] = ssq;
        } else if (want_ssq) {
          // uniform over the tile: the threads of a row add their parts, which pass through the column parameters' place
          float* parts = col_sw;  // [TN / 64 - 1][128]
          static_assert((TN / PIECE_COLS - 1) * 128 * 4 <= TN * 8, "partial sums");
          asm volatile("bar.sync 1, %0;" ::"n"(ET) : "memory");
          if (part != 0) parts[(part - 1) * 128 + q * 32 + lane] = ssq;
          asm volatile("bar.sync 1, %0;" ::"n"(ET) : "memory");
          if (part == 0 && row_ok) {
#pragma unroll
            for (int i = 0; i < TN / PIECE_COLS - 1; ++i) ssq += parts[i * 128 + q * 32 + lane];
            g.tile_sumsq[static_cast<int64_t>(tn) * g.M + row] = ssq;
          }
        }
      }
      if (SCATTER) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 2) mbar_arrive_cluster_relaxed(tempty_even + 8 * acc); else mbar_arrive(tempty0 + 8 * acc);
        }
      }
      if (!failed) fetch_resid(tile + workers);
    }
    if (!SCATTER && failed && lane == 0) mbar_wait(my_resid, resid_phase, p.status, (KERNEL_ID << 16) | 6);  // a residual on its way lands before the block leaves
    bulk_wait_all();  // no bulk copy of this thread may outlive the kernel's shared memory
  }

  // ------------------------------------------------------------------ common exit
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    if (CTAS == 2) tmem_dealloc_pair(tmem_base, C::TMEM_COLS); else tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

}  // namespace gemm
}  // namespace ksb

using namespace ksb;

// 0: every CTA on its own (cta_group::1); 1: CTA pairs (cta_group::2).
// The pair form is the default: same bits, 2 - 20 % less time at the 75 600-token shapes under the power cap.
static int g_pair_mode = 1;

extern "C" int ksb_gemm_pair_mode(int mode) {
  const int previous = g_pair_mode;
  if (mode == 0 || mode == 1) g_pair_mode = mode;
  return previous;
}

namespace ksb {
namespace gemm {

template <typename T, int CTAS, int TN, bool SCATTER>
static int launch_as(const Params& p, int grid, bool chained, cudaStream_t st) {
  using C = Cfg<CTAS, TN, SCATTER>;
  auto kernel = fp8_gemm_kernel<T, CTAS, TN, SCATTER>;
  static DeviceOnce smem_limit;
  if (int rc = smem_limit.raise_smem(reinterpret_cast<const void*>(kernel), C::SMEM_BYTES)) return rc;
  return launch_kernel("fp8 gemm", reinterpret_cast<const void*>(kernel), dim3((unsigned)grid), dim3(C::THREADS), C::SMEM_BYTES, st, CTAS, chained, p);
}

template <int CTAS, int TN, bool SCATTER>
static int launch_form(const Params& p, int dtype, bool chained, cudaStream_t st) {
  const int workers = CTAS == 2 ? sm_count() / 2 : sm_count();
  const int grid = CTAS * (p.num_tiles < workers ? p.num_tiles : workers);
  return dtype == KSB_BF16 ? launch_as<__nv_bfloat16, CTAS, TN, SCATTER>(p, grid, chained, st) : launch_as<__half, CTAS, TN, SCATTER>(p, grid, chained, st);
}

// Fills the launch parameters for tiles of (ctas * 128) x tn.
static int fill(Params& p, const Problem* pr, int count, int64_t K, int ctas, int tn, bool scatter) {
  p.n_groups = count;
  p.K = (int)K;
  p.num_tiles = 0;
  p.status = status_words();
  if (!p.status) return fail(KSB_ERR_CUDA, "status words unavailable");
  p.group_m = 64;
  while (p.group_m > 8 && (int64_t)p.group_m * BM * K > (32ll << 20)) p.group_m >>= 1;
  if (ctas == 2) p.group_m >>= 1;  // counted in 256-row tiles
  for (int i = 0; i < count; ++i) {
    const Problem& q = pr[i];
    Group& g = p.g[i];
    if (int rc = encode_tmap_2d(&g.ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q.a, (uint64_t)K, (uint64_t)q.M, (uint64_t)K, BK, BM)) return rc;
    if (int rc = encode_tmap_2d(&g.tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q.w, (uint64_t)K, (uint64_t)q.N, (uint64_t)K, BK, (uint32_t)(tn / ctas))) return rc;
    auto pieces = [&](CUtensorMap& whole, CUtensorMap& half, const void* x, int64_t ld) -> int {
      if (int rc = encode_tmap_2d(&whole, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, x, (uint64_t)q.N, (uint64_t)q.M, (uint64_t)ld * 2, PIECE_COLS, 32)) return rc;
      return tn % PIECE_COLS == 0 ? 0 : encode_tmap_2d(&half, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, x, (uint64_t)q.N, (uint64_t)q.M, (uint64_t)ld * 2, PIECE_COLS / 2, 32);
    };
    if (!scatter)
      if (int rc = pieces(g.to, g.to_half, q.out, q.ldo)) return rc;
    if (q.epilogue == KSB_EPI_GATE_RESIDUAL)
      if (int rc = pieces(g.tr, g.tr_half, q.resid, q.ldr)) return rc;
    g.M = (int)q.M; g.N = (int)q.N;
    g.tiles_m = (int)((q.M + ctas * BM - 1) / (ctas * BM)); g.tiles_n = (int)((q.N + tn - 1) / tn);
    g.tile0 = p.num_tiles;
    p.num_tiles += g.tiles_m * g.tiles_n;
    g.epilogue = q.epilogue;
    g.sa = q.sa; g.sw = q.sw; g.bias = q.bias;
    g.gate = q.gate; g.gate_stride = q.gate_stride; g.gate_index = q.gate_index; g.gate_rows = q.gate_rows; g.rows_per_gate = q.rows_per_gate > 0 ? q.rows_per_gate : 1;
    g.gate_bcast = q.gate && !q.gate_index && q.rows_per_gate == 0;
    g.tile_sumsq = q.tile_sumsq; g.sumsq_cols = q.sumsq_cols; g.fine = q.fine;
  }
  return 0;
}

static int64_t tile_count(const Problem* pr, int count, int tm, int tn) {
  int64_t n = 0;
  for (int i = 0; i < count; ++i) n += ((pr[i].M + tm - 1) / tm) * ((pr[i].N + tn - 1) / tn);
  return n;
}

int validate(const Problem& p, int64_t K, int dtype) {
  if (dtype != KSB_BF16 && dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  if (p.M <= 0 || p.N <= 0 || K <= 0 || p.M > INT32_MAX || p.N > INT32_MAX || K > INT32_MAX)
    return fail(KSB_ERR_INVALID, "bad shape M=%lld N=%lld K=%lld", (long long)p.M, (long long)p.N, (long long)K);
  if (K % 16 != 0 || p.N % 8 != 0) return fail(KSB_ERR_INVALID, "K must be a multiple of 16 and N of 8 (K=%lld N=%lld)", (long long)K, (long long)p.N);
  if ((!p.x && (!p.a || !p.sa)) || !p.w || !p.sw || !p.out) return fail(KSB_ERR_INVALID, "null pointer");
  if (p.ldo < p.N || p.ldo % 8 != 0 || !aligned16(p.out)) return fail(KSB_ERR_INVALID, "out must be 16-byte aligned with ldo >= N, ldo %% 8 == 0");
  if (p.epilogue < KSB_EPI_NONE || p.epilogue > KSB_EPI_GATE_RESIDUAL) return fail(KSB_ERR_INVALID, "unknown epilogue %d", p.epilogue);
  if (p.epilogue == KSB_EPI_GATE_RESIDUAL) {
    if (!p.resid || !p.gate) return fail(KSB_ERR_INVALID, "gate-residual epilogue needs resid and gate");
    if (p.ldr < p.N || p.ldr % 8 != 0 || !aligned16(p.resid) || !aligned16(p.gate) || p.gate_stride % 8 != 0) return fail(KSB_ERR_INVALID, "resid/gate alignment");
  }
  if (p.tile_sumsq && (p.sumsq_cols <= 0 || p.sumsq_cols > p.N || p.sumsq_cols % BN != 0))
    return fail(KSB_ERR_INVALID, "sumsq_cols must be a positive multiple of %d and <= N", BN);
  return 0;
}

// The form of a launch: 0 = split (its plan in sp), 128, 192, 224 or 256 = columns per tile of CTA pairs, -1 = CTAs on their own.
static int choose_form(const Problem* pr, int count, int64_t K, SplitPlan& sp) {
  if (g_pair_mode == 0 || sm_count() < 2) return -1;
  bool stats256 = false, stats = false;
  for (int i = 0; i < count; ++i) stats256 = stats256 || (pr[i].tile_sumsq != nullptr && !pr[i].fine), stats = stats || pr[i].tile_sumsq != nullptr;
  // Estimated time in microseconds = waves x main loop of a tile + what a launch and its last epilogue cost (6).
  // A k-step (128 of K) takes a CTA pair 0.36 at 256 columns (tensor-bound) and 0.28 at 128, so narrow tiles pay only where
  // they save more than a third of the waves.
  const double num_k = (double)((K + BK - 1) / BK);
  const int pairs = sm_count() / 2;
  // Rows of one tile only stream the weight, and these forms do that at 3 - 4.5 TB/s (their pairs wait for each other's loads), the
  // split form at 5 - 6: 1 x 36864 x 3072 38.0 us against 22.2, 16 rows 32.5 / 23.0, 128 rows 29.4 / 29.1; 1 x 36864 x 5120
  // 63.6 / 33.9; 1 x 18432 x 15360 73.7 / 49.3; 128 x 18432 x 8960 39.9 / 37.0.
  double stream_us = 0;
  int64_t most = 0;
  for (int i = 0; i < count; ++i) {
    stream_us += (double)pr[i].N * (double)K / 4.2e6;
    most = pr[i].M > most ? pr[i].M : most;
  }
  auto tiles_us = [&](int tn, double step) {
    const double t = (double)((tile_count(pr, count, 2 * BM, tn) + pairs - 1) / pairs) * num_k * step + 6.0;
    return most <= BM && t < stream_us ? stream_us : t;
  };
  const double t256 = tiles_us(256, 0.36), t128 = tiles_us(128, 0.28);
  sp = plan_split(pr, count, K, stats256);
  const int form = (!stats256 && t128 < 0.97 * t256) ? 128 : 256;
  if (sp.us > 0.f && sp.us < 0.97 * (form == 128 ? t128 : t256)) return 0;
  // Launches of a few waves: tiles of 224 or 192 columns (112 and 96 rows of W per CTA; sums per 64 columns need the latter), where
  // the same or one more wave of shorter k-steps takes less.  A k-step of 256 / 224 / 192 columns takes 0.285 / 0.252 / 0.246 us (the
  // last two bound by L2 -> shared memory), the rest of a launch 7.0 / 6.9 / 6.5.  us, 256 / 224 / 192 columns: 1560 x 1536 x 1536 gated
  // 10.5 / 9.9 / 9.5; 1560 x 1536 x 8960 gated 27.0 / 24.5 / 23.7; 1560 x 8960 x 1536, GELU 26.7 / 24.7 / 27.3; 1101 x 9216 x 3072 29.6 / 28.1 /
  // 32.1; 1101 x 3072 x 12288 gated 37.3 / 35.6 / 57.5.  Beyond four waves, where L2 has to carry all pairs at once, this no longer holds:
  // a little is left at five (4000 x 5120 x 5120 79.2 / 76.8 / 82.1), at ten they lose (7145 x 12288 x 3072, GELU 198 / 244 / 253).  With one
  // k-step a tile's output is what takes its time, and a wave more costs more than it gives (with the row quantiser, 256 / 192 columns:
  // 357 x 8960 x 128, GELU 10.4 / 12.3 in one wave and two, 1420 x 12288 x 128, GELU 23.5 / 27.0 in four and six).
  const int64_t waves = (tile_count(pr, count, 2 * BM, 256) + pairs - 1) / pairs;
  if (form == 256 && !stats256 && waves <= 4 && most > BM) {
    auto steps_us = [&](int tn, double step, double rest) {
      const int64_t w = (tile_count(pr, count, 2 * BM, tn) + pairs - 1) / pairs;
      return num_k < 2 && w > waves ? 1e9 : (double)w * num_k * step + rest;
    };
    const double wide = 0.98 * steps_us(256, 0.285, 7.0), t192 = steps_us(192, 0.246, 6.5), t224 = stats ? wide : steps_us(224, 0.252, 6.9);
    if (t192 < wide && t192 <= t224) return 192;
    if (t224 < wide) return 224;
  }
  return form;
}

bool launch_quantises(const Problem& p, int64_t K) {
  SplitPlan sp{};
  return choose_form(&p, 1, K, sp) == 0 && split_quantises(p, K, sp);
}

int run(const Problem* pr, int count, int64_t K, int dtype, bool chained, cudaStream_t st) {
  if (count < 1 || count > MAX_GROUPS) return fail(KSB_ERR_INVALID, "1..%d problems per launch", MAX_GROUPS);
  for (int i = 0; i < count; ++i)
    if (int rc = validate(pr[i], K, dtype)) return rc;
  SplitPlan sp{};
  const int form = choose_form(pr, count, K, sp);
  if (form == 0) return run_split(pr, count, K, dtype, chained, st, sp);
  Params p{};
  p.early_w = chained ? 1 : 0;
  if (int rc = fill(p, pr, count, K, form < 0 ? 1 : 2, form < 0 ? BN : form, false)) return rc;
  switch (form) {
    case -1: return launch_form<1, BN, false>(p, dtype, chained, st);
    case 128: return launch_form<2, 128, false>(p, dtype, chained, st);
    case 192: return launch_form<2, 192, false>(p, dtype, chained, st);
    case 224: return launch_form<2, 224, false>(p, dtype, chained, st);
    default: return launch_form<2, BN, false>(p, dtype, chained, st);
  }
}

}  // namespace gemm
}  // namespace ksb

extern "C" int ksb_gemm_form(int count, const int64_t* M, const int64_t* N, int64_t K, int sums) {
  if (count < 1 || count > gemm::MAX_GROUPS || !M || !N || K <= 0 || (sums != 0 && sums != 64 && sums != 256)) return fail(KSB_ERR_INVALID, "bad launch");
  gemm::Problem pr[gemm::MAX_GROUPS]{};
  float table = 0.f;
  for (int i = 0; i < count; ++i) {
    if (M[i] <= 0 || N[i] <= 0) return fail(KSB_ERR_INVALID, "bad shape M=%lld N=%lld", (long long)M[i], (long long)N[i]);
    pr[i].M = M[i]; pr[i].N = N[i]; pr[i].tile_sumsq = sums ? &table : nullptr; pr[i].fine = sums == 64;
  }
  gemm::SplitPlan sp{};
  const int form = gemm::choose_form(pr, count, K, sp);
  return form < 0 ? 1 : form;
}

extern "C" int ksb_fp8_gemm_qkv_scatter(const void* a, const float* a_scale, const void* w, const float* w_scale,
                                        const void* bias, int64_t M, int64_t C, int64_t K, int dtype, void* const* peer_out,
                                        int n_peers, int rank, int64_t heads, float* tile_sumsq, ksb_stream_t stream) {
  if (dtype != KSB_BF16 && dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  if (M <= 0 || C <= 0 || K <= 0 || M > INT32_MAX / 4 || C > INT32_MAX / 4 || K > INT32_MAX) return fail(KSB_ERR_INVALID, "bad shape");
  if (K % 16 != 0 || C % 256 != 0 || heads * 128 != C) return fail(KSB_ERR_INVALID, "need K %% 16 == 0, C %% 256 == 0 and C == heads * 128");
  if (n_peers < 1 || n_peers > KSB_MAX_PEERS || rank < 0 || rank >= n_peers || heads % n_peers != 0)
    return fail(KSB_ERR_INVALID, "n_peers must be 1..%d, rank inside it, heads divisible by it", KSB_MAX_PEERS);
  if (!a || !a_scale || !w || !w_scale || !peer_out || !tile_sumsq) return fail(KSB_ERR_INVALID, "null pointer");
  gemm::Params p{};
  for (int i = 0; i < n_peers; ++i) {
    if (!peer_out[i] || !aligned16(peer_out[i])) return fail(KSB_ERR_INVALID, "peer buffer %d null or unaligned", i);
    p.peers[i] = peer_out[i];
  }
  p.n_peers = n_peers; p.rank = rank; p.heads_per_peer = (int)(heads / n_peers); p.C = (int)C;
  gemm::Problem q{};
  q.a = a; q.sa = a_scale; q.w = w; q.sw = w_scale; q.bias = bias; q.M = M; q.N = 3 * C; q.epilogue = KSB_EPI_SCATTER_HEADS;
  q.tile_sumsq = tile_sumsq; q.sumsq_cols = (int)(2 * C);
  const bool pair = g_pair_mode == 1 && sm_count() >= 2;
  if (int rc = gemm::fill(p, &q, 1, K, pair ? 2 : 1, gemm::BN, true)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return pair ? gemm::launch_form<2, gemm::BN, true>(p, dtype, false, st) : gemm::launch_form<1, gemm::BN, true>(p, dtype, false, st);
}

extern "C" int ksb_fp8_gemm(const void* a, const float* a_scale, const void* w, const float* w_scale,
                            const void* bias, int64_t M, int64_t N, int64_t K, void* out, int dtype, int64_t ldo,
                            int epilogue, const void* resid, int64_t ldr, const void* gate, int64_t gate_rows,
                            ksb_stream_t stream) {
  gemm::Problem q{};
  q.a = a; q.sa = a_scale; q.w = w; q.sw = w_scale; q.bias = bias; q.M = M > 0 ? M : 1; q.N = N; q.out = out; q.ldo = ldo; q.epilogue = epilogue;
  if (M == 0 && N > 0 && K > 0 && K % 16 == 0 && N % 8 == 0 && (dtype == KSB_BF16 || dtype == KSB_FP16)) return 0;
  if (M <= 0) return fail(KSB_ERR_INVALID, "bad shape M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
  if (epilogue == KSB_EPI_GATE_RESIDUAL) {
    q.resid = resid; q.ldr = ldr; q.gate = gate; q.gate_stride = N;
    if (gate && (gate_rows < 1 || gate_rows > M || M % gate_rows != 0)) return fail(KSB_ERR_INVALID, "gate_rows must divide M");
    q.rows_per_gate = gate_rows > 1 ? (int)(M / gate_rows) : 0;
  }
  return gemm::run(&q, 1, K, dtype, false, static_cast<cudaStream_t>(stream));
}

extern "C" int ksb_fp8_gemm_rowstats(const void* a, const float* a_scale, const void* w, const float* w_scale,
                                     const void* bias, int64_t M, int64_t N, int64_t K, void* out, int dtype, int64_t ldo,
                                     float* tile_sumsq, int64_t sumsq_cols, ksb_stream_t stream) {
  if (!tile_sumsq) return fail(KSB_ERR_INVALID, "null pointer");
  if (sumsq_cols > INT32_MAX) return fail(KSB_ERR_INVALID, "bad sumsq_cols");
  gemm::Problem q{};
  q.a = a; q.sa = a_scale; q.w = w; q.sw = w_scale; q.bias = bias; q.M = M; q.N = N; q.out = out; q.ldo = ldo; q.epilogue = KSB_EPI_NONE;
  q.tile_sumsq = tile_sumsq; q.sumsq_cols = (int)sumsq_cols;
  return gemm::run(&q, 1, K, dtype, false, static_cast<cudaStream_t>(stream));
}
