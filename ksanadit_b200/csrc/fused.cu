// Whole operators as one call: quantise + GEMM, the attention with its pre-pass, and the fused Wan and Qwen-Image blocks.
//
// A denoise step at image sizes is bound by the host when every kernel is its own call from Python (20 - 25 us each with
// argument conversion, allocation and launch, against 3 - 20 us on the GPU).  Here one call queues the kernels of an
// operator back to back (about 2 us each), every one as a programmatic dependent of the one before it, into a workspace
// the caller allocates once per call.
#include <algorithm>

#include "../../include/ksana_b200.h"
#include "attn.h"
#include "common.cuh"
#include "gemm.h"
#include "host_utils.h"
#include "prep.h"
#include "rowwise.h"

namespace ksb {
namespace fused {

// Hands out 256-byte aligned pieces of the workspace; with a null base it only adds up their sizes.
struct Arena {
  char* base;
  int64_t used = 0;
  explicit Arena(void* b) : base(static_cast<char*>(b)) {}
  template <typename T> T* take(int64_t n) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (n * static_cast<int64_t>(sizeof(T)) + 255) / 256 * 256;
    return p;
  }
};

typedef uint16_t half_t;  // bf16 or fp16 storage

#define KSB_TRY(expr) do { if (int rc_ = (expr)) return rc_; } while (0)

// ---------------------------------------------------------------------------------- pieces
static gemm::Problem problem(const ksb_linear& l, const void* xq, const float* sx, int64_t M, void* out, int64_t ldo) {
  gemm::Problem q{};
  q.a = xq; q.sa = sx; q.w = l.w; q.sw = l.w_scale; q.bias = l.bias; q.M = M; q.N = l.N; q.out = out; q.ldo = ldo;
  return q;
}
static void gated(gemm::Problem& q, const void* resid, int64_t ldr, const void* gate, int64_t gate_stride, int rows_per_gate, const int64_t* index = nullptr,
                  int64_t index_rows = 0) {
  q.epilogue = KSB_EPI_GATE_RESIDUAL;
  q.resid = resid; q.ldr = ldr; q.gate = gate; q.gate_stride = gate_stride; q.rows_per_gate = rows_per_gate; q.gate_index = index; q.gate_rows = index_rows;
}

static int quant_rows(const void* x, int64_t M, int64_t K, int64_t ldx, void* q, float* s, int dtype, cudaStream_t st) {
  rq::Params p{};
  p.segs = 1; p.seg[0].x = x; p.seg[0].rows = M; p.seg[0].ldx = ldx; p.K = K; p.q = static_cast<uint8_t*>(q); p.qscale = s;
  KSB_TRY(rq::validate(p, dtype));
  return rq::run(rq::PLAIN, p, dtype, true, st);
}

static prep::Operand operand(const void* x, int64_t L, int64_t H, int64_t ts, int64_t hs) {
  prep::Operand op{};
  op.x = x; op.L = (int)L; op.H = (int)H; op.ts = ts; op.hs = hs; op.split = INT32_MAX;
  return op;
}

// K mean and V maxima of up to six (K, V) pairs in one launch; the sums over the chunks are left to the quantisers
// unless so many of them would repeat the work.  A K with a norm is stored normalised on the way (where
// the attention's output goes later): 2 bytes per value against a second normalisation, of 10 instructions, in a quantiser that issue bounds.
struct KvStats {
  prep::Operand k, v;
  void* knorm = nullptr;  // room for the normalised K
  float* kpart;
  float* vpart;
  int chunks;
  float k_scale;  // mean = (sum over the chunks left) * k_scale
  int left;       // chunks the quantisers have to add up
};
static int stat_chunks(int64_t L, int64_t H) { return prep::plan_chunks(L, H, prep::MAX_STAT_CHUNKS); }
static int64_t stat_floats(int64_t L, int64_t H) { return stat_chunks(L, H) * H * prep::D; }

static int kv_stats(KvStats* s, int n, int dtype, cudaStream_t st) {
  prep::StatsJob j[prep::MAX_JOBS];
  for (int i = 0; i < n; ++i) {
    s[i].chunks = stat_chunks(s[i].k.L, s[i].k.H);
    for (int w = 0; w < 2; ++w) {
      prep::StatsJob& job = j[2 * i + w];
      job = prep::StatsJob{};
      job.op = w ? s[i].v : s[i].k; job.is_max = w; job.normed_out = w ? nullptr : s[i].knorm; job.part = w ? s[i].vpart : s[i].kpart; job.chunks = s[i].chunks;
    }
  }
  KSB_TRY(prep::run_stats(j, 2 * n, dtype, true, st));
  for (int i = 0; i < n; ++i) {
    if (s[i].knorm) s[i].k = operand(s[i].knorm, s[i].k.L, s[i].k.H, s[i].k.H * prep::D, prep::D);
    const int64_t HD = (int64_t)s[i].k.H * prep::D;
    s[i].k_scale = 1.0f / (float)s[i].k.L;
    s[i].left = s[i].chunks;
    // 64 tiles: a quantiser CTA adds up to a dozen chunks next to its 32 KB tile without being slowed down; many more
    // tiles would read the partial sums many times over
    if (s[i].chunks > 1 && s[i].k.L > 64 * 128) {
      KSB_TRY(prep::run_finish(s[i].kpart, s[i].chunks, HD, 1.f, false, s[i].kpart, true, st));
      KSB_TRY(prep::run_finish(s[i].vpart, s[i].chunks, HD, 1.f, true, s[i].vpart, true, st));
      s[i].left = 1;
    }
  }
  return 0;
}

// The INT8 / FP8 operands of one attention.
struct Operands {
  int8_t* q8;
  float* qs;
  int8_t* k8;
  float* ks;
  uint8_t* vt;
  float* vs;
};
static void take_q(Arena& a, Operands& o, int64_t H, int64_t Lq) {
  const int64_t p = prep::pad128(Lq);
  o.q8 = a.take<int8_t>(H * p * 128);
  o.qs = a.take<float>(H * (p / 128));
}
static void take_kv(Arena& a, Operands& o, int64_t H, int64_t Lk) {
  const int64_t p = prep::pad128(Lk);
  o.k8 = a.take<int8_t>(H * p * 128);
  o.ks = a.take<float>(H * (p / 64));
  o.vt = a.take<uint8_t>(H * p * 128);
  o.vs = a.take<float>(H * 128);
}
// The slots of sample b of a batch whose heads follow one another.
static prep::QuantJob q_job(const prep::Operand& q, const Operands& o, int64_t b, float premul) {
  const int64_t p = prep::pad128(q.L), h0 = b * q.H;
  prep::QuantJob j{};
  j.op = q; j.kind = prep::QUANT_Q; j.premul = premul; j.out = o.q8 + h0 * p * 128; j.scale = o.qs + h0 * (p / 128);
  return j;
}
static prep::QuantJob k_job(const KvStats& s, const Operands& o, int64_t b) {
  const int64_t p = prep::pad128(s.k.L), h0 = b * s.k.H;
  prep::QuantJob j{};
  j.op = s.k; j.kind = prep::QUANT_K; j.part = s.kpart; j.chunks = s.left; j.inv_l = s.k_scale;
  j.out = o.k8 + h0 * p * 128; j.scale = o.ks + h0 * (p / 64);
  return j;
}
static prep::QuantJob v_job(const KvStats& s, const Operands& o, int64_t b) {
  const int64_t p = prep::pad128(s.v.L), h0 = b * s.v.H;
  prep::QuantJob j{};
  j.op = s.v; j.kind = prep::QUANT_V; j.part = s.vpart; j.chunks = s.left;
  j.out = o.vt + h0 * p * 128; j.scale = o.vs + h0 * 128;
  return j;
}

static attn::Call attention(const Operands& o, int64_t H, int64_t Lq, int64_t Lk, void* out, int64_t out_ts, int64_t out_hs) {
  attn::Call c{};
  c.q8 = o.q8; c.qs = o.qs; c.k8 = o.k8; c.ks = o.ks; c.vt = o.vt; c.vs = o.vs; c.H = H; c.Lq = Lq; c.Lk = Lk;
  c.out = out; c.out_ts = out_ts; c.out_hs = out_hs;
  return c;
}
static void lists(attn::Call& c, const ksb_tile_lists* l) {
  if (!l) return;
  c.tile_offsets = l->offsets; c.tile_entries = l->entries; c.order = l->order; c.pair_lists = l->pairs != 0;
}

// ---------------------------------------------------------------------------------- attention
struct AttentionPlan {
  Operands o;
  float* kpart;
  float* vpart;
  int64_t part;  // floats per sample and statistic
  int64_t bytes;
};
static AttentionPlan plan_attention(void* ws, int64_t B, int64_t Lq, int64_t Lk, int64_t H) {
  Arena a(ws);
  AttentionPlan p;
  take_q(a, p.o, B * H, Lq);
  take_kv(a, p.o, B * H, Lk);
  p.part = stat_floats(Lk, H);
  p.kpart = a.take<float>(B * p.part);
  p.vpart = a.take<float>(B * p.part);
  p.bytes = a.used;
  return p;
}

// ---------------------------------------------------------------------------------- modulation of a Wan block
// em[r][i] = round(modulation[i] + e[r][i]) for the rows of e, and a row of ones (the gate of the cross-attention's output).
template <typename T, typename E>
__global__ void __launch_bounds__(256) modulation_kernel(const T* modulation, const E* e, T* em, T* ones, int64_t rows, int C) {
  pdl_wait();
  pdl_release();
  const int64_t n = rows * 6 * C;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n + C; i += (int64_t)gridDim.x * blockDim.x) {
    if (i < n) {
      float v;
      if constexpr (sizeof(E) == 4) v = e[i]; else v = HalfOps<E>::to_f(e[i]);
      em[i] = HalfOps<T>::from_f(HalfOps<T>::to_f(modulation[i % (6 * C)]) + v);
    } else {
      ones[i - n] = HalfOps<T>::from_f(1.f);
    }
  }
}
template <typename T> static int launch_modulation(const void* modulation, const void* e, int e_dtype, half_t* em, half_t* ones, int64_t rows, int C, cudaStream_t st) {
  const T* mod = static_cast<const T*>(modulation);
  T* out = reinterpret_cast<T*>(em);
  T* one = reinterpret_cast<T*>(ones);
  const int64_t blocks = (rows * 6 * C + C + 255) / 256, cap = 8 * (int64_t)sm_count();
  const void* fn = e_dtype == KSB_FP32 ? (const void*)modulation_kernel<T, float> : e_dtype == KSB_BF16 ? (const void*)modulation_kernel<T, __nv_bfloat16> : (const void*)modulation_kernel<T, __half>;
  return launch_kernel("modulation", fn, dim3((unsigned)std::min(blocks, cap)), dim3(256), 0, st, 1, true, mod, e, out, one, rows, C);
}

// ---------------------------------------------------------------------------------- Wan block
constexpr int64_t RSTD_TABLE_ROWS = 8192;  // from here on 1 / rms comes from a table (one more launch) instead of being summed per tile and head

struct WanPlan {
  half_t *em, *ones, *big, *attn;
  uint8_t *xq, *cq;
  float *sx, *cs, *ssq, *cssq, *rstd, *kpart, *vpart, *ckpart, *cvpart;
  half_t *ck, *cv, *ckn;
  Operands self;
  int64_t part, cpart, bytes;
};
static WanPlan plan_wan(void* ws, const ksb_wan_block& b, int64_t B, int64_t L, int64_t Lc, int64_t e_rows) {
  const int64_t C = b.dim, H = b.heads, F = b.ffn_up.N, M = B * L;
  Arena a(ws);
  WanPlan p;
  p.em = a.take<half_t>(B * e_rows * 6 * C);
  p.ones = a.take<half_t>(C);
  p.xq = a.take<uint8_t>(M * std::max(C, F));
  p.sx = a.take<float>(M);
  p.big = a.take<half_t>(M * std::max(3 * C, F));  // q | k | v; the cross-attention's q; the FFN's hidden rows
  p.attn = a.take<half_t>(M * C);
  p.ssq = a.take<float>(2 * C / 64 * M);
  p.rstd = a.take<float>(2 * M);
  take_q(a, p.self, B * H, L);
  take_kv(a, p.self, B * H, L);
  p.part = stat_floats(L, H);
  p.kpart = a.take<float>(B * p.part);
  p.vpart = a.take<float>(B * p.part);
  p.cq = a.take<uint8_t>(B * Lc * C);
  p.cs = a.take<float>(B * Lc);
  p.ck = a.take<half_t>(B * Lc * C);
  p.cv = a.take<half_t>(B * Lc * C);
  p.ckn = a.take<half_t>(B * Lc * C);  // K normalised
  p.cssq = a.take<float>(C / 64 * B * Lc);
  p.cpart = stat_floats(Lc, H);
  p.ckpart = a.take<float>(B * p.cpart);
  p.cvpart = a.take<float>(B * p.cpart);
  p.bytes = a.used;
  return p;
}
static Operands context_operands(void* ctx, int64_t B, int64_t H, int64_t Lc, int64_t* bytes) {
  Arena a(ctx);
  Operands o{};
  take_kv(a, o, B * H, Lc);
  if (bytes) *bytes = a.used;
  return o;
}

// The norm of an operand over all C channels of rows [row0, row0 + L) of a projection.
static prep::NormSpec row_norm(const float* w, const float* ssq, int64_t rows, int64_t row0, int64_t C, float eps, const float* rstd) {
  prep::NormSpec n{};
  n.w = w; n.eps = eps; n.c = (float)C;
  if (rstd) n.row_rstd = rstd + row0;
  else { n.ssq = ssq + row0; n.ssq_tiles = (int)(C / 64); n.ssq_stride = rows; }
  return n;
}

static int adaln_rows(const WanPlan& p, const ksb_wan_block& b, const void* x, const half_t* shift, const half_t* scale, int64_t B, int64_t L, int64_t e_rows, int dtype, cudaStream_t st) {
  const int64_t C = b.dim;
  for (int64_t b0 = 0; b0 < B; b0 += rq::MAX_SEGS) {  // one segment per sample
    rq::Params r{};
    r.segs = (int)std::min<int64_t>(rq::MAX_SEGS, B - b0);
    for (int i = 0; i < r.segs; ++i) {
      rq::Segment& g = r.seg[i];
      g.x = static_cast<const half_t*>(x) + (b0 + i) * L * C; g.rows = L; g.ldx = C;
      g.shift = shift + (b0 + i) * e_rows * 6 * C; g.scale = scale + (b0 + i) * e_rows * 6 * C; g.mod_stride = 6 * C; g.rows_per_mod = e_rows == 1 ? 0 : 1;
    }
    r.K = C; r.eps = b.eps; r.q = p.xq + b0 * L * C; r.qscale = p.sx + b0 * L;
    KSB_TRY(rq::validate(r, dtype));
    KSB_TRY(rq::run(rq::ADALN, r, dtype, true, st));
  }
  return 0;
}

static int run_wan(const ksb_wan_block& b, const ksb_wan_call& c, int first, int last, void* ws, cudaStream_t st) {
  const int dtype = c.dtype;
  const int64_t B = c.batch, L = c.tokens, Lc = c.text, C = b.dim, H = b.heads, F = b.ffn_up.N, M = B * L;
  const WanPlan p = plan_wan(ws, b, B, L, Lc, c.e_rows);
  const Operands ctx = context_operands(c.context_operands, B, H, Lc, nullptr);
  const bool fresh = c.compute_context != 0;
  Operands cross = p.self;  // Q goes to the self-attention's buffers
  cross.k8 = ctx.k8; cross.ks = ctx.ks; cross.vt = ctx.vt; cross.vs = ctx.vs;
  half_t* out = static_cast<half_t*>(c.out);
  auto step = [&](int s) { return first <= s && s <= last; };
  const int per_row = c.e_rows == 1 ? (B == 1 ? 0 : (int)L) : 1;  // rows of x per modulation row (0: one for all)
  prep::RopeGrid rg;
  KSB_TRY(prep::make_rope_grid(rg, c.rope_table, c.rope_len, c.rope_nf, c.rope_nh, c.grid_f, c.grid_h, c.grid_w, 0, 0));
  prep::RopeGrid none{};
  const float* rstd = M > RSTD_TABLE_ROWS ? p.rstd : nullptr;

  if (step(KSB_WAN_PRE)) {
    KSB_TRY(dtype == KSB_BF16 ? launch_modulation<__nv_bfloat16>(b.modulation, c.e, c.e_dtype, p.em, p.ones, B * c.e_rows, (int)C, st)
                              : launch_modulation<__half>(b.modulation, c.e, c.e_dtype, p.em, p.ones, B * c.e_rows, (int)C, st));
    if (fresh) KSB_TRY(quant_rows(c.context, B * Lc, C, C, p.cq, p.cs, dtype, st));
    KSB_TRY(adaln_rows(p, b, c.x, p.em, p.em + C, B, L, c.e_rows, dtype, st));
  }
  if (step(KSB_WAN_QKV)) {
    // the context's K and V ride along: on their own they would fill a tenth of the GPU
    gemm::Problem g[3];
    g[0] = problem(b.qkv, p.xq, p.sx, M, p.big, 3 * C);
    g[0].tile_sumsq = p.ssq; g[0].sumsq_cols = (int)(2 * C); g[0].fine = 1;
    if (fresh) {
      g[1] = problem(b.cross_k, p.cq, p.cs, B * Lc, p.ck, C);
      g[1].tile_sumsq = p.cssq; g[1].sumsq_cols = (int)C; g[1].fine = 1;
      g[2] = problem(b.cross_v, p.cq, p.cs, B * Lc, p.cv, C);
    }
    KSB_TRY(gemm::run(g, fresh ? 3 : 1, C, dtype, true, st));
  }
  if (step(KSB_WAN_SELF_PREP)) {
    if (rstd) KSB_TRY(prep::run_rstd(p.ssq, (int)(C / 64), 2, (int)M, (int)C, b.eps, p.rstd, true, st));
    for (int64_t s0 = 0; s0 < B; s0 += 2) {  // two samples per launch: self and context K and V of each
      const int n = (int)std::min<int64_t>(2, B - s0);
      KvStats kv[4];
      prep::QuantJob j[prep::MAX_JOBS];
      int m = 0, count = 0;
      for (int i = 0; i < n; ++i) {
        const int64_t s = s0 + i, row0 = s * L;
        const half_t* qkv = p.big + row0 * 3 * C;
        KvStats& self = kv[m++];
        self.k = operand(qkv + C, L, H, 3 * C, 128);
        self.k.normed = 1;
        self.k.ns[0] = row_norm(b.norm_k, p.ssq + (C / 64) * M, M, row0, C, b.eps, rstd ? rstd + M : nullptr);
        KSB_TRY(prep::finish_norm(self.k.ns[0], L, rg));
        self.v = operand(qkv + 2 * C, L, H, 3 * C, 128);
        self.knorm = p.attn + row0 * C;
        self.kpart = p.kpart + s * p.part; self.vpart = p.vpart + s * p.part;
        if (!fresh) continue;
        KvStats& text = kv[m++];
        text.k = operand(p.ck + s * Lc * C, Lc, H, C, 128);
        text.k.normed = 1;
        text.k.ns[0] = row_norm(b.cross_norm_k, p.cssq, B * Lc, s * Lc, C, b.eps, nullptr);
        KSB_TRY(prep::finish_norm(text.k.ns[0], Lc, none));
        text.v = operand(p.cv + s * Lc * C, Lc, H, C, 128);
        text.knorm = p.ckn + s * Lc * C;
        text.kpart = p.ckpart + s * p.cpart; text.vpart = p.cvpart + s * p.cpart;
      }
      KSB_TRY(kv_stats(kv, m, dtype, st));
      m = 0;
      for (int i = 0; i < n; ++i) {
        const int64_t s = s0 + i, row0 = s * L;
        prep::Operand q = operand(p.big + row0 * 3 * C, L, H, 3 * C, 128);
        q.normed = 1;
        q.ns[0] = row_norm(b.norm_q, p.ssq, M, row0, C, b.eps, rstd);
        KSB_TRY(prep::finish_norm(q.ns[0], L, rg));
        j[count++] = q_job(q, p.self, s, c.premul);
        j[count++] = k_job(kv[m], p.self, s);
        j[count++] = v_job(kv[m++], p.self, s);
        if (!fresh) continue;
        j[count++] = k_job(kv[m], ctx, s);
        j[count++] = v_job(kv[m++], ctx, s);
      }
      KSB_TRY(prep::run_quant(j, count, dtype, true, st));
    }
  }
  if (step(KSB_WAN_SELF_ATTN)) {
    attn::Call a = attention(p.self, B * H, L, L, p.attn, C, 128);
    a.heads_per_batch = H; a.out_bs = L * C;
    lists(a, c.lists);
    KSB_TRY(attn::run(a, dtype, true, st));
  }
  if (step(KSB_WAN_SELF_POST)) KSB_TRY(quant_rows(p.attn, M, C, C, p.xq, p.sx, dtype, st));
  if (step(KSB_WAN_O)) {
    gemm::Problem g = problem(b.o, p.xq, p.sx, M, out, C);
    gated(g, c.x, C, p.em + 2 * C, 6 * C, per_row, nullptr);
    KSB_TRY(gemm::run(&g, 1, C, dtype, true, st));
  }
  if (step(KSB_WAN_CROSS_PRE)) {
    if (b.norm3_w) {
      rq::Params r{};
      r.segs = 1; r.seg[0].x = out; r.seg[0].rows = M; r.seg[0].ldx = C; r.K = C; r.w = b.norm3_w; r.b = b.norm3_b; r.eps = b.eps; r.q = p.xq; r.qscale = p.sx;
      KSB_TRY(rq::validate(r, dtype));
      KSB_TRY(rq::run(rq::LN_AFFINE, r, dtype, true, st));
    } else {
      KSB_TRY(quant_rows(out, M, C, C, p.xq, p.sx, dtype, st));
    }
  }
  if (step(KSB_WAN_CROSS_Q)) {
    gemm::Problem g = problem(b.cross_q, p.xq, p.sx, M, p.big, C);
    g.tile_sumsq = p.ssq; g.sumsq_cols = (int)C; g.fine = 1;
    KSB_TRY(gemm::run(&g, 1, C, dtype, true, st));
  }
  if (step(KSB_WAN_CROSS_PREP)) {
    if (rstd) KSB_TRY(prep::run_rstd(p.ssq, (int)(C / 64), 1, (int)M, (int)C, b.eps, p.rstd, true, st));
    for (int64_t s0 = 0; s0 < B; s0 += prep::MAX_JOBS) {
      const int n = (int)std::min<int64_t>(prep::MAX_JOBS, B - s0);
      prep::QuantJob j[prep::MAX_JOBS];
      for (int i = 0; i < n; ++i) {
        const int64_t row0 = (s0 + i) * L;
        prep::Operand q = operand(p.big + row0 * C, L, H, C, 128);
        q.normed = 1;
        q.ns[0] = row_norm(b.cross_norm_q, p.ssq, M, row0, C, b.eps, rstd);
        KSB_TRY(prep::finish_norm(q.ns[0], L, none));
        j[i] = q_job(q, cross, s0 + i, c.premul);
      }
      KSB_TRY(prep::run_quant(j, n, dtype, true, st));
    }
  }
  if (step(KSB_WAN_CROSS_ATTN)) {
    attn::Call a = attention(cross, B * H, L, Lc, p.attn, C, 128);
    a.heads_per_batch = H; a.out_bs = L * C;
    KSB_TRY(attn::run(a, dtype, true, st));
  }
  if (step(KSB_WAN_CROSS_POST)) KSB_TRY(quant_rows(p.attn, M, C, C, p.xq, p.sx, dtype, st));
  if (step(KSB_WAN_CROSS_O)) {
    gemm::Problem g = problem(b.cross_o, p.xq, p.sx, M, out, C);
    gated(g, out, C, p.ones, 0, 0, nullptr);
    KSB_TRY(gemm::run(&g, 1, C, dtype, true, st));
  }
  if (step(KSB_WAN_FFN_PRE)) KSB_TRY(adaln_rows(p, b, out, p.em + 3 * C, p.em + 4 * C, B, L, c.e_rows, dtype, st));
  if (step(KSB_WAN_FFN_UP)) {
    gemm::Problem g = problem(b.ffn_up, p.xq, p.sx, M, p.big, F);
    g.epilogue = KSB_EPI_GELU_TANH;
    KSB_TRY(gemm::run(&g, 1, C, dtype, true, st));
  }
  if (step(KSB_WAN_FFN_MID)) KSB_TRY(quant_rows(p.big, M, F, F, p.xq, p.sx, dtype, st));
  if (step(KSB_WAN_FFN_DOWN)) {
    gemm::Problem g = problem(b.ffn_down, p.xq, p.sx, M, out, C);
    gated(g, out, C, p.em + 5 * C, 6 * C, per_row, nullptr);
    KSB_TRY(gemm::run(&g, 1, F, dtype, true, st));
  }
  return 0;
}

// ---------------------------------------------------------------------------------- Qwen-Image dual-stream block
// Both streams share every launch: their rows follow one another ([text; image]) in the activations, the row passes take
// one segment per stream, the GEMMs one problem per stream, the quantisers switch norm and rotation at the first image row.
struct QwenPlan {
  half_t *big, *attn;
  uint8_t* xq;
  float *sx, *kpart, *vpart;
  Operands o;
  int64_t bytes;
};
static QwenPlan plan_qwen(void* ws, const ksb_qwen_block& b, int64_t Lt, int64_t Li) {
  const int64_t C = b.dim, H = b.heads, F = b.img_up.N, M = Lt + Li;
  Arena a(ws);
  QwenPlan p;
  p.xq = a.take<uint8_t>(M * std::max(C, F));
  p.sx = a.take<float>(M);
  p.big = a.take<half_t>(M * std::max(3 * C, F));
  p.attn = a.take<half_t>(M * C);
  take_q(a, p.o, H, M);
  take_kv(a, p.o, H, M);
  p.kpart = a.take<float>(stat_floats(M, H));
  p.vpart = a.take<float>(stat_floats(M, H));
  p.bytes = a.used;
  return p;
}

static int run_qwen(const ksb_qwen_block& b, const ksb_qwen_call& c, int first, int last, void* ws, cudaStream_t st) {
  const int dtype = c.dtype;
  const int64_t Lt = c.text_tokens, Li = c.img_tokens, C = b.dim, H = b.heads, F = b.img_up.N, M = Lt + Li;
  const QwenPlan p = plan_qwen(ws, b, Lt, Li);
  half_t* out = static_cast<half_t*>(c.out);
  const half_t* mods = static_cast<const half_t*>(c.mods);  // [rows][image 6C | text 6C], 6C = two of (shift, scale, gate)
  auto step = [&](int s) { return first <= s && s <= last; };
  const void* in[2] = {c.txt, c.img};
  const int64_t rows[2] = {Lt, Li}, row0[2] = {0, Lt};
  // modulation vector `which` (0..5) of a stream; the image's may come from one row per token
  auto mod = [&](int stream, int which) { return mods + (stream == 0 ? 6 * C : 0) + which * C; };
  const int64_t* index[2] = {nullptr, c.mod_index};
  auto modulate = [&](const void* const (&x)[2], int which) -> int {
    rq::Params r{};
    r.segs = 2;
    for (int i = 0; i < 2; ++i) {
      rq::Segment& g = r.seg[i];
      g.x = x[i]; g.rows = rows[i]; g.ldx = C; g.shift = mod(i, which); g.scale = mod(i, which + 1); g.mod_stride = 12 * C; g.mod_index = index[i]; g.mod_rows = c.mod_rows;
    }
    r.K = C; r.eps = b.eps; r.round_product = 1; r.q = p.xq; r.qscale = p.sx;
    KSB_TRY(rq::validate(r, dtype));
    return rq::run(rq::ADALN, r, dtype, true, st);
  };
  // one problem per stream over the rows in xq (`K` wide); resid == nullptr: no gate
  auto project = [&](const ksb_linear& txt, const ksb_linear& img, int64_t K, half_t* dst, int64_t ldo, int epilogue, const void* const* resid, int which) -> int {
    gemm::Problem g[2];
    for (int i = 0; i < 2; ++i) {
      gemm::Problem& q = g[i];
      q = problem(i == 0 ? txt : img, p.xq + row0[i] * K, p.sx + row0[i], rows[i], dst + row0[i] * ldo, ldo);
      q.epilogue = epilogue;
      if (resid) gated(q, resid[i], C, mod(i, which), 12 * C, 0, index[i], c.mod_rows);
    }
    return gemm::run(g, 2, K, dtype, true, st);
  };
  const void* residual[2] = {out, out + Lt * C};

  if (step(KSB_QWEN_PRE)) KSB_TRY(modulate(in, 0));
  if (step(KSB_QWEN_QKV)) KSB_TRY(project(b.txt_qkv, b.img_qkv, C, p.big, 3 * C, KSB_EPI_NONE, nullptr, 0));
  if (step(KSB_QWEN_PREP)) {
    prep::RopeGrid rt, ri;
    KSB_TRY(prep::make_rope_grid(rt, c.txt_rope, c.txt_rope_len, c.rope_nf, c.rope_nh, c.txt_grid, 1, 1, 0, 1));
    KSB_TRY(prep::make_rope_grid(ri, c.img_rope, c.img_rope_len, c.rope_nf, c.rope_nh, c.img_f, c.img_h, c.img_w, 0, c.img_diag));
    auto normed = [&](int64_t col, const float* wt, const float* wi, prep::Operand& op) -> int {
      op = operand(p.big + col, M, H, 3 * C, 128);
      op.normed = 1;
      op.split = (int)Lt;
      const float* w[2] = {wt, wi};
      for (int i = 0; i < 2; ++i) {
        op.ns[i].w = w[i]; op.ns[i].per_head = 1; op.ns[i].eps = b.eps;
        KSB_TRY(prep::finish_norm(op.ns[i], rows[i], i == 0 ? rt : ri));
      }
      return 0;
    };
    KvStats kv{};
    prep::Operand q;
    KSB_TRY(normed(C, b.txt_norm_k, b.img_norm_k, kv.k));
    KSB_TRY(normed(0, b.txt_norm_q, b.img_norm_q, q));
    kv.v = operand(p.big + 2 * C, M, H, 3 * C, 128);
    kv.knorm = p.attn;
    kv.kpart = p.kpart; kv.vpart = p.vpart;
    KSB_TRY(kv_stats(&kv, 1, dtype, st));
    prep::QuantJob j[3] = {q_job(q, p.o, 0, c.premul), k_job(kv, p.o, 0), v_job(kv, p.o, 0)};
    KSB_TRY(prep::run_quant(j, 3, dtype, true, st));
  }
  if (step(KSB_QWEN_ATTN)) KSB_TRY(attn::run(attention(p.o, H, M, M, p.attn, C, 128), dtype, true, st));
  if (step(KSB_QWEN_POST)) KSB_TRY(quant_rows(p.attn, M, C, C, p.xq, p.sx, dtype, st));
  if (step(KSB_QWEN_OUT)) KSB_TRY(project(b.txt_out, b.img_out, C, out, C, KSB_EPI_NONE, in, 2));
  if (step(KSB_QWEN_MLP_PRE)) KSB_TRY(modulate(residual, 3));
  if (step(KSB_QWEN_MLP_UP)) KSB_TRY(project(b.txt_up, b.img_up, C, p.big, F, KSB_EPI_GELU_TANH, nullptr, 0));
  if (step(KSB_QWEN_MLP_MID)) KSB_TRY(quant_rows(p.big, M, F, F, p.xq, p.sx, dtype, st));
  if (step(KSB_QWEN_MLP_DOWN)) KSB_TRY(project(b.txt_down, b.img_down, F, out, C, KSB_EPI_NONE, residual, 5));
  return 0;
}

}  // namespace fused
}  // namespace ksb

using namespace ksb;

extern "C" {

int64_t ksb_linear_workspace(int64_t M, int64_t K) { return M > 0 && K > 0 ? rq::workspace_bytes(M, K) : 0; }

int ksb_linear_forward(const ksb_linear* lin, const void* x, int dtype, int64_t M, int64_t ldx, int static_input, const float* in_scale,
                       void* out, int epilogue, const void* resid, int64_t ldr, const void* gate, int64_t gate_rows, void* workspace,
                       ksb_stream_t stream) {
  if (M < 0) return fail(KSB_ERR_INVALID, "bad shape M=%lld", (long long)M);
  if (M == 0) return 0;
  if (!lin || !workspace) return fail(KSB_ERR_INVALID, "null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t K = lin->K;
  const int before = launch_count();
  void* q = workspace;
  float* s = reinterpret_cast<float*>(static_cast<char*>(workspace) + rq::scale_offset(M, K));
  rq::Params p{};
  p.segs = 1; p.seg[0].x = x; p.seg[0].rows = M; p.seg[0].ldx = ldx; p.K = K; p.q = static_cast<uint8_t*>(q); p.qscale = s; p.scale_input = in_scale;
  if (int rc = rq::validate(p, dtype)) return rc;
  gemm::Problem g = fused::problem(*lin, q, s, M, out, lin->N);
  g.epilogue = epilogue;
  if (epilogue == KSB_EPI_GATE_RESIDUAL) {
    if (gate && (gate_rows < 1 || gate_rows > M || M % gate_rows != 0)) return fail(KSB_ERR_INVALID, "gate_rows must divide M");
    fused::gated(g, resid, ldr, gate, lin->N, gate_rows > 1 ? (int)(M / gate_rows) : 0);
  }
  if (int rc = gemm::validate(g, K, dtype)) return rc;
  // A launch that quantises its rows reads them in every CTA, while others may be storing: `out` over `x` (or over the scale) takes two.
  const char *o0 = static_cast<const char*>(out), *o1 = o0 + M * lin->N * sizeof(fused::half_t);
  auto in_place = [&](const void* p, int64_t bytes) { return p && static_cast<const char*>(p) < o1 && static_cast<const char*>(p) + bytes > o0; };
  const bool apart = !in_place(x, ((M - 1) * ldx + K) * sizeof(fused::half_t)) && !(static_input && in_place(in_scale, sizeof(float)));
  if (apart && gemm::launch_quantises(g, K)) {
    g.x = x; g.x_ld = ldx; g.x_static = static_input; g.x_scale = static_input ? in_scale : nullptr;
  } else if (int rc = rq::run(static_input ? rq::STATIC : rq::PLAIN, p, dtype, true, st)) return rc;
  if (int rc = gemm::run(&g, 1, K, dtype, true, st)) return rc;
  return launch_count() - before;
}

int64_t ksb_sage_attention_workspace(int64_t B, int64_t Lq, int64_t Lk, int64_t H) {
  if (B <= 0 || Lq <= 0 || Lk <= 0 || H <= 0) return 0;
  return fused::plan_attention(nullptr, B, Lq, Lk, H).bytes;
}

int ksb_sage_attention(const void* q, const void* k, const void* v, int dtype, int64_t B, int64_t Lq, int64_t Lk, int64_t H,
                       const int64_t* strides, float premul, const ksb_tile_lists* lists, void* out, void* workspace, ksb_stream_t stream) {
  if (!strides || !workspace) return fail(KSB_ERR_INVALID, "null pointer");
  if (B <= 0) return fail(KSB_ERR_INVALID, "bad batch %lld", (long long)B);
  const int64_t *sq = strides, *sk = strides + 3, *sv = strides + 6, *so = strides + 9;  // batch, token, head
  if (int rc = prep::check_operand(q, dtype, Lq, H, 128, sq[1], sq[2])) return rc;
  if (int rc = prep::check_operand(k, dtype, Lk, H, 128, sk[1], sk[2])) return rc;
  if (int rc = prep::check_operand(v, dtype, Lk, H, 128, sv[1], sv[2])) return rc;
  if (B > 1 && (sq[0] | sk[0] | sv[0] | so[0]) % 8 != 0) return fail(KSB_ERR_INVALID, "batch strides must be multiples of 8 elements");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int before = launch_count();
  const fused::AttentionPlan p = fused::plan_attention(workspace, B, Lq, Lk, H);
  auto at = [](const void* x, int64_t off) { return static_cast<const void*>(static_cast<const fused::half_t*>(x) + off); };
  constexpr int GROUP = prep::MAX_JOBS / 3;
  for (int64_t b0 = 0; b0 < B; b0 += GROUP) {
    const int n = (int)std::min<int64_t>(GROUP, B - b0);
    fused::KvStats kv[GROUP];
    prep::QuantJob j[prep::MAX_JOBS];
    for (int i = 0; i < n; ++i) {
      const int64_t b = b0 + i;
      kv[i].k = fused::operand(at(k, b * sk[0]), Lk, H, sk[1], sk[2]);
      kv[i].v = fused::operand(at(v, b * sv[0]), Lk, H, sv[1], sv[2]);
      kv[i].kpart = p.kpart + b * p.part;
      kv[i].vpart = p.vpart + b * p.part;
    }
    if (int rc = fused::kv_stats(kv, n, dtype, st)) return rc;
    for (int i = 0; i < n; ++i) {
      const int64_t b = b0 + i;
      j[3 * i] = fused::q_job(fused::operand(at(q, b * sq[0]), Lq, H, sq[1], sq[2]), p.o, b, premul);
      j[3 * i + 1] = fused::k_job(kv[i], p.o, b);
      j[3 * i + 2] = fused::v_job(kv[i], p.o, b);
    }
    if (int rc = prep::run_quant(j, 3 * n, dtype, true, st)) return rc;
  }
  attn::Call c = fused::attention(p.o, B * H, Lq, Lk, out, so[1], so[2]);
  c.heads_per_batch = H; c.out_bs = B > 1 ? so[0] : 0;  // one sample's stride says nothing
  fused::lists(c, lists);
  if (int rc = attn::run(c, dtype, true, st)) return rc;
  return launch_count() - before;
}

int64_t ksb_wan_block_workspace(const ksb_wan_block* block, int64_t batch, int64_t tokens, int64_t text, int64_t e_rows) {
  if (!block || block->heads <= 0 || batch <= 0 || tokens <= 0 || text <= 0 || e_rows <= 0) return 0;
  return fused::plan_wan(nullptr, *block, batch, tokens, text, e_rows).bytes;
}
int64_t ksb_wan_context_bytes(const ksb_wan_block* block, int64_t batch, int64_t text) {
  if (!block || block->heads <= 0 || batch <= 0 || text <= 0) return 0;
  int64_t bytes = 0;
  fused::context_operands(nullptr, batch, block->heads, text, &bytes);
  return bytes;
}
int ksb_wan_block_forward(const ksb_wan_block* block, const ksb_wan_call* call, int first, int last, void* workspace, ksb_stream_t stream) {
  if (!block || !call || !workspace || !call->x || !call->e || !call->out || !call->context_operands || !block->modulation) return fail(KSB_ERR_INVALID, "null pointer");
  if (call->batch <= 0 || call->tokens <= 0 || call->text <= 0) return fail(KSB_ERR_INVALID, "bad shape");
  if (call->dtype != KSB_BF16 && call->dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  if (block->dim % 256 != 0 || block->dim != block->heads * 128) return fail(KSB_ERR_INVALID, "need dim %% 256 == 0 and dim == heads * 128");
  if (call->e_rows != 1 && call->e_rows != call->tokens) return fail(KSB_ERR_INVALID, "e_rows must be 1 or the token count");
  const int before = launch_count();
  if (int rc = fused::run_wan(*block, *call, first, last, workspace, static_cast<cudaStream_t>(stream))) return rc;
  return launch_count() - before;
}

int64_t ksb_qwen_block_workspace(const ksb_qwen_block* block, int64_t text_tokens, int64_t img_tokens) {
  if (!block || block->heads <= 0 || text_tokens < 0 || img_tokens < 0 || text_tokens + img_tokens == 0) return 0;
  return fused::plan_qwen(nullptr, *block, text_tokens, img_tokens).bytes;
}
int ksb_qwen_block_forward(const ksb_qwen_block* block, const ksb_qwen_call* call, int first, int last, void* workspace, ksb_stream_t stream) {
  if (!block || !call || !workspace || !call->img || !call->txt || !call->mods || !call->out) return fail(KSB_ERR_INVALID, "null pointer");
  if (call->text_tokens <= 0 || call->img_tokens <= 0) return fail(KSB_ERR_INVALID, "bad shape");
  if (call->dtype != KSB_BF16 && call->dtype != KSB_FP16) return fail(KSB_ERR_INVALID, "dtype must be KSB_BF16 or KSB_FP16");
  if (call->mod_rows < 1) return fail(KSB_ERR_INVALID, "bad mod_rows");
  if (block->dim % 128 != 0 || block->dim != block->heads * 128) return fail(KSB_ERR_INVALID, "need dim == heads * 128");
  const int before = launch_count();
  if (int rc = fused::run_qwen(*block, *call, first, last, workspace, static_cast<cudaStream_t>(stream))) return rc;
  return launch_count() - before;
}

}  // extern "C"
