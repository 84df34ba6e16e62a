// Exact (fp32) backward of the token-by-token recurrence, for fp32 activations and for head widths
// the chunked kernels do not cover.
//   o = S^T qs            ->  dqs = S do,            dS += qs do^T
//   S = S' + w e^T        ->  dw = dS e,  de = dS^T w
//   e = v - S'^T k        ->  dv = de,   dS' = dS - k de^T,  dk_read = -S' de
//   S' = diag(exp g) S_-  ->  dg = rowsum(dS' * S'),  dS_- = exp(g) dS'
// followed per token by the write-key / preconditioner / gate chain rule.
//
// Only two things are sequential in t: the state (forward) and its cotangent dS.  Neither needs the
// other, and both are independent per value column, so each is a column-sliced scan of its own
// (pkda_recurrent_kernel, pkda_recurrent_dscan_kernel) that leaves checkpoints every 32 tokens and
// the residuals e, de of every token.  With e and de known, S and dS of a 32-token block follow from
// its checkpoints elementwise, without any sum over rows, so all row sums and the chain rule run
// block-parallel (pkda_recurrent_grad_kernel; S' comes from the state before the token, which keeps the
// digits that S - w e^T loses under strong decay).  The preconditioner's cotangent, a diagonal scan
// backwards over the tokens, and the terms that depend on it close the pass.
// (One CTA per (sequence, head) that replayed and walked back every token with the whole state took
// 1655 us for 2 x 4 units of 512 tokens at D = 64, fp32, behind a 551 us forward; these take 88 us, behind 72.)
#include <type_traits>

#include "pkda_launch.h"
#include "pkda_recurrent.cuh"

namespace pkda {

struct RecBwdParams {
  Geo geo;
  const void *q, *k, *g;
  const float* g_atk;
  const void *beta_atk, *beta;
  const float *A_log, *dt_bias, *log_atk_scale, *A0;
  RecSaved s;
  const void* d_o;
  const float* dST;
  float* dSck;                 // dS behind the last token of every 32-token block [blocks][H][D][D]
  float *de, *lam, *dkp;       // [tokens][H][D]
  float *carry, *decay;        // per (block, head): lam leaving / entering the block [D], its total decay
  void *dq, *dk, *dv, *dg, *dbeta_atk, *dbeta;
  float* dg_atk;
  float *partA, *partB, *partC;  // per (block, head): [blocks][H], [blocks][H][D], [blocks][H]
  float *dS0, *dA0;
  ScanWarps warps;  // consumer and producer warps of a scan CTA
  int groups;       // CTAs per (sequence, head)
  float scale, ln_x, eps;
};

// ---------------------------------------------------------------- state cotangent, last token first
// The mirror image of the forward scan: same column slices, same producer / consumer split.
template <int D, typename T, bool kTwoAhead>
__global__ void __launch_bounds__(ScanLay<D, 1>::kProd + 32 * ScanLay<D, 1>::kMaxConsumers)
pkda_recurrent_dscan_kernel(const RecBwdParams p) {
  after_previous();
  using L = ScanLay<D, 1>;
  constexpr int TB = L::kTB, TPG = L::kTPG, RG = L::kRG, R = L::kR, RUNS = L::kR / L::kU, VEC = L::kVecs * D;
  extern __shared__ __align__(16) float stage[];  // [2][TB][5][D]: scale q, w, -k, exp(g), do
  const int H = p.geo.heads;
  const int unit = blockIdx.x / p.groups, cg = blockIdx.x - unit * p.groups;
  const int n = unit / H, h = unit - n * H;
  const SeqInfo sq = seq_info(p.geo, n);
  const int nblk = (sq.len + TB - 1) / TB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = p.warps.nw, nthreads = 32 * nw + L::kProd;
  const size_t tstep = (size_t)H * D;

  if (p.warps.idle(warp)) return;
  if (warp >= nw) {
    const int ptid = 32 * p.warps.producer(warp) + lane;
    const int grp = ptid / L::kProdPerGroup, c = ptid - grp * L::kProdPerGroup;
    const bool act = D >= 32 || c < D;
    // (running pointers, 32-bit offsets and no checks in a whole block, as in the forward)
    const int step = H * D;
    const size_t at = ((size_t)sq.bos * H + h) * D + (act ? c : 0) + (size_t)(nblk > 0 ? (nblk - 1) * TB + TPG * grp : 0) * step;
    const T *kp = static_cast<const T*>(p.k) + at, *qp = static_cast<const T*>(p.q) + at, *dop = static_cast<const T*>(p.d_o) + at;
    const float *alp = p.s.al + at, *wp = p.s.w + at;
    typename Raw<T>::type qr[TPG], kr[TPG], dr[TPG];
    float wr[TPG], ar[TPG];
    auto fetch_block = [&](int left, auto whole) {  // left: tokens from the block's first one on
      constexpr bool kWhole = decltype(whole)::value;
#pragma unroll
      for (int i = 0; i < TPG; ++i) {
        const bool ok = act && (kWhole || TPG * grp + i < left);
        qr[i] = ok ? Raw<T>::load(qp + i * step) : 0;
        wr[i] = ok ? wp[i * step] : 0.f;
        kr[i] = ok ? Raw<T>::load(kp + i * step) : 0;
        dr[i] = ok ? Raw<T>::load(dop + i * step) : 0;
        ar[i] = ok ? alp[i * step] : 1.f;  // a token past the end leaves dS as it is
      }
    };
    auto fetch = [&](int t0) {
      const int left = sq.len - t0;
      if (left >= TB) fetch_block(left, std::true_type{});
      else fetch_block(left, std::false_type{});
      kp -= TB * step;
      qp -= TB * step;
      dop -= TB * step;
      alp -= TB * step;
      wp -= TB * step;
    };
    if (nblk > 0) fetch((nblk - 1) * TB);
    for (int it = 0; it < nblk; ++it) {
      const int s = it & 1;
      float qc[TPG], wc[TPG], kc[TPG], ac[TPG], dc[TPG];
#pragma unroll
      for (int i = 0; i < TPG; ++i) { qc[i] = Raw<T>::value(qr[i]); wc[i] = wr[i]; kc[i] = Raw<T>::value(kr[i]); ac[i] = ar[i]; dc[i] = Raw<T>::value(dr[i]); }
      if (it + 1 < nblk) fetch((nblk - 2 - it) * TB);
      if (it >= 2) bar_sync_n(3 + s, nthreads);
      if (act) {
        float* row = stage + s * L::kStage + TPG * grp * VEC + c;
#pragma unroll
        for (int i = 0; i < TPG; ++i) {
          row[0] = qc[i] * p.scale;
          row[D] = wc[i];
          row[2 * D] = -kc[i];
          row[3 * D] = ac[i];
          row[4 * D] = dc[i];
          row += VEC;
        }
      }
      bar_arrive_n(1 + s, nthreads);
    }
    return;
  }

  const int rg = lane & (RG - 1);
  const int col0 = (cg * nw + warp) * L::kCols + lane / RG;
  const size_t sbase = (size_t)unit * D * D + col0;
  float2 S[R / 2];
#pragma unroll
  for (int b = 0; b < RUNS; ++b)
#pragma unroll
    for (int u = 0; u < L::kU; ++u) {
      const float x = p.dST ? p.dST[sbase + (size_t)(L::row(b, rg) + u) * D] : 0.f;
      float2& d = S[(b * L::kU + u) / 2];
      if (u & 1) d.y = x; else d.x = x;
    }
  auto store_state = [&](float* dst) {
#pragma unroll
    for (int b = 0; b < RUNS; ++b)
#pragma unroll
      for (int u = 0; u < L::kU; ++u) {
        const float2 d = S[(b * L::kU + u) / 2];
        dst[(size_t)(L::row(b, rg) + u) * D] = (u & 1) ? d.y : d.x;
      }
  };
  T* dv = static_cast<T*>(p.dv);
  const size_t tbase = ((size_t)sq.bos * H + h) * D + col0;
  struct Rows { float2 qs[R / 2], w[R / 2], nk[R / 2], al[R / 2]; float dot; };  // the vectors of a token, and its dO (kTwoAhead)
  Rows ahead[kTwoAhead ? 2 : 1];
  auto load_token = [&](Rows& x, uint32_t vec) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x.dot) : "r"(vec + 16 * D + 4 * col0));
    load_rows<L>(vec, rg, x.qs);
    load_rows<L>(vec + 4 * D, rg, x.w);
    load_rows<L>(vec + 8 * D, rg, x.nk);
    load_rows<L>(vec + 12 * D, rg, x.al);
  };
  if (kTwoAhead && nblk > 0) {
    bar_sync_n(1, nthreads);
    load_token(ahead[kTwoAhead], smem_u32(stage) + 4 * (TB - 1) * VEC);
    load_token(ahead[0], smem_u32(stage) + 4 * (TB - 2) * VEC);
  }
  for (int it = 0; it < nblk; ++it) {
    const int s = it & 1, blk = nblk - 1 - it, t0 = blk * TB;
    float keep[L::kSums];
    if (it == 0 || ((t0 + TB) & (kCkpt - 1)) == 0)
      store_state(p.dSck + ((ckpt_base(p.geo, n, sq.bos) + t0 / kCkpt) * H + h) * (size_t)(D * D) + col0);
    if (!kTwoAhead) bar_sync_n(1 + s, nthreads);
    const uint32_t st = smem_u32(stage + s * L::kStage);
    if constexpr (kTwoAhead) {
      const uint32_t nx = smem_u32(stage + (s ^ 1) * L::kStage);
#pragma unroll
      for (int t = TB - 1; t >= 0; --t) {
        Rows& x = ahead[t & 1];
        float2 a0 = make_float2(0.f, 0.f), a1 = a0;
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
          S[i] = __ffma2_rn(x.qs[i], make_float2(x.dot, x.dot), S[i]);
          if (i & 1) a1 = __ffma2_rn(x.w[i], S[i], a1);
          else a0 = __ffma2_rn(x.w[i], S[i], a0);
        }
        float de = (a0.x + a0.y) + (a1.x + a1.y);
#pragma unroll
        for (int o = RG / 2; o >= 1; o >>= 1) de += xor_lane(de, o);
        if (rg == t / L::kSums) keep[t % L::kSums] = de;
#pragma unroll
        for (int i = 0; i < R / 2; ++i)
          S[i] = __fmul2_rn(x.al[i], __ffma2_rn(x.nk[i], make_float2(de, de), S[i]));
        if (t == 1 && it + 1 < nblk) bar_sync_n(1 + (s ^ 1), nthreads);
        if (t >= 2) load_token(x, st + 4 * (t - 2) * VEC);
        else if (it + 1 < nblk) load_token(x, nx + 4 * (t - 2 + TB) * VEC);
      }
    } else {
    float2 qs[R / 2], w[R / 2];
    float dot;
    auto load_do = [&](int t) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(dot) : "r"(st + 4 * (t * VEC + 4 * D + col0))); };
    load_do(TB - 1);
    load_rows<L>(st + 4 * (TB - 1) * VEC, rg, qs);
    load_rows<L>(st + 4 * ((TB - 1) * VEC + D), rg, w);
#pragma unroll
    for (int t = TB - 1; t >= 0; --t) {
      const uint32_t vec = st + 4 * t * VEC;
      float2 a0 = make_float2(0.f, 0.f), a1 = a0;
#pragma unroll
      for (int i = 0; i < R / 2; ++i) {
        S[i] = __ffma2_rn(qs[i], make_float2(dot, dot), S[i]);
        if (i & 1) a1 = __ffma2_rn(w[i], S[i], a1);
        else a0 = __ffma2_rn(w[i], S[i], a0);
      }
      // the token's other vectors and the next token's first ones are asked for between the rounds of shuffles
      float2 nk[R / 2], al[R / 2];
      float de = (a0.x + a0.y) + (a1.x + a1.y);
      float r = xor_lane(de, RG / 2);
      load_rows<L>(vec + 8 * D, rg, nk);
      load_rows<L>(vec + 12 * D, rg, al);
      de += r;
      r = xor_lane(de, RG / 4);
      if (t > 0) {
        load_do(t - 1);
        load_rows<L>(vec - 4 * VEC, rg, qs);
        if (RG < 8) load_rows<L>(vec - 4 * VEC + 4 * D, rg, w);
      }
      de += r;
      if (RG == 8) {
        r = xor_lane(de, 1);
        if (t > 0) load_rows<L>(vec - 4 * VEC + 4 * D, rg, w);
        de += r;
      }
      if (rg == t / L::kSums) keep[t % L::kSums] = de;
#pragma unroll
      for (int i = 0; i < R / 2; ++i)
        S[i] = __fmul2_rn(al[i], __ffma2_rn(nk[i], make_float2(de, de), S[i]));
    }
    }
    if (it + 2 < nblk) bar_arrive_n(3 + s, nthreads);
#pragma unroll
    for (int i = 0; i < L::kSums; ++i) {
      const int t = t0 + rg * L::kSums + i;
      if (t < sq.len) {
        const size_t idx = tbase + (size_t)t * tstep;
        p.de[idx] = keep[i];
        dv[idx] = from_f<T>(keep[i]);
      }
    }
  }
  if (p.dS0) store_state(p.dS0 + sbase);
}

// ------------------------------------------------------------- row sums and chain rule, block-parallel
// One CTA owns 32 tokens of one (sequence, head): thread = row of the state x quarter of a 16-column
// group.  Tokens are taken 8 at a time, last first: the eight states of a sub-block are rebuilt from
// the checkpoint into registers (for the later sub-blocks by running over the earlier tokens without
// keeping them: one multiply and one multiply-add per element), then dS walks back over them.
template <int D> struct GradLay {
  static constexpr int kNS = D >= 16 ? 4 : 2;      // lanes that share a row
  static constexpr int kGC = 4 * kNS;              // columns of a group
  static constexpr int kNG = D / kGC;              // column groups
  static constexpr int kActive = D * kNS;
  static constexpr int kThreads = kActive < 32 ? 32 : kActive;
  static constexpr int kWarps = kThreads / 32;
  static constexpr int kSub = 8;                   // tokens of a sub-block
  static constexpr int kTPS = kSub / kNS;          // tokens whose chain rule a lane takes
  static constexpr int kFloats = kCkpt * D * 4 + 3 * kCkpt * D + kNG * kThreads * 4 + kCkpt * D + kWarps * kCkpt + 2 * kWarps + kCkpt;
};

// Sequence and first token of checkpoint block j; false where the axis has a hole (packed only).
__device__ __forceinline__ bool block_lookup(const Geo& g, long j, int& n, int& t0, SeqInfo& sq) {
  if (g.cu_seqlens) {
    int lo = 0, hi = g.n_seqs - 1;
    while (lo < hi) {  // last sequence that starts at or before j
      const int mid = (lo + hi + 1) >> 1;
      if (ckpt_base(g, mid, g.cu_seqlens[mid]) <= j) lo = mid; else hi = mid - 1;
    }
    n = lo;
  } else {
    n = (int)(j / ((g.seq_len + kCkpt - 1) / kCkpt));
  }
  sq = seq_info(g, n);
  t0 = (int)(j - ckpt_base(g, n, sq.bos)) * kCkpt;
  return t0 < sq.len;
}

template <int D, typename T>
__global__ void __launch_bounds__(GradLay<D>::kThreads)
pkda_recurrent_grad_kernel(const RecBwdParams p) {
  after_previous();
  using L = GradLay<D>;
  // The next column group's state and the chain rule's inputs are asked for ahead where the registers are there (up to 64 rows:
  // 32 checkpoint blocks of 4 heads x 64 33.6 -> 29 us).
  constexpr bool kAhead = D <= 64;
  constexpr int NS = L::kNS, NG = L::kNG, SUB = L::kSub, TPS = L::kTPS;
  extern __shared__ __align__(16) float sm[];
  float4* s_row = reinterpret_cast<float4*>(sm);  // [32][D]: exp(g), w, k, scale q
  float* s_e = sm + kCkpt * D * 4;                // [32][D]
  float* s_de = s_e + kCkpt * D;
  float* s_do = s_de + kCkpt * D;
  float4* s_dS = reinterpret_cast<float4*>(s_do + kCkpt * D);  // [NG][threads]
  float* s_u = reinterpret_cast<float*>(s_dS + NG * L::kThreads);  // [32][D]
  float* s_db = s_u + kCkpt * D;                  // [warps][32]
  float* s_red = s_db + L::kWarps * kCkpt;        // [2][warps]
  float* s_dec = s_red + 2 * L::kWarps;           // [32] exp(gP)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, H = p.geo.heads;
  const size_t slot = (size_t)blockIdx.x * H + h;
  const bool act = tid < L::kActive;   // (D = 8: the upper half warp shadows the lower one)
  const int r = (tid / NS) % D, sub = tid & (NS - 1);
  int n, t0;
  SeqInfo sq;
  if (!block_lookup(p.geo, blockIdx.x, n, t0, sq)) {
    if (tid < D) p.partB[slot * D + tid] = p.carry[slot * D + tid] = 0.f;
    if (tid == 0) { p.partA[slot] = 0.f; p.partC[slot] = 0.f; p.decay[slot] = 1.f; }
    return;
  }
  const int nt = min(kCkpt, sq.len - t0);
  const size_t tstep = (size_t)H * D;
  const size_t tbase = ((size_t)(sq.bos + t0) * H + h) * D;
#pragma unroll 4
  for (int i = tid; i < kCkpt * D; i += L::kThreads) {  // (28 loads in flight)
    const int t = i / D, c = i - t * D;
    const bool ok = t < nt;
    const size_t idx = tbase + (size_t)t * tstep + c;
    s_row[i] = ok ? make_float4(p.s.al[idx], p.s.w[idx], to_f(static_cast<const T*>(p.k)[idx]),
                                to_f(static_cast<const T*>(p.q)[idx]) * p.scale)
                  : make_float4(1.f, 0.f, 0.f, 0.f);
    s_e[i] = ok ? p.s.e[idx] : 0.f;
    s_de[i] = ok ? p.de[idx] : 0.f;
    s_do[i] = ok ? to_f(static_cast<const T*>(p.d_o)[idx]) : 0.f;
  }
  if (tid < kCkpt) s_dec[tid] = tid < nt ? expf(p.g_atk[(size_t)(sq.bos + t0 + tid) * H + h]) : 1.f;
  const float* S0 = p.s.S + slot * D * D + (size_t)r * D + 4 * sub;
  const float* dS1 = p.dSck + slot * D * D + (size_t)r * D + 4 * sub;
#pragma unroll
  for (int cg = 0; cg < NG; ++cg) s_dS[cg * L::kThreads + tid] = *reinterpret_cast<const float4*>(dS1 + cg * L::kGC);
  __syncthreads();

  const float ea = expf(p.A_log[h]), centre = p.log_atk_scale[h], bias = p.dt_bias[h * D + r];
  float accA = 0.f, accB = 0.f, accC = 0.f;
  float4 S4n = kAhead ? *reinterpret_cast<const float4*>(S0) : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int sb = (nt - 1) / SUB; sb >= 0; --sb) {
    // what the chain rule below needs of memory
    float An_n[TPS], bw_n[TPS], g_n[TPS];
    auto chain_inputs = [&](int i) {
      const int t = min(SUB * sb + TPS * sub + i, nt - 1);
      const size_t sidx = (size_t)(sq.bos + t0 + t) * H + h;
      An_n[i] = p.s.A[sidx * D + r];
      bw_n[i] = to_f(static_cast<const T*>(p.beta)[sidx]);
      g_n[i] = to_f(static_cast<const T*>(p.g)[sidx * D + r]);
    };
    if (kAhead) {
#pragma unroll
      for (int i = 0; i < TPS; ++i) chain_inputs(i);
    }
    float acc[4 * SUB];  // [token][dqs, dw, dk_read, dg]
#pragma unroll
    for (int i = 0; i < 4 * SUB; ++i) acc[i] = 0.f;
#pragma unroll 1
    for (int cg = 0; cg < NG; ++cg) {
      const float4 S4 = kAhead ? S4n : *reinterpret_cast<const float4*>(S0 + cg * L::kGC);
      if (kAhead) S4n = *reinterpret_cast<const float4*>(S0 + (cg + 1 < NG ? cg + 1 : 0) * L::kGC);
      float2 S[2] = {make_float2(S4.x, S4.y), make_float2(S4.z, S4.w)};
      const float* ec = s_e + cg * L::kGC + 4 * sub;
      const float* dec = s_de + cg * L::kGC + 4 * sub;
      const float* doc = s_do + cg * L::kGC + 4 * sub;
#pragma unroll 4
      for (int t = 0; t < SUB * sb; ++t) {
        const float2 aw = *reinterpret_cast<const float2*>(&s_row[t * D + r]);
        const float4 e = *reinterpret_cast<const float4*>(ec + t * D);
        const float2 a2 = make_float2(aw.x, aw.x), w2 = make_float2(aw.y, aw.y);
        S[0] = __ffma2_rn(w2, make_float2(e.x, e.y), __fmul2_rn(a2, S[0]));
        S[1] = __ffma2_rn(w2, make_float2(e.z, e.w), __fmul2_rn(a2, S[1]));
      }
      float2 St[SUB][2];
      const float2 Sin[2] = {S[0], S[1]};
#pragma unroll
      for (int t = 0; t < SUB; ++t) {
        const int tt = SUB * sb + t;
        const float2 aw = *reinterpret_cast<const float2*>(&s_row[tt * D + r]);
        const float4 e = *reinterpret_cast<const float4*>(ec + tt * D);
        const float2 a2 = make_float2(aw.x, aw.x), w2 = make_float2(aw.y, aw.y);
        St[t][0] = S[0] = __ffma2_rn(w2, make_float2(e.x, e.y), __fmul2_rn(a2, S[0]));
        St[t][1] = S[1] = __ffma2_rn(w2, make_float2(e.z, e.w), __fmul2_rn(a2, S[1]));
      }
      const float4 d4 = s_dS[cg * L::kThreads + tid];
      float2 dS[2] = {make_float2(d4.x, d4.y), make_float2(d4.z, d4.w)};
#pragma unroll
      for (int t = SUB - 1; t >= 0; --t) {
        const int tt = SUB * sb + t;
        const float4 rw = s_row[tt * D + r];
        const float4 e4 = *reinterpret_cast<const float4*>(ec + tt * D);
        const float4 de4 = *reinterpret_cast<const float4*>(dec + tt * D);
        const float4 do4 = *reinterpret_cast<const float4*>(doc + tt * D);
        const float2 e[2] = {make_float2(e4.x, e4.y), make_float2(e4.z, e4.w)};
        const float2 de[2] = {make_float2(de4.x, de4.y), make_float2(de4.z, de4.w)};
        const float2 dd[2] = {make_float2(do4.x, do4.y), make_float2(do4.z, do4.w)};
        float2 x = make_float2(0.f, 0.f), y = x, z = x, g = x;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          x = __ffma2_rn(St[t][i], dd[i], x);
          dS[i] = __ffma2_rn(make_float2(rw.w, rw.w), dd[i], dS[i]);
          y = __ffma2_rn(dS[i], e[i], y);
          const float2 Sp = __fmul2_rn(make_float2(rw.x, rw.x), t > 0 ? St[t > 0 ? t - 1 : 0][i] : Sin[i]);  // S'
          z = __ffma2_rn(Sp, de[i], z);
          dS[i] = __ffma2_rn(make_float2(-rw.z, -rw.z), de[i], dS[i]);
          g = __ffma2_rn(dS[i], Sp, g);
          dS[i] = __fmul2_rn(make_float2(rw.x, rw.x), dS[i]);
        }
        acc[4 * t] += x.x + x.y;
        acc[4 * t + 1] += y.x + y.y;
        acc[4 * t + 2] -= z.x + z.y;
        acc[4 * t + 3] += g.x + g.y;
      }
      s_dS[cg * L::kThreads + tid] = make_float4(dS[0].x, dS[0].y, dS[1].x, dS[1].y);
    }
    rg_sum_transposed<NS, 4 * SUB>(acc, sub);  // lane `sub`: tokens TPS * sub ..
    // ---- per-channel chain rule of the lane's tokens
#pragma unroll
    for (int i = 0; i < TPS; ++i) {
      const int t = SUB * sb + TPS * sub + i;
      const bool ok = t < nt;
      float x_db = 0.f;
      if (ok) {
        const size_t idx = ((size_t)(sq.bos + t0 + t) * H + h) * D + r;
        const float kc = s_row[t * D + r].z;
        if (!kAhead) chain_inputs(i);
        const float An = An_n[i], bw = bw_n[i];
        const float rawz = g_n[i] + bias;
        const float dev = logf(An + p.eps) - centre, den = 1.f + fabsf(dev);
        const float Bf = expf(-p.ln_x * dev / den);
        const float dw = acc[4 * i + 1], dgl = acc[4 * i + 3];
        x_db = dw * (kc * Bf);                // d beta = <dw, kt>
        const float dkt = bw * dw;
        const float ddev = -p.ln_x * dkt * kc * Bf / (den * den);
        const float gn = -ea * softplus_acc(rawz);
        const float dr = dgl * (-ea) / (1.f + expf(-rawz));
        accA += dgl * gn;
        accB += dr;
        accC -= ddev;
        if (act) {
          s_u[t * D + r] = ddev / (An + p.eps);
          p.dkp[idx] = acc[4 * i + 2] + dkt * Bf;
          static_cast<T*>(p.dq)[idx] = from_f<T>(acc[4 * i] * p.scale);
          static_cast<T*>(p.dg)[idx] = from_f<T>(dr);
        }
      }
      if (!act) x_db = 0.f;
#pragma unroll
      for (int o = 16; o >= NS; o >>= 1) x_db += __shfl_xor_sync(0xffffffffu, x_db, o);
      if (lane < NS) s_db[warp * kCkpt + SUB * sb + TPS * sub + i] = x_db;
    }
  }
  // ---- sums over the rows (d beta) and over the block (parameter gradients), in a fixed order
  if (!act) accA = accB = accC = 0.f;
#pragma unroll
  for (int o = NS / 2; o >= 1; o >>= 1) accB += __shfl_xor_sync(0xffffffffu, accB, o);
  if (act && sub == 0) p.partB[slot * D + r] = accB;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    accA += __shfl_xor_sync(0xffffffffu, accA, o);
    accC += __shfl_xor_sync(0xffffffffu, accC, o);
  }
  if (lane == 0) { s_red[warp] = accA; s_red[L::kWarps + warp] = accC; }
  __syncthreads();
  // the preconditioner's cotangent inside the block (lam behind its last token taken as zero):
  //   lam_t = exp(gP_{t+1}) lam_{t+1} + ddev_t / (A_t + eps)
  if (tid < D) {
    float lam = 0.f;
    for (int t = nt - 1; t >= 0; --t) {
      lam += s_u[t * D + tid];
      p.lam[tbase + (size_t)t * tstep + tid] = lam;
      lam *= s_dec[t];
    }
    p.carry[slot * D + tid] = lam;
  }
  if (tid == 0) {
    float d = 1.f;
    for (int t = 0; t < kCkpt; ++t) d *= s_dec[t];
    p.decay[slot] = d;
  }
  if (tid < nt) {
    float s = 0.f;
    for (int w = 0; w < L::kWarps; ++w) s += s_db[w * kCkpt + tid];
    static_cast<T*>(p.dbeta)[(size_t)(sq.bos + t0 + tid) * H + h] = from_f<T>(s);
  }
  if (tid < 2) {
    float s = 0.f;
    for (int w = 0; w < L::kWarps; ++w) s += s_red[tid * L::kWarps + w];
    (tid == 0 ? p.partA : p.partC)[slot] = s;
  }
}

// ------------------------------------------------- preconditioner cotangent across blocks, last first
// Replaces every block's outgoing lam by the one that enters it from behind.  One thread per channel.
template <int D>
__global__ void __launch_bounds__(D < 32 ? 32 : D) pkda_recurrent_carry_kernel(const RecBwdParams p) {
  after_previous();
  constexpr int kAhead = 8;
  const int H = p.geo.heads, unit = blockIdx.x, n = unit / H, h = unit - n * H, c = threadIdx.x;
  const SeqInfo sq = seq_info(p.geo, n);
  if (c >= D) return;
  const size_t slot0 = (size_t)ckpt_base(p.geo, n, sq.bos) * H + h;
  float lam = 0.f;
  for (int j1 = (sq.len + kCkpt - 1) / kCkpt; j1 > 0; j1 -= kAhead) {
    float out[kAhead], dec[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int j = j1 - 1 - i;
      const size_t slot = slot0 + (size_t)(j < 0 ? 0 : j) * H;
      out[i] = p.carry[slot * D + c];
      dec[i] = p.decay[slot];
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int j = j1 - 1 - i;
      if (j >= 0) {
        p.carry[(slot0 + (size_t)j * H) * D + c] = lam;
        lam = out[i] + dec[i] * lam;
      }
    }
  }
  if (p.dA0) p.dA0[(size_t)unit * D + c] = lam;
}

// ------------------------------------------------------------------ the terms that depend on lam
// One warp per token: dk, d beta_atk = <lam, k^2>, d g_atk = exp(gP) <lam, A before the token>.
template <int D, typename T>
__global__ void __launch_bounds__(256) pkda_recurrent_close_kernel(const RecBwdParams p) {
  after_previous();
  const int H = p.geo.heads, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int n, t0;
  SeqInfo sq;
  if (!block_lookup(p.geo, blockIdx.x, n, t0, sq)) return;
  const int nt = min(kCkpt, sq.len - t0);
  const size_t slot = (size_t)blockIdx.x * H + h;
  // decay from behind the block's end to each of its tokens: product of exp(gP) over the later tokens
  float suffix = __shfl_down_sync(0xffffffffu, lane < nt ? expf(p.g_atk[(size_t)(sq.bos + t0 + lane) * H + h]) : 1.f, 1);
  if (lane == 31) suffix = 1.f;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y = __shfl_down_sync(0xffffffffu, suffix, o);
    if (lane + o < 32) suffix *= y;
  }
  // a warp's four tokens: every load of all four is issued before the first is used
  constexpr int N = (D + 31) / 32;
  typename Raw<T>::type kr[4][N], br[4];
  float lm[4][N], ap[4][N], dp[4][N], cr[N];
#pragma unroll
  for (int j = 0; j < N; ++j) cr[j] = lane + 32 * j < D ? p.carry[slot * D + lane + 32 * j] : 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int tl = warp + 8 * u, t = t0 + tl;
    br[u] = 0;
    const size_t sidx = (size_t)(sq.bos + t) * H + h;
    if (tl < nt) br[u] = Raw<T>::load(static_cast<const T*>(p.beta_atk) + sidx);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int c = lane + 32 * j;
      const size_t idx = sidx * D + c;
      kr[u][j] = 0;
      lm[u][j] = ap[u][j] = dp[u][j] = 0.f;
      if (tl < nt && c < D) {
        kr[u][j] = Raw<T>::load(static_cast<const T*>(p.k) + idx);
        lm[u][j] = p.lam[idx];
        dp[u][j] = p.dkp[idx];
        if (t > 0) ap[u][j] = p.s.A[idx - (size_t)H * D];
        else if (p.A0) ap[u][j] = p.A0[((size_t)n * H + h) * D + c];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int tl = warp + 8 * u;
    if (tl >= nt) break;
    const float fade = __shfl_sync(0xffffffffu, suffix, tl);
    const size_t sidx = (size_t)(sq.bos + t0 + tl) * H + h;
    const float bp = Raw<T>::value(br[u]);
    float sb = 0.f, sg = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int c = lane + 32 * j;
      if (c < D) {
        const float kc = Raw<T>::value(kr[u][j]), lam = lm[u][j] + fade * cr[j];
        static_cast<T*>(p.dk)[sidx * D + c] = from_f<T>(dp[u][j] + 2.f * lam * bp * kc);
        sb += lam * kc * kc;
        sg += lam * ap[u][j];
      }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      sb += __shfl_xor_sync(0xffffffffu, sb, o);
      sg += __shfl_xor_sync(0xffffffffu, sg, o);
    }
    if (lane == 0) {
      static_cast<T*>(p.dbeta_atk)[sidx] = from_f<T>(sb);
      p.dg_atk[sidx] = sg * expf(p.g_atk[sidx]);
    }
  }
}

// Sums the per-block partials: grid (H), D channels x 256 / D slices of the block axis, fixed order.
__global__ void __launch_bounds__(256)
pkda_recurrent_bwd_reduce_kernel(int blocks, int H, int D, const float* partA, const float* partB, const float* partC,
                                 float* dA_log, float* ddt_bias, float* dcentre) {
  launch_dependents();  // (it needs nothing of the pass in front of it and runs beside it; what it reads, see launch_rec_bwd)
  __shared__ float s[3][256];
  const int h = blockIdx.x, tid = threadIdx.x, c = tid % D, sl = tid / D, ns = 256 / D;
  float b = 0.f, a = 0.f, cc = 0.f;
  for (int j = sl; j < blocks; j += ns) b += partB[((size_t)j * H + h) * D + c];
  for (int j = tid; j < blocks; j += 256) { a += partA[(size_t)j * H + h]; cc += partC[(size_t)j * H + h]; }
  s[0][tid] = b; s[1][tid] = a; s[2][tid] = cc;
  __syncthreads();
  if (tid < D) {
    float x = 0.f;
    for (int i = 0; i < ns; ++i) x += s[0][i * D + tid];
    ddt_bias[h * D + tid] = x;
  }
  for (int o = 128; o >= 1; o >>= 1) {
    if (tid < o) { s[1][tid] += s[1][tid + o]; s[2][tid] += s[2][tid + o]; }
    __syncthreads();
  }
  if (tid == 0) { dA_log[h] = s[1][0]; dcentre[h] = s[2][0]; }
  wait_prerequisites();
}

struct RecBwdWorkspace {
  float *dSck, *de, *lam, *dkp, *carry, *decay, *partA, *partB, *partC;
  void* saved;      // what a saving forward would have left (unless the caller hands it in)
  void* o_scratch;  // output of the forward that is run again (its contents are not used)
  size_t bytes;
};

// `with_saved`: the forward's leavings are part of the workspace.
static RecBwdWorkspace carve_rec_bwd(const pkda_problem& p, void* base, bool with_saved) {
  RecBwdWorkspace w;
  const size_t H = p.heads, D = p.head_dim, units = (size_t)p.total_tokens * H, blocks = ckpt_bound(p);
  size_t off = 0;
  unsigned char* b = static_cast<unsigned char*>(base);
  auto take = [&](size_t bytes) { void* ptr = b + off; off += align_up(bytes); return ptr; };
  w.dSck = static_cast<float*>(take(blocks * H * D * D * 4));
  w.de = static_cast<float*>(take(units * D * 4));
  w.lam = static_cast<float*>(take(units * D * 4));
  w.dkp = static_cast<float*>(take(units * D * 4));
  w.carry = static_cast<float*>(take(blocks * H * D * 4));
  w.decay = static_cast<float*>(take(blocks * H * 4));
  w.partA = static_cast<float*>(take(blocks * H * 4));
  w.partB = static_cast<float*>(take(blocks * H * D * 4));
  w.partC = static_cast<float*>(take(blocks * H * 4));
  w.saved = w.o_scratch = nullptr;
  if (with_saved) {
    w.saved = take(recurrent_saved_bytes(p));
    w.o_scratch = take(units * D * 4);
  }
  w.bytes = off;
  return w;
}

size_t recurrent_bwd_workspace(const pkda_problem& p) { return carve_rec_bwd(p, nullptr, true).bytes; }
size_t recurrent_bwd_saved_workspace(const pkda_problem& p) { return carve_rec_bwd(p, nullptr, false).bytes; }

template <int D, typename T>
static int launch_rec_bwd(RecBwdParams bp, size_t blocks, cudaStream_t st) {
  using L = ScanLay<D, 1>;
  using G = GradLay<D>;
  const int units = bp.geo.n_seqs * bp.geo.heads, H = bp.geo.heads;
  const int nw = scan_consumers(units, L::kWarps, L::kMaxConsumers, sm_count());
  bp.groups = L::kWarps / nw;
  bp.warps = {nw, spread_producers(nw, units * bp.groups, sm_count())};
  constexpr int kMost = two_ahead_reverse<D>();
  auto dscan = nw <= kMost ? pkda_recurrent_dscan_kernel<D, T, (kMost > 0)> : pkda_recurrent_dscan_kernel<D, T, false>;
  if (!ensure_dynamic_smem(dscan, L::kSmem) ||
      !ensure_dynamic_smem(pkda_recurrent_grad_kernel<D, T>, G::kFloats * 4))
    return PKDA_ERR_LAUNCH;
  begin_stage(kStageRecurrent, st);
  // Set up while the forward's scan still runs, its CTAs come to lie two on an SM beside idle ones (512 tokens of 40 units at 64 rows,
  // one token ahead: 188 us against 106; 76 units at 32 rows: 108 against 66), unless two do not fit: two tokens ahead they do not,
  // by their registers (exact step of 2 x 512 tokens of 4 heads x 64: 158 us early, 160 behind the forward).
  int rc = launch_kernel(nw <= kMost, dscan, units * bp.groups, bp.warps.threads(L::kProd), L::kSmem, st, bp);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  const dim3 grid((unsigned)blocks, (unsigned)H);
  begin_stage(kStageRecurrent, st);
  rc = launch_kernel(pkda_recurrent_grad_kernel<D, T>, grid, G::kThreads, G::kFloats * 4, st, bp);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageRecurrent, st);
  // (An ordinary launch: the reduction that runs beside the closing pass reads the partial sums without a wait of its own, so the
  // pass that leaves them has to have ended in front of a launch in between.)
  rc = launch_kernel(false, pkda_recurrent_carry_kernel<D>, units, D < 32 ? 32 : D, 0, st, bp);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageRecurrent, st);
  rc = launch_kernel(pkda_recurrent_close_kernel<D, T>, grid, 256, 0, st, bp);
  end_stage(st);
  return rc;
}

template <typename T>
static int dispatch_rec_bwd(int D, const RecBwdParams& bp, size_t blocks, cudaStream_t st) {
  switch (D) {
    case 8: return launch_rec_bwd<8, T>(bp, blocks, st);
    case 16: return launch_rec_bwd<16, T>(bp, blocks, st);
    case 32: return launch_rec_bwd<32, T>(bp, blocks, st);
    case 64: return launch_rec_bwd<64, T>(bp, blocks, st);
    case 128: return launch_rec_bwd<128, T>(bp, blocks, st);
    default: return PKDA_ERR_SHAPE;
  }
}

// `saved`: what pkda_recurrent_fwd_saving left for the same problem, or NULL (it is made again).
int recurrent_bwd(const pkda_recurrent_bwd_args* a, const void* saved, size_t saved_bytes, cudaStream_t st) {
  const pkda_problem& p = a->p;
  int rc = check_problem(p);
  if (rc != PKDA_OK) return rc;
  if (p.n_seqs == 0 || p.total_tokens == 0) return PKDA_OK;
  if (!a->d_o || !a->dq || !a->dk || !a->dv || !a->dg || !a->dg_atk || !a->dbeta_atk || !a->dbeta || !a->dA_log ||
      !a->ddt_bias || !a->dlog_atk_scale)
    return PKDA_ERR_NULL;
  const RecBwdWorkspace ws = carve_rec_bwd(p, a->workspace, saved == nullptr);
  if (!a->workspace || a->workspace_bytes < ws.bytes) return PKDA_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(a->workspace) | reinterpret_cast<uintptr_t>(saved)) & 15) return PKDA_ERR_ALIGN;
  if (saved && saved_bytes < recurrent_saved_bytes(p)) return PKDA_ERR_WORKSPACE;
  RecBwdParams bp;
  bp.geo = make_geo(p, nullptr);
  bp.s = carve_rec_saved(p, saved ? const_cast<void*>(saved) : ws.saved, nullptr);
  if (!saved) {
    rc = recurrent_fwd_saving(p, ws.o_scratch, bp.s, st);
    if (rc != PKDA_OK) return rc;
  }
  bp.q = p.q; bp.k = p.k; bp.g = p.g; bp.g_atk = p.g_atk; bp.beta_atk = p.beta_atk; bp.beta = p.beta;
  bp.A_log = p.A_log; bp.dt_bias = p.dt_bias; bp.log_atk_scale = p.log_atk_scale; bp.A0 = p.initial_A_state;
  bp.d_o = a->d_o; bp.dST = a->d_final_state;
  bp.dSck = ws.dSck; bp.de = ws.de; bp.lam = ws.lam; bp.dkp = ws.dkp;
  bp.carry = ws.carry; bp.decay = ws.decay;
  bp.dq = a->dq; bp.dk = a->dk; bp.dv = a->dv; bp.dg = a->dg; bp.dbeta_atk = a->dbeta_atk; bp.dbeta = a->dbeta;
  bp.dg_atk = a->dg_atk; bp.partA = ws.partA; bp.partB = ws.partB; bp.partC = ws.partC;
  bp.dS0 = a->d_initial_state; bp.dA0 = a->d_initial_A_state;
  bp.warps = {0, 0};
  bp.groups = 0;
  bp.scale = p.scale; bp.ln_x = logf(p.squash_x); bp.eps = p.squash_eps;
  const size_t blocks = ckpt_bound(p);
  rc = p.dtype == PKDA_BF16 ? dispatch_rec_bwd<bf16>(p.head_dim, bp, blocks, st)
                            : dispatch_rec_bwd<float>(p.head_dim, bp, blocks, st);
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageParamReduce, st);
  rc = launch_kernel(pkda_recurrent_bwd_reduce_kernel, p.heads, 256, 0, st, (int)blocks, p.heads, p.head_dim, ws.partA, ws.partB,
                     ws.partC, a->dA_log, a->ddt_bias, a->dlog_atk_scale);
  end_stage(st);
  return rc;
}

}  // namespace pkda
