// Token-by-token PKDA recurrence: short cached prefill, packed short sequences, and the exact fp32
// forward (fp32 activations, head widths other than 128).  Single-token steps on a cached state run
// in pkda_decode_step.cu.
//
// Follows delta_feedback_experiment/pkda.py:390-410:
//   A  <- exp(gP) A + bP k^2 ;  kw = k * precond_factor(A)
//   S  <- diag(exp(g)) S ;  e = v - S^T k ;  S <- S + (beta kw) e^T ;  o = S^T (scale q)
//
// What bounds it: the chain of dependent tokens.  The value columns of S are independent of one
// another, so each warp takes 4 columns (16 once the one-column warps fill the chip, 8 at D = 8) with all D
// rows (ScanLay) and the step's only exchange is log2(8) = 3 shuffles for e (7 for four columns per lane);
// with one CTA holding the whole state the step crossed three block barriers and two shared-memory reductions.  The row vectors (exp(g), k, beta kw, q) do not depend
// on S: producer warps make them for 8 tokens at a time, double buffered, while the consumer warps
// run the chain; the sum for o is off the chain and is reduced for 8 tokens at once.
// The output of a token and the decay of the state are taken while the next token's sum goes through its shuffles.
// Measured, against one CTA with the whole state: 4 x 16 units, 48 tokens, D = 128, bf16: 67 -> 21.7 us; 2 x 4 units, 512
// tokens, D = 64, fp32: 548 -> 64 us (72 when it leaves what the backward needs).
#include <type_traits>

#include "pkda_launch.h"
#include "pkda_recurrent.cuh"

namespace pkda {

struct RecParams {
  Geo geo;
  const void *q, *k, *v, *g;
  const float* g_atk;
  const void *beta_atk, *beta;
  const float *A_log, *dt_bias, *log_atk_scale;
  const float *S0, *A0;
  void* o;
  float *ST, *AT;
  RecSaved save;     // kSave only
  ScanWarps warps;   // consumer and producer warps of a CTA
  int groups;        // CTAs per (sequence, head)
  int inplace_A;     // AT aliases A0: written only after every CTA of the unit has read it (a cluster)
  float scale, ln_x, eps;
};

template <int D, int kCPL, typename T, bool kSave, bool kTwoAhead>
__global__ void __launch_bounds__(ScanLay<D, kCPL>::kProd + 32 * ScanLay<D, kCPL>::kMaxConsumers)
pkda_recurrent_kernel(const RecParams p) {
  after_previous();
  using L = ScanLay<D, kCPL>;
  constexpr int TB = L::kTB, TPG = L::kTPG, RG = L::kRG, R = L::kR, VEC = L::kVecs * D;
  extern __shared__ __align__(16) float stage[];  // [2][TB][5][D]: exp(g) k, exp(g), beta kw, scale q, v
  const int H = p.geo.heads;
  const int unit = blockIdx.x / p.groups, cg = blockIdx.x - unit * p.groups;
  const int n = unit / H, h = unit - n * H;
  const SeqInfo sq = seq_info(p.geo, n);
  const int nblk = (sq.len + TB - 1) / TB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = p.warps.nw, nthreads = 32 * nw + L::kProd;

  if (p.warps.idle(warp)) return;
  if (warp >= nw) {
    // ------------------------------------------------ producers: row vectors of TB tokens at a time
    const int ptid = 32 * p.warps.producer(warp) + lane;
    const int grp = ptid / L::kProdPerGroup, c = ptid - grp * L::kProdPerGroup;
    const bool act = D >= 32 || c < D;
    const float ea = expf(p.A_log[h]), centre = p.log_atk_scale[h];
    const float bias = act ? p.dt_bias[h * D + c] : 0.f;
    float A = (act && p.A0) ? p.A0[(size_t)unit * D + c] : 0.f;
    if (p.inplace_A) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    // The producers set the pace of a scan that has its SM to itself, and the addresses and checks of a block's 16 loads were 1,000 of their
    // 2,600 cycles: running pointers, 32-bit offsets, no checks in a whole block.  (The vectors that the backward needs are
    // written by all CTAs of the unit in turn, a block each: by the first one alone, that one was late.)
    const int step = H * D;
    const size_t first = (size_t)sq.bos * H + h, base = first * D + (act ? c : 0), own = base + (size_t)(TPG * grp) * step;
    const T *kp = static_cast<const T*>(p.k) + base, *qp = static_cast<const T*>(p.q) + own, *gp = static_cast<const T*>(p.g) + own,
            *vp = static_cast<const T*>(p.v) + own;
    const int kind = lane >> 3;  // of the lane's scalar: lane = 8 * kind + token
    const float* pdp = p.g_atk + first + (size_t)(lane & 7) * H;
    const T* bp = static_cast<const T*>(kind == 1 ? p.beta_atk : p.beta) + first + (size_t)(lane & 7) * H;
    typename Raw<T>::type kr[TB], qr[TPG], gr[TPG], vr[TPG], bt;
    float sc;
    auto fetch_block = [&](int left, auto whole) {  // left: tokens from the block's first one on
      constexpr bool kWhole = decltype(whole)::value;
#pragma unroll
      for (int i = 0; i < TB; ++i) kr[i] = act && (kWhole || i < left) ? Raw<T>::load(kp + i * step) : 0;
#pragma unroll
      for (int i = 0; i < TPG; ++i) {
        const bool ok = act && (kWhole || TPG * grp + i < left);
        qr[i] = ok ? Raw<T>::load(qp + i * step) : 0;
        gr[i] = ok ? Raw<T>::load(gp + i * step) : 0;
        vr[i] = ok ? Raw<T>::load(vp + i * step) : 0;
      }
      const bool ok = kWhole || (lane & 7) < left;
      sc = 0.f;
      bt = 0;
      if (ok && kind == 0) sc = *pdp;
      if (ok && kind != 0) bt = Raw<T>::load(bp);  // (the last eight lanes' are not used)
    };
    auto fetch = [&](int t0) {
      const int left = sq.len - t0;
      if (left >= TB) fetch_block(left, std::true_type{});
      else fetch_block(left, std::false_type{});
      kp += TB * step;
      qp += TB * step;
      gp += TB * step;
      vp += TB * step;
      pdp += TB * H;
      bp += TB * H;
    };
    if (nblk > 0) fetch(0);
    for (int b = 0; b < nblk; ++b) {
      const int s = b & 1, t0 = b * TB;
      float kc[TPG], An[TPG], qc[TPG], gc[TPG], vc[TPG];
      const float scal = lane < 8 ? expf(sc) : Raw<T>::value(bt);
#pragma unroll
      for (int i = 0; i < TB; ++i) {
        const float pd = __shfl_sync(0xffffffffu, scal, i), ba = __shfl_sync(0xffffffffu, scal, 8 + i);
        const float kf = Raw<T>::value(kr[i]);
        A = pd * A + ba * kf * kf;
        if (i < TPG || grp == i / TPG) { An[i % TPG] = A; kc[i % TPG] = kf; }
      }
#pragma unroll
      for (int i = 0; i < TPG; ++i) { qc[i] = Raw<T>::value(qr[i]); gc[i] = Raw<T>::value(gr[i]); vc[i] = Raw<T>::value(vr[i]); }
      if (b + 1 < nblk) fetch(t0 + TB);
      if (b >= 2) bar_sync_n(3 + s, nthreads);
      float* st = stage + s * L::kStage;
#pragma unroll
      for (int i = 0; i < TPG; ++i) {
        const int tl = TPG * grp + i;
        const float bw = __shfl_sync(0xffffffffu, scal, 16 + tl);
        const bool ok = t0 + tl < sq.len;  // tokens past the end leave the state as it is
        // The same two functions as in the few-token and decoding kernels, so that a token's factors do not depend
        // on the kernel.  (A branch-free log1p series and approximate quotients here saved 2% of a call, 193.6
        // against 197.8 us at 2 x 512 tokens of 4 heads x 64, and cost 4% in the error against 64 bits.)
        float al = expf(-ea * softplus_acc(gc[i] + bias));
        al = ok ? al : 1.f;
        const float wk = bw * (kc[i] * precond_factor(An[i], p.eps, centre, p.ln_x));
        if (act) {
          float* row = st + tl * VEC + c;
          row[0] = al * kc[i];
          row[D] = al;
          row[2 * D] = wk;
          row[3 * D] = qc[i] * p.scale;
          row[4 * D] = vc[i];
          if (kSave && b % p.groups == cg && ok) {
            const size_t idx = base + (size_t)(t0 + tl) * step;
            p.save.al[idx] = al;
            p.save.w[idx] = wk;
            p.save.A[idx] = An[i];
          }
        }
      }
      bar_arrive_n(1 + s, nthreads);
    }
    if (p.inplace_A) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (p.AT && cg == 0 && grp == 0 && act) p.AT[(size_t)unit * D + c] = A;
    return;
  }

  // ---------------------------------------------------- consumers: the chain over tokens
  if (p.inplace_A) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  const int rg = lane & (RG - 1);
  const int col0 = (cg * nw + warp) * L::kCols + (lane / RG) * kCPL;
  const size_t sbase = (size_t)unit * D * D + col0;
  float2 S[kCPL][R / 2];
  // element (row, column c) of the lane's part of the state
  auto elem = [&](int row, int c) -> float& { return (row & 1) ? S[c][row / 2].y : S[c][row / 2].x; };
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float* src = p.S0 + sbase + (size_t)(L::row(i / L::kU, rg) + i % L::kU) * D;
    float x[kCPL];
#pragma unroll
    for (int c = 0; c < kCPL; ++c) x[c] = 0.f;
    if (p.S0) {
      if (kCPL == 4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(src);
      else x[0] = *src;
    }
#pragma unroll
    for (int c = 0; c < kCPL; ++c) elem(i, c) = x[c];
  }
  auto store_state = [&](float* base) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float* dst = base + (size_t)(L::row(i / L::kU, rg) + i % L::kU) * D;
      if (kCPL == 4) *reinterpret_cast<float4*>(dst) = make_float4(elem(i, 0), elem(i, 1 % kCPL), elem(i, 2 % kCPL), elem(i, 3 % kCPL));
      else *dst = elem(i, 0);
    }
  };
  const size_t tstep = (size_t)H * D;
  const size_t tbase = ((size_t)sq.bos * H + h) * D + col0;
  T* const o_row = static_cast<T*>(p.o) + tbase;
  // The vectors of a token, and its value (kTwoAhead).
  struct Rows { float2 kx[R / 2], al[R / 2], wk[R / 2], qs[R / 2]; float v; };
  Rows ahead[kTwoAhead ? 2 : 1];
  auto load_token = [&](Rows& x, uint32_t vec) {
    load_rows<L>(vec, rg, x.kx);
    load_rows<L>(vec + 4 * D, rg, x.al);
    load_rows<L>(vec + 8 * D, rg, x.wk);
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x.v) : "r"(vec + 16 * D + 4 * col0));
    load_rows<L>(vec + 12 * D, rg, x.qs);
  };
  if (kTwoAhead && nblk > 0) {
    bar_sync_n(1, nthreads);
    load_token(ahead[0], smem_u32(stage));
    load_token(ahead[kTwoAhead], smem_u32(stage) + 4 * VEC);
  }
  for (int b = 0; b < nblk; ++b) {
    const int s = b & 1, t0 = b * TB;
    if (kSave && (t0 & (kCkpt - 1)) == 0)
      store_state(p.save.S + ((ckpt_base(p.geo, n, sq.bos) + t0 / kCkpt) * H + h) * (size_t)(D * D) + col0);
    if (!kTwoAhead) bar_sync_n(1 + s, nthreads);
    const uint32_t st = smem_u32(stage + s * L::kStage);
    float oacc[L::kTO * kCPL], ekeep[L::kSums];  // [token][column]
    // Two vectors of rows are held at a time.  x: exp(g) k, then exp(g) of a token; y: beta kw, then scale q.
    float2 x[R / 2], y[R / 2];
    auto out_sum = [&](int u) {  // the sum for o of token u (of the block)
#pragma unroll
      for (int c = 0; c < kCPL; ++c) {
        float2 a0 = __fmul2_rn(y[0], S[c][0]);
#pragma unroll
        for (int i = 1; i < R / 2; ++i) a0 = __ffma2_rn(y[i], S[c][i], a0);
        oacc[(u % L::kTO) * kCPL + c] = a0.x + a0.y;
      }
    };
    auto out_round = [&](int u, int o) {  // a round over the lanes for the kTO tokens that end with u; behind the last they leave
      if ((u + 1) % L::kTO) return;
      rg_sum_round(oacc, rg, o, L::kTO * kCPL * o / RG);
      if (o > 1) return;
#pragma unroll
      for (int i = 0; i < L::kSums; ++i) {
        const int n = rg * L::kSums + i, to = t0 + u + 1 - L::kTO + n / kCPL;
        if (to < sq.len) o_row[(size_t)to * tstep + n % kCPL] = from_f<T>(oacc[i]);
      }
    };
    if constexpr (kTwoAhead) {
      const uint32_t nx = smem_u32(stage + (s ^ 1) * L::kStage);
#pragma unroll
      for (int t = 0; t < TB; ++t) {
        Rows& w = ahead[t & 1];
        float2 a0 = __fmul2_rn(w.kx[0], S[0][0]), a1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 1; i < R / 2; ++i) {
          if (i & 1) a1 = __ffma2_rn(w.kx[i], S[0][i], a1);
          else a0 = __ffma2_rn(w.kx[i], S[0][i], a0);
        }
        float e = (a0.x + a0.y) + (a1.x + a1.y);
#pragma unroll
        for (int i = 0; i < R / 2; ++i) S[0][i] = __fmul2_rn(w.al[i], S[0][i]);
#pragma unroll
        for (int o = RG / 2; o >= 1; o >>= 1) e += xor_lane(e, o);
        e = w.v - e;
        if (kSave && rg == t / L::kSums) ekeep[t % L::kSums] = e;
#pragma unroll
        for (int i = 0; i < R / 2; ++i) S[0][i] = __ffma2_rn(w.wk[i], make_float2(e, e), S[0][i]);
#pragma unroll
        for (int i = 0; i < R / 2; ++i) y[i] = w.qs[i];
        out_sum(t);
        if (t == TB - 2 && b + 1 < nblk) bar_sync_n(1 + (s ^ 1), nthreads);
        if (t + 2 < TB) load_token(w, st + 4 * (t + 2) * VEC);
        else if (b + 1 < nblk) load_token(w, nx + 4 * (t + 2 - TB) * VEC);
      }
      if (b + 2 < nblk) bar_arrive_n(3 + s, nthreads);
    } else {
    load_rows<L>(st, rg, x);
#pragma unroll
    for (int t = 0; t < TB; ++t) {
      // e's sum over the lane's rows, then rounds of shuffles; behind each round's shuffles stands what does not depend on
      // them: the output of the token before, the decay of the state, the loads.
      const uint32_t vec = st + 4 * t * VEC;
      float e[kCPL], r[kCPL], vt[kCPL];
#pragma unroll
      for (int c = 0; c < kCPL; ++c) {
        float2 a0 = __fmul2_rn(x[0], S[c][0]), a1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 1; i < R / 2; ++i) {
          if (i & 1) a1 = __ffma2_rn(x[i], S[c][i], a1);
          else a0 = __ffma2_rn(x[i], S[c][i], a0);
        }
        e[c] = (a0.x + a0.y) + (a1.x + a1.y);
      }
      auto round = [&](int o) {
#pragma unroll
        for (int c = 0; c < kCPL; ++c) r[c] = xor_lane(e[c], o);
      };
      auto add = [&]() {
#pragma unroll
        for (int c = 0; c < kCPL; ++c) e[c] += r[c];
      };
      round(RG / 2);
      load_rows<L>(vec + 4 * D, rg, x);
      if (t > 0) out_sum(t - 1);
      add();
      round(RG / 4);
      if (t > 0) out_round(t - 1, RG / 2);
      load_rows<L>(vec + 8 * D, rg, y);
#pragma unroll
      for (int c = 0; c < kCPL; ++c)
#pragma unroll
        for (int i = 0; i < R / 2; ++i) S[c][i] = __fmul2_rn(x[i], S[c][i]);
      add();
      if (RG == 8) round(1);
      if (t > 0) out_round(t - 1, RG / 4);
      if (kCPL == 4) {
        float2 v[2];
        load_run<4>(vec + 16 * D + 4 * col0, v);
        vt[0] = v[0].x; vt[1 % kCPL] = v[0].y; vt[2 % kCPL] = v[1].x; vt[3 % kCPL] = v[1].y;
      } else {
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(vt[0]) : "r"(vec + 16 * D + 4 * col0));
      }
      if (t + 1 < TB) load_rows<L>(vec + 4 * VEC, rg, x);
      if (RG == 8) add();
#pragma unroll
      for (int c = 0; c < kCPL; ++c) e[c] = vt[c] - e[c];
      if (kSave && rg == t / L::kSums) ekeep[t % L::kSums] = e[0];
#pragma unroll
      for (int c = 0; c < kCPL; ++c)
#pragma unroll
        for (int i = 0; i < R / 2; ++i) S[c][i] = __ffma2_rn(y[i], make_float2(e[c], e[c]), S[c][i]);
      load_rows<L>(vec + 12 * D, rg, y);
      if (RG == 8 && t > 0) out_round(t - 1, 1);
    }
    out_sum(TB - 1);
    if (b + 2 < nblk) bar_arrive_n(3 + s, nthreads);
    }
#pragma unroll
    for (int o = RG / 2; o >= 1; o >>= 1) out_round(TB - 1, o);
    if (kSave) {  // (one column per lane)
#pragma unroll
      for (int i = 0; i < L::kSums; ++i) {
        const int t = t0 + rg * L::kSums + i;
        if (t < sq.len) p.save.e[tbase + (size_t)t * tstep] = ekeep[i];
      }
    }
  }
  if (p.ST) store_state(p.ST + sbase);
  if (p.inplace_A) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// A few tokens for more (sequence, head) units than SMs, e.g. a speculative block of a large batch:
// reading and writing the states is most of the call.  One CTA keeps the whole state in registers
// (thread = 16 rows x 4 columns, state rows moved in full 512-byte lines, two CTAs per SM), as the
// decode step does, and crosses three block barriers per token.  D = 128, bf16, us a call at 2 / 7 / 13 / 16 tokens:
// 256 units (one wave of this kernel, two of the sliced one) 10.3 / 18.4 / 28.7 / 33.8 against 22.6 / 22.6 / 32.8 /
// 32.8; 512 units 16 / 35 / 57 / 70 against 41 / 43 / 62 / 62; 1024 units 41 / 86 / 142 / 166 against 78 / 78 / 113 / 113.
template <int D, typename T>
__global__ void __launch_bounds__(RecCfg<D>::kThreads, D == 128 ? 2 : 1)
pkda_recurrent_few_kernel(const RecParams p) {
  after_previous();
  using Cfg = RecCfg<D>;
  constexpr int VQ = Cfg::kVQ, KW = Cfg::kKW, R = Cfg::kR;
  const int tid = threadIdx.x;
  const int n = blockIdx.x / p.geo.heads;
  const int h = blockIdx.x - n * p.geo.heads;
  const SeqInfo sq = seq_info(p.geo, n);
  const int H = p.geo.heads;

  __shared__ float s_k[D], s_wk[D], s_q[D], s_al[D];
  __shared__ __align__(16) float s_v[D];
  __shared__ __align__(16) float s_red[2][KW][D];

  const bool active = tid < Cfg::kActive;
  const int kq = tid / VQ, vq = tid - kq * VQ;
  const int krow0 = kq * R;

  float4 S[R];
  const size_t sbase = ((size_t)n * H + h) * D * D;
  if (active) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (p.S0) S[r] = *reinterpret_cast<const float4*>(p.S0 + sbase + (size_t)(krow0 + r) * D + 4 * vq);
      else S[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  // per-channel persistent values (threads tid < D)
  float A = 0.f, bias = 0.f;
  const float ea = expf(p.A_log[h]);
  const float centre = p.log_atk_scale[h];
  if (tid < D) {
    A = p.A0 ? p.A0[((size_t)n * H + h) * D + tid] : 0.f;
    bias = p.dt_bias[h * D + tid];
  }
  const T* q = static_cast<const T*>(p.q);
  const T* k = static_cast<const T*>(p.k);
  const T* v = static_cast<const T*>(p.v);
  const T* g = static_cast<const T*>(p.g);
  const T* bA = static_cast<const T*>(p.beta_atk);
  const T* bW = static_cast<const T*>(p.beta);
  T* o = static_cast<T*>(p.o);

  for (int t = 0; t < sq.len; ++t) {
    const size_t tok = (size_t)(sq.bos + t);
    const size_t sidx = tok * H + h;
    if (tid < D) {
      const size_t idx = sidx * D + tid;
      const float kc = to_f(k[idx]);
      const float pd = expf(p.g_atk[sidx]);
      A = pd * A + to_f(bA[sidx]) * kc * kc;
      const float kw = kc * precond_factor(A, p.eps, centre, p.ln_x);
      s_k[tid] = kc;
      s_wk[tid] = to_f(bW[sidx]) * kw;
      s_q[tid] = to_f(q[idx]) * p.scale;
      s_al[tid] = expf(-ea * softplus_acc(to_f(g[idx]) + bias));
      s_v[tid] = to_f(v[idx]);
    }
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float al = s_al[krow0 + r], kk = s_k[krow0 + r];
        S[r].x *= al; S[r].y *= al; S[r].z *= al; S[r].w *= al;
        acc.x += S[r].x * kk; acc.y += S[r].y * kk; acc.z += S[r].z * kk; acc.w += S[r].w * kk;
      }
      *reinterpret_cast<float4*>(&s_red[0][kq][4 * vq]) = acc;
    }
    __syncthreads();
    if (active) {
      float4 e = *reinterpret_cast<const float4*>(&s_v[4 * vq]);
#pragma unroll
      for (int w = 0; w < KW; ++w) {
        const float4 pr = *reinterpret_cast<const float4*>(&s_red[0][w][4 * vq]);
        e.x -= pr.x; e.y -= pr.y; e.z -= pr.z; e.w -= pr.w;
      }
      acc = make_float4(0.f, 0.f, 0.f, 0.f);
      const bool last = p.ST && t == sq.len - 1;  // final state rows leave as soon as they are final
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float wk = s_wk[krow0 + r], qq = s_q[krow0 + r];
        S[r].x += wk * e.x; S[r].y += wk * e.y; S[r].z += wk * e.z; S[r].w += wk * e.w;
        acc.x += S[r].x * qq; acc.y += S[r].y * qq; acc.z += S[r].z * qq; acc.w += S[r].w * qq;
        if (last) *reinterpret_cast<float4*>(p.ST + sbase + (size_t)(krow0 + r) * D + 4 * vq) = S[r];
      }
      *reinterpret_cast<float4*>(&s_red[1][kq][4 * vq]) = acc;
    }
    __syncthreads();
    if (tid < D) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < KW; ++w) sum += s_red[1][w][tid];
      o[sidx * D + tid] = from_f<T>(sum);
    }
  }
  if (p.ST && active && sq.len == 0) {  // no token: the state passes through
#pragma unroll
    for (int r = 0; r < R; ++r)
      *reinterpret_cast<float4*>(p.ST + sbase + (size_t)(krow0 + r) * D + 4 * vq) = S[r];
  }
  if (p.AT && tid < D) p.AT[((size_t)n * H + h) * D + tid] = A;
}

template <int D, int kCPL, typename T, bool kSave>
static int launch_rec(RecParams rp, cudaStream_t st) {
  using L = ScanLay<D, kCPL>;
  const int units = rp.geo.n_seqs * rp.geo.heads;
  int nw = scan_consumers(units, L::kWarps, L::kMaxConsumers, sm_count());
  if (rp.inplace_A)  // the unit's CTAs form one cluster: at most eight of them
    while (L::kWarps / nw > 8) nw *= 2;
  rp.groups = L::kWarps / nw;
  if (rp.groups == 1) rp.inplace_A = 0;
  constexpr int kMost = kCPL == 1 ? two_ahead_forward<D>() : 0;
  auto kernel = nw <= kMost ? pkda_recurrent_kernel<D, kCPL, T, kSave, (kMost > 0)> : pkda_recurrent_kernel<D, kCPL, T, kSave, false>;
  rp.warps = {nw, spread_producers(nw, units * rp.groups, sm_count()) && !rp.inplace_A};  // (every thread takes part in the cluster's barrier)
  if (!ensure_dynamic_smem(kernel, L::kSmem)) return PKDA_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units * rp.groups));
  cfg.blockDim = dim3((unsigned)rp.warps.threads(L::kProd));
  cfg.dynamicSmemBytes = L::kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)rp.groups;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = rp.inplace_A ? 2 : 1;
  begin_stage(kStageRecurrent, st);
  const int rc = launch_code(cudaLaunchKernelEx(&cfg, kernel, rp));
  end_stage(st);
  return rc;
}

template <int D, typename T>
static int launch_rec_d(const RecParams& rp, bool save, cudaStream_t st) {
  if (save) return launch_rec<D, 1, T, true>(rp, st);
  const long units = (long)rp.geo.n_seqs * rp.geo.heads;
  const int few = units <= 2L * sm_count() ? 14 : 8;  // break-even in tokens, see that kernel
  if (rp.geo.seq_len > 0 && rp.geo.seq_len < few && units > sm_count()) {
    if (!aligned({rp.ST}, 16)) return PKDA_ERR_ALIGN;  // (here, with four columns per lane and in the single step: states by float4)
    begin_stage(kStageRecurrent, st);
    const int rc = launch_kernel(pkda_recurrent_few_kernel<D, T>, (unsigned)units, RecCfg<D>::kThreads, 0, st, rp);
    end_stage(st);
    return rc;
  }
  // Four columns per lane once the one-column warps number more than two per scheduler (4 per SM).
  constexpr bool kFour = D >= 64;
  const long warps = units * ScanLay<D, 1>::kWarps;
  if (kFour && warps > 8L * sm_count()) return aligned({rp.ST}, 16) ? launch_rec<D, kFour ? 4 : 1, T, false>(rp, st) : PKDA_ERR_ALIGN;
  return launch_rec<D, 1, T, false>(rp, st);
}

template <typename T>
static int dispatch_rec(int D, const RecParams& rp, bool save, cudaStream_t st) {
  switch (D) {
    case 8: return launch_rec_d<8, T>(rp, save, st);
    case 16: return launch_rec_d<16, T>(rp, save, st);
    case 32: return launch_rec_d<32, T>(rp, save, st);
    case 64: return launch_rec_d<64, T>(rp, save, st);
    case 128: return launch_rec_d<128, T>(rp, save, st);
    default: return PKDA_ERR_SHAPE;
  }
}

RecSaved carve_rec_saved(const pkda_problem& p, void* base, size_t* bytes) {
  RecSaved s;
  const size_t units = (size_t)p.total_tokens * p.heads, D = p.head_dim;
  size_t off = 0;
  unsigned char* b = static_cast<unsigned char*>(base);
  auto take = [&](size_t n) { float* x = reinterpret_cast<float*>(b + off); off += align_up(n * 4); return x; };
  s.al = take(units * D);
  s.w = take(units * D);
  s.A = take(units * D);
  s.e = take(units * D);
  s.S = take(ckpt_bound(p) * p.heads * D * D);
  if (bytes) *bytes = off;
  return s;
}

static int run_rec(const pkda_problem& p, void* o, float* ST, float* AT, const RecSaved* save, cudaStream_t st) {
  RecParams rp;
  rp.geo = make_geo(p, nullptr);
  rp.q = p.q; rp.k = p.k; rp.v = p.v; rp.g = p.g; rp.g_atk = p.g_atk;
  rp.beta_atk = p.beta_atk; rp.beta = p.beta;
  rp.A_log = p.A_log; rp.dt_bias = p.dt_bias; rp.log_atk_scale = p.log_atk_scale;
  rp.S0 = p.initial_state; rp.A0 = p.initial_A_state;
  rp.o = o; rp.ST = ST; rp.AT = AT;
  rp.save = save ? *save : RecSaved{};
  rp.inplace_A = AT && AT == p.initial_A_state;
  rp.scale = p.scale; rp.ln_x = logf(p.squash_x); rp.eps = p.squash_eps;
  if (p.dtype == PKDA_BF16) return dispatch_rec<bf16>(p.head_dim, rp, save != nullptr, st);
  if (p.dtype == PKDA_F32) return dispatch_rec<float>(p.head_dim, rp, save != nullptr, st);
  return PKDA_ERR_DTYPE;
}

int recurrent_fwd(const pkda_recurrent_args* a, void* saved, size_t saved_bytes, cudaStream_t st) {
  const pkda_problem& p = a->p;
  int rc = check_problem(p);
  if (rc != PKDA_OK) return rc;
  if (p.n_seqs == 0 || p.total_tokens == 0) return PKDA_OK;
  if (!a->o) return PKDA_ERR_NULL;
  if (saved) {
    if (reinterpret_cast<uintptr_t>(saved) & 15) return PKDA_ERR_ALIGN;  // (states move four values at a time)
    size_t need = 0;
    const RecSaved s = carve_rec_saved(p, saved, &need);
    if (saved_bytes < need) return PKDA_ERR_WORKSPACE;
    return run_rec(p, a->o, a->final_state, a->final_A_state, &s, st);
  }
  // One token per sequence on a cached state: the decode-step kernel (all loads of the step issued
  // up front), without its convolution and gate stages.
  if (!p.cu_seqlens && p.seq_len == 1 && p.initial_state && a->final_state &&
      (p.dtype == PKDA_BF16 || p.dtype == PKDA_F32)) {
    if (!aligned({a->final_state}, 16)) return PKDA_ERR_ALIGN;
    return decode_direct(p, a->o, a->final_state, a->final_A_state, st);
  }
  return run_rec(p, a->o, a->final_state, a->final_A_state, nullptr, st);
}

// Forward pass that only leaves what the exact backward needs (its output goes to scratch).
int recurrent_fwd_saving(const pkda_problem& p, void* o_scratch, const RecSaved& save, cudaStream_t st) {
  return run_rec(p, o_scratch, nullptr, nullptr, &save, st);
}

size_t recurrent_saved_bytes(const pkda_problem& p) {
  size_t bytes = 0;
  carve_rec_saved(p, nullptr, &bytes);
  return bytes;
}

}  // namespace pkda
