// Reverse scan of the state cotangent dS for few units.  Eight, four or (beside a recompute pass's scan) two CTAs per
// (sequence, head), 16, 32 or 64 value columns each.  Per chunk (last first) and group of 16 columns (transposed, see pkda_scan.cuh):
//   chain warp    d     = bf16(dS)                      registers, A operand as they stand
//                 dF^T  = d^T kg^T + dO^T P             64 + 20 mma.sync
//                 dE    = -beta * bf16(dF)              registers, A operand as they stand
//                 dS^T  = Gam_last dS^T + dO^T qg + dE^T W     64 + 64 mma.sync
//   store warp    stores d (the saved dh) and dF
//   copy warp     kg, W, qg, dO, P, beta, Gam_last by TMA, up to three chunks ahead
// The chain warp leaves d and dF for the store warp in shared memory, two slots deep.  T = 4096, 24 units:
// 163 -> 109 us.  Every wait is bounded.
// Rows of a ragged last chunk past its end hold the next sequence's tokens (or zero fill past the end of
// the tensor): dO is masked there, beta is zero there, nothing else of those rows reaches a kept result.
#include "pkda_scan.cuh"

namespace pkda {

struct ScanBwdColsParams {
  Geo geo;
  const float *beta_c, *gc, *dST;
  bf16 *dh, *dF;
  float* dS0;
  int* status;
  int beside;  // the recompute pass's scan, launched in front of this one, may still run
};

// NW: column groups (of 16) per CTA.
template <int NW> struct ScanBwdLay {
  static constexpr int kSplit = 8 / NW;               // CTAs per unit
  static constexpr int kThreads = 32 * (2 * NW + 1);
  static constexpr int oKg = 0, oW = oKg + scanw::kTile, oQg = oW + scanw::kTile, oDo = oQg + scanw::kTile;  // dO: one block
  static constexpr int oP = oDo + scanw::kBlk, oBeta = oP + scanw::kBlk, oGc = oBeta + 256;
  static constexpr int kTx = oGc + 512;
  static constexpr int kStage = (kTx + 1023) / 1024 * 1024;
  static constexpr int kStages = NW == 4 ? 2 : 3;
  static constexpr int kSlot = 4096 + 2048;           // d and dF fragments of one group
  static constexpr int oSlots = kStages * kStage;     // [NW][2]
  static constexpr int oBar = oSlots + NW * 2 * kSlot;
  static constexpr int kSmem = oBar + 8 * (2 * kStages + 4 * NW) + 1024;
  static_assert(kSmem <= 232448, "shared memory of one SM");
};

template <int NW>
__global__ void __launch_bounds__(ScanBwdLay<NW>::kThreads, 1)
pkda_scan_bwd_cols_kernel(const __grid_constant__ CUtensorMap tm_kg, const __grid_constant__ CUtensorMap tm_w,
                          const __grid_constant__ CUtensorMap tm_qg, const __grid_constant__ CUtensorMap tm_do,
                          const __grid_constant__ CUtensorMap tm_p, const ScanBwdColsParams p) {
  if (!p.beside) wait_prerequisites();
  launch_dependents();
  using namespace scanw;
  using Y = ScanBwdLay<NW>;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* const sm = smem_raw + (base - smem_u32(smem_raw));
  const int unit = blockIdx.x / Y::kSplit, grp0 = (blockIdx.x % Y::kSplit) * NW;
  const int H = p.geo.heads, n = unit / H, h = unit - n * H;
  const SeqInfo sq = seq_info(p.geo, n);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto bar_full = [&](int s) { return base + Y::oBar + 8 * s; };
  auto bar_empty = [&](int s) { return base + Y::oBar + 8 * (Y::kStages + s); };
  auto bar_ready = [&](int w, int s) { return base + Y::oBar + 8 * (2 * Y::kStages + 4 * w + s); };
  auto bar_free = [&](int w, int s) { return base + Y::oBar + 8 * (2 * Y::kStages + 4 * w + 2 + s); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < Y::kStages; ++s) {
      tc::mbar_init(bar_full(s), 1);
      tc::mbar_init(bar_empty(s), NW);
    }
    for (int w = 0; w < NW; ++w)
      for (int s = 0; s < 2; ++s) {
        tc::mbar_init(bar_ready(w, s), 1);
        tc::mbar_init(bar_free(w, s), 1);
      }
    tc::fence_barrier_init();
  }
  __syncthreads();
  bool ok = true;
  const int last = sq.nchunks - 1;  // j counts processed chunks, chunk index = last - j

  if (warp == 2 * NW) {
    // ---------------------------------------------------------------- the copies
    if (lane == 0) {
      for (int j = 0; j < sq.nchunks; ++j) {
        const int s = j % Y::kStages, i = last - j;
        if (j >= Y::kStages && !tc::mbar_wait(bar_empty(s), (j / Y::kStages - 1) & 1)) { ok = false; break; }
        const uint32_t st = base + s * Y::kStage, bar = bar_full(s);
        const int tok0 = sq.bos + i * kChunk;
        const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
        tc::mbar_expect_tx(bar, Y::kTx);
        tma_load_4d(st + Y::oKg, &tm_kg, bar, 0, tok0, 0, h);
        tc::bulk_load(st + Y::oGc, p.gc + chh * kD, 512, bar);
        tma_load_4d(st + Y::oDo, &tm_do, bar, 0, tok0, grp0 >> 2, h);
        tc::tma_load_3d(st + Y::oP, &tm_p, bar, 0, h, tok0);
        tma_load_4d(st + Y::oQg, &tm_qg, bar, 0, tok0, 0, h);
        tc::bulk_load(st + Y::oBeta, p.beta_c + chh * kChunk, 256, bar);
        tma_load_4d(st + Y::oW, &tm_w, bar, 0, tok0, 0, h);
      }
      if (!ok) atomicExch(p.status, 1);
    }
    return;
  }

  const Lane L(lane);
  const int cw = warp % NW;
  const int v0 = 16 * (grp0 + cw), piece = 2 * ((grp0 + cw) & 3);
  unsigned char* const slot0 = sm + Y::oSlots + cw * 2 * Y::kSlot + 16 * lane;
  const size_t gld = (size_t)H * kD;
  // fragments of P (k = tok', n = tok), k step jj: only column tiles up to the k step's own
  auto load_p = [&](Frags& b, uint32_t tile, const Lane& l, int jj) {
#pragma unroll
    for (int np = 0; np < 4; ++np)
      if (np <= jj) ldb_t(b.r[np], tile, l, jj, np);
  };

  if (warp >= NW) {
    // ----------------------------------------------------------------------- the stores
    for (int j = 0; j < sq.nchunks; ++j) {
      const int i = last - j;
      const unsigned char* sl = slot0 + (j & 1) * Y::kSlot;
      const int tok0 = sq.bos + i * kChunk, valid = min(kChunk, sq.len - i * kChunk);
      const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
      ok = tc::mbar_wait(bar_ready(cw, j & 1), (j >> 1) & 1);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      uint32_t a[8][4], e[4][4];
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) get4(sl + ks * 512, a[ks]);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) get4(sl + 4096 + jj * 512, e[jj]);
      warp_arrive(bar_free(cw, j & 1), lane);
#pragma unroll
      for (int ks = 0; ks < 8; ks += 2)
        store_a2(p.dh + (chh * kD + 16 * ks + L.g) * kD + v0, 8 * kD, 0, kD, a[ks], a[ks + 1], L.t);
#pragma unroll
      for (int jj = 0; jj < 4; jj += 2)
        store_a2(p.dF + ((size_t)(tok0 + 16 * jj + L.g) * H + h) * kD + v0, 8 * gld, 16 * jj + L.g, valid, e[jj],
                 e[jj + 1], L.t);
    }
  } else {
    // ------------------------------------------------------------------------ the chain
    float S[16][4];  // dS^T: rows v0 + g, v0 + g + 8, columns k = 8 nt + 2 t, + 1
    const size_t sbase = (size_t)unit * kD * kD + v0 + L.g;
#pragma unroll
    for (int nt = 0; nt < 16; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        S[nt][e] = p.dST ? p.dST[sbase + (size_t)(8 * nt + 2 * L.t + (e & 1)) * kD + 8 * (e >> 1)] : 0.f;
    bool tried = false;
    for (int j = 0; j < sq.nchunks; ++j) {
      const int s = j % Y::kStages, i = last - j;
      const uint32_t st = base + s * Y::kStage;
      unsigned char *stp = sm + s * Y::kStage, *sl = slot0 + (j & 1) * Y::kSlot;
      const int valid = min(kChunk, sq.len - i * kChunk);
      // (for the first two chunks the slot is free as it stands: the parity of the phase before the first)
      ok = mbar_wait2(tried, bar_full(s), (j / Y::kStages) & 1, bar_free(cw, j & 1), ((j >> 1) - 1) & 1);
      if (!ok) break;
      Frags b[2];
      load_n(b[0], st + Y::oKg, L, 0);
      uint32_t ad[4][4];  // dO^T as an A operand; nothing past the end of the sequence
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        ld_cols(ad[jj], st + Y::oDo, L, jj, piece);
        if (valid < kChunk) {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int tok = 16 * jj + 8 * (x >> 1) + 2 * L.t;
            if (tok >= valid) ad[jj][x] = 0;
            else if (tok + 1 >= valid) ad[jj][x] &= 0xFFFFu;
          }
        }
      }
      float acc[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t a[4];
        if (ks < 7) load_n(b[(ks + 1) & 1], st + Y::oKg, L, ks + 1);
        else load_p(b[0], st + Y::oP, L, 0);
        pack_a(a, S, ks);
        mma4(acc, a, b[ks & 1]);
        put4(sl + ks * 512, a);
#pragma unroll
        for (int half = 0; half < 2; ++half) {  // dS *= Gam_last
          const float2 gl = get2f(stp + Y::oGc + (16 * ks + 8 * half + 2 * L.t) * 4);
          float(&x)[4] = S[2 * ks + half];
          x[0] *= gl.x; x[1] *= gl.y; x[2] *= gl.x; x[3] *= gl.y;
        }
      }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        if (jj < 3) load_p(b[(jj + 1) & 1], st + Y::oP, L, jj + 1);
        else load_t(b[0], st + Y::oQg, L, 0);
#pragma unroll
        for (int np = 0; np <= jj; ++np) {  // P[tok'][tok] is zero for tok > tok'
          mma_bf16(acc[2 * np], ad[jj], b[jj & 1].r[np][0], b[jj & 1].r[np][1]);
          mma_bf16(acc[2 * np + 1], ad[jj], b[jj & 1].r[np][2], b[jj & 1].r[np][3]);
        }
      }
      update_state(S, ad, st + Y::oQg, L, b[0]);  // (independent of dF: the rounding below runs beside it)
      load_t(b[0], st + Y::oW, L, 0);
      uint32_t f[4][4];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        uint32_t e[4];
        pack_a(e, acc, jj);
        const float2 b0 = get2f(stp + Y::oBeta + (16 * jj + 2 * L.t) * 4), b1 = get2f(stp + Y::oBeta + (16 * jj + 8 + 2 * L.t) * 4);
        const float2 n0 = make_float2(-b0.x, -b0.y), n1 = make_float2(-b1.x, -b1.y);
        f[jj][0] = scale_pair(e[0], n0);
        f[jj][1] = scale_pair(e[1], n0);
        f[jj][2] = scale_pair(e[2], n1);
        f[jj][3] = scale_pair(e[3], n1);
        put4(sl + 4096 + jj * 512, e);
      }
      warp_arrive(bar_ready(cw, j & 1), lane);
      tried = mbar_try2(bar_full((j + 1) % Y::kStages), ((j + 1) / Y::kStages) & 1, bar_free(cw, (j + 1) & 1),
                        (((j + 1) >> 1) - 1) & 1);
      update_state(S, f, st + Y::oW, L, b[0]);
      warp_arrive(bar_empty(s), lane);
    }
    if (ok && p.dS0) {
#pragma unroll
      for (int nt = 0; nt < 16; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          p.dS0[sbase + (size_t)(8 * nt + 2 * L.t + (e & 1)) * kD + 8 * (e >> 1)] = S[nt][e];
    }
  }
  if (!ok && lane == 0) atomicExch(p.status, 1);
  wait_prerequisites();  // (what follows on the stream also reads what a scan beside this one leaves)
}

template <int NW>
static int launch(const CUtensorMap (&tm)[5], const ScanBwdColsParams& sp, int units, cudaStream_t st) {
  using Y = ScanBwdLay<NW>;
  if (!ensure_dynamic_smem(pkda_scan_bwd_cols_kernel<NW>, Y::kSmem)) return PKDA_ERR_LAUNCH;
  return launch_kernel(pkda_scan_bwd_cols_kernel<NW>, units * Y::kSplit, Y::kThreads, Y::kSmem, st, tm[0], tm[1], tm[2], tm[3],
                       tm[4], sp);
}

int launch_scan_bwd_cols(const Geo& geo, int total_tokens, int units, const bf16* kg, const bf16* w, const bf16* qg,
                         const bf16* d_o, const bf16* Aqk, const float* beta_c, const float* gc, const float* dST,
                         bf16* dh, bf16* dF, float* dS0, int* status, int split, bool beside, cudaStream_t st) {
  const uint64_t H = geo.heads, tok = total_tokens;
  CUtensorMap tm[5];
  if (!scanw::rows_map(&tm[0], kg, H, tok, 2) || !scanw::rows_map(&tm[1], w, H, tok, 2) ||
      !scanw::rows_map(&tm[2], qg, H, tok, 2) || !scanw::rows_map(&tm[3], d_o, H, tok, 1) ||
      !scanw::pairs_map(&tm[4], Aqk, H, tok))
    return PKDA_ERR_LAUNCH;
  ScanBwdColsParams sp;
  sp.geo = geo; sp.beta_c = beta_c; sp.gc = gc; sp.dST = dST; sp.dh = dh; sp.dF = dF; sp.dS0 = dS0; sp.status = status;
  sp.beside = beside;
  return split == 8   ? launch<1>(tm, sp, units, st)
         : split == 4 ? launch<2>(tm, sp, units, st)
                      : launch<4>(tm, sp, units, st);
}

}  // namespace pkda
