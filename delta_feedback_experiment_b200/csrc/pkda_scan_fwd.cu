// Forward state scan for few units, with the output formed on the way.  Eight, four or (a recompute pass beside the
// backward's scan) two CTAs per (sequence, head), 16, 32 or 64 value columns each.  Per 64-token chunk and group of 16 columns
// (transposed, see pkda_scan.cuh):
//   chain warp    h    = bf16(S)                   registers, A operand as they stand
//                 S   *= Gam_last (per k)
//                 E^T  = U^T I - h^T W^T           64 + 8 mma.sync
//                 F    = beta * bf16(E)            registers, A operand as they stand
//                 S^T += F^T kg                    64 mma.sync
//   output warp   O^T  = h^T qg^T + E^T (P diag beta)^T   84 mma.sync, stores o
//   store warp    stores h and E (v_new)
//   copy warp     W, kg, U, qg, P, beta, Gam_last by TMA, up to three chunks ahead
// The chain warp leaves h and E for the other two in shared memory, two slots deep.  A step takes 1.05 us with
// one column group per CTA and 1.45 us with two (the SM's shared memory then moves 1,700 of the 2,700 cycles);
// T = 8192, 16 units: 360 -> 141 us, T = 4096, 24 units: 180 -> 100 us.  Every wait is bounded: on a timeout the
// warp sets the status word and leaves.
#include "pkda_scan.cuh"

namespace pkda {

struct ScanFwdParams {
  Geo geo;
  const float *beta_c, *gc, *S0;
  bf16 *h, *v_new;
  float* ST;
  bf16* o;
  int* status;
};

// NW: column groups (of 16) per CTA.
template <int NW, bool kOut> struct ScanFwdLay {
  static constexpr int kSplit = 8 / NW;                      // CTAs per unit
  static constexpr int kReaders = kOut ? 2 : 1;              // of the h / E slots, per group
  static constexpr int kWorkers = NW * (1 + kReaders);
  static constexpr int kStageUsers = NW * (kOut ? 2 : 1);
  static constexpr int kThreads = 32 * (kWorkers + 1);
  static constexpr int oW = 0, oKg = oW + scanw::kTile, oU = oKg + scanw::kTile;  // U: the CTA's 64-column block
  static constexpr int oQg = oU + scanw::kBlk, oP = oQg + (kOut ? scanw::kTile : 0);
  static constexpr int oBeta = oP + (kOut ? scanw::kBlk : 0), oGc = oBeta + 256;
  static constexpr int kTx = oGc + 512;                      // bytes that land per stage
  static constexpr int kStage = (kTx + 1023) / 1024 * 1024;
  static constexpr int kStages = 3;
  static constexpr int kSlot = 4096 + 2048;                  // h and E fragments of one group
  static constexpr int oSlots = kStages * kStage;            // [NW][2]
  static constexpr int oBar = oSlots + NW * 2 * kSlot;       // full, empty [kStages]; ready, free [NW][2]
  static constexpr int kSmem = oBar + 8 * (2 * kStages + 4 * NW) + 1024;
  static_assert(kSmem <= 232448, "shared memory of one SM");
};

template <int NW, bool kOut>
__global__ void __launch_bounds__(ScanFwdLay<NW, kOut>::kThreads, 1)
pkda_scan_fwd_cols_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_kg,
                          const __grid_constant__ CUtensorMap tm_u, const __grid_constant__ CUtensorMap tm_qg,
                          const __grid_constant__ CUtensorMap tm_p, const ScanFwdParams p) {
  after_previous();
  using namespace scanw;
  using Y = ScanFwdLay<NW, kOut>;
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
      tc::mbar_init(bar_empty(s), Y::kStageUsers);
    }
    for (int w = 0; w < NW; ++w)
      for (int s = 0; s < 2; ++s) {
        tc::mbar_init(bar_ready(w, s), 1);
        tc::mbar_init(bar_free(w, s), Y::kReaders);
      }
    tc::fence_barrier_init();
  }
  __syncthreads();
  bool ok = true;

  if (warp == Y::kWorkers) {
    // ---------------------------------------------------------------- the copies
    if (lane == 0) {
      for (int i = 0; i < sq.nchunks; ++i) {
        const int s = i % Y::kStages;
        if (i >= Y::kStages && !tc::mbar_wait(bar_empty(s), (i / Y::kStages - 1) & 1)) { ok = false; break; }
        const uint32_t st = base + s * Y::kStage, bar = bar_full(s);
        const int tok0 = sq.bos + i * kChunk;
        const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
        tc::mbar_expect_tx(bar, Y::kTx);
        tma_load_4d(st + Y::oW, &tm_w, bar, 0, tok0, 0, h);
        tc::bulk_load(st + Y::oGc, p.gc + chh * kD, 512, bar);
        tma_load_4d(st + Y::oU, &tm_u, bar, 0, tok0, grp0 >> 2, h);
        tc::bulk_load(st + Y::oBeta, p.beta_c + chh * kChunk, 256, bar);
        tma_load_4d(st + Y::oKg, &tm_kg, bar, 0, tok0, 0, h);
        if (kOut) {
          tma_load_4d(st + Y::oQg, &tm_qg, bar, 0, tok0, 0, h);
          tc::tma_load_3d(st + Y::oP, &tm_p, bar, 0, h, tok0);
        }
      }
      if (!ok) atomicExch(p.status, 1);
    }
    return;
  }

  const Lane L(lane);
  const int role = warp / NW;                 // 0: chain, 1: output (kOut), last: store
  const int cw = warp - role * NW;            // column group inside the CTA
  const int v0 = 16 * (grp0 + cw);               // first value column of the warp
  const int piece = 2 * ((grp0 + cw) & 3);       // its 16-byte piece inside the 64-column block
  unsigned char* const slot0 = sm + Y::oSlots + cw * 2 * Y::kSlot + 16 * lane;
  const size_t gld = (size_t)H * kD;
  if (role == 0) {
    // ------------------------------------------------------------------------ the chain
    float S[16][4];  // S^T: rows v0 + g, v0 + g + 8, columns k = 8 nt + 2 t, + 1
    const size_t sbase = (size_t)unit * kD * kD + v0 + L.g;
#pragma unroll
    for (int nt = 0; nt < 16; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        S[nt][e] = p.S0 ? p.S0[sbase + (size_t)(8 * nt + 2 * L.t + (e & 1)) * kD + 8 * (e >> 1)] : 0.f;
    const uint32_t one = identity_b(L);
    bool tried = false;
    for (int i = 0; i < sq.nchunks; ++i) {
      const int s = i % Y::kStages;
      const uint32_t st = base + s * Y::kStage;
      unsigned char *stp = sm + s * Y::kStage, *sl = slot0 + (i & 1) * Y::kSlot;
      // (for the first two chunks the slot is free as it stands: the parity of the phase before the first)
      ok = mbar_wait2(tried, bar_full(s), (i / Y::kStages) & 1, bar_free(cw, i & 1), ((i >> 1) - 1) & 1);
      if (!ok) break;
      Frags b[2];
      load_n(b[0], st + Y::oW, L, 0);
      uint32_t u[4][4];
      float acc[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t a[4], na[4];
        if (ks < 7) load_n(b[(ks + 1) & 1], st + Y::oW, L, ks + 1);
        else load_t(b[0], st + Y::oKg, L, 0);  // the state update's first fragments
        if (ks >= 4) ld_cols(u[ks - 4], st + Y::oU, L, ks - 4, piece);
        pack_a(a, S, ks);
#pragma unroll
        for (int x = 0; x < 4; ++x) na[x] = a[x] ^ 0x80008000u;
        mma4(acc, na, b[ks & 1]);
        put4(sl + ks * 512, a);
#pragma unroll
        for (int half = 0; half < 2; ++half) {  // S *= Gam_last
          const float2 gl = get2f(stp + Y::oGc + (16 * ks + 8 * half + 2 * L.t) * 4);
          float(&x)[4] = S[2 * ks + half];
          x[0] *= gl.x; x[1] *= gl.y; x[2] *= gl.x; x[3] *= gl.y;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // + U^T I (the other k steps of these tiles would add zeros)
        mma_bf16(acc[2 * j], u[j], one, 0u);
        mma_bf16(acc[2 * j + 1], u[j], 0u, one);
      }
      uint32_t e[4][4], f[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        pack_a(e[j], acc, j);
        const float2 b0 = get2f(stp + Y::oBeta + (16 * j + 2 * L.t) * 4), b1 = get2f(stp + Y::oBeta + (16 * j + 8 + 2 * L.t) * 4);
        f[j][0] = scale_pair(e[j][0], b0);
        f[j][1] = scale_pair(e[j][1], b0);
        f[j][2] = scale_pair(e[j][2], b1);
        f[j][3] = scale_pair(e[j][3], b1);
        put4(sl + 4096 + j * 512, e[j]);
      }
      warp_arrive(bar_ready(cw, i & 1), lane);
      tried = mbar_try2(bar_full((i + 1) % Y::kStages), ((i + 1) / Y::kStages) & 1, bar_free(cw, (i + 1) & 1),
                        (((i + 1) >> 1) - 1) & 1);
      update_state(S, f, st + Y::oKg, L, b[0]);
      warp_arrive(bar_empty(s), lane);
    }
    if (ok && p.ST) {
#pragma unroll
      for (int nt = 0; nt < 16; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          p.ST[sbase + (size_t)(8 * nt + 2 * L.t + (e & 1)) * kD + 8 * (e >> 1)] = S[nt][e];
    }
  } else {
    // -------------------------------------------------------------- the output and the stores
    // (One loop for both: with a loop of its own for each the chain's step takes 2 to 6% longer.)
    const bool out = kOut && role == 1;
    for (int i = 0; i < sq.nchunks; ++i) {
      const int s = i % Y::kStages;
      const uint32_t st = base + s * Y::kStage;
      const unsigned char *stp = sm + s * Y::kStage, *sl = slot0 + (i & 1) * Y::kSlot;
      const int tok0 = sq.bos + i * kChunk, valid = min(kChunk, sq.len - i * kChunk);
      const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
      if (out) {  // (the chunk's tiles stood before the chain could write its h: the first wait only orders the reads)
        const bool tried = mbar_try2(bar_full(s), (i / Y::kStages) & 1, bar_ready(cw, i & 1), (i >> 1) & 1);
        ok = mbar_wait2(tried, bar_full(s), (i / Y::kStages) & 1, bar_ready(cw, i & 1), (i >> 1) & 1);
      } else {
        // The store warp reads the slots alone.  It is no user of the stages, which go on to later chunks without
        // it, so it must not wait for their barriers: its chunk's phase may be two behind and look like one to come.
        ok = __all_sync(0xffffffffu, tc::mbar_wait(bar_ready(cw, i & 1), (i >> 1) & 1));
      }
      if (!ok) break;
      uint32_t a[8][4], e[4][4];
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) get4(sl + ks * 512, a[ks]);
#pragma unroll
      for (int j = 0; j < 4; ++j) get4(sl + 4096 + j * 512, e[j]);
      if (!out) {
        warp_arrive(bar_free(cw, i & 1), lane);
#pragma unroll
        for (int ks = 0; ks < 8; ks += 2)
          store_a2(p.h + (chh * kD + 16 * ks + L.g) * kD + v0, 8 * kD, 0, kD, a[ks], a[ks + 1], L.t);
#pragma unroll
        for (int j = 0; j < 4; j += 2)
          store_a2(p.v_new + ((size_t)(tok0 + 16 * j + L.g) * H + h) * kD + v0, 8 * gld, 16 * j + L.g, valid, e[j],
                   e[j + 1], L.t);
        continue;
      }
      float acc[8][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
      Frags b[2];
      load_n(b[0], st + Y::oQg, L, 0);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if (ks < 7) load_n(b[(ks + 1) & 1], st + Y::oQg, L, ks + 1);
        else load_n(b[0], st + Y::oP, L, 0);
        mma4(acc, a[ks], b[ks & 1]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 b0 = get2f(stp + Y::oBeta + (16 * j + 2 * L.t) * 4), b1 = get2f(stp + Y::oBeta + (16 * j + 8 + 2 * L.t) * 4);
        if (j < 3) load_n(b[(j + 1) & 1], st + Y::oP, L, j + 1);
        const Frags& pf = b[j & 1];
#pragma unroll
        for (int np = j; np < 4; ++np) {  // P is lower triangular: tokens before the k step's own see none of it
          mma_bf16(acc[2 * np], e[j], scale_pair(pf.r[np][0], b0), scale_pair(pf.r[np][1], b1));
          mma_bf16(acc[2 * np + 1], e[j], scale_pair(pf.r[np][2], b0), scale_pair(pf.r[np][3], b1));
        }
      }
      warp_arrive(bar_free(cw, i & 1), lane);
      if (lane == 0) mbar_arrive(bar_empty(s));
      uint32_t lo[8], hi[8];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        lo[nt] = pack_bf16(acc[nt][0], acc[nt][1]);
        hi[nt] = pack_bf16(acc[nt][2], acc[nt][3]);
      }
      store_pairs<8>(p.o + ((size_t)(tok0 + L.g) * H + h) * kD + v0, 8 * gld, L.g, valid, lo, hi, L.t);
    }
  }
  if (!ok && lane == 0) {
    atomicExch(p.status, 1);
    __threadfence();
  }
  __syncwarp();
  // This is the forward's last kernel when it forms the output.  If any kernel of the call gave up
  // (this one included), the first output row of this (sequence, head) becomes NaN, so that a caller
  // who never reads the status word cannot take a partial result for a complete one.
  if (kOut && role == 1 && sq.len > 0 && *reinterpret_cast<volatile int*>(p.status) != 0 && lane < 16)
    p.o[((size_t)sq.bos * H + h) * kD + v0 + lane] = __float2bfloat16(__int_as_float(0x7fc00000));
}

template <int NW, bool kOut>
static int launch(const CUtensorMap (&tm)[5], const ScanFwdParams& sp, int units, cudaStream_t st) {
  using Y = ScanFwdLay<NW, kOut>;
  if (!ensure_dynamic_smem(pkda_scan_fwd_cols_kernel<NW, kOut>, Y::kSmem)) return PKDA_ERR_LAUNCH;
  return launch_kernel(false, pkda_scan_fwd_cols_kernel<NW, kOut>, units * Y::kSplit, Y::kThreads, Y::kSmem, st, tm[0], tm[1], tm[2], tm[3],
                tm[4], sp);
}

// o == NULL: h, v_new and the final state only.  split: CTAs per unit, 8, 4 or (without o) 2.
int launch_scan_fwd_cols(const Geo& geo, int total_tokens, int units, const bf16* w, const bf16* kg, const bf16* u,
                         const float* beta_c, const float* gc, const float* S0, bf16* h, bf16* v_new, float* ST,
                         int* status, const bf16* qg, const bf16* Aqk, bf16* o, int split, cudaStream_t st) {
  const uint64_t H = geo.heads, tok = total_tokens;
  CUtensorMap tm[5];
  if (!scanw::rows_map(&tm[0], w, H, tok, 2) || !scanw::rows_map(&tm[1], kg, H, tok, 2) ||
      !scanw::rows_map(&tm[2], u, H, tok, 1) || !scanw::rows_map(&tm[3], o ? qg : w, H, tok, 2))
    return PKDA_ERR_LAUNCH;
  if (o) {
    if (!scanw::pairs_map(&tm[4], Aqk, H, tok)) return PKDA_ERR_LAUNCH;
  } else {
    tm[4] = tm[3];  // unused
  }
  ScanFwdParams sp;
  sp.geo = geo; sp.beta_c = beta_c; sp.gc = gc; sp.S0 = S0; sp.h = h; sp.v_new = v_new; sp.ST = ST; sp.o = o;
  sp.status = status;
  if (o) return split == 8 ? launch<1, true>(tm, sp, units, st) : launch<2, true>(tm, sp, units, st);
  return split == 8   ? launch<1, false>(tm, sp, units, st)
         : split == 4 ? launch<2, false>(tm, sp, units, st)
                      : launch<4, false>(tm, sp, units, st);
}

}  // namespace pkda
