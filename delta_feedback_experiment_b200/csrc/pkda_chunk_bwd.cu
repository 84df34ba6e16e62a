// Chunked PKDA backward for D = 128, chunk 64, bf16 activations.
//
// With the forward's per-chunk quantities (see pkda_chunk_fwd.cu)
//   E = Tm (V - Kd S0), F = beta E, O = qg S0 + P F, S1 = Gam_last S0 + kg^T F
// the cotangents are
//   dF = kg dS1 + P^T dO,  dE = beta dF,  dS0 = Gam_last dS1 + qg^T dO - W^T dE
//   dR = Tm^T dE (= dV),  dKd = -dR S0^T,  d(tril M) = -tril(dR E^T) diag(beta)
//   dP = scale tril(dO F^T),  dkg = F dS1^T,  dqg = dO S0^T
// and the gated pair products are differentiated strip by strip with the same
// rounded operands on both sides, so that each pair's +/- contributions to the
// log-decay gradient cancel exactly under the reverse cumulative sum.
//
// Pipeline:  [recompute forward stages]  scan_bwd (sequential over chunks)
//   -> intra_bwd (per chunk; the preconditioner's reverse scan inside it too) -> atk_bwd
//   carry / final (the same over chunks) -> param_reduce.
#include <algorithm>

#include "pkda_chunk.cuh"
#include "pkda_tc.cuh"

namespace pkda {

// ------------------------------------------------------------------ reverse state scan
struct ScanBwdParams {
  Geo geo;
  const bf16 *kg, *qg, *w, *Aqk, *d_o;
  const float *beta_c, *gc;
  const float* dST;
  bf16 *dh, *dF;
  float* dS0;
};

namespace scanb {
template <int VB> __host__ __device__ constexpr int threads() { return 128 * (VB / 32); }  // 4 warps per 32 value columns
template <int VB> struct L {
  static constexpr int ldv = VB + kPad;
  static constexpr int oKg = 0;
  static constexpr int oP = oKg + kTileBytes;            // bf16 [64][72]
  static constexpr int oBeta = oP + kChunk * kLdC * 2;   // f32 [64]
  static constexpr int oQg = oBeta + kChunk * 4;
  static constexpr int oW = oQg + kTileBytes;
  static constexpr int oGc = oW + kTileBytes;            // f32 [128]
  static constexpr int oDo = oGc + kD * 4;               // 2 x bf16 [64][ldv]
  static constexpr int kDoBytes = kChunk * ldv * 2;
  static constexpr int oD = oDo + 2 * kDoBytes;          // bf16 [128][ldv]
  static constexpr int oDE = oD + kD * ldv * 2;          // bf16 [64][ldv]
  static constexpr int kSmem = oDE + kChunk * ldv * 2;
};
}  // namespace scanb

template <int VB>
__global__ void __launch_bounds__(scanb::threads<VB>())
pkda_scan_bwd_kernel(const ScanBwdParams p) {
  after_previous();
  using Lay = scanb::L<VB>;
  constexpr int ldv = Lay::ldv, NT = 4, kT = scanb::threads<VB>();
  extern __shared__ __align__(128) unsigned char smem[];
  const int VS = kD / VB;
  const int vs = blockIdx.x % VS;
  const int nh = blockIdx.x / VS;
  const int n = nh / p.geo.heads, h = nh - n * p.geo.heads, H = p.geo.heads;
  const SeqInfo sq = seq_info(p.geo, n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int wr = warp & 3, c0 = 32 * (warp >> 2);  // this warp: rows [32 wr, +32), columns [c0, +32) of the slice
  const int v0 = vs * VB;
  const long gld = (long)H * kD;
  const size_t sbase = ((size_t)n * H + h) * kD * kD;

  bf16* sKg = reinterpret_cast<bf16*>(smem + Lay::oKg);
  bf16* sP = reinterpret_cast<bf16*>(smem + Lay::oP);
  float* sBeta = reinterpret_cast<float*>(smem + Lay::oBeta);
  bf16* sQg = reinterpret_cast<bf16*>(smem + Lay::oQg);
  bf16* sW = reinterpret_cast<bf16*>(smem + Lay::oW);
  float* sGc = reinterpret_cast<float*>(smem + Lay::oGc);
  bf16* sD = reinterpret_cast<bf16*>(smem + Lay::oD);
  bf16* sDE = reinterpret_cast<bf16*>(smem + Lay::oDE);

  auto prefetchA = [&](int i) {
    const int tok0 = sq.bos + i * kChunk;
    const int valid = min(kChunk, sq.len - i * kChunk);
    const size_t row0 = ((size_t)tok0 * H + h) * kD;
    const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
    tile_load_async(sKg, kLdD, p.kg + row0, gld, kChunk, kD, valid, kT);
    tile_load_async(sP, kLdC, p.Aqk + ((size_t)tok0 * H + h) * kChunk, (long)H * kChunk, kChunk, kChunk, valid,
                    kT);
    tile_load_async(reinterpret_cast<bf16*>(smem + Lay::oDo + (i & 1) * Lay::kDoBytes), ldv, p.d_o + row0 + v0, gld,
                    kChunk, VB, valid, kT);
    if (tid < 16) cp_async16(smem + Lay::oBeta + tid * 16, p.beta_c + chh * kChunk + tid * 4, true);
  };
  auto prefetchB = [&](int i) {
    const int tok0 = sq.bos + i * kChunk;
    const int valid = min(kChunk, sq.len - i * kChunk);
    const size_t row0 = ((size_t)tok0 * H + h) * kD;
    const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
    tile_load_async(sQg, kLdD, p.qg + row0, gld, kChunk, kD, valid, kT);
    tile_load_async(sW, kLdD, p.w + row0, gld, kChunk, kD, valid, kT);
    if (tid < 32) cp_async16(smem + Lay::oGc + tid * 16, p.gc + chh * kD + tid * 4, true);
  };

  float dS[2][NT][4];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = 32 * wr + 16 * mt + gq + 8 * half, c = v0 + c0 + 8 * nt + 2 * tq;
        float2 s2 = make_float2(0.f, 0.f);
        if (p.dST) s2 = *reinterpret_cast<const float2*>(p.dST + sbase + (size_t)r * kD + c);
        dS[mt][nt][2 * half] = s2.x;
        dS[mt][nt][2 * half + 1] = s2.y;
      }

  const int last = sq.nchunks - 1;
  if (last >= 0) {
    prefetchA(last);
    cp_async_commit();
    prefetchB(last);
    cp_async_commit();
  }
  for (int i = last; i >= 0; --i) {
    const int tok0 = sq.bos + i * kChunk;
    const int valid = min(kChunk, sq.len - i * kChunk);
    const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
    const bf16* sdO = reinterpret_cast<const bf16*>(smem + Lay::oDo + (i & 1) * Lay::kDoBytes);
    cp_async_wait<1>();  // group A(i) has landed
    // a. chunk-exit state cotangent -> bf16 operand tile (and the saved dh)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 32 * wr + 16 * mt + gq + 8 * half, c = c0 + 8 * nt + 2 * tq;
          *reinterpret_cast<uint32_t*>(sD + r * ldv + c) = pack_bf16(dS[mt][nt][2 * half], dS[mt][nt][2 * half + 1]);
        }
    __syncthreads();
    {
      constexpr int cpr = VB / 8;
      for (int j = tid; j < kD * cpr; j += kT) {
        const int r = j / cpr, c = (j - r * cpr) * 8;
        *reinterpret_cast<uint4*>(p.dh + (chh * kD + r) * kD + v0 + c) =
            *reinterpret_cast<const uint4*>(sD + r * ldv + c);
      }
    }
    // c. dF = kg dS1 + P^T dO ;  -dE = -beta dF
    {
      float f[1][NT][4];
      zero_acc(f);
      warp_gemm<1, NT, false, true>(f, sKg, kLdD, 16 * wr, sD, ldv, c0, 0, kD);
      warp_gemm<1, NT, true, true>(f, sP, kLdC, 16 * wr, sdO, ldv, c0, 16 * wr, kChunk);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 16 * wr + gq + 8 * half, c = c0 + 8 * nt + 2 * tq;
          const uint32_t fk = pack_bf16(f[0][nt][2 * half], f[0][nt][2 * half + 1]);
          if (r < valid) *reinterpret_cast<uint32_t*>(p.dF + ((size_t)(tok0 + r) * H + h) * kD + v0 + c) = fk;
          const float2 fr = unpack_bf16(fk);
          const float b = sBeta[r];
          *reinterpret_cast<uint32_t*>(sDE + r * ldv + c) = pack_bf16(-b * fr.x, -b * fr.y);
        }
    }
    __syncthreads();  // group-A buffers free
    if (i > 0) prefetchA(i - 1);
    cp_async_commit();
    cp_async_wait<1>();  // group B(i) has landed
    __syncthreads();
    // d. dS0 = Gam_last dS1 + qg^T dO - W^T dE
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float gcv = sGc[32 * wr + 16 * mt + gq + 8 * half];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          dS[mt][nt][2 * half] *= gcv;
          dS[mt][nt][2 * half + 1] *= gcv;
        }
      }
    warp_gemm<2, NT, true, true>(dS, sQg, kLdD, 32 * wr, sdO, ldv, c0, 0, kChunk);
    warp_gemm<2, NT, true, true>(dS, sW, kLdD, 32 * wr, sDE, ldv, c0, 0, kChunk);
    __syncthreads();  // group-B buffers, sD and sDE free
    if (i > 0) prefetchB(i - 1);
    cp_async_commit();
  }
  cp_async_wait<0>();
  if (p.dS0) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 32 * wr + 16 * mt + gq + 8 * half, c = v0 + c0 + 8 * nt + 2 * tq;
          *reinterpret_cast<float2*>(p.dS0 + sbase + (size_t)r * kD + c) =
              make_float2(dS[mt][nt][2 * half], dS[mt][nt][2 * half + 1]);
        }
  }
}

// ------------------------------------------------------------------ chunk-parallel backward
// Tensor maps of the phase-A tiles.  Each box is wider than the data it needs (136
// or 72 columns for 128 or 64) so that the rows land in shared memory with the
// padded pitch the ldmatrix reads want; the surplus columns are the neighbouring
// head's data or, past the end of a row, zero fill.
// The four output maps are [token][head][channel] with a box of one head and 136
// columns: a store clips the eight columns past the head, so the padded pitch of
// the shared-memory tile never reaches the neighbouring head.
struct IntraBwdMaps {
  CUtensorMap d_o, dF, h, dh, Akk, E;
  CUtensorMap q, k, kt, g;
  CUtensorMap dq, dv, dk_read, dkt;
};

namespace ib {
constexpr int kThreads = 512;
constexpr int oA0 = 0;                        // dO          | later q
constexpr int oA1 = kTileBytes;               // S0 [128][136] | E | later k, kt
constexpr int oG = oA1 + 2 * kTileBytes;      // f32 [64][kLdG] log2-domain cumulative decay
constexpr int oTm = oG + kChunk * kLdG * 4;   // bf16 [64][72]
constexpr int oDE = oTm + kChunk * kLdC * 2;  // dE | later F = beta E
constexpr int oDR = oDE + kTileBytes;
constexpr int oStage = oTm;                   // the gated q and k tiles, then the strip factors | later dG f32 [64][128]
constexpr int oStrip = oStage + 2 * kTileBytes;  // f32 [36][128]
constexpr int oDP = oStrip + 36 * kD * 4;     // bf16 [64][72]
constexpr int oDM = oDP + kChunk * kLdC * 2;
constexpr int oFac = oDM + kChunk * kLdC * 2; // f32 [64][kLdY]: kt 2^(z - G)
constexpr int kLdY = kD + 4;                  // = 4 (mod 32): rows 2 t and channels g of a fragment lie in different banks
constexpr int oSmall = oFac + kChunk * kLdG * 4;
// small: beta[64] db[64] hdh[128] gcv[128] col[4][128] rb[4][64] red[16] bias[2][128] worst[4][3] diag[64] there[36]
constexpr int kSmallFloats = 64 + 64 + 128 + 128 + 512 + 256 + 16 + 256 + 12 + 64 + 36;
constexpr int oBar = oSmall + kSmallFloats * 4;  // three mbarriers: the tiles of phase A, those of phase B, what comes ahead
constexpr int oRaw = (oBar + 32 + 127) / 128 * 128;  // bf16 [64][136]: the raw gate of a full chunk, asked for while the item before ends
constexpr int kSmem = oRaw + kTileBytes;
static_assert(kSmem <= 232448, "shared memory of one SM");
// A copy takes its issuing thread some 500 cycles, so every one has a warp of its own (the first lane arrives with its bytes).
constexpr int kCopiesA = 6, kCopiesB = 3, kCopiesAhead = 2;
static_assert(2 * kChunk * kLdC * 2 >= kTileBytes && oDP % 128 == 0, "E waits in the pair-gradient tiles");
static_assert(oBar % 8 == 0 && oA1 % 128 == 0 && oTm % 128 == 0 && oDE % 128 == 0 && oFac % 128 == 0,
              "TMA destinations and the mbarrier must be aligned");
static_assert(oDR + kTileBytes <= oDP, "phase-A tiles must not reach the pair-gradient tiles");
static_assert(oDE + kD * kLdD * 2 <= oDP, "dS1 tile must fit");
// The preconditioner's part: what its row blocks exchange, in a region that is dead after the pairs.
constexpr int kAtkBlocks = kThreads / 32, kAtkRows = kChunk / kAtkBlocks;  // one row block per warp
constexpr int oAtkEx = oDP;    // f32: end[16][128] part[16][128] dec[16] centre[16]
static_assert((2 * kAtkBlocks * kD + 2 * kAtkBlocks) * 4 <= 2 * kChunk * kLdC * 2,
              "dead region");

// ---- The local part of the preconditioner's backward, with the chunk's dkt and dk_read still in shared memory:
//   dkt <- dA_local = d(loss)/dA_t through the write-key factor B alone,  dk_read <- dk_read + dkt B,
//   the chunk's outgoing carry sum_r (prod_{j<=r} decay_j) dA_local_r and its share of the centre gradient.
// Warp w owns rows 4 w .. 4 w + 3, lane l channels 4 l .. 4 l + 3, and the scan A_t = decay_t A_(t-1) + beta_t k_t^2 is
// blocked: the row blocks exchange (decay product, end value).  Five special-function operations an element
// (2,600 cycles of the unit per chunk), while the gradients' reverse sum runs on four of the warps.  Against a kernel of its own,
// which read both gradients and k again and wrote the gradients a second time (225 MB in 37 us for 1,536 chunks): this kernel
// 253 -> 281 us, the pass 838 -> 829 us.  (Plain row stores instead of TMA from the tiles: 284.)
struct AtkIn {
  uint2 k[kAtkRows];
  float4 a0;      // the state in front of the chunk
  float lg, beta; // of row lane % 4 of the warp's
  float centre;
};
__device__ __forceinline__ void atk_request(AtkIn& a, const IntraBwdParams& p, size_t chh, int tok0, int valid, int h, int w,
                                            int lane) {
  const int r = kAtkRows * w + (lane & (kAtkRows - 1));
  a.lg = a.beta = 0.f;  // rows past the end: decay 1, beta 0: the state passes through
  if (r < valid) {
    const size_t s = (size_t)(tok0 + r) * p.geo.heads + h;
    a.lg = p.g_atk[s];
    a.beta = __bfloat162float(p.beta_atk[s]);
  }
  a.centre = p.log_atk_scale[h];
  a.a0 = *reinterpret_cast<const float4*>(p.a_start + chh * kD + 4 * lane);
}
// Before the barrier: the row block's end value from a zero start.
__device__ __forceinline__ void atk_block_end(const AtkIn& in, int w, int lane, float* ex) {
  const int c4 = 4 * lane;
  const float pd_l = __expf(in.lg);
  float A[4] = {0.f, 0.f, 0.f, 0.f}, dblk = 1.f;
#pragma unroll
  for (int i = 0; i < kAtkRows; ++i) {
    const float2 x = unpack_bf16(in.k[i].x), y = unpack_bf16(in.k[i].y);
    const float kc[4] = {x.x, x.y, y.x, y.y};
    const float pd = __shfl_sync(0xffffffffu, pd_l, i), bp = __shfl_sync(0xffffffffu, in.beta, i);
    dblk *= pd;
#pragma unroll
    for (int e = 0; e < 4; ++e) A[e] = pd * A[e] + bp * kc[e] * kc[e];
  }
  *reinterpret_cast<float4*>(ex + w * kD + c4) = make_float4(A[0], A[1], A[2], A[3]);
  if (lane == 0) ex[2 * kAtkBlocks * kD + w] = dblk;
}
// Behind it: the true states, the gradients.
__device__ __forceinline__ void atk_local(const AtkIn& in, const IntraBwdParams& p, size_t row0, long gld, int valid, int w,
                                          int lane, float* sOutKt, float* sOutK, float* ex, bool out_tma) {
  const int r0 = kAtkRows * w, c4 = 4 * lane;
  const float pd_l = __expf(in.lg);
  float* const sDec = ex + 2 * kAtkBlocks * kD;
  float A[4] = {in.a0.x, in.a0.y, in.a0.z, in.a0.w};
#pragma unroll 4
  for (int b = 0; b < w; ++b) {  // the state before this block's first row
    const float d = sDec[b];
    const float4 e4 = *reinterpret_cast<const float4*>(ex + b * kD + c4);
    A[0] = d * A[0] + e4.x; A[1] = d * A[1] + e4.y; A[2] = d * A[2] + e4.z; A[3] = d * A[3] + e4.w;
  }
  float wt = 1.f, part[4] = {0.f, 0.f, 0.f, 0.f}, dc = 0.f;
#pragma unroll
  for (int i = 0; i < kAtkRows; ++i) {
    const int r = r0 + i;
    const bool ok = r < valid;
    const float2 x = unpack_bf16(in.k[i].x), y = unpack_bf16(in.k[i].y);
    const float kc[4] = {x.x, x.y, y.x, y.y};
    const float pd = __shfl_sync(0xffffffffu, pd_l, i), bp = __shfl_sync(0xffffffffu, in.beta, i);
    float4 dkt_i = *reinterpret_cast<float4*>(sOutKt + r * kLdG + c4), dkr_i = *reinterpret_cast<float4*>(sOutK + r * kLdG + c4);
    float* dk_t = reinterpret_cast<float*>(&dkt_i);
    float* dk_r = reinterpret_cast<float*>(&dkr_i);
    wt *= pd;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float An = pd * A[e] + bp * kc[e] * kc[e];
      const float dev = __logf(An + p.eps) - in.centre;
      const float rden = __fdividef(1.f, 1.f + fabsf(dev));
      const float Bf = __expf(-p.ln_x * dev * rden);
      const float ddev = -p.ln_x * dk_t[e] * kc[e] * Bf * rden * rden;
      dk_r[e] += dk_t[e] * Bf;
      dk_t[e] = ok ? __fdividef(ddev, An + p.eps) : 0.f;
      if (ok) dc -= ddev;
      part[e] += wt * dk_t[e];
      A[e] = An;
    }
    if (out_tma) {
      *reinterpret_cast<float4*>(sOutKt + r * kLdG + c4) = dkt_i;
      *reinterpret_cast<float4*>(sOutK + r * kLdG + c4) = dkr_i;
    } else if (ok) {
      *reinterpret_cast<float4*>(p.dkt + row0 + (size_t)r * gld + c4) = dkt_i;
      *reinterpret_cast<float4*>(p.dk_read + row0 + (size_t)r * gld + c4) = dkr_i;
    }
  }
  *reinterpret_cast<float4*>(ex + (kAtkBlocks + w) * kD + c4) = make_float4(part[0], part[1], part[2], part[3]);
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) dc += __shfl_xor_sync(0xffffffffu, dc, o);
  if (lane == 0) sDec[kAtkBlocks + w] = dc;
}
// Behind a barrier: one thread per channel.
__device__ __forceinline__ void atk_carry(const float* ex, const IntraBwdParams& p, size_t chh, int c) {
  const float* const sDec = ex + 2 * kAtkBlocks * kD;
  float acc = 0.f, wt = 1.f, dc = 0.f;
#pragma unroll 4
  for (int b = 0; b < kAtkBlocks; ++b) {
    acc += wt * ex[(kAtkBlocks + b) * kD + c];
    wt *= sDec[b];
    dc += sDec[kAtkBlocks + b];
  }
  p.c_loc[chh * kD + c] = acc;
  if (c == 0) p.partC[chh] = dc;
}
}  // namespace ib

// Chunk, head, first token and valid tokens of an item (chunk * heads + head); chunk -1 for none.  Packed: all lanes of a warp
// together.
__device__ __forceinline__ int4 describe_item(const Geo& geo, int item) {
  int n, tok0, valid;
  const int chunk = item / geo.heads;
  if (item < 0 || !chunk_lookup_warp(geo, chunk, n, tok0, valid)) return make_int4(-1, 0, 0, 0);
  return make_int4(chunk, item - chunk * geo.heads, tok0, valid);
}
// What a full chunk needs first, asked for while the item before it ends: the raw gate, beta, Gam_last and the gate's bias.  All of it
// lands in shared memory: in registers, the tail of the item before waited for it.  phase: the barrier's for that chunk.  With the
// next item drawn on the way and a warp for every copy, the first 8,000 of an item's 47,000 cycles are 5,000 (1,408 items 289 -> 280 us,
// 256 92 -> 86, 7,168 1,300 -> 1,276).
__device__ __forceinline__ void intra_bwd_ahead(const IntraBwdParams& p, const IntraBwdMaps& maps, int4 it, uint32_t phase) {
  using namespace ib;
  extern __shared__ __align__(128) unsigned char smem[];
  if (it.x < 0 || !p.use_tma || it.w != kChunk) return;
  const int tid = threadIdx.x, h = it.y;
  const uint32_t bar = smem_u32(smem + oBar) + 16;
  float* sBeta = reinterpret_cast<float*>(smem + oSmall);
  if (tid == kThreads - 64) {
    tc::mbar_expect_tx(bar, kTileBytes);
    tc::tma_load_2d(smem_u32(smem + oRaw), &maps.g, bar, h * kD, it.z);
  }
  if (tid == kThreads - 96) {
    const size_t chh = (size_t)it.x * p.geo.heads + h;
    tc::mbar_expect_tx(bar, (kChunk + kD) * 4);
    tc::bulk_load(smem_u32(sBeta), p.beta_c + chh * kChunk, kChunk * 4, bar);
    tc::bulk_load(smem_u32(sBeta + 256), p.gc + chh * kD, kD * 4, bar);
  }
  if (tid >= kD && tid < 2 * kD)  // (dt_bias may start at any float)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(sBeta + 64 + 64 + 128 + 128 + 512 + 256 + 16 + phase * kD + tid - kD)),
                 "l"(p.dt_bias + h * kD + tid - kD));
  cp_async_commit();
}

// The item in s_next (chunk, head, first token, valid tokens); every thread of the CTA takes part.  With a work list one thread draws
// the CTA's next item near the end, in steps that nothing waits for, and leaves it in s_next (chunk -1: none).  (Drawn early, the last turn
// is less even: 290 -> 302 us for 1,408 items.)  A word behind the barriers holds their phase, which changes with every full chunk; in a
// register it cost spills and the whole gain.
__device__ __forceinline__ void intra_bwd_item(const IntraBwdParams& p, const IntraBwdMaps& maps, int4* s_next) {
  using namespace ib;
  extern __shared__ __align__(128) unsigned char smem[];
  bf16* sdO = reinterpret_cast<bf16*>(smem + oA0);
  bf16* sS0 = reinterpret_cast<bf16*>(smem + oA1);
  bf16* sE = reinterpret_cast<bf16*>(smem + oA1);
  bf16* sF = reinterpret_cast<bf16*>(smem + oDE);  // F = beta E takes the dE tile once that is dead
  float* sG = reinterpret_cast<float*>(smem + oG);
  bf16* sTm = reinterpret_cast<bf16*>(smem + oTm);
  bf16* sdE = reinterpret_cast<bf16*>(smem + oDE);
  bf16* sdR = reinterpret_cast<bf16*>(smem + oDR);
  bf16* sdP = reinterpret_cast<bf16*>(smem + oDP);
  bf16* sdM = reinterpret_cast<bf16*>(smem + oDM);
  float* sY = reinterpret_cast<float*>(smem + oFac);
  float* sStrip = reinterpret_cast<float*>(smem + oStrip);
  float* sBeta = reinterpret_cast<float*>(smem + oSmall);
  float* sDb = sBeta + 64;
  float* sHdh = sDb + 64;
  float* sGcv = sHdh + 128;
  float* sCol = sGcv + 128;  // [4][128]
  float* sRb = sCol + 512;   // [4][64]
  float* sRed = sRb + 256;   // [16]
  float* sWorst = sRed + 16 + 256;    // [4][3]
  float* sDiag = sWorst + 12;     // [64] diagonal of dP
  int* sThere = reinterpret_cast<int*>(sDiag + 64);  // [36]

  volatile uint32_t* const s_phase = reinterpret_cast<volatile uint32_t*>(smem + oBar + 24);
  const int bx = s_next->x, h = s_next->y, tok0 = s_next->z, valid = s_next->w, H = p.geo.heads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int I = warp & 3, cq = warp >> 2;
  const size_t chh = (size_t)bx * H + h;
  const size_t row0 = ((size_t)tok0 * H + h) * kD;
  const long gld = (long)H * kD;
  const size_t crow0 = ((size_t)tok0 * H + h) * kChunk;
  const long cld = (long)H * kChunk;

  // ================= phase A: state-coupled terms =================
  const bool by_tma = p.use_tma && valid == kChunk;
  const bool drawer = p.slow_list && tid == kThreads - 32;
  // (a ragged chunk takes the half of the bias that the full chunk behind it does not)
  auto bias = [&]() { return sRed + 16 + (by_tma ? *s_phase : *s_phase ^ 1) * kD; };  // [128]
  GateRaw<kThreads> graw;
  float s_small = 0.f;
  if (!by_tma) {
    if (tid < kChunk) s_small = p.beta_c[chh * kChunk + tid];
    else if (tid >= 2 * kD && tid < 3 * kD) s_small = p.gc[chh * kD + tid - 2 * kD];
    else if (tid >= kD && tid < 2 * kD) s_small = p.dt_bias[h * kD + tid - kD];
    gate_load(graw, p.g + row0, gld, valid, tid);
  }
  // dS1 waits where the strips' kt goes later until the dkg product, E in the (not yet
  // used) pair-gradient tiles until S0 has left the tile E belongs in
  bf16* sdSC = reinterpret_cast<bf16*>(smem + oFac);
  bf16* sEarly = reinterpret_cast<bf16*>(smem + oDP);
  // Full chunks: six warps start a TMA tile copy each and everybody goes on to the
  // gate computation while they land.  Ragged chunks (rows past the sequence end must
  // read as zero) take 16-byte cp.async copies.
  const bool out_tma = by_tma && p.out_tma;  // gradients of full chunks leave by TMA from padded tiles
  const uint32_t bar = smem_u32(smem + oBar), bar_b = bar + 8;
  auto copy = [&](uint32_t b, const void* dst, const CUtensorMap* map, int bytes, int c0, int c1) {
    tc::mbar_expect_tx(b, bytes);
    tc::tma_load_2d(smem_u32(dst), map, b, c0, c1);
  };
  if (by_tma) {
    if (lane == 0) {
      switch (warp) {
        case 0: copy(bar, sdO, &maps.d_o, kTileBytes, h * kD, tok0); break;
        case 1: copy(bar, sS0, &maps.h, 2 * kTileBytes, 0, (int)(chh * kD)); break;
        case 2: copy(bar, sTm, &maps.Akk, kChunk * kLdC * 2, h * kChunk, tok0); break;
        case 3: copy(bar, sdE, &maps.dF, kTileBytes, h * kD, tok0); break;  // raw dF; scaled by beta below
        case 4: copy(bar, sdSC, &maps.dh, 2 * kTileBytes, 0, (int)(chh * kD)); break;
        case 5: copy(bar, sEarly, &maps.E, kTileBytes, h * kD, tok0); break;
        default: break;
      }
    }
  } else {
    tile_load_async(sdO, kLdD, p.d_o + row0, gld, kChunk, kD, valid, kThreads);
    tile_load_async(sS0, kLdD, p.h + chh * kD * kD, kD, kD, kD, kD, kThreads);
    tile_load_async(sTm, kLdC, p.Akk + crow0, cld, kChunk, kChunk, valid, kThreads);
    tile_load_async(sdE, kLdD, p.dF + row0, gld, kChunk, kD, valid, kThreads);
    tile_load_async(sdSC, kLdD, p.dh + chh * kD * kD, kD, kD, kD, kD, kThreads);
    tile_load_async(sEarly, kLdD, p.v_new + row0, gld, kChunk, kD, valid, kThreads);
    cp_async_commit();
    if (tid < kChunk) sBeta[tid] = s_small;
    else if (tid >= 2 * kD && tid < 3 * kD) sGcv[tid - 2 * kD] = s_small;
    else if (tid >= kD && tid < 2 * kD) bias()[tid - kD] = s_small;
  }
  if (by_tma) {
    cp_async_wait<0>();
    if (!tc::mbar_wait(bar_b + 8, *s_phase) && tid == 0) atomicExch(p.status, 1);
    gate_load(graw, reinterpret_cast<const bf16*>(smem + oRaw), kLdD, kChunk, tid);
  }
  __syncthreads();
  // log2-domain cumulative log-decay, exactly as the forward computes it
  gate_apply(graw, sG, valid, bias(), __expf(p.A_log[h]) * kLog2e, tid);
  __syncthreads();
  if (tid < kD) {
    gate_cumsum(sG, tid);
    // worst decays of a strip of 8 rows: all of it, and what strip_decays says
    float worst[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < kChunk; r += 8) {
      const float g0 = sG[r * kLdG + tid], g7 = sG[(r + 7) * kLdG + tid];
      const float2 d = strip_decays(g0, sG[(r + 2) * kLdG + tid], sG[(r + kHalfRow) * kLdG + tid], sG[(r + 5) * kLdG + tid], g7);
      worst[0] = fmaxf(worst[0], g0 - g7);
      worst[1] = fmaxf(worst[1], d.x);
      worst[2] = fmaxf(worst[2], d.y);
    }
#pragma unroll
    for (int e = 0; e < 3; ++e) {  // (not negative, so their bit patterns have their order)
      const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(worst[e]));
      if (lane == 0) sWorst[warp * 3 + e] = __uint_as_float(m);
    }
  }
  if (by_tma) {
    if (!tc::mbar_wait(bar, *s_phase) && tid == 0) atomicExch(p.status, 1);  // gave up: flag it, results are void
  } else {
    cp_async_wait<0>();
  }
  __syncthreads();
  // the direct part of dbeta, rowsum(dF * E), while dF is still unscaled; dE = beta * dF in place;
  // hdh[k] = sum_v S0[k][v] dS1[k][v] (four threads per state row)
  for (int i = tid; i < kChunk * kD / 8; i += kThreads) {
    const int r = i >> 4, c = (i & 15) << 3;
    const float b = sBeta[r];
    const float f[8] = {b, b, b, b, b, b, b, b};
    uint4 x = *reinterpret_cast<const uint4*>(sdE + r * kLdD + c);
    const uint4 ev = *reinterpret_cast<const uint4*>(sEarly + r * kLdD + c);
    const uint32_t* e32 = reinterpret_cast<const uint32_t*>(&ev);
    const uint32_t* f32 = reinterpret_cast<const uint32_t*>(&x);
    float part = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 xe = unpack_bf16(e32[j]), y = unpack_bf16(f32[j]);
      part += xe.x * y.x + xe.y * y.y;
    }
    part += __shfl_xor_sync(0xffffffffu, part, 8);
    part += __shfl_xor_sync(0xffffffffu, part, 4);
    part += __shfl_xor_sync(0xffffffffu, part, 2);
    part += __shfl_xor_sync(0xffffffffu, part, 1);
    if ((i & 15) == 0) sDb[r] = part;
    scale8(x, f);
    *reinterpret_cast<uint4*>(sdE + r * kLdD + c) = x;
  }
  {
    const int row = tid >> 2, part = tid & 3;
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 a = *reinterpret_cast<const uint4*>(sS0 + row * kLdD + part * 32 + 8 * j);
      const uint4 b = *reinterpret_cast<const uint4*>(sdSC + row * kLdD + part * 32 + 8 * j);
      const uint32_t* a32 = reinterpret_cast<const uint32_t*>(&a);
      const uint32_t* b32 = reinterpret_cast<const uint32_t*>(&b);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = unpack_bf16(a32[e]), y = unpack_bf16(b32[e]);
        acc += x.x * y.x + x.y * y.y;
      }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    if (part == 0) sHdh[row] = acc;
  }
  __syncthreads();

  float dQ[1][4][4], dK[1][4][4], dKt[1][4][4], dG[1][4][4];
  float t[1][4][4];
  // dqg = dO S0^T  ->  dq_a = scale * Gam * dqg
  zero_acc(t);
  warp_gemm<1, 4, false, false>(t, sdO, kLdD, 16 * I, sS0, kLdD, 32 * cq, 0, kD);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float2 g = *reinterpret_cast<const float2*>(sG + (16 * I + gq + 8 * half) * kLdG + 32 * cq + 8 * nt + 2 * tq);
      dQ[0][nt][2 * half] = t[0][nt][2 * half] * p.scale * ex2(g.x);
      dQ[0][nt][2 * half + 1] = t[0][nt][2 * half + 1] * p.scale * ex2(g.y);
    }
  // dR = Tm^T dE  (= dV)
  zero_acc(t);
  warp_gemm<1, 4, true, true>(t, sTm, kLdC, 16 * I, sdE, kLdD, 32 * cq, 16 * I, kChunk);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r = 16 * I + gq + 8 * half, c = 32 * cq + 8 * nt + 2 * tq;
      const uint32_t pk = pack_bf16(t[0][nt][2 * half], t[0][nt][2 * half + 1]);
      if (!out_tma && r < valid) *reinterpret_cast<uint32_t*>(p.dv + row0 + (size_t)r * gld + c) = pk;
      *reinterpret_cast<uint32_t*>(sdR + r * kLdD + c) = pk;
    }
  if (out_tma) tc::fence_proxy_async();
  __syncthreads();
  if (out_tma && tid == kThreads - 32) {  // dv is the dR tile as it stands
    tc::tma_store_3d(&maps.dv, smem_u32(sdR), 0, h, tok0);
    tc::bulk_commit();
  }
  // dKd = -dR S0^T  ->  dk_a = Gam * dKd
  zero_acc(t);
  warp_gemm<1, 4, false, false>(t, sdR, kLdD, 16 * I, sS0, kLdD, 32 * cq, 0, kD);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float2 g = *reinterpret_cast<const float2*>(sG + (16 * I + gq + 8 * half) * kLdG + 32 * cq + 8 * nt + 2 * tq);
      dK[0][nt][2 * half] = -t[0][nt][2 * half] * ex2(g.x);
      dK[0][nt][2 * half + 1] = -t[0][nt][2 * half + 1] * ex2(g.y);
    }
  __syncthreads();  // S0 no longer needed
  // E moves into its operand tile (S0 has left it) and F = beta E into the dead dE tile
  for (int i = tid; i < kChunk * kD / 8; i += kThreads) {
    const int r = i >> 4, c = (i & 15) << 3;
    const uint4 ev = *reinterpret_cast<const uint4*>(sEarly + r * kLdD + c);
    const float b = sBeta[r];
    const uint32_t* e32 = reinterpret_cast<const uint32_t*>(&ev);
    uint4 bf;
    uint32_t* bf32 = reinterpret_cast<uint32_t*>(&bf);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16(e32[j]);
      bf32[j] = pack_bf16(b * x.x, b * x.y);
    }
    *reinterpret_cast<uint4*>(sE + r * kLdD + c) = ev;
    *reinterpret_cast<uint4*>(sF + r * kLdD + c) = bf;
  }
  __syncthreads();
  // pair-weight gradients: dM = -tril(dR E^T, -1) diag(beta),  dP = scale tril(dO F^T)
  {
    const int J = cq;
    float t2[1][2][4];
    zero_acc(t2);
    if (J <= I) warp_gemm<1, 2, false, false>(t2, sdR, kLdD, 16 * I, sE, kLdD, 16 * J, 0, kD);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int i = 16 * I + gq + 8 * half, j = 16 * J + 8 * nt + 2 * tq;
        const float m0 = (j < i) ? -t2[0][nt][2 * half] * sBeta[j] : 0.f;
        const float m1 = (j + 1 < i) ? -t2[0][nt][2 * half + 1] * sBeta[j + 1] : 0.f;
        *reinterpret_cast<uint32_t*>(sdM + i * kLdC + j) = pack_bf16(m0, m1);
      }
    zero_acc(t2);
    if (J <= I) warp_gemm<1, 2, false, false>(t2, sdO, kLdD, 16 * I, sF, kLdD, 16 * J, 0, kD);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int i = 16 * I + gq + 8 * half, j = 16 * J + 8 * nt + 2 * tq;
        // (the diagonal is ungated and stays out of the products)
        const float p0 = (j <= i) ? t2[0][nt][2 * half] * p.scale : 0.f;
        const float p1 = (j + 1 <= i) ? t2[0][nt][2 * half + 1] * p.scale : 0.f;
        if (j == i) sDiag[i] = to_f(__float2bfloat16(p0));
        if (j + 1 == i) sDiag[i] = to_f(__float2bfloat16(p1));
        *reinterpret_cast<uint32_t*>(sdP + i * kLdC + j) = pack_bf16(j < i ? p0 : 0.f, j + 1 < i ? p1 : 0.f);
      }
  }
  if (out_tma && tid == kThreads - 32) tc::bulk_wait_read();  // the dv store has read the dR tile
  tc::fence_proxy_async();
  __syncthreads();  // dO, dR, E no longer needed
  // dkg = F dS1^T  ->  dkt_a = exp(G_last - G) * dkg
  // q, k and kt tiles of the pair-product phase land while the dkg product runs
  if (by_tma) {
    if (lane == 0) {
      if (warp == 0) copy(bar_b, smem + oA0, &maps.q, kTileBytes, h * kD, tok0);
      if (warp == 1) copy(bar_b, smem + oA1, &maps.k, kTileBytes, h * kD, tok0);
      if (warp == 2) copy(bar_b, smem + oA1 + kTileBytes, &maps.kt, kTileBytes, h * kD, tok0);
    }
  } else {
    tile_load_async(reinterpret_cast<bf16*>(smem + oA0), kLdD, p.q + row0, gld, kChunk, kD, valid, kThreads);
    tile_load_async(reinterpret_cast<bf16*>(smem + oA1), kLdD, p.k + row0, gld, kChunk, kD, valid, kThreads);
    tile_load_async(reinterpret_cast<bf16*>(smem + oA1 + kTileBytes), kLdD, p.kt + row0, gld, kChunk, kD, valid, kThreads);
    cp_async_commit();
  }
  zero_acc(t);
  warp_gemm<1, 4, false, false>(t, sF, kLdD, 16 * I, sdSC, kLdD, 32 * cq, 0, kD);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int c = 32 * cq + 8 * nt + 2 * tq;
    const float2 gl = *reinterpret_cast<const float2*>(sG + (kChunk - 1) * kLdG + c);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float2 g = *reinterpret_cast<const float2*>(sG + (16 * I + gq + 8 * half) * kLdG + c);
      dKt[0][nt][2 * half] = t[0][nt][2 * half] * ex2(gl.x - g.x);
      dKt[0][nt][2 * half + 1] = t[0][nt][2 * half + 1] * ex2(gl.y - g.y);
    }
  }
  __syncthreads();

  // ================= phase B: gated pair products =================
  bf16* sQ = reinterpret_cast<bf16*>(smem + oA0);
  bf16* sK = reinterpret_cast<bf16*>(smem + oA1);
  bf16* sKt = reinterpret_cast<bf16*>(smem + oA1 + kTileBytes);
  bf16* sXq = reinterpret_cast<bf16*>(smem + oStage);
  bf16* sXk = sXq + kChunk * kLdD;
  if (by_tma) {
    if (!tc::mbar_wait(bar_b, *s_phase) && tid == 0) atomicExch(p.status, 1);
  } else {
    cp_async_wait<0>();
    __syncthreads();
  }
  {
    // dG starts from the state-coupled parts; column sums of kt * dkt_a feed the
    // chunk's last row (d/dG_last of exp(G_last - G_j)).
    float cs[4][2];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      cs[nt][0] = cs[nt][1] = 0.f;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int at = (16 * I + gq + 8 * half) * kLdD + 32 * cq + 8 * nt + 2 * tq;
        const float2 qv = unpack_bf16(*reinterpret_cast<const uint32_t*>(sQ + at));
        const float2 kv = unpack_bf16(*reinterpret_cast<const uint32_t*>(sK + at));
        const float2 ktv = unpack_bf16(*reinterpret_cast<const uint32_t*>(sKt + at));
        const float kd0 = ktv.x * dKt[0][nt][2 * half], kd1 = ktv.y * dKt[0][nt][2 * half + 1];
        dG[0][nt][2 * half] = qv.x * dQ[0][nt][2 * half] + kv.x * dK[0][nt][2 * half] - kd0;
        dG[0][nt][2 * half + 1] = qv.y * dQ[0][nt][2 * half + 1] + kv.y * dK[0][nt][2 * half + 1] - kd1;
        cs[nt][0] += kd0;
        cs[nt][1] += kd1;
      }
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        float v = cs[nt][b];
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (gq == 0) sCol[I * kD + 32 * cq + 8 * nt + 2 * tq + b] = v;
      }
  }
  // ---- The pairs, strip by strip (8 rows; the factors 2^(G_i - x(I)), 2^(x(I) - z(J)), 2^(z(J) - G_j) and their reference rows
  // are those of pairs_of_strip in pkda_intra_fwd_tc.cu).  Staged: Xq = bf16(q 2^(G - x)), Xk likewise, y = kt 2^(z - G) in fp32;
  // the operand of a strip pair is Y = bf16(y 2^(x(I) - z(J))), and both sides of a pair see the same X and Y.
  //   rows of strip I     t  = [dP_I; dM_I] Y     (8 + 8 rows, K = the tokens)   dq, dk_read += 2^(G - x) t,  dG += Xq t, Xk t
  //   columns of strip J  u_I = dP_I^T Xq + dM_I^T Xk  (K = 8 + 8 rows of I)     dkt += 2^(z - G) sum_I 2^(x(I) - z(J)) u_I,  dG -= Y u_I
  // Chunks whose strips decay too much for that take their pairs inside a strip level by level (lvl = 4, 2, 1, every row with a
  // reference of its own, one staging each) after those between strips.
  // Against staged pairing levels (operands, factors and masked weights of up to seven levels a chunk): 304 -> 247 us for
  // 1,460 strongly decaying chunks, 35 -> 29 for 40.
  float rb[2] = {0.f, 0.f};
  float worst[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) worst[e] = fmaxf(fmaxf(sWorst[e], sWorst[3 + e]), fmaxf(sWorst[6 + e], sWorst[9 + e]));
  const bool first_last = worst[0] <= kDirectLimit, bounded = worst[1] <= kDirectLimit && worst[2] <= kOuterLimit;
  const bool by_level = p.direct_cap < 8 || !(first_last || bounded);
  auto pairs = [&](auto halves) {
  constexpr bool kHalves = decltype(halves)::value;
  constexpr int xo = kHalves ? kHalfRow : 0, zo = kHalves ? kHalfRow : 7;  // reference rows of a strip: x of the second half (of the first: 0), z
#pragma unroll 1
  for (int lvl = 0;;) {
    // (a warp takes a row, four channels a lane: fp32 rows then move without bank conflicts)
#pragma unroll 2
    for (int r = warp; r < kChunk; r += kThreads / 32) {
      const int c4 = lane << 2, own = lvl ? (r & ~(2 * lvl - 1)) + lvl : r & ~7;
      const float4 g = *reinterpret_cast<const float4*>(sG + r * kLdG + c4);
      const float4 gx = *reinterpret_cast<const float4*>(sG + (lvl ? own : own + (r & xo)) * kLdG + c4);
      const float4 gz = *reinterpret_cast<const float4*>(sG + (lvl ? own : own + zo) * kLdG + c4);
      float4 x = make_float4(ex2(g.x - gx.x), ex2(g.y - gx.y), ex2(g.z - gx.z), ex2(g.w - gx.w));
      float4 z = make_float4(ex2(gz.x - g.x), ex2(gz.y - g.y), ex2(gz.z - g.z), ex2(gz.w - g.w));
      if (lvl) {  // the row is on one side of its pairs only
        if (r & lvl) z = make_float4(0.f, 0.f, 0.f, 0.f);
        else x = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      const uint2 qr = *reinterpret_cast<const uint2*>(sQ + r * kLdD + c4), kr = *reinterpret_cast<const uint2*>(sK + r * kLdD + c4);
      const uint2 ktr = *reinterpret_cast<const uint2*>(sKt + r * kLdD + c4);
      const float2 q0 = unpack_bf16(qr.x), q1 = unpack_bf16(qr.y), k0 = unpack_bf16(kr.x), k1 = unpack_bf16(kr.y);
      const float2 t0 = unpack_bf16(ktr.x), t1 = unpack_bf16(ktr.y);
      *reinterpret_cast<uint2*>(sXq + r * kLdD + c4) = make_uint2(pack_bf16(q0.x * x.x, q0.y * x.y), pack_bf16(q1.x * x.z, q1.y * x.w));
      *reinterpret_cast<uint2*>(sXk + r * kLdD + c4) = make_uint2(pack_bf16(k0.x * x.x, k0.y * x.y), pack_bf16(k1.x * x.z, k1.y * x.w));
      *reinterpret_cast<float4*>(sY + r * kLdY + c4) = make_float4(t0.x * z.x, t0.y * z.y, t1.x * z.z, t1.y * z.w);
    }
    // The factor of every strip pair, and whether it is there at all (nonzero in some channel).
    for (int pr = warp; pr < 36; pr += kThreads / 32) {
      const int Is = (pr >= 1) + (pr >= 3) + (pr >= 6) + (pr >= 10) + (pr >= 15) + (pr >= 21) + (pr >= 28);
      const int Js = pr - Is * (Is + 1) / 2;
      float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lvl) {
        if (Is == Js) d = make_float4(1.f, 1.f, 1.f, 1.f);
      } else if (!by_level || Js < Is) {
        const float4 a = *reinterpret_cast<const float4*>(sG + 8 * Is * kLdG + 4 * lane);
        const float4 b = *reinterpret_cast<const float4*>(sG + (8 * Js + zo) * kLdG + 4 * lane);
        d = make_float4(ex2(a.x - b.x), ex2(a.y - b.y), ex2(a.z - b.z), ex2(a.w - b.w));
      }
      *reinterpret_cast<float4*>(sStrip + pr * kD + 4 * lane) = d;
      const bool there = __any_sync(0xffffffffu, fmaxf(fmaxf(d.x, d.y), fmaxf(d.z, d.w)) > 0.f);
      if (lane == 0) sThere[pr] = there;
    }
    __syncthreads();
    const int m8 = lane >> 3, r7 = lane & 7;
    // rows of the strips 2 I and 2 I + 1
#pragma unroll
    for (int sub = 0; sub < 2; ++sub) {
      const int Is = 2 * I + sub, tri = Is * (Is + 1) / 2;
      zero_acc(t);
#pragma unroll 1
      for (int K = 0; K <= I; ++K) {
        const bool two = 2 * K + 1 <= Is;  // (the second strip of the step may be the one behind)
        if (!sThere[tri + 2 * K] && !(two && sThere[tri + 2 * K + 1])) continue;
        uint32_t a[4];
        ldsm_x4(a, smem_u32(((m8 & 1) ? sdM : sdP) + (8 * Is + r7) * kLdC + 16 * K + 8 * (m8 >> 1)));
        if (lvl) {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int i = 8 * Is + gq, j = 16 * K + 2 * tq + 8 * (x >> 1);
            a[x] &= (level_pair_ok(i, j, lvl) ? 0x0000ffffu : 0u) | (level_pair_ok(i, j + 1, lvl) ? 0xffff0000u : 0u);
          }
        }
        const float* y = sY + (16 * K + 2 * tq) * kLdY + 32 * cq + gq;
        const float* d = sStrip + (tri + 2 * K) * kD + 32 * cq + gq;
        // part 0: all rows; by halves 1: those of the first with their factors, 2: those of the second with theirs.  (The
        // second half's columns of the strip itself have no rows in the first, and their factor no bound.)
        auto take = [&](auto part) {
          constexpr int kPart = decltype(part)::value;
          const bool in = kPart == 0 || (gq < kHalfRow) == (kPart == 1);
          const uint32_t ap[4] = {in ? a[0] : 0u, in ? a[1] : 0u, in ? a[2] : 0u, in ? a[3] : 0u};
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            float d0 = d[8 * nt], d1 = two ? d[kD + 8 * nt] : 0.f;
            if (kPart == 1 && 2 * tq >= kHalfRow) {
              if (2 * K == Is) d0 = 0.f;
              if (2 * K + 1 == Is) d1 = 0.f;
            }
            if (kPart == 2) {
              const float self = sStrip[(tri + Is) * kD + 32 * cq + gq + 8 * nt];
              d0 = __fdividef(d0, self);
              d1 = __fdividef(d1, self);
            }
            mma_bf16(t[0][nt], ap, pack_bf16(y[8 * nt] * d0, y[kLdY + 8 * nt] * d0),
                     pack_bf16(y[8 * kLdY + 8 * nt] * d1, y[9 * kLdY + 8 * nt] * d1));
          }
        };
        if (!kHalves) {
          take(std::integral_constant<int, 0>{});
        } else {
          take(std::integral_constant<int, 1>{});
          take(std::integral_constant<int, 2>{});
        }
      }
      const int i = 8 * Is + gq, ref = lvl ? (i & ~(2 * lvl - 1)) + lvl : 8 * Is + (gq & xo);
      if (!lvl || (i & lvl)) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const int c = 32 * cq + 8 * nt + 2 * tq;
          const float2 g = *reinterpret_cast<const float2*>(sG + i * kLdG + c), gr = *reinterpret_cast<const float2*>(sG + ref * kLdG + c);
          const float2 xq = unpack_bf16(*reinterpret_cast<const uint32_t*>(sXq + i * kLdD + c));
          const float2 xk = unpack_bf16(*reinterpret_cast<const uint32_t*>(sXk + i * kLdD + c));
          const float f0 = ex2(g.x - gr.x), f1 = ex2(g.y - gr.y);
          dQ[0][nt][2 * sub] += f0 * t[0][nt][0];
          dQ[0][nt][2 * sub + 1] += f1 * t[0][nt][1];
          dK[0][nt][2 * sub] += f0 * t[0][nt][2];
          dK[0][nt][2 * sub + 1] += f1 * t[0][nt][3];
          dG[0][nt][2 * sub] += xq.x * t[0][nt][0] + xk.x * t[0][nt][2];
          dG[0][nt][2 * sub + 1] += xq.y * t[0][nt][1] + xk.y * t[0][nt][3];
        }
      }
    }
    // columns of the strips 2 I and 2 I + 1, two tiles of 8 channels at a time
#pragma unroll
    for (int np = 0; np < 2; ++np) {
      float2 y[2][2];
      float w[2][4];
      const int c = 32 * cq + 16 * np + 2 * tq;
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          y[x][half] = *reinterpret_cast<const float2*>(sY + (16 * I + gq + 8 * half) * kLdY + c + 8 * x);
          w[x][2 * half] = w[x][2 * half + 1] = 0.f;
        }
#pragma unroll 1
      for (int Is = 2 * I; Is < 8; ++Is) {
        const int tri = Is * (Is + 1) / 2 + 2 * I;
        const bool two = Is > 2 * I;  // (the second strip of the columns is the one behind)
        if (!sThere[tri] && !(two && sThere[tri + 1])) {
          if (two && !by_level) break;  // strips further behind decay by more
          continue;
        }
        uint32_t a[4], b[4];
        ldsm_x4_t(a, smem_u32(((m8 >> 1) ? sdM : sdP) + (8 * Is + r7) * kLdC + 16 * I + 8 * (m8 & 1)));
        ldsm_x4_t(b, smem_u32(((m8 & 1) ? sXk : sXq) + (8 * Is + r7) * kLdD + 32 * cq + 16 * np + 8 * (m8 >> 1)));
        if (lvl) {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int j = 16 * I + gq + 8 * (x & 1), i = 8 * Is + 2 * tq;
            a[x] &= (level_pair_ok(i, j, lvl) ? 0x0000ffffu : 0u) | (level_pair_ok(i + 1, j, lvl) ? 0xffff0000u : 0u);
          }
        }
        auto take = [&](auto part) {
          constexpr int kPart = decltype(part)::value;
          const bool in = kPart == 0 || (2 * tq < kHalfRow) == (kPart == 1);
          const uint32_t ap[4] = {in ? a[0] : 0u, in ? a[1] : 0u, in ? a[2] : 0u, in ? a[3] : 0u}, am[4] = {0u, 0u, ap[2], ap[3]};
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            float u[4] = {0.f, 0.f, 0.f, 0.f}, um[4] = {0.f, 0.f, 0.f, 0.f};
            mma_bf16(u, ap, b[2 * x], b[2 * x + 1]);
            mma_bf16(um, am, b[2 * x], b[2 * x + 1]);  // the part through M: its product with Y is dbeta's
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              float2 d = make_float2(0.f, 0.f);
              if (!half || two) d = *reinterpret_cast<const float2*>(sStrip + (tri + half) * kD + c + 8 * x);
              if (kPart == 1 && 2 * I + half == Is && gq >= kHalfRow) d = make_float2(0.f, 0.f);
              if (kPart == 2) {
                const float2 self = *reinterpret_cast<const float2*>(sStrip + Is * (Is + 3) / 2 * kD + c + 8 * x);
                d = make_float2(__fdividef(d.x, self.x), __fdividef(d.y, self.y));
              }
              const float2 Y = unpack_bf16(pack_bf16(y[x][half].x * d.x, y[x][half].y * d.y));
              const float u0 = u[2 * half], u1 = u[2 * half + 1];
              w[x][2 * half] += d.x * u0;
              w[x][2 * half + 1] += d.y * u1;
              dG[0][2 * np + x][2 * half] -= Y.x * u0;
              dG[0][2 * np + x][2 * half + 1] -= Y.y * u1;
              rb[half] += Y.x * um[2 * half] + Y.y * um[2 * half + 1];
            }
          }
        };
        if (!kHalves) {
          take(std::integral_constant<int, 0>{});
        } else {
          take(std::integral_constant<int, 1>{});
          take(std::integral_constant<int, 2>{});
        }
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int j = 16 * I + gq + 8 * half, ref = lvl ? (j & ~(2 * lvl - 1)) + lvl : (j & ~7) + zo;
        if (lvl && (j & lvl)) continue;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float2 g = *reinterpret_cast<const float2*>(sG + j * kLdG + c + 8 * x);
          const float2 gr = *reinterpret_cast<const float2*>(sG + ref * kLdG + c + 8 * x);
          dKt[0][2 * np + x][2 * half] += ex2(gr.x - g.x) * w[x][2 * half];
          dKt[0][2 * np + x][2 * half + 1] += ex2(gr.y - g.y) * w[x][2 * half + 1];
        }
      }
    }
    __syncthreads();
    if (kHalves || !by_level || lvl == 1) break;
    lvl = lvl ? lvl >> 1 : 4;
  }
  };
  if (first_last || by_level) pairs(std::false_type{});
  else pairs(std::true_type{});
  int next = 0;  // the drawer's: position in the list, then the item
  if (drawer) next = atomicAdd(p.fast_count + 2, 1);
  AtkIn atk;  // what the preconditioner's part below needs
  atk_request(atk, p, chh, tok0, valid, h, warp, lane);
  // ungated diagonal of P
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int i = 16 * I + gq + 8 * half;
    const float d = sDiag[i];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int at = i * kLdD + 32 * cq + 8 * nt + 2 * tq;
      const float2 qv = unpack_bf16(*reinterpret_cast<const uint32_t*>(sQ + at));
      const float2 ktv = unpack_bf16(*reinterpret_cast<const uint32_t*>(sKt + at));
      dQ[0][nt][2 * half] += d * ktv.x;
      dQ[0][nt][2 * half + 1] += d * ktv.y;
      dKt[0][nt][2 * half] += d * qv.x;
      dKt[0][nt][2 * half + 1] += d * qv.y;
    }
  }
  // dbeta: direct part + <kt_j, dkt_j(M path)> / beta_j
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float v = rb[half];
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    if (tq == 0) sRb[cq * kChunk + 16 * I + gq + 8 * half] = v;
  }
  // outputs of this stage, through padded tiles in dead regions; dG for the reverse cumulative sum, dkt and dk_read
  // for the preconditioner's part.  Full chunks send dq, dk_read and dkt from there by TMA: scattered fragment
  // stores cost more issue slots than the rest of this phase together.
  float* sdG = reinterpret_cast<float*>(smem + oStage);
  float *sOutKt = sG, *sOutK = reinterpret_cast<float*>(smem + oA1);  // (the decay tile is dead after the pairs)
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = 16 * I + gq + 8 * half, c = 32 * cq + 8 * nt + 2 * tq;
      *reinterpret_cast<float2*>(sOutKt + i * kLdG + c) = make_float2(dKt[0][nt][2 * half], dKt[0][nt][2 * half + 1]);
      *reinterpret_cast<float2*>(sdG + i * kLdG + c) = make_float2(dG[0][nt][2 * half], dG[0][nt][2 * half + 1]);
    }
#pragma unroll
  for (int i = 0; i < kAtkRows; ++i)
    atk.k[i] = *reinterpret_cast<const uint2*>(sK + (kAtkRows * warp + i) * kLdD + 4 * lane);
  __syncthreads();
  if (drawer) next = next < p.fast_count[1] ? p.slow_list[next] : -1;
  if (by_tma && tid == 0) *s_phase ^= 1;
  // every warp is past its reads of q, k and kt: their tiles take dq and dk_read
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = 16 * I + gq + 8 * half, c = 32 * cq + 8 * nt + 2 * tq;
      const uint32_t dq = pack_bf16(dQ[0][nt][2 * half], dQ[0][nt][2 * half + 1]);
      if (out_tma) *reinterpret_cast<uint32_t*>(sQ + i * kLdD + c) = dq;
      else if (i < valid) *reinterpret_cast<uint32_t*>(p.dq + row0 + (size_t)i * gld + c) = dq;
      *reinterpret_cast<float2*>(sOutK + i * kLdG + c) = make_float2(dK[0][nt][2 * half], dK[0][nt][2 * half + 1]);
    }
  tc::fence_proxy_async();
  // The raw gate of the tail phase is requested here, with the accumulators gone and the
  // reverse cumulative sum still to run: loaded where it is used, it cost the tail a full
  // memory round trip.
  constexpr int kIter = kChunk * kD / 8 / kThreads;
  uint4 raws[kIter];
#pragma unroll
  for (int it = 0; it < kIter; ++it) {
    const int r = (tid + it * kThreads) >> 4;
    raws[it] = make_uint4(0, 0, 0, 0);
    if (r < valid) raws[it] = *reinterpret_cast<const uint4*>(p.g + row0 + (size_t)r * gld + ((tid & 15) << 3));
  }
  if (tid < kChunk && tid < valid) {
    const float b = sBeta[tid];
    const float s = sRb[tid] + sRb[kChunk + tid] + sRb[2 * kChunk + tid] + sRb[3 * kChunk + tid];
    const float db = sDb[tid] + (b != 0.f ? s / b : 0.f);
    p.dbeta[(size_t)(tok0 + tid) * H + h] = __float2bfloat16(db);
  }
  atk_block_end(atk, warp, lane, reinterpret_cast<float*>(smem + oAtkEx));
  __syncthreads();
  if (out_tma && tid == kThreads - 32) {
    tc::tma_store_3d(&maps.dq, smem_u32(sQ), 0, h, tok0);
    tc::bulk_commit();
  }
  // reverse cumulative sum over the chunk (one channel per thread, in place), beside the preconditioner's part ...
  if (tid < kD) {
    const int c = tid;
    float run = sCol[c] + sCol[kD + c] + sCol[2 * kD + c] + sCol[3 * kD + c] + sGcv[c] * sHdh[c];
#pragma unroll 8
    for (int r = kChunk - 1; r >= 0; --r) {
      run += sdG[r * kLdG + c];
      sdG[r * kLdG + c] = run;
    }
  }
  atk_local(atk, p, row0, gld, valid, warp, lane, sOutKt, sOutK,
            reinterpret_cast<float*>(smem + oAtkEx), out_tma);
  if (p.slow_list && !p.geo.cu_seqlens) {
    if (drawer) *s_next = describe_item(p.geo, next);
  } else if (p.slow_list && warp == kThreads / 32 - 1) {  // packed: the drawer's warp looks the sequence up together
    const int4 d = describe_item(p.geo, __shfl_sync(0xffffffffu, next, 0));
    if (drawer) *s_next = d;
  }
  tc::fence_proxy_async();
  __syncthreads();
  if (p.slow_list) intra_bwd_ahead(p, maps, *s_next, *s_phase);
  if (out_tma && (tid == kThreads - 32 || tid == kThreads - 64)) {
    if (tid == kThreads - 32) tc::tma_store_3d(&maps.dkt, smem_u32(sOutKt), 0, h, tok0);
    else tc::tma_store_3d(&maps.dk_read, smem_u32(sOutK), 0, h, tok0);
    tc::bulk_commit();
  }
  // ... then the gate's own backward, elementwise over the tile with all threads:
  //   g = -exp(A_log) softplus(raw + bias);  draw = dg * (-exp(A_log)) sigmoid(raw + bias)
  // Per-thread partial sums (dA_log: scalar; ddt_bias: per channel) are reduced in a fixed order.
  const float* sBias = sRed + 16 + (*s_phase ^ 1) * kD;
  float* sPart = sY;  // [32][kLdG] per-(row group, channel) partials of ddt_bias (y is dead)
  {
    const float ea = __expf(p.A_log[h]);
    float pa = 0.f;
    float pb[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) pb[j] = 0.f;
    const int c8 = (tid & 15) << 3;
#pragma unroll
    for (int it = 0; it < kIter; ++it) {
      const int r = (tid + it * kThreads) >> 4;
      if (r < valid) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(&raws[it]);
        const float4 d0 = *reinterpret_cast<const float4*>(sdG + r * kLdG + c8);
        const float4 d1 = *reinterpret_cast<const float4*>(sdG + r * kLdG + c8 + 4);
        const float dgv[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
        uint4 outv;
        uint32_t* o32 = reinterpret_cast<uint32_t*>(&outv);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 x = unpack_bf16(w[j]);
          const float z0 = x.x + sBias[c8 + 2 * j], z1 = x.y + sBias[c8 + 2 * j + 1];
          // sigmoid and softplus from one exp(-|z|): 1/(1+e) (or e/(1+e)) and max(z,0) - log(1/(1+e))
          const float e0 = __expf(-fabsf(z0)), e1 = __expf(-fabsf(z1));
          const float i0 = __fdividef(1.f, 1.f + e0), i1 = __fdividef(1.f, 1.f + e1);
          const float sg0 = z0 >= 0.f ? i0 : e0 * i0, sg1 = z1 >= 0.f ? i1 : e1 * i1;
          const float sp0 = fmaxf(z0, 0.f) - __logf(i0), sp1 = fmaxf(z1, 0.f) - __logf(i1);
          const float dr0 = dgv[2 * j] * (-ea) * sg0, dr1 = dgv[2 * j + 1] * (-ea) * sg1;
          pa += dgv[2 * j] * (-ea * sp0) + dgv[2 * j + 1] * (-ea * sp1);
          pb[2 * j] += dr0;
          pb[2 * j + 1] += dr1;
          o32[j] = pack_bf16(dr0, dr1);
        }
        *reinterpret_cast<uint4*>(p.dg + row0 + (size_t)r * gld + c8) = outv;
      }
    }
    // thread (tid >> 4) in 0..31 covers rows (tid >> 4) and (tid >> 4) + 32 of channel group c8
    *reinterpret_cast<float4*>(sPart + (tid >> 4) * kLdG + c8) = make_float4(pb[0], pb[1], pb[2], pb[3]);
    *reinterpret_cast<float4*>(sPart + (tid >> 4) * kLdG + c8 + 4) = make_float4(pb[4], pb[5], pb[6], pb[7]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) pa += __shfl_xor_sync(0xffffffffu, pa, o);
    if (lane == 0) sRed[warp] = pa;
  }
  __syncthreads();
  if (tid < kD) {
    float acc = 0.f;
#pragma unroll 8
    for (int g = 0; g < 32; ++g) acc += sPart[g * kLdG + tid];
    p.partB[chh * kD + tid] = acc;
    atk_carry(reinterpret_cast<const float*>(smem + oAtkEx), p, chh, tid);
  }
  if (tid == 0) {
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) acc += sRed[w];
    p.partA[chh] = acc;
  }
  if (out_tma && (tid == kThreads - 32 || tid == kThreads - 64)) tc::bulk_wait_read();  // the tiles stay in place until the stores have read them
}

// grid (chunks, heads): one item per CTA; or, with a work list, a few persistent CTAs that walk it.
__global__ void __launch_bounds__(ib::kThreads, 1)
pkda_intra_bwd_kernel(const IntraBwdParams p, const __grid_constant__ IntraBwdMaps maps) {
  // With a work list it runs beside the tensor-memory kernel, an ordinary launch behind the classifier and the scans whose results both
  // read: no launch may come between the two.
  if (!p.slow_list) wait_prerequisites();
  launch_dependents();
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int4 s_next;  // the item: chunk, head, first token, valid tokens
  // with a work list items differ in cost (how many strip pairs are left, and how they are taken, follows the decay): CTAs draw them one
  // at a time
  if (threadIdx.x == 0) {
    tc::mbar_init(smem_u32(smem + ib::oBar), ib::kCopiesA);
    tc::mbar_init(smem_u32(smem + ib::oBar) + 8, ib::kCopiesB);
    tc::mbar_init(smem_u32(smem + ib::oBar) + 16, ib::kCopiesAhead);
    *reinterpret_cast<uint32_t*>(smem + ib::oBar + 24) = 0;
    tc::fence_barrier_init();
  }
  if (threadIdx.x < 32) {
    int item = blockIdx.x * p.geo.heads + blockIdx.y;
    if (p.slow_list) {
      if (threadIdx.x == 0) {
        const int at = atomicAdd(p.fast_count + 2, 1);
        item = at < p.fast_count[1] ? p.slow_list[at] : -1;
      }
      item = __shfl_sync(0xffffffffu, item, 0);
    }
    const int4 d = describe_item(p.geo, item);
    if (threadIdx.x == 0) s_next = d;
  }
  __syncthreads();
  intra_bwd_ahead(p, maps, s_next, 0);
  while (s_next.x >= 0) {
    intra_bwd_item(p, maps, &s_next);
    if (!p.slow_list) break;
    tc::fence_proxy_async();  // the sums of ddt_bias lie where the next item's copies land
    __syncthreads();  // the next item reuses every shared-memory region
  }
  wait_prerequisites();
}

// ------------------------------------------------------------------ preconditioner backward
struct AtkBwdParams {
  Geo geo;
  const bf16* k;
  const float* g_atk;
  const bf16* beta_atk;
  const float* a_start;
  const float* dkt;      // dA_local: d(loss)/dA_t through the write-key factor
  const float* dk_read;  // d(loss)/dk without the part through A_t
  const float* lam_in;
  bf16* dk;
  float* dg_atk;
  bf16* dbeta_atk;
};

// One (chunk, head) per CTA, 256 threads, everything in registers.  Warp w owns
// rows 8w..8w+7 of the chunk, lane l owns channels 4l..4l+3, so a whole token row
// lives in one warp (128-bit loads of the fp32 gradients, 64-bit loads of k) and a
// thread holds its 8 x 4 elements for the whole kernel; all global loads are
// issued before the first use.  Both first-order scans over the 64 rows (A_t
// forward, lam = dL/dA backward) are blocked: a thread scans its 8 rows, the
// eight row blocks exchange one (decay product, end value) pair through shared
// memory, and each block continues from the carry it is owed -- every factor is a
// product of decays <= 1, so nothing overflows.  The per-row channel sums are
// transposed butterfly reductions (9 shuffles for 8 rows).
// The chunk kernels leave dA_local, the lam-free part of dk and the outgoing carries; with the incoming carry given
// this is the reverse scan of dA_local and all gradients.  No transcendental per element: the states A_t are
// rebuilt with multiply-adds.
namespace atkb {
constexpr int kThreads = 256;
constexpr int kRows = 8;  // rows per warp
}  // namespace atkb

// Thread-private prefetch slots in dynamic shared memory (a thread only reads back
// what it copied itself, so they need no barrier): per row k (8 B), dkt (16 B),
// dk_read (16 B); per tile the chunk's entry state and incoming carry (16 B each).
namespace atkb {
constexpr int kSmem = kThreads * (kRows * (8 + 16 + 16) + 16 + 16);
}  // namespace atkb

__global__ void __launch_bounds__(atkb::kThreads, 2)
pkda_atk_bwd_kernel(const AtkBwdParams p, int n_tiles) {
  after_previous();
  using namespace atkb;
  extern __shared__ __align__(16) unsigned char slots[];
  __shared__ __align__(16) float sEnd[8][kD];  // per row block: end value of its zero-start scan
  __shared__ float sDec[8];                    // per row block: product of its decays
  const int H = p.geo.heads, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c4 = lane << 2, r0 = warp * kRows;
  const long gld = (long)H * kD;
  // slot layout: arrays of [kRows][kThreads] (then [kThreads]) so that a warp's accesses are contiguous
  uint2* sK = reinterpret_cast<uint2*>(slots);
  float4* sDkt = reinterpret_cast<float4*>(slots + kThreads * kRows * 8);
  float4* sDkr = sDkt + kThreads * kRows;
  float4* sA0 = sDkr + kThreads * kRows;
  float4* sLin = sA0 + kThreads;

  // A persistent CTA walks tiles blockIdx.x, blockIdx.x + gridDim.x, ...; a tile is one (chunk, head).
  // The next tile's data is requested before the current tile is computed.
  int tok0_n = 0, valid_n = 0;
  bool live_n = false;
  // The next tile's beta_atk and log-decay (lane i of a warp holds the values of the warp's row i),
  // by plain loads that nothing consumes before the next iteration.
  uint32_t bpraw_n = 0;
  float lg_n = 0.f;  // lg_n: the same for the row's log-decay
  static_assert(kRows <= 32 && (kRows & (kRows - 1)) == 0, "one lane per row");
  auto request = [&](int tile) {
    int n;
    live_n = tile < n_tiles && chunk_lookup_warp(p.geo, tile / H, n, tok0_n, valid_n);
    if (live_n) {
      const int hh = tile % H;
      const size_t col0 = ((size_t)tok0_n * H + hh) * kD + c4;
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int r = r0 + i;
        const bool ok = r < valid_n;
        const size_t off = ok ? col0 + (size_t)r * gld : 0;
        // 8-byte copy as two 4-byte pieces (cp.async sizes are 4, 8 or 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(sK + i * kThreads + tid)),
                     "l"(p.k + off), "r"(ok ? 8 : 0));
        cp_async16(sDkt + i * kThreads + tid, p.dkt + off, ok);
        cp_async16(sDkr + i * kThreads + tid, p.dk_read + off, ok);
      }
      {
        const int r = r0 + (lane & (kRows - 1));
        bpraw_n = 0;
        lg_n = 0.f;  // rows past the end: decay 1
        if (r < valid_n) {
          bpraw_n = *reinterpret_cast<const unsigned short*>(p.beta_atk + (size_t)(tok0_n + r) * H + hh);
          lg_n = p.g_atk[(size_t)(tok0_n + r) * H + hh];
        }
      }
      cp_async16(sA0 + tid, p.a_start + (size_t)tile * kD + c4, true);
      cp_async16(sLin + tid, p.lam_in + (size_t)tile * kD + c4, true);
    }
    cp_async_commit();
  };
  request(blockIdx.x);
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
  const bool live = live_n;
  const int tok0 = tok0_n, valid = valid_n, h = tile % H;
  const size_t col0 = ((size_t)tok0 * H + h) * kD + c4;
  cp_async_wait<0>();
  // ---- this tile's data: shared-memory slots -> registers
  uint2 kraw[kRows];
  float4 dkt[kRows], dkr[kRows];
  float pd[kRows], bp[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    kraw[i] = sK[i * kThreads + tid];
    dkt[i] = sDkt[i * kThreads + tid];
    dkr[i] = sDkr[i * kThreads + tid];
    pd[i] = __shfl_sync(0xffffffffu, lg_n, i);  // the log-decay for now
    bp[i] = __uint_as_float(__shfl_sync(0xffffffffu, bpraw_n, i) << 16);
  }
  const float4 a0 = sA0[tid];
  const float4 lin = sLin[tid];
  request(tile + gridDim.x);  // the slots are free again, the next tile's copies fly during the computation
  if (!live) continue;        // (uniform) index past the last real chunk of a packed batch
  float dblk = 1.f;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    pd[i] = __expf(pd[i]);  // rows past the end: exp(0) = 1, beta 0: the state passes through
    dblk *= pd[i];
  }
  // ---- forward scan, pass 1: the block's end value from a zero start
  {
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const float2 x = unpack_bf16(kraw[i].x), y = unpack_bf16(kraw[i].y);
      const float kc[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = pd[i] * a[e] + bp[i] * kc[e] * kc[e];
    }
    *reinterpret_cast<float4*>(&sEnd[warp][c4]) = make_float4(a[0], a[1], a[2], a[3]);
    if (lane == 0) sDec[warp] = dblk;
  }
  __syncthreads();
  float A[4] = {a0.x, a0.y, a0.z, a0.w};  // state before this block's first row
  for (int b = 0; b < warp; ++b) {
    const float d = sDec[b];
    const float4 e4 = *reinterpret_cast<const float4*>(&sEnd[b][c4]);
    A[0] = d * A[0] + e4.x; A[1] = d * A[1] + e4.y; A[2] = d * A[2] + e4.z; A[3] = d * A[3] + e4.w;
  }
  const float Ain[4] = {A[0], A[1], A[2], A[3]};
  // ---- reverse scan: block-local lam from a zero incoming value (into dkt), outgoing value exchanged
  {
    float l[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = kRows - 1; i >= 0; --i) {
      float* d = reinterpret_cast<float*>(&dkt[i]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        l[e] += d[e];
        d[e] = l[e];
        l[e] *= pd[i];
      }
    }
    __syncthreads();  // every warp has read the forward end values
    *reinterpret_cast<float4*>(&sEnd[warp][c4]) = make_float4(l[0], l[1], l[2], l[3]);
  }
  __syncthreads();
  float L[4] = {lin.x, lin.y, lin.z, lin.w};  // lam arriving at the end of this block
  for (int b = 7; b > warp; --b) {
    const float d = sDec[b];
    const float4 e4 = *reinterpret_cast<const float4*>(&sEnd[b][c4]);
    L[0] = d * L[0] + e4.x; L[1] = d * L[1] + e4.y; L[2] = d * L[2] + e4.z; L[3] = d * L[3] + e4.w;
  }
  // suffix[i] = product of the decays of rows i+1 .. 7 of this block
  float suf[kRows];
  suf[kRows - 1] = 1.f;
#pragma unroll
  for (int i = kRows - 2; i >= 0; --i) suf[i] = suf[i + 1] * pd[i + 1];
  // ---- pass 2: outputs, walking the rows forward again for the state before each row
  float x1[kRows], x2[kRows];
  A[0] = Ain[0]; A[1] = Ain[1]; A[2] = Ain[2]; A[3] = Ain[3];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int r = r0 + i;
    const float2 x = unpack_bf16(kraw[i].x), y = unpack_bf16(kraw[i].y);
    const float kc[4] = {x.x, x.y, y.x, y.y};
    const float* ll = reinterpret_cast<const float*>(&dkt[i]);
    const float* t2 = reinterpret_cast<const float*>(&dkr[i]);
    float o[4];
    x1[i] = 0.f;
    x2[i] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float lam = ll[e] + suf[i] * L[e];
      o[e] = t2[e] + 2.f * lam * bp[i] * kc[e];
      const float k2 = kc[e] * kc[e];
      x1[i] += lam * k2;
      x2[i] += lam * A[e];
      A[e] = pd[i] * A[e] + bp[i] * k2;
    }
    x2[i] *= pd[i];
    if (r < valid)
      *reinterpret_cast<uint2*>(p.dk + col0 + (size_t)r * gld) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
  }
  row_sums8(x1, lane);
  row_sums8(x2, lane);
  if ((lane & 3) == 0) {
    const int r = r0 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    if (r < valid) {
      const size_t s = (size_t)(tok0 + r) * H + h;
      p.dbeta_atk[s] = __float2bfloat16(x1[0]);
      p.dg_atk[s] = x2[0];
    }
  }
  __syncthreads();  // the exchange arrays are reused by the next tile
  }  // tile loop
  cp_async_wait<0>();
}

// Sequential carry over a sequence's chunks, last to first.
__global__ void __launch_bounds__(kD)
pkda_atk_bwd_carry_kernel(Geo geo, const float* c_loc, const float* sa, float* lam_in, float* dA0) {
  after_previous();
  const int n = blockIdx.x, h = blockIdx.y, H = geo.heads, c = threadIdx.x;
  const SeqInfo sq = seq_info(geo, n);
  float lam = 0.f;
  constexpr int kBatch = 16;  // loads of 16 chunks in flight before the dependent multiply-adds
  for (int i0 = sq.nchunks - 1; i0 >= 0; i0 -= kBatch) {
    float dec[kBatch], loc[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const bool ok = i0 - j >= 0;
      const size_t ch = (size_t)(sq.chunk0 + (ok ? i0 - j : 0)) * H + h;
      dec[j] = ok ? sa[ch] : 0.f;
      loc[j] = ok ? c_loc[ch * kD + c] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (i0 - j >= 0) {
        lam_in[((size_t)(sq.chunk0 + i0 - j) * H + h) * kD + c] = lam;
        lam = loc[j] + __expf(dec[j]) * lam;
      }
    }
  }
  if (dA0) dA0[((size_t)n * H + h) * kD + c] = lam;
}

// Deterministic reduction of the per-chunk partial sums of the three per-head
// parameter gradients.  grid (H), 1024 threads: eight sub-ranges of the chunk axis are
// summed side by side per channel and then added in order.
constexpr int kReduceSubs = 8;
__global__ void __launch_bounds__(kD * kReduceSubs)
pkda_param_reduce_kernel(Geo geo, const float* partA, const float* partB, const float* partC, float* dA_log,
                         float* ddt_bias, float* dcentre, const int* status, bf16* g0, bf16* g1, bf16* g2, size_t guard_n) {
  // It runs beside the pass in front of it, and the carry in front of that is an ordinary launch behind the kernels that leave the
  // partial sums: no launch may come between those two.
  launch_dependents();
  __shared__ float sSub[kReduceSubs][kD];
  __shared__ float sR[2][4];
  const int h = blockIdx.x, H = geo.heads, tid = threadIdx.x, c = tid % kD, sub = tid / kD;
  const int warp = tid >> 5, lane = tid & 31;
  const int nreal = geo.cu_seqlens ? geo.chunk_offsets[geo.n_seqs] : geo.total_chunks;
  const int per = (nreal + kReduceSubs - 1) / kReduceSubs;
  const int lo = sub * per, hi = min(nreal, lo + per);
  float b = 0.f;
  for (int ch = lo; ch < hi; ++ch) b += partB[((size_t)ch * H + h) * kD + c];
  sSub[sub][c] = b;
  float a = 0.f, cc = 0.f;
  if (tid < kD) {
    for (int ch = c; ch < nreal; ch += kD) {
      a += partA[(size_t)ch * H + h];
      cc += partC[(size_t)ch * H + h];
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      cc += __shfl_xor_sync(0xffffffffu, cc, o);
    }
    if (lane == 0) { sR[0][warp] = a; sR[1][warp] = cc; }
  }
  __syncthreads();
  if (tid < kD) {
    float t = 0.f;
#pragma unroll
    for (int s2 = 0; s2 < kReduceSubs; ++s2) t += sSub[s2][c];
    ddt_bias[h * kD + c] = t;
  }
  if (tid == 0) {
    dA_log[h] = sR[0][0] + sR[0][1] + sR[0][2] + sR[0][3];
    dcentre[h] = sR[1][0] + sR[1][1] + sR[1][2] + sR[1][3];
  }
  // The backward's last kernel: if any kernel of the call gave up, the heads of dq, dk and dv become
  // NaN, so that a caller who never reads the status word cannot take partial gradients for complete ones.
  wait_prerequisites();
  if (blockIdx.x == 0 && *reinterpret_cast<const volatile int*>(status) != 0) {
    const bf16 nan = __float2bfloat16(__int_as_float(0x7fc00000));
    for (size_t i = tid; i < guard_n; i += blockDim.x) {
      g0[i] = nan;
      g1[i] = nan;
      g2[i] = nan;
    }
  }
}

// ------------------------------------------------------------------ host side
struct BwdWorkspace {
  int* chunk_offsets;
  float* beta_c;
  bf16 *u, *dF, *dh;
  float *dk_read, *dkt, *partA, *partB, *partC, *c_loc, *lam_in;
  int2* fast_list;
  int *slow_list, *counts;
  int* fwd_cursor;  // item cursor of the recompute pass (lean backward)
  int* status;
  size_t bytes;
};

static BwdWorkspace carve_bwd(const pkda_problem& p, void* base) {
  BwdWorkspace w;
  const size_t chunks = (size_t)chunk_bound(p), H = p.heads, tok = p.total_tokens;
  size_t off = 0;
  unsigned char* b = static_cast<unsigned char*>(base);
  auto take = [&](size_t bytes) {
    void* ptr = b + off;
    off += align_up(bytes);
    return ptr;
  };
  w.chunk_offsets = static_cast<int*>(take((size_t)(p.n_seqs + 1) * sizeof(int)));
  w.beta_c = static_cast<float*>(take(chunks * H * kChunk * 4));
  w.u = static_cast<bf16*>(take(tok * H * kD * 2));
  w.dF = static_cast<bf16*>(take(tok * H * kD * 2));
  w.dh = static_cast<bf16*>(take(chunks * H * kD * kD * 2));
  w.dk_read = static_cast<float*>(take(tok * H * kD * 4));
  w.dkt = static_cast<float*>(take(tok * H * kD * 4));
  w.partA = static_cast<float*>(take(chunks * H * 4));
  w.partB = static_cast<float*>(take(chunks * H * kD * 4));
  w.partC = static_cast<float*>(take(chunks * H * 4));
  w.c_loc = static_cast<float*>(take(chunks * H * kD * 4));
  w.lam_in = static_cast<float*>(take(chunks * H * kD * 4));
  w.fast_list = static_cast<int2*>(take(chunks * H * sizeof(int2)));
  w.slow_list = static_cast<int*>(take(chunks * H * sizeof(int)));
  w.status = static_cast<int*>(take(16 * sizeof(int)));  // status word, then lengths and cursors of the work lists
  w.counts = w.status + 1;       // [0] fast, [1] slow, [2] cursor
  w.fwd_cursor = w.status + 5;
  w.bytes = off;
  return w;
}

size_t chunk_bwd_workspace(const pkda_problem& p) { return carve_bwd(p, nullptr).bytes; }
size_t chunk_bwd_status_offset(const pkda_problem& p) {
  return (size_t)(reinterpret_cast<unsigned char*>(carve_bwd(p, nullptr).status) - static_cast<unsigned char*>(nullptr));
}

template <typename K>
static bool set_smem(K kernel, int bytes) {
  return ensure_dynamic_smem(kernel, bytes);
}

template <int VB>
static int launch_scan_bwd(const ScanBwdParams& sp, int units, cudaStream_t st) {
  if (!set_smem(pkda_scan_bwd_kernel<VB>, scanb::L<VB>::kSmem)) return PKDA_ERR_LAUNCH;
  return launch_kernel(pkda_scan_bwd_kernel<VB>, units * (kD / VB), scanb::threads<VB>(), scanb::L<VB>::kSmem, st, sp);
}

int chunk_bwd(const pkda_chunk_bwd_args* a, cudaStream_t st) {
  const pkda_problem& p = a->p;
  int rc = check_chunk_problem(p);
  if (rc != PKDA_OK) return rc;
  if (p.n_seqs == 0 || p.total_tokens == 0) return PKDA_OK;
  if (!a->d_o || !a->Aqk || !a->Akk || !a->k_precond || !a->ac_atk || !a->a_atk || !a->sa_atk || !a->w ||
      !a->kg || !a->v_new || !a->h || !a->qg || !a->dq || !a->dk || !a->dv || !a->dg || !a->dg_atk ||
      !a->dbeta_atk || !a->dbeta || !a->dA_log || !a->ddt_bias || !a->dlog_atk_scale)
    return PKDA_ERR_NULL;
  if (!a->workspace || a->workspace_bytes < chunk_bwd_workspace(p)) return PKDA_ERR_WORKSPACE;
  // What moves several values at a time or by TMA, as in the forward.  (The column scans touch the states' cotangents by scalars.)
  if (!aligned({a->d_o, a->Aqk, a->Akk, a->k_precond, a->ac_atk, a->a_atk, a->w, a->kg, a->v_new, a->h, a->qg, a->dv, a->dg,
                a->workspace, a->recompute ? p.dt_bias : nullptr}, 16) ||
      !aligned({a->dk}, 8) || !aligned({a->dq}, 4))
    return PKDA_ERR_ALIGN;
  if (!scan_columns(p.n_seqs * p.heads) && !aligned({a->d_final_state, a->d_initial_state}, 16)) return PKDA_ERR_ALIGN;
  BwdWorkspace ws = carve_bwd(p, a->workspace);
  Geo geo;
  // On the default path the classifier of the intra stage runs first and packs beta on the way.
  const bool tc_intra = stage_variant(kStageIntraBwd) == 0;
  rc = run_prologue(p, ws.chunk_offsets, tc_intra ? nullptr : ws.beta_c, &geo, st);
  if (rc != PKDA_OK) return rc;

  const bf16* Aqk = static_cast<const bf16*>(a->Aqk);
  const bf16* Akk = static_cast<const bf16*>(a->Akk);
  const bf16* kt = static_cast<const bf16*>(a->k_precond);
  const float* gc = a->ac_atk;
  bf16* w = static_cast<bf16*>(a->w);
  bf16* kg = static_cast<bf16*>(a->kg);
  bf16* v_new = static_cast<bf16*>(a->v_new);
  bf16* h = static_cast<bf16*>(a->h);
  bf16* qg = static_cast<bf16*>(a->qg);
  if (cudaMemsetAsync(ws.status, 0, 16 * sizeof(int), st) != cudaSuccess) return PKDA_ERR_LAUNCH;
  if (tc_intra) {
    rc = launch_bwd_classify(geo, gc, direct_block_cap(), ws.fast_list, ws.slow_list, ws.counts,
                             static_cast<const bf16*>(p.beta), ws.beta_c, st);
    if (rc != PKDA_OK) return rc;
  }
  const int units = p.n_seqs * p.heads;
  // The older mma.sync scans run only when they are pinned (pkda_set_variant).
  const bool scan_mma = stage_variant(kStageScanBwd) == 1;
  // The recompute pass ends with its scan, an ordinary launch, which leaves h and v_new; the reverse scan, the very next launch, reads
  // neither, so the two run side by side, unless the caller lets the state's gradient take the place of the state, which the first one still reads.
  const uintptr_t S0 = reinterpret_cast<uintptr_t>(p.initial_state), dS0 = reinterpret_cast<uintptr_t>(a->d_initial_state);
  const bool in_place = S0 && dS0 && (S0 < dS0 ? dS0 - S0 : S0 - dS0) < (size_t)units * kD * kD * sizeof(float);
  const ScanPair pair = a->recompute && !in_place && !scan_mma && stage_variant(kStageScanFwd) != 1 ? scan_pair(units) : ScanPair{0, 0};
  if (a->recompute) {
    // The recompute kernels only read the products, write keys and decay totals.
    rc = run_forward_stages(p, geo, ws.beta_c, ws.u, const_cast<bf16*>(Aqk), const_cast<bf16*>(Akk),
                            const_cast<bf16*>(kt), const_cast<float*>(gc), a->a_atk, w, kg, v_new, h, qg,
                            nullptr, true, ws.status, ws.fwd_cursor, st, nullptr, nullptr, nullptr, pair.fwd);
    if (rc != PKDA_OK) return rc;
  }

  ScanBwdParams sp;
  sp.geo = geo; sp.kg = kg; sp.qg = qg; sp.w = w; sp.Aqk = Aqk; sp.d_o = static_cast<const bf16*>(a->d_o);
  sp.beta_c = ws.beta_c; sp.gc = gc; sp.dST = a->d_final_state; sp.dh = ws.dh; sp.dF = ws.dF;
  sp.dS0 = a->d_initial_state;
  {
    const int vb = units >= 120 ? 128 : (units >= 60 ? 64 : 32);  // value columns per CTA of the mma.sync kernel
    // Columns over eight, four or (beside the recompute pass's scan) two SMs for few units, else tcgen05 / TMEM / TMA, as
    // in the forward.
    begin_stage(kStageScanBwd, st);
    if (!scan_mma && scan_columns(units))
      rc = launch_scan_bwd_cols(geo, p.total_tokens, units, kg, w, qg, sp.d_o, Aqk, ws.beta_c, gc, a->d_final_state, ws.dh,
                                ws.dF, a->d_initial_state, ws.status, pair.bwd ? pair.bwd : scan_columns(units), pair.bwd != 0, st);
    else if (!scan_mma)
      rc = launch_scan_bwd_tc(geo, p.total_tokens, units, kg, w, qg, sp.d_o, Aqk, ws.beta_c, gc, a->d_final_state,
                              ws.dh, ws.dF, a->d_initial_state, ws.status, pair.bwd != 0, st);
    else if (vb == 128) rc = launch_scan_bwd<128>(sp, units, st);
    else if (vb == 64) rc = launch_scan_bwd<64>(sp, units, st);
    else rc = launch_scan_bwd<32>(sp, units, st);
    end_stage(st);
    if (rc != PKDA_OK) return rc;
  }

  dim3 gridc(geo.total_chunks, p.heads);
  IntraBwdParams ip;
  ip.geo = geo;
  ip.q = static_cast<const bf16*>(p.q); ip.k = static_cast<const bf16*>(p.k); ip.kt = kt;
  ip.g = static_cast<const bf16*>(p.g); ip.A_log = p.A_log; ip.dt_bias = p.dt_bias;
  ip.beta_c = ws.beta_c; ip.gc = gc; ip.Akk = Akk; ip.v_new = v_new; ip.h = h; ip.dh = ws.dh; ip.dF = ws.dF;
  ip.d_o = static_cast<const bf16*>(a->d_o);
  ip.dq = static_cast<bf16*>(a->dq); ip.dk_read = ws.dk_read; ip.dv = static_cast<bf16*>(a->dv);
  ip.dg = static_cast<bf16*>(a->dg); ip.dbeta = static_cast<bf16*>(a->dbeta); ip.dkt = ws.dkt;
  ip.partA = ws.partA; ip.partB = ws.partB; ip.scale = p.scale; ip.direct_cap = direct_block_cap();
  ip.g_atk = p.g_atk; ip.beta_atk = static_cast<const bf16*>(p.beta_atk); ip.log_atk_scale = p.log_atk_scale;
  ip.a_start = a->a_atk; ip.c_loc = ws.c_loc; ip.partC = ws.partC;
  ip.ln_x = logf(p.squash_x); ip.eps = p.squash_eps;
  IntraBwdMaps maps;
  {
    const uint64_t H = p.heads, tok = p.total_tokens, rows = (uint64_t)geo.total_chunks * H * kD;
    const uint64_t act_dims[2] = {H * kD, tok}, act_str[1] = {H * kD * 2};
    const uint32_t act_box[2] = {kLdD, kChunk};
    const uint64_t st_dims[2] = {kD, rows}, st_str[1] = {kD * 2};
    const uint32_t st_box[2] = {kLdD, kD};
    const uint64_t pr_dims[2] = {H * kChunk, tok}, pr_str[1] = {H * kChunk * 2};
    const uint32_t pr_box[2] = {kLdC, kChunk};
    ip.use_tma = tok >= kChunk && encode_bf16_map(&maps.d_o, ip.d_o, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.dF, ip.dF, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.E, ip.v_new, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.q, ip.q, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.k, ip.k, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.kt, ip.kt, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.g, ip.g, 2, act_dims, act_str, act_box, false) &&
                 encode_bf16_map(&maps.h, ip.h, 2, st_dims, st_str, st_box, false) &&
                 encode_bf16_map(&maps.dh, ip.dh, 2, st_dims, st_str, st_box, false) &&
                 encode_bf16_map(&maps.Akk, ip.Akk, 2, pr_dims, pr_str, pr_box, false);
    const uint64_t o_dims[3] = {kD, H, tok}, o_str2[2] = {kD * 2, H * kD * 2}, o_str4[2] = {kD * 4, H * kD * 4};
    const uint32_t o_box[3] = {kLdD, 1, kChunk};
    ip.out_tma = ip.use_tma && encode_bf16_map(&maps.dq, ip.dq, 3, o_dims, o_str2, o_box, false) &&
                 encode_bf16_map(&maps.dv, ip.dv, 3, o_dims, o_str2, o_box, false) &&
                 encode_f32_map(&maps.dk_read, ip.dk_read, 3, o_dims, o_str4, o_box) &&
                 encode_f32_map(&maps.dkt, ip.dkt, 3, o_dims, o_str4, o_box);
    ip.status = ws.status;
  }
  // Full chunks that are one direct block run on tcgen05 / tensor memory; a classifier in front sorts
  // the chunks into two work lists and the mma.sync kernel works off the second one (every chunk, one
  // CTA each, when it is pinned).
  ip.fast_list = nullptr;
  ip.slow_list = ip.fast_count = nullptr;
  const int sms = sm_count();
  if (tc_intra) {
    ip.fast_list = ws.fast_list; ip.slow_list = ws.slow_list; ip.fast_count = ws.counts;
    rc = launch_intra_bwd_tc(ip, st);
    if (rc != PKDA_OK) return rc;
    const int items = geo.total_chunks * p.heads;
    gridc = dim3(items < sms ? items : sms, 1);
  }
  if (!set_smem(pkda_intra_bwd_kernel, ib::kSmem)) return PKDA_ERR_LAUNCH;
  begin_stage(ip.slow_list ? kStageIntraBwdRest : kStageIntraBwd, st);
  rc = launch_kernel(pkda_intra_bwd_kernel, gridc, ib::kThreads, ib::kSmem, st, ip, maps);
  end_stage(st);
  if (rc != PKDA_OK) return rc;

  AtkBwdParams ap;
  ap.geo = geo; ap.k = static_cast<const bf16*>(p.k); ap.g_atk = p.g_atk;
  ap.beta_atk = static_cast<const bf16*>(p.beta_atk);
  ap.a_start = a->a_atk; ap.dkt = ws.dkt; ap.dk_read = ws.dk_read; ap.lam_in = ws.lam_in;
  ap.dk = static_cast<bf16*>(a->dk); ap.dg_atk = a->dg_atk; ap.dbeta_atk = static_cast<bf16*>(a->dbeta_atk);
  const int atk_tiles = geo.total_chunks * p.heads;
  const int atk_grid = atk_tiles < 2 * sms ? atk_tiles : 2 * sms;  // persistent: two CTAs per SM
  begin_stage(kStageAtkBwdCarry, st);
  rc = launch_kernel(false, pkda_atk_bwd_carry_kernel, dim3(p.n_seqs, p.heads), kD, 0, st, geo, ws.c_loc, a->sa_atk, ws.lam_in,
                a->d_initial_A_state);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageAtkBwdFinal, st);
  if (!set_smem(pkda_atk_bwd_kernel, atkb::kSmem)) return PKDA_ERR_LAUNCH;
  rc = launch_kernel(pkda_atk_bwd_kernel, atk_grid, atkb::kThreads, atkb::kSmem, st, ap, atk_tiles);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageParamReduce, st);
  const size_t guard_n = std::min<size_t>((size_t)p.total_tokens * p.heads * kD, 4096);
  rc = launch_kernel(pkda_param_reduce_kernel, p.heads, kD * kReduceSubs, 0, st, geo, ws.partA, ws.partB, ws.partC, a->dA_log,
                a->ddt_bias, a->dlog_atk_scale, ws.status, static_cast<bf16*>(a->dq), static_cast<bf16*>(a->dk),
                static_cast<bf16*>(a->dv), guard_n);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  return PKDA_OK;
}

}  // namespace pkda

