// Chunked PKDA forward for D = 128, chunk 64, bf16 activations.
//
// Pipeline (one launch each, all on the caller's stream):
//   offsets   packed input only: cumulative chunk counts per sequence
//   pack_beta beta -> fp32 [chunks][H][64], zero for rows past a sequence end
//   atk_local chunk-local preconditioner accumulation (from A = 0) and decay sums
//   atk_carry sequential over a sequence's chunks: A at every chunk start
//   intra     per chunk: log-decay cumsum, write keys, gated pair products
//             M (k x kt) and P (q x kt), relative to one reference row or strip by strip,
//             Tm = (I + tril(M) diag(beta))^-1, W = Tm (k*Gam), U = Tm v,
//             kg = kt * exp(G_last - G), qg = scale q * Gam
//   scan      sequential over chunks, V split across CTAs: h_n, E = U - W h_n,
//             S <- Gam_last * S + kg^T (beta E)
//   out       per chunk: o = qg h_n + P (beta E)
// With per-channel decay exp(G_i - G_j) cannot be factored as exp(G_i)exp(-G_j)
// (overflow after a few tokens), hence the reference rows (pkda_intra_fwd_tc.cu).
#include <algorithm>

#include "pkda_chunk.cuh"

namespace pkda {

// ------------------------------------------------------------------ small kernels
// First chunk of every packed sequence: a prefix sum over the sequences' chunk counts, 1,024 of them a turn.  (One thread that walks
// them waits for memory on the way: 4,000 sequences 222 -> 10 us, 44 6 -> 3.)
__global__ void __launch_bounds__(1024) pkda_chunk_offsets_kernel(const int* cu, int n_seqs, int* offs) {
  after_previous();
  __shared__ int s_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int acc = 0;  // chunks of the turns before
  if (tid == 0) offs[0] = 0;
  for (int n0 = 0; n0 < n_seqs; n0 += 1024) {
    const int n = n0 + tid;
    int x = n < n_seqs ? (cu[n + 1] - cu[n] + kChunk - 1) / kChunk : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_sum[warp] = x;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < 32; ++w) {
      const int y = s_sum[w];
      before += w < warp ? y : 0;
      all += y;
    }
    if (n < n_seqs) offs[n + 1] = acc + before + x;
    acc += all;
    __syncthreads();  // (the sums are rewritten by the next turn)
  }
}

__global__ void pkda_pack_beta_kernel(Geo geo, const bf16* beta, float* beta_c) {
  after_previous();
  int n, tok0, valid;
  if (!chunk_lookup(geo, blockIdx.x, n, tok0, valid)) return;
  const int H = geo.heads;
  for (int i = threadIdx.x; i < H * kChunk; i += blockDim.x) {
    int h = i / kChunk, r = i - h * kChunk;
    float b = r < valid ? to_f(beta[(size_t)(tok0 + r) * H + h]) : 0.f;
    beta_c[((size_t)blockIdx.x * H + h) * kChunk + r] = b;
  }
}

// Chunk-local preconditioner scan from A = 0: loc[c] = sum_j (prod_{m>j} d_m) bP_j k_j[c]^2
// and the chunk's summed log-decay; also the chunk-major fp32 copy of beta (when beta_c is
// given), which saves a launch.  grid chunks * H, the heads of a chunk next to each other (they share the
// sectors of the per-token scalars and lie side by side in k), 256 threads: warp w scans rows 8w..8w+7 with
// lane l holding channels 4l..4l+3 (64-bit loads, one token row per warp request), then the
// eight row blocks are chained in order through shared memory.
__global__ void __launch_bounds__(256)
pkda_atk_local_kernel(Geo geo, const bf16* k, const float* g_atk, const bf16* beta_atk, const bf16* beta,
                      float* ac_local, float* sa, float* beta_c, int* zero) {
  after_previous();
  __shared__ __align__(16) float sEnd[8][kD];
  __shared__ float sDec[8], sSum[8];
  if (blockIdx.x == 0 && threadIdx.x < 8) zero[threadIdx.x] = 0;  // status word and cursors of the kernels behind
  int n, tok0, valid;
  const int H = geo.heads, chunk = blockIdx.x / H, h = blockIdx.x % H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (geo.cu_seqlens) {
    // The whole CTA compares the last 256 candidates at once, one round trip instead of one per step of a binary
    // search; beyond that many sequences the candidates are halved first.  (Counting through all of them takes
    // 412 us for 4,000 sequences and 2,894 for 16,000, 64,000 tokens of 16 heads each, against 291 and 1,125.)
    int lo = 0, len = geo.n_seqs;  // the sequence is one of [lo, lo + len)
    while (len > 256) {
      const int half = len >> 1;
      if (geo.chunk_offsets[lo + half] <= chunk) {
        lo += half;
        len -= half;
      } else {
        len = half;
      }
    }
    n = lo - 1 + __syncthreads_count(tid < len && geo.chunk_offsets[lo + tid] <= chunk);
    const int total = geo.chunk_offsets[geo.n_seqs], first = geo.chunk_offsets[n];
    const int bos = geo.cu_seqlens[n], eos = geo.cu_seqlens[n + 1];
    if (chunk >= total) return;
    tok0 = bos + (chunk - first) * kChunk;
    valid = min(kChunk, eos - tok0);
  } else if (!chunk_lookup(geo, chunk, n, tok0, valid)) {
    return;
  }
  const size_t chh = blockIdx.x;
  const int c4 = lane << 2, r0 = warp * 8;
  uint2 kraw[8];
  float lg_l = 0.f, bp_l = 0.f;  // lane i < 8: the scalars of row r0 + i
  if (lane < 8 && r0 + lane < valid) {  // all loads first
    const size_t s = (size_t)(tok0 + r0 + lane) * H + h;
    lg_l = g_atk[s];
    bp_l = to_f(beta_atk[s]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const bool ok = r0 + i < valid;
    const size_t s = (size_t)(tok0 + (ok ? r0 + i : 0)) * H + h;
    kraw[i] = ok ? *reinterpret_cast<const uint2*>(k + s * kD + c4) : make_uint2(0, 0);
  }
  if (beta_c && tid < kChunk)
    beta_c[chh * kChunk + tid] = tid < valid ? to_f(beta[(size_t)(tok0 + tid) * H + h]) : 0.f;
  float a[4] = {0.f, 0.f, 0.f, 0.f}, dblk = 1.f, gsum = 0.f;
  const float pd_l = __expf(lg_l);  // rows past the end: decay 1, beta 0
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 x = unpack_bf16(kraw[i].x), y = unpack_bf16(kraw[i].y);
    const float pd = __shfl_sync(0xffffffffu, pd_l, i), bp = __shfl_sync(0xffffffffu, bp_l, i);
    a[0] = pd * a[0] + bp * x.x * x.x;
    a[1] = pd * a[1] + bp * x.y * x.y;
    a[2] = pd * a[2] + bp * y.x * y.x;
    a[3] = pd * a[3] + bp * y.y * y.y;
    dblk *= pd;
    gsum += __shfl_sync(0xffffffffu, lg_l, i);
  }
  *reinterpret_cast<float4*>(&sEnd[warp][c4]) = make_float4(a[0], a[1], a[2], a[3]);
  if (lane == 0) { sDec[warp] = dblk; sSum[warp] = gsum; }
  __syncthreads();
  if (tid < kD) {
    float acc = 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) acc = sDec[b] * acc + sEnd[b][tid];
    ac_local[chh * kD + tid] = acc;
  }
  if (tid == 0) {
    float g = 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) g += sSum[b];
    sa[chh] = g;
  }
}

// Sequential carry over the chunks of one (sequence, head): A at each chunk start.
__global__ void __launch_bounds__(kD)
pkda_atk_carry_kernel(Geo geo, const float* ac_local, const float* sa, const float* A0,
                      float* a_start, float* AT) {
  after_previous();
  const int n = blockIdx.x, h = blockIdx.y, H = geo.heads, c = threadIdx.x;
  const SeqInfo sq = seq_info(geo, n);
  float A = A0 ? A0[((size_t)n * H + h) * kD + c] : 0.f;
  constexpr int kBatch = 16;  // loads of 16 chunks in flight before the dependent multiply-adds
  for (int i0 = 0; i0 < sq.nchunks; i0 += kBatch) {
    float dec[kBatch], loc[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const bool ok = i0 + j < sq.nchunks;
      const size_t ch = (size_t)(sq.chunk0 + (ok ? i0 + j : 0)) * H + h;
      dec[j] = ok ? sa[ch] : 0.f;
      loc[j] = ok ? ac_local[ch * kD + c] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (i0 + j < sq.nchunks) {
        a_start[((size_t)(sq.chunk0 + i0 + j) * H + h) * kD + c] = A;
        A = __expf(dec[j]) * A + loc[j];
      }
    }
  }
  if (AT) AT[((size_t)n * H + h) * kD + c] = A;
}

// ------------------------------------------------------------------ forward state scan
struct ScanParams {
  Geo geo;
  const bf16 *w, *u, *kg;
  const float *beta_c, *gc;
  const float* S0;
  bf16 *h, *v_new;
  float* ST;
};

namespace scan {
template <int VB> __host__ __device__ constexpr int threads() { return 128 * (VB / 32); }  // 4 warps per 32 value columns
template <int VB> struct L {
  static constexpr int ldv = VB + kPad;
  static constexpr int oW = 0;
  static constexpr int oKg = oW + kTileBytes;
  static constexpr int oU = oKg + kTileBytes;            // bf16 [64][ldv]
  static constexpr int oBeta = oU + kChunk * ldv * 2;    // f32 [64]
  static constexpr int oGc = oBeta + kChunk * 4;         // f32 [128]
  static constexpr int kStage = oGc + kD * 4;
  static constexpr int oH = 2 * kStage;                  // bf16 [128][ldv]
  static constexpr int oF = oH + kD * ldv * 2;           // bf16 [64][ldv]
  static constexpr int kSmem = oF + kChunk * ldv * 2;
};
}  // namespace scan

template <int VB, bool kRecompute>
__global__ void __launch_bounds__(scan::threads<VB>())
pkda_scan_fwd_kernel(const ScanParams p) {
  after_previous();
  using Lay = scan::L<VB>;
  constexpr int ldv = Lay::ldv, NT = 4, kT = scan::threads<VB>();
  extern __shared__ __align__(128) unsigned char smem[];
  const int VS = kD / VB;
  const int vs = blockIdx.x % VS;
  const int nh = blockIdx.x / VS;
  const int n = nh / p.geo.heads, h = nh - n * p.geo.heads, H = p.geo.heads;
  const SeqInfo sq = seq_info(p.geo, n);
  if (sq.nchunks == 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int wr = warp & 3, c0 = 32 * (warp >> 2);  // this warp: state rows [32 wr, +32), columns [c0, +32) of the slice
  const int v0 = vs * VB;
  const long gld = (long)H * kD;
  bf16* sH = reinterpret_cast<bf16*>(smem + Lay::oH);
  bf16* sF = reinterpret_cast<bf16*>(smem + Lay::oF);

  auto prefetch = [&](int i) {
    unsigned char* st = smem + (i & 1) * Lay::kStage;
    const int tok0 = sq.bos + i * kChunk;
    const int valid = min(kChunk, sq.len - i * kChunk);
    const size_t row0 = ((size_t)tok0 * H + h) * kD;
    const size_t chh = (size_t)(sq.chunk0 + i) * H + h;
    tile_load_async(reinterpret_cast<bf16*>(st + Lay::oW), kLdD, p.w + row0, gld, kChunk, kD, valid, kT);
    tile_load_async(reinterpret_cast<bf16*>(st + Lay::oKg), kLdD, p.kg + row0, gld, kChunk, kD, valid, kT);
    tile_load_async(reinterpret_cast<bf16*>(st + Lay::oU), ldv, p.u + row0 + v0, gld, kChunk, VB, valid, kT);
    if (tid < 16) cp_async16(st + Lay::oBeta + tid * 16, p.beta_c + chh * kChunk + tid * 4, true);
    else if (tid < 48) cp_async16(st + Lay::oGc + (tid - 16) * 16, p.gc + chh * kD + (tid - 16) * 4, true);
  };

  // state rows [32*warp, +32) x VB columns, fp32 fragments
  float S[2][NT][4];
  const size_t sbase = ((size_t)n * H + h) * kD * kD;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = 32 * wr + 16 * mt + gq + 8 * half, c = v0 + c0 + 8 * nt + 2 * tq;
        float2 s2 = make_float2(0.f, 0.f);
        if (p.S0) s2 = *reinterpret_cast<const float2*>(p.S0 + sbase + (size_t)r * kD + c);
        S[mt][nt][2 * half] = s2.x;
        S[mt][nt][2 * half + 1] = s2.y;
      }

  prefetch(0);
  cp_async_commit();
  for (int i = 0; i < sq.nchunks; ++i) {
    if (i + 1 < sq.nchunks) prefetch(i + 1);
    cp_async_commit();
    cp_async_wait<1>();
    unsigned char* st = smem + (i & 1) * Lay::kStage;
    const bf16* sW = reinterpret_cast<const bf16*>(st + Lay::oW);
    const bf16* sKg = reinterpret_cast<const bf16*>(st + Lay::oKg);
    const bf16* sU = reinterpret_cast<const bf16*>(st + Lay::oU);
    const float* sBeta = reinterpret_cast<const float*>(st + Lay::oBeta);
    const float* sGc = reinterpret_cast<const float*>(st + Lay::oGc);
    const int tok0 = sq.bos + i * kChunk;
    const int valid = min(kChunk, sq.len - i * kChunk);
    const size_t chh = (size_t)(sq.chunk0 + i) * H + h;

    // a. chunk-entry state -> bf16 operand tile (and the saved chunk states)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 32 * wr + 16 * mt + gq + 8 * half, c = c0 + 8 * nt + 2 * tq;
          *reinterpret_cast<uint32_t*>(sH + r * ldv + c) = pack_bf16(S[mt][nt][2 * half], S[mt][nt][2 * half + 1]);
        }
    __syncthreads();  // sH complete; stage i landed for every thread
    {
      constexpr int cpr = VB / 8;
      for (int j = tid; j < kD * cpr; j += kT) {
        const int r = j / cpr, c = (j - r * cpr) * 8;
        *reinterpret_cast<uint4*>(p.h + (chh * kD + r) * kD + v0 + c) =
            *reinterpret_cast<const uint4*>(sH + r * ldv + c);
      }
    }
    // b. E = U - W h ; F = beta * E
    {
      float e[1][NT][4];
      zero_acc(e);
      warp_gemm<1, NT, false, true>(e, sW, kLdD, 16 * wr, sH, ldv, c0, 0, kD);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 16 * wr + gq + 8 * half, c = c0 + 8 * nt + 2 * tq;
          const float2 uu = unpack_bf16(*reinterpret_cast<const uint32_t*>(sU + r * ldv + c));
          const uint32_t ek = pack_bf16(uu.x - e[0][nt][2 * half], uu.y - e[0][nt][2 * half + 1]);
          if (r < valid)
            *reinterpret_cast<uint32_t*>(p.v_new + ((size_t)(tok0 + r) * H + h) * kD + v0 + c) = ek;
          const float2 er = unpack_bf16(ek);
          const float b = sBeta[r];
          *reinterpret_cast<uint32_t*>(sF + r * ldv + c) = pack_bf16(b * er.x, b * er.y);
        }
    }
    __syncthreads();
    // c. S <- Gam_last * S + kg^T F
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float gcv = sGc[32 * wr + 16 * mt + gq + 8 * half];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          S[mt][nt][2 * half] *= gcv;
          S[mt][nt][2 * half + 1] *= gcv;
        }
      }
    warp_gemm<2, NT, true, true>(S, sKg, kLdD, 32 * wr, sF, ldv, c0, 0, kChunk);
    __syncthreads();  // everyone done with stage i and sF before they are refilled
  }
  cp_async_wait<0>();
  if (!kRecompute && p.ST) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 32 * wr + 16 * mt + gq + 8 * half, c = v0 + c0 + 8 * nt + 2 * tq;
          *reinterpret_cast<float2*>(p.ST + sbase + (size_t)r * kD + c) =
              make_float2(S[mt][nt][2 * half], S[mt][nt][2 * half + 1]);
        }
  }
}

// ------------------------------------------------------------------ output kernel
struct OutParams {
  Geo geo;
  const bf16 *qg, *h, *Aqk, *v_new;
  const float* beta_c;
  bf16* o;
};

namespace outk {
constexpr int kThreads = 256;
constexpr int oQg = 0;
constexpr int oH = oQg + kTileBytes;              // bf16 [128][136]
constexpr int oP = oH + kD * kLdD * 2;            // bf16 [64][72]
constexpr int oF = oP + kChunk * kLdC * 2;        // bf16 [64][136]
constexpr int kSmem = oF + kTileBytes;
}  // namespace outk

__global__ void __launch_bounds__(outk::kThreads)
pkda_out_fwd_kernel(const OutParams p) {
  after_previous();
  using namespace outk;
  extern __shared__ __align__(128) unsigned char smem[];
  bf16* sQg = reinterpret_cast<bf16*>(smem + oQg);
  bf16* sH = reinterpret_cast<bf16*>(smem + oH);
  bf16* sP = reinterpret_cast<bf16*>(smem + oP);
  bf16* sF = reinterpret_cast<bf16*>(smem + oF);
  int n, tok0, valid;
  if (!chunk_lookup(p.geo, blockIdx.x, n, tok0, valid)) return;
  const int h = blockIdx.y, H = p.geo.heads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const size_t chh = (size_t)blockIdx.x * H + h;
  const size_t row0 = ((size_t)tok0 * H + h) * kD;
  const long gld = (long)H * kD;

  tile_load_async(sQg, kLdD, p.qg + row0, gld, kChunk, kD, valid, kThreads);
  tile_load_async(sH, kLdD, p.h + chh * kD * kD, kD, kD, kD, kD, kThreads);
  tile_load_async(sP, kLdC, p.Aqk + ((size_t)tok0 * H + h) * kChunk, (long)H * kChunk, kChunk, kChunk, valid, kThreads);
  cp_async_commit();
  // F = beta * E (E read from global, rounded exactly as the scan rounded it)
  for (int i = tid; i < kChunk * kD / 8; i += kThreads) {
    const int r = i >> 4, c = (i & 15) << 3;
    uint4 ev = make_uint4(0, 0, 0, 0);
    if (r < valid) ev = *reinterpret_cast<const uint4*>(p.v_new + row0 + (size_t)r * gld + c);
    const float b = p.beta_c[chh * kChunk + r];
    uint32_t* e32 = reinterpret_cast<uint32_t*>(&ev);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16(e32[j]);
      e32[j] = pack_bf16(b * x.x, b * x.y);
    }
    *reinterpret_cast<uint4*>(sF + r * kLdD + c) = ev;
  }
  cp_async_wait<0>();
  __syncthreads();

  const int I = warp & 3, n0 = 64 * (warp >> 2);
  float acc[1][8][4];
  zero_acc(acc);
  warp_gemm<1, 8, false, true>(acc, sQg, kLdD, 16 * I, sH, kLdD, n0, 0, kD);
  warp_gemm<1, 8, false, true>(acc, sP, kLdC, 16 * I, sF, kLdD, n0, 0, 16 * (I + 1));
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = 16 * I + gq + 8 * half;
      if (i < valid)
        *reinterpret_cast<uint32_t*>(p.o + row0 + (size_t)i * gld + n0 + 8 * nt + 2 * tq) =
            pack_bf16(acc[0][nt][2 * half], acc[0][nt][2 * half + 1]);
    }
}

// ------------------------------------------------------------------ host side
struct FwdWorkspace {
  int* chunk_offsets;
  float* beta_c;
  bf16* u;
  int* status;  // device status word: 0 = ok, 1 = a bounded wait in a kernel gave up; then the item cursor
  size_t bytes;
};

static FwdWorkspace carve_fwd(const pkda_problem& p, void* base) {
  FwdWorkspace w;
  const size_t chunks = (size_t)chunk_bound(p);
  size_t off = 0;
  unsigned char* b = static_cast<unsigned char*>(base);
  w.chunk_offsets = reinterpret_cast<int*>(b + off);
  off += align_up((size_t)(p.n_seqs + 1) * sizeof(int));
  w.beta_c = reinterpret_cast<float*>(b + off);
  off += align_up(chunks * p.heads * kChunk * sizeof(float));
  w.u = reinterpret_cast<bf16*>(b + off);
  off += align_up((size_t)p.total_tokens * p.heads * kD * sizeof(bf16));
  w.status = reinterpret_cast<int*>(b + off);
  off += align_up(8 * sizeof(int));
  w.bytes = off;
  return w;
}

size_t chunk_fwd_workspace(const pkda_problem& p) { return carve_fwd(p, nullptr).bytes; }

// True where the forward runs in chained mode (no preconditioner kernels in front of the intra stage).  Asked once a call:
// it looks at the process-wide testing switches, and what runs in front of the intra stage and the stage itself must agree.
static bool forward_chain_possible(const pkda_problem& p) {
  if (p.cu_seqlens || stage_variant(kStageIntraFwd) != 0 || direct_block_cap() < 64) return false;
  // A hand-over from one chunk of a chain to the next takes about 0.6 us, an item 0.05 us of the chip: with a dozen
  // (row, head) units side by side the hand-overs hide, and the chain spares two kernels in front of the intra stage.
  // The fewer the units, the less there is to hide behind, and what a chain loses at one level it never makes up for, so the
  // limit is one of length.  Whole forward, unchained -> chained, us (chunks that decay mildly; the strongly decaying ones, whose items
  // take longer, lose less):
  //   1 unit of 1,536 tokens 63.5 -> 59.5, 7 of 1,536 67.6 -> 65.5;        4 of 4,096 109 -> 119, 5 of 3,072 92 -> 98
  //   8 units of 16,384 418 -> 412, 12 471 -> 462, 16 522 -> 496;          12 of 24,576 688 -> 696, 16 of 65,536 1,980 -> 2,074
  //   24 units of 65,536 2,772 -> 2,650, 28 2,965 -> 2,805;                24 of 131,072 5,467 -> 5,623
  //   32 units of 65,536 3,176 -> 2,996, of 131,072 6,325 -> 5,965
  // The state is the same bit for bit either way.  (A packed batch goes sequence after
  // sequence, a chain per head side by side: 65,536 tokens of 32 heads 1,740 -> 1,731 us, of 12 heads 682 -> 768.)
  const long units = (long)p.n_seqs * p.heads, chunks = ((long)p.seq_len + kChunk - 1) / kChunk;
  return units >= 32 || chunks <= (units >= 24 ? 1024 : units >= 8 ? 256 : 24);
}
size_t chunk_fwd_status_offset(const pkda_problem& p) {
  return (size_t)(reinterpret_cast<unsigned char*>(carve_fwd(p, nullptr).status) - static_cast<unsigned char*>(nullptr));
}

template <typename K>
static bool set_smem(K kernel, int bytes) {
  return ensure_dynamic_smem(kernel, bytes);
}

int check_chunk_problem(const pkda_problem& p) {
  int rc = check_problem(p);
  if (rc != PKDA_OK) return rc;
  if (p.head_dim != kD) return PKDA_ERR_SHAPE;
  if (p.dtype != PKDA_BF16) return PKDA_ERR_DTYPE;
  return PKDA_OK;
}

int scan_columns(int units) {
  const int sms = sm_count();
  return 8L * units <= sms ? 8 : 4L * units <= sms ? 4 : 0;
}

// A scan is a chain of chunk steps that keeps few SMs busy, so two side by side cost little more than the longer one.  Each CTA
// takes an SM of its own (two do not fit its shared memory), so the rule is the most CTAs a unit with which both run in one wave,
// the backward's, whose step is the longer, before the forward's.  Lean step, one scan after the other -> side by side, us: 4,096
// tokens of 8 units 467 -> 403, 16 643 -> 584, 24 828 -> 761, 36 1,057 -> 1,028; 2,048 tokens of 64 units 950 -> 874; 1,024 of 72
// 551 -> 510.  From 75 units on the tensor-memory scans fill more than half the chip each.
ScanPair scan_pair(int units) {
  static constexpr ScanPair kPairs[] = {{8, 8}, {4, 8}, {4, 4}, {2, 4}, {2, 2}, {1, 1}};
  for (const ScanPair& s : kPairs)
    if (units * (s.fwd + s.bwd) <= sm_count()) return s;
  return {0, 0};
}

template <int VB, bool kRecompute>
static int launch_scan_fwd(const ScanParams& sp, int units, cudaStream_t st) {
  if (!set_smem(pkda_scan_fwd_kernel<VB, kRecompute>, scan::L<VB>::kSmem)) return PKDA_ERR_LAUNCH;
  return launch_kernel(pkda_scan_fwd_kernel<VB, kRecompute>, units * (kD / VB), scan::threads<VB>(), scan::L<VB>::kSmem, st, sp);
}

// Shared by the forward and by the backward's recompute mode.
int run_forward_stages(const pkda_problem& p, const Geo& geo, const float* beta_c, bf16* u_ws,
                       bf16* Aqk, bf16* Akk, bf16* kt, float* gc, const float* a_start,
                       bf16* w, bf16* kg, bf16* v_new, bf16* h, bf16* qg, float* ST,
                       bool recompute, int* status, int* cursor, cudaStream_t st, bf16* o,
                       bool* o_done, const ChainArgs* chain, int scan_split) {
  IntraParams ip;
  ip.geo = geo;
  ip.q = static_cast<const bf16*>(p.q); ip.k = static_cast<const bf16*>(p.k);
  ip.v = static_cast<const bf16*>(p.v); ip.g = static_cast<const bf16*>(p.g);
  ip.g_atk = p.g_atk; ip.beta_atk = static_cast<const bf16*>(p.beta_atk);
  ip.A_log = p.A_log; ip.dt_bias = p.dt_bias; ip.log_atk_scale = p.log_atk_scale;
  ip.beta_c = beta_c; ip.a_start = a_start;
  ip.Aqk = Aqk; ip.Akk = Akk; ip.kt = kt; ip.gc = gc;
  ip.w = w; ip.u = u_ws; ip.kg = kg; ip.qg = qg;
  ip.scale = p.scale; ip.ln_x = logf(p.squash_x); ip.eps = p.squash_eps;
  ip.direct_cap = direct_block_cap();
  ip.by_strip = stage_variant(kStageIntraFwd) != 0 || ip.direct_cap < 64;
  ip.status = status; ip.cursor = cursor;
  ip.chain = 0;
  ip.beta = static_cast<const bf16*>(p.beta); ip.A0 = p.initial_A_state;
  ip.beta_c_w = ip.a_chain = ip.sa = ip.AT = nullptr;
  if (chain) {
    ip.chain = 1;
    ip.beta_c_w = chain->beta_c_w; ip.a_chain = chain->a_chain; ip.sa = chain->sa; ip.AT = chain->AT;
  }
  begin_stage(kStageIntraFwd, st);
  int rc = launch_intra_fwd_tc(ip, recompute, st);
  end_stage(st);
  if (rc != PKDA_OK) return rc;

  ScanParams sp;
  sp.geo = geo; sp.w = w; sp.u = u_ws; sp.kg = kg; sp.beta_c = beta_c; sp.gc = gc;
  sp.S0 = p.initial_state; sp.h = h; sp.v_new = v_new; sp.ST = ST;
  // Few units (scan_columns: while four or eight CTAs per unit run in one wave; scan_split of them, two at least, where the
  // backward's scan runs beside this one): the value columns of a unit spread over that many SMs, with the state in
  // mma.sync accumulators.  More units: tcgen05 / TMEM / TMA,
  // one CTA per (sequence, head).  The older mma.sync kernel, which slices the value columns when there are
  // fewer units than SMs, runs only when it is pinned (pkda_set_variant).  Same bits from the first two.
  const int units = p.n_seqs * p.heads;
  const int vb = units >= 120 ? 128 : (units >= 60 ? 64 : 32);
  const bool scan_mma = stage_variant(kStageScanFwd) == 1;
  // The tcgen05 scan also produces the output (it holds h and E of every chunk) unless a separate
  // output kernel is asked for (pkda_set_variant("out_fwd", 1: mma.sync, 2: tcgen05)).
  const bool fuse_out = o && !recompute && stage_variant(kStageOutFwd) == 0;
  if (o_done) *o_done = false;
  begin_stage(kStageScanFwd, st);
  if (status && !scan_mma && scan_columns(units)) {
    rc = launch_scan_fwd_cols(geo, p.total_tokens, units, w, kg, u_ws, beta_c, gc, p.initial_state, h, v_new,
                              recompute ? nullptr : ST, status, qg, Aqk, fuse_out ? o : nullptr,
                              scan_split ? scan_split : scan_columns(units), st);
    if (o_done) *o_done = fuse_out;
  } else if (status && !scan_mma) {
    rc = launch_scan_fwd_tc(geo, p.total_tokens, units, w, kg, u_ws, beta_c, gc, p.initial_state, h, v_new, ST,
                            status, recompute, qg, Aqk, fuse_out ? o : nullptr, st);
    if (o_done) *o_done = fuse_out;
  }
  else if (vb == 128) rc = recompute ? launch_scan_fwd<128, true>(sp, units, st) : launch_scan_fwd<128, false>(sp, units, st);
  else if (vb == 64) rc = recompute ? launch_scan_fwd<64, true>(sp, units, st) : launch_scan_fwd<64, false>(sp, units, st);
  else rc = recompute ? launch_scan_fwd<32, true>(sp, units, st) : launch_scan_fwd<32, false>(sp, units, st);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  return PKDA_OK;
}

int run_prologue(const pkda_problem& p, int* chunk_offsets, float* beta_c, Geo* geo, cudaStream_t st) {
  int rc = PKDA_OK;
  // beta_c == nullptr: the caller fills the chunk-major beta itself (the forward does, in its first kernel)
  if (p.cu_seqlens) {
    begin_stage(kStageOffsets, st);
    rc = launch_kernel(pkda_chunk_offsets_kernel, 1, 1024, 0, st, p.cu_seqlens, p.n_seqs, chunk_offsets);
    end_stage(st);
    if (rc != PKDA_OK) return rc;
  }
  *geo = make_geo(p, chunk_offsets);
  if (beta_c) {
    begin_stage(kStagePackBeta, st);
    rc = launch_kernel(pkda_pack_beta_kernel, geo->total_chunks, 256, 0, st, *geo, static_cast<const bf16*>(p.beta), beta_c);
    end_stage(st);
  }
  return rc;
}

int chunk_fwd(const pkda_chunk_fwd_args* a, cudaStream_t st) {
  const pkda_problem& p = a->p;
  int rc = check_chunk_problem(p);
  if (rc != PKDA_OK) return rc;
  if (p.n_seqs == 0 || p.total_tokens == 0) return PKDA_OK;
  if (!a->o || !a->Aqk || !a->Akk || !a->k_precond || !a->ac_atk || !a->a_atk || !a->sa_atk || !a->w ||
      !a->kg || !a->v_new || !a->h || !a->qg)
    return PKDA_ERR_NULL;
  if (!a->workspace || a->workspace_bytes < chunk_fwd_workspace(p)) return PKDA_ERR_WORKSPACE;
  // What moves sixteen or eight bytes at a time or by TMA.  (The column scans write o, h and v_new in eights and the
  // states by scalars; a_atk, sa_atk and the preconditioner's states are scalars everywhere.)
  if (!aligned({p.dt_bias, a->Aqk, a->Akk, a->ac_atk, a->w, a->kg, a->qg, a->workspace}, 16) || !aligned({a->k_precond}, 8))
    return PKDA_ERR_ALIGN;
  if (scan_columns(p.n_seqs * p.heads) ? !aligned({a->o, a->h, a->v_new}, 8) : !aligned({a->h, a->v_new, a->final_state}, 16))
    return PKDA_ERR_ALIGN;
  FwdWorkspace ws = carve_fwd(p, a->workspace);
  Geo geo;
  rc = run_prologue(p, ws.chunk_offsets, nullptr, &geo, st);
  if (rc != PKDA_OK) return rc;

  // Dense batches on the default kernels: the intra stage carries the preconditioner state across
  // chunks itself (and packs beta).  Otherwise two small kernels in front do.
  const bool chained = forward_chain_possible(p);
  if (!chained) {
    begin_stage(kStageAtkLocal, st);
    rc = launch_kernel(pkda_atk_local_kernel, geo.total_chunks * p.heads, 256, 0, st, geo, static_cast<const bf16*>(p.k), p.g_atk,
                  static_cast<const bf16*>(p.beta_atk), static_cast<const bf16*>(p.beta), a->ac_atk, a->sa_atk, ws.beta_c,
                  ws.status);
    end_stage(st);
    if (rc != PKDA_OK) return rc;
    begin_stage(kStageAtkCarry, st);
    rc = launch_kernel(pkda_atk_carry_kernel, dim3(p.n_seqs, p.heads), kD, 0, st, geo, a->ac_atk, a->sa_atk, p.initial_A_state, a->a_atk,
                  a->final_A_state);
    end_stage(st);
    if (rc != PKDA_OK) return rc;
  }

  // (The local scan also zeroes the status word and the cursor when it runs.)
  if (chained && (rc = launch_chain_init(a->a_atk, (size_t)geo.total_chunks * p.heads, ws.status, st)) != PKDA_OK) return rc;
  ChainArgs chain_args;
  chain_args.beta_c_w = ws.beta_c; chain_args.a_chain = a->a_atk; chain_args.sa = a->sa_atk;
  chain_args.AT = a->final_A_state;
  bool o_done = false;
  rc = run_forward_stages(p, geo, ws.beta_c, ws.u, static_cast<bf16*>(a->Aqk), static_cast<bf16*>(a->Akk),
                          static_cast<bf16*>(a->k_precond), a->ac_atk, a->a_atk, static_cast<bf16*>(a->w),
                          static_cast<bf16*>(a->kg), static_cast<bf16*>(a->v_new), static_cast<bf16*>(a->h),
                          static_cast<bf16*>(a->qg), a->final_state, false, ws.status, ws.status + 1, st,
                          static_cast<bf16*>(a->o), &o_done, chained ? &chain_args : nullptr);
  if (rc != PKDA_OK) return rc;

  // Output stage, when the scan has not produced o already: tcgen05 + TMA unless the mma.sync kernel is
  // pinned (pkda_set_variant).
  const size_t guard_n = std::min<size_t>((size_t)p.total_tokens * p.heads * kD, 4096);
  if (o_done) return PKDA_OK;  // (that kernel also marks the output if any kernel gave up)
  if (stage_variant(kStageOutFwd) != 1) {
    rc = launch_out_fwd_tc(geo, p.total_tokens, static_cast<const bf16*>(a->qg), static_cast<const bf16*>(a->h),
                           static_cast<const bf16*>(a->Aqk), static_cast<const bf16*>(a->v_new), ws.beta_c,
                           static_cast<bf16*>(a->o), ws.status, st);
    if (rc != PKDA_OK) return rc;
    return launch_status_guard(ws.status, a->o, nullptr, nullptr, guard_n, st);
  }
  OutParams op;
  op.geo = geo;
  op.qg = static_cast<const bf16*>(a->qg); op.h = static_cast<const bf16*>(a->h);
  op.Aqk = static_cast<const bf16*>(a->Aqk); op.v_new = static_cast<const bf16*>(a->v_new);
  op.beta_c = ws.beta_c; op.o = static_cast<bf16*>(a->o);
  if (!set_smem(pkda_out_fwd_kernel, outk::kSmem)) return PKDA_ERR_LAUNCH;
  begin_stage(kStageOutFwd, st);
  rc = launch_kernel(pkda_out_fwd_kernel, dim3(geo.total_chunks, p.heads), outk::kThreads, outk::kSmem, st, op);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  return launch_status_guard(ws.status, a->o, nullptr, nullptr, guard_n, st);
}

}  // namespace pkda

