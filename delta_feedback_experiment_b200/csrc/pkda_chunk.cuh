// Pieces shared by the chunked forward and backward kernels (D = 128, chunk 64).
#pragma once

#include "pkda_common.cuh"
#include "pkda_launch.h"

namespace pkda {

constexpr int kD = 128;                       // head width handled by the chunked kernels
constexpr int kLdD = kD + kPad;               // smem row stride of a [*][128] bf16 tile
constexpr int kLdC = kChunk + kPad;           // smem row stride of a [*][64] bf16 tile
constexpr int kTileBytes = kChunk * kLdD * 2; // one [64][128] bf16 tile

// Level `lvl` (4, 2 or 1, inside a strip of 8 rows) pairs row i (bit lvl set) with row j (bit
// lvl clear) of the same 2*lvl block, relative to the first row of the upper half.
__device__ __forceinline__ bool level_pair_ok(int i, int j, int lvl) {
  return (((i ^ j) & ~(2 * lvl - 1)) == 0) && (i & lvl) && !(j & lvl);
}

constexpr int kLdG = kD + 8;                  // smem row stride of a [64][128] fp32 array

// "Direct" pairing: all pairs j < i of a block of rows use ONE reference row: row factor
// 2^(G_i - G_ref) <= 1, column factor 2^(G_ref - G_j) >= 1.  That is only safe while the decay across
// the block stays far inside the fp32 / bf16 exponent range: the whole chunk is one block where it decays by
// at most kDirectLimit (log2 units), else strips of 8 rows have reference rows of their own.
// With the limit at 112 the column operand kt 2^112 (|kt| <= 1.5 |k|) and the fp32 sums of up to 128
// masked products of that size stay below 2^127, and the row operand k 2^-112 only loses (to the
// flush of denormals) channels with |k| < 2^-14, whose products are below the bf16 rounding of the
// others; chunks of the benchmark's gate distribution (about 75 +- 6 log2 units of decay per 64
// tokens) then practically always form one block.
constexpr float kDirectLimit = 112.f;
// Where a strip decays by more than that, each half of it (4 rows) is taken relative to its own first row and all columns
// relative to the strip's fifth row, as long as 5 tokens decay by at most kDirectLimit, the 2 outer ones by at most this and the 3
// behind the fifth row by twice this (log2 units): strip_decays.
constexpr float kOuterLimit = 45.f;
constexpr int kHalfRow = 4;
// {decay that kDirectLimit bounds, decay that kOuterLimit bounds} of a strip from the G of its rows.
__device__ __forceinline__ float2 strip_decays(float g0, float g2, float g4, float g5, float g7) {
  return make_float2(fmaxf(g0 - g5, g2 - g7), fmaxf(fmaxf(g0 - g2, g5 - g7), 0.5f * (g4 - g7)));
}

// 2^x by the hardware approximation (flushes denormal results to zero, which is
// what the gating factors want: every argument here is <= 0).
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void scale8(uint4& x, const float (&f)[8]) {
  uint32_t* w = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 v = unpack_bf16(w[j]);
    w[j] = pack_bf16(v.x * f[2 * j], v.y * f[2 * j + 1]);
  }
}

// Elementwise part of the decay gate for one chunk, all kNThreads threads: log2-domain
// per-token log-decay  -exp(A_log) log2(e) softplus(raw + bias)  into sG (zero for
// rows past the sequence end).  The cumulative sum over rows follows separately.
// The raw gate of the tile is fetched first (gate_load, at the top of a kernel, so
// that the loads fly while other data is set up) and converted later (gate_apply).
template <int kNThreads>
struct GateRaw {
  static constexpr int kIter = kChunk * kD / 8 / kNThreads;
  static_assert(kIter * kNThreads * 8 == kChunk * kD, "tile must divide evenly");
  uint4 raw[kIter];
};

template <int kNThreads>
__device__ __forceinline__ void gate_load(GateRaw<kNThreads>& gr, const bf16* g_row0, long gld, int valid, int tid) {
#pragma unroll
  for (int it = 0; it < GateRaw<kNThreads>::kIter; ++it) {
    const int idx = tid + it * kNThreads, r = idx >> 4, c8 = (idx & 15) << 3;
    gr.raw[it] = make_uint4(0, 0, 0, 0);
    if (r < valid) gr.raw[it] = *reinterpret_cast<const uint4*>(g_row0 + (size_t)r * gld + c8);
  }
}

template <int kNThreads>
__device__ __forceinline__ void gate_apply(const GateRaw<kNThreads>& gr, float* sG, int valid, const float* bias_h,
                                           float ea2, int tid) {
#pragma unroll
  for (int it = 0; it < GateRaw<kNThreads>::kIter; ++it) {
    const int idx = tid + it * kNThreads, r = idx >> 4, c8 = (idx & 15) << 3;
    float o[8];
    if (r < valid) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&gr.raw[it]);
      const float4 bA = *reinterpret_cast<const float4*>(bias_h + c8);
      const float4 bB = *reinterpret_cast<const float4*>(bias_h + c8 + 4);
      const float bb[8] = {bA.x, bA.y, bA.z, bA.w, bB.x, bB.y, bB.z, bB.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 v = unpack_bf16(w[j]);
        o[2 * j] = -ea2 * softplus_fast(v.x + bb[2 * j]);
        o[2 * j + 1] = -ea2 * softplus_fast(v.y + bb[2 * j + 1]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = 0.f;
    }
    *reinterpret_cast<float4*>(sG + r * kLdG + c8) = make_float4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<float4*>(sG + r * kLdG + c8 + 4) = make_float4(o[4], o[5], o[6], o[7]);
  }
}

// In-place cumulative sum over the 64 rows of sG, one channel per thread (tid < 128).
__device__ __forceinline__ void gate_cumsum(float* sG, int c) {
  float run = 0.f;
#pragma unroll 8
  for (int r = 0; r < kChunk; ++r) {
    run += sG[r * kLdG + c];
    sG[r * kLdG + c] = run;
  }
}

// One doubling step of the triangular inverse: for every pair of inverted diagonal
// blocks T11, T22 of size N (16 or 32) and their coupling block L21,
// T21 = -T22 (L21 T11), on the tensor cores: both products as
// mma.sync m16n8k8 TF32 with every fp32 operand split into a high and a low TF32
// part (three MMAs per step: lo*hi + hi*lo + hi*hi), which keeps fp32-level
// accuracy (the dropped lo*lo term is 2^-22 relative).  One warp per 16 x 8
// output tile; operands come straight from the fp32 arrays in shared memory.
//
// Rounding to TF32 (nearest, ties away from zero: what cvt.rna.tf32.f32 returns for
// finite values and infinities) is an integer add and a mask on the bit pattern; both
// run at full rate, the conversion instruction does not.  It would turn the NaN that arithmetic
// produces, 0x7fffffff, into -0.  The difference of a NaN and that is a NaN still, and for the low part the add
// is kept from overflowing: one instruction more, 546 -> 550 us for the intra kernel at 8 x 4,096 tokens of 16 heads.
__device__ __forceinline__ uint32_t tf32_rna(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }

__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo) {
  hi = tf32_rna(x);
  lo = tf32_rna(__int_as_float(min(__float_as_int(x - __uint_as_float(hi)), 0x7fffefff)));
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// d[16 x 8] += A[16 x K] B[K x 8] over the k range [kbeg, kend) (multiples of 8),
// A(r, m) = Ap[r * lda + m],  B(m, c) = Bp[m * ldb + c].  The fragment loads of A are
// free of bank conflicts when lda = 4 (mod 8), those of B when ldb = 8 (mod 16); with an
// odd stride (65) every one of them is a 4-way conflict, and the merge is bound by them.
template <int K>
__device__ __forceinline__ void tile_mma_3xtf32(float (&d)[4], const float* Ap, int lda, const float* Bp, int ldb,
                                                int lane, int kbeg, int kend) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 8) {
    if (k0 < kbeg || k0 >= kend) continue;
    const float a[4] = {Ap[g * lda + k0 + t], Ap[(g + 8) * lda + k0 + t], Ap[g * lda + k0 + t + 4],
                        Ap[(g + 8) * lda + k0 + t + 4]};
    const float b[2] = {Bp[(k0 + t) * ldb + g], Bp[(k0 + t + 4) * ldb + g]};
    uint32_t ah[4], al[4], bh[2], bl[2];
#pragma unroll
    for (int e = 0; e < 4; ++e) tf32_split(a[e], ah[e], al[e]);
#pragma unroll
    for (int e = 0; e < 2; ++e) tf32_split(b[e], bh[e], bl[e]);
    mma_tf32(d, al, bh);
    mma_tf32(d, ah, bl);
    mma_tf32(d, ah, bh);
  }
}

// kYPad widens the rows of the scratch Y to N + kYPad floats (8 makes the second
// product's B loads conflict-free; the scratch then holds 2 * 16 * 24 or 32 * 40 floats).
// The k-steps in which a triangular factor is all zero (the rows of T11 above the output
// tile's columns, the columns of T22 right of the output tile's rows) are left out: the
// sums lose only exact zeros.
template <int N, int kYPad>
__device__ __forceinline__ void inverse_merge_tc(const float* sL, float* sT, float* sY2, int ldl, int ldt, int tid) {
  constexpr int kMT = N / 16, kNT = N / 8, kTiles = (32 / N) * kMT * kNT;  // N = 32: 8 tiles, N = 16: 4 tiles
  constexpr int ldy = N + kYPad;
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int pr = warp / (kMT * kNT), mt = (warp / kNT) % kMT, nt = warp % kNT;
  const int base = pr * 2 * N;
  if (warp < kTiles) {  // Y = L21 T11
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    tile_mma_3xtf32<N>(d, sL + (base + N + 16 * mt) * ldl + base, ldl, sT + base * ldt + base + 8 * nt, ldt, lane,
                       8 * nt, N);
    float* y = sY2 + pr * N * ldy + (16 * mt + g) * ldy + 8 * nt + 2 * t;
    *reinterpret_cast<float2*>(y) = make_float2(d[0], d[1]);
    *reinterpret_cast<float2*>(y + 8 * ldy) = make_float2(d[2], d[3]);
  }
  __syncthreads();
  if (warp < kTiles) {  // T21 = -T22 Y
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    tile_mma_3xtf32<N>(d, sT + (base + N + 16 * mt) * ldt + base + N, ldt, sY2 + pr * N * ldy + 8 * nt, ldy, lane, 0,
                       16 * mt + 16);
    float* o = sT + (base + N + 16 * mt + g) * ldt + base + 8 * nt + 2 * t;
    o[0] = -d[0];
    o[1] = -d[1];
    o[8 * ldt] = -d[2];
    o[8 * ldt + 1] = -d[3];
  }
  __syncthreads();
}

// T = (I + L)^-1 for a 64 x 64 strictly lower triangular L (fp32; row strides ldl of L, a
// multiple of 4, and ldt of T), all nthreads threads of the CTA (at least 256): the 16 x 16
// diagonal blocks by forward substitution, one column per thread of two warps with the column in
// registers, while the other warps zero the blocks above them; then two doubling steps on the
// tensor cores.  (Substitution only up to 4 x 4 and two fp32 doubling steps more are six block
// barriers and about 1,500 cycles of dependent shared-memory round trips instead of 500.)
// sY2 is a scratch of 1024 floats (kYPad = 0) or 1280 (kYPad = 8).  The result does not depend on
// the strides or on kYPad.  L must be visible to every thread on entry (a barrier after its
// last write); ends with a __syncthreads().
template <int kYPad = 0>
__device__ __forceinline__ void unit_lower_inverse_64(const float* sL, float* sT, float* sY2, int ldl, int ldt, int tid,
                                                      int nthreads) {
  if (tid < 64) {
    const int base = tid & 48, col = tid & 15;
    const float* L = sL + base * ldl + base;
    float* T = sT + base * ldt + base + col;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s = (i == col) ? 1.f : 0.f, s2 = 0.f;
#pragma unroll
      for (int m = 0; m < i; m += 4) {
        const float4 l = *reinterpret_cast<const float4*>(L + i * ldl + m);
        s -= l.x * x[m];
        if (m + 1 < i) s2 -= l.y * x[m + 1];
        if (m + 2 < i) s -= l.z * x[m + 2];
        if (m + 3 < i) s2 -= l.w * x[m + 3];
      }
      x[i] = s + s2;
      T[i * ldt] = x[i];
    }
  } else {
    // the 16 x 16 blocks above the diagonal: block rows 0..2, four columns per thread and step
    for (int i = tid - 64; i < 48 * 16; i += nthreads - 64) {
      const int r = i >> 4, c4 = (i & 15) << 2;
      if ((c4 >> 4) > (r >> 4)) *reinterpret_cast<float4*>(sT + r * ldt + c4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __syncthreads();
  inverse_merge_tc<16, kYPad>(sL, sT, sY2, ldl, ldt, tid);
  inverse_merge_tc<32, kYPad>(sL, sT, sY2, ldl, ldt, tid);
}

// Sums each of v[0..7] over the 32 lanes.  On return lane l holds in v[0] the
// total of entry ((l >> 4) & 1) * 4 + ((l >> 3) & 1) * 2 + ((l >> 2) & 1).
__device__ __forceinline__ void row_sums8(float (&v)[8], int lane) {
  const bool hi16 = lane & 16, hi8 = lane & 8, hi4 = lane & 4;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float keep = hi16 ? v[j + 4] : v[j], send = hi16 ? v[j] : v[j + 4];
    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float keep = hi8 ? v[j + 2] : v[j], send = hi8 ? v[j] : v[j + 2];
    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  {
    const float keep = hi4 ? v[1] : v[0], send = hi4 ? v[0] : v[1];
    v[0] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The same for v[0..3], in the same order; lane l holds the total of entry ((l >> 4) & 1) * 2 + ((l >> 3) & 1).
__device__ __forceinline__ void row_sums4(float (&v)[4], int lane) {
  const bool hi16 = lane & 16, hi8 = lane & 8;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float keep = hi16 ? v[j + 2] : v[j], send = hi16 ? v[j] : v[j + 2];
    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  const float keep = hi8 ? v[1] : v[0], send = hi8 ? v[0] : v[1];
  v[0] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

// Tail of the classifier kernel: a CTA has put the kind of its 64 items into sKind (-1: none, 0:
// tensor-memory kernel, 1: mma.sync kernel) and their first tokens into sTok, and appends them to the two
// work lists with one atomic per list, keeping their order.  One warp per list, two items per lane.
__device__ __forceinline__ void append_work_items(const int* sKind, const int* sTok, int2* fast_list, int* slow_list,
                                                  int* counts, int first_item, int tid) {
  __syncthreads();
  const int list = tid >> 5, lane = tid & 31;
  if (list >= 2) return;
  const bool in0 = sKind[lane] == list, in1 = sKind[lane + 32] == list;
  const uint32_t m0 = __ballot_sync(0xffffffffu, in0), m1 = __ballot_sync(0xffffffffu, in1);
  const int n0 = __popc(m0), n1 = __popc(m1);
  int at = 0;
  if (lane == 0 && n0 + n1) at = atomicAdd(counts + list, n0 + n1);
  at = __shfl_sync(0xffffffffu, at, 0);
  const uint32_t below = (1u << lane) - 1;
  const int p0 = at + __popc(m0 & below), p1 = at + n0 + __popc(m1 & below);
  if (list) {
    if (in0) slow_list[p0] = first_item + lane;
    if (in1) slow_list[p1] = first_item + lane + 32;
  } else {
    if (in0) fast_list[p0] = make_int2(first_item + lane, sTok[lane]);
    if (in1) fast_list[p1] = make_int2(first_item + lane + 32, sTok[lane + 32]);
  }
}

// Arguments of the intra-chunk forward stage (both implementations).
struct IntraParams {
  Geo geo;
  const bf16 *q, *k, *v, *g;
  const float* g_atk;
  const bf16* beta_atk;
  const float *A_log, *dt_bias, *log_atk_scale;
  const float* beta_c;
  const float* a_start;
  bf16 *Aqk, *Akk, *kt;
  float* gc;  // [chunks][H][D] exp of the chunk's total log-decay
  bf16 *w, *u, *kg, *qg;
  float scale, ln_x, eps;
  int direct_cap;  // below 64: every chunk by strips; below 8: by levels inside them
  int* status;     // device status word (tcgen05 kernel): set to 1 when a bounded wait gives up
  int* cursor;     // the CTAs draw their items with it (zeroed before every call)
  int by_strip;    // nonzero: every chunk is paired strip by strip, whatever it decays by
  // Preconditioner state across chunks inside the tensor-memory kernel (dense batches; chain != 0):
  // every item computes its chunk's local scan anyway, so it takes its chunk-entry state from the item
  // of the chunk before (a_chain, which is the saved "state at chunk starts" tensor; launch_chain_init
  // has marked all of it as not there yet), and publishes the next chunk's.  The items are
  // then drawn chunk level by chunk level across all (row, head) units, so that an item's predecessor
  // started long before it.  beta (raw) is packed to beta_c_w on the way; sa takes the chunk's summed
  // preconditioner log-decay, A0 / AT are the initial / final preconditioner states (may be NULL).
  int chain;
  const bf16* beta;
  float *beta_c_w, *a_chain, *sa, *AT;
  const float* A0;
};

// tcgen05 / tensor-memory intra-chunk forward stage (pkda_intra_fwd_tc.cu).
int launch_intra_fwd_tc(const IntraParams& ip, bool recompute, cudaStream_t st);
// What a chained launch finds: no entry of a_chain there yet, the status word and the cursors zero.
int launch_chain_init(float* a_chain, size_t items, int* zero, cudaStream_t st);

// Arguments of the chunk-parallel backward stage (both implementations).
struct IntraBwdParams {
  Geo geo;
  const bf16 *q, *k, *kt, *g;
  const float *A_log, *dt_bias;
  const float *beta_c, *gc;
  const bf16 *Akk, *v_new, *h, *dh, *dF, *d_o;
  bf16 *dq, *dv, *dg, *dbeta;
  float *dk_read, *dkt;
  float *partA, *partB;
  float scale;
  int direct_cap;
  int use_tma;   // the five phase-A tiles of full chunks arrive by TMA (tensor maps valid)
  int out_tma;   // dq, dv, dk_read and dkt of full chunks leave by TMA from padded shared-memory tiles
  int* status;   // set to 1 if a bounded wait gives up
  // The local part of the preconditioner's backward runs inside the chunk kernels: with B the write-key factor kt = k B(A_t),
  //   dkt buffer <- dA_local = d(loss)/dA_t through B alone,  dk_read buffer <- dk_read + dkt B,
  //   c_loc[chunk] = sum_r (prod_{j<=r} decay_j) dA_local_r,  partC[chunk] = d(loss)/d(centre).
  const float* g_atk;
  const bf16* beta_atk;
  const float* log_atk_scale;
  const float* a_start;
  float *c_loc, *partC;
  float ln_x, eps;
  // Work lists of (chunk * heads + head) items written by pkda_bwd_classify_kernel: fast_list for the
  // tensor-memory kernel (each with its chunk's first token: a full chunk is all that this kernel takes),
  // slow_list for the mma.sync kernel; fast_count[0] / fast_count[1] are their
  // lengths and fast_count[2] the cursor the mma.sync CTAs draw items with (all zeroed before every
  // call).  slow_list == NULL: the mma.sync kernel takes every chunk, one CTA per (chunk, head).
  int2* fast_list;
  int *slow_list, *fast_count;
};

// tcgen05 / tensor-memory chunk-parallel backward stage (pkda_intra_bwd_tc.cu).
int launch_intra_bwd_tc(const IntraBwdParams& ip, cudaStream_t st);
// The backward's first kernel on the default path: sorts the items into the two work lists (counts zeroed
// before) and packs beta chunk-major.
int launch_bwd_classify(const Geo& geo, const float* gc, int direct_cap, int2* fast_list, int* slow_list, int* counts,
                        const bf16* beta, float* beta_c, cudaStream_t st);

// tcgen05 / TMA output stage (pkda_out_tc.cu).
int launch_out_fwd_tc(const Geo& geo, int total_tokens, const bf16* qg, const bf16* h, const bf16* Aqk,
                      const bf16* v_new, const float* beta_c, bf16* o, int* status, cudaStream_t st);

// tcgen05 / TMA forward state scan (pkda_scan_tc.cu): one CTA per (sequence, head).
int launch_scan_fwd_tc(const Geo& geo, int total_tokens, int units, const bf16* w, const bf16* kg, const bf16* u,
                       const float* beta_c, const float* gc, const float* S0, bf16* h, bf16* v_new, float* ST,
                       int* status, bool recompute, const bf16* qg, const bf16* Aqk, bf16* o, cudaStream_t st);

// tcgen05 / TMA reverse state scan of the backward (pkda_scan_bwd_tc.cu): one CTA per (sequence, head).
int launch_scan_bwd_tc(const Geo& geo, int total_tokens, int units, const bf16* kg, const bf16* w, const bf16* qg,
                       const bf16* d_o, const bf16* Aqk, const float* beta_c, const float* gc, const float* dST,
                       bf16* dh, bf16* dF, float* dS0, int* status, bool beside, cudaStream_t st);

// The same two scans with the value columns spread over `split` SMs (pkda_scan_fwd.cu, pkda_scan_bwd.cu).
int launch_scan_fwd_cols(const Geo& geo, int total_tokens, int units, const bf16* w, const bf16* kg, const bf16* u,
                         const float* beta_c, const float* gc, const float* S0, bf16* h, bf16* v_new, float* ST,
                         int* status, const bf16* qg, const bf16* Aqk, bf16* o, int split, cudaStream_t st);
int launch_scan_bwd_cols(const Geo& geo, int total_tokens, int units, const bf16* kg, const bf16* w, const bf16* qg,
                         const bf16* d_o, const bf16* Aqk, const float* beta_c, const float* gc, const float* dST,
                         bf16* dh, bf16* dF, float* dS0, int* status, int split, bool beside, cudaStream_t st);
// CTAs per unit, 0 where the tensor-memory scans are taken: as many as still run in one wave (one per SM).
int scan_columns(int units);
// CTAs per unit of the two state scans of a lean backward, which need nothing of each other and run side by side while
// both fit the chip; {0, 0} where they run one after the other.  (1: the tensor-memory scans.)
struct ScanPair { int fwd, bwd; };
ScanPair scan_pair(int units);

// Host-side pieces defined in pkda_chunk_fwd.cu and reused by the backward.
int check_chunk_problem(const pkda_problem& p);
int run_prologue(const pkda_problem& p, int* chunk_offsets, float* beta_c, Geo* geo, cudaStream_t st);
// cursor: a zeroed int.
// o / o_done: the forward's output tensor; *o_done says whether the state scan has already written it.
// What the tensor-memory intra kernel needs to carry the preconditioner state across chunks itself
// (dense batches; NULL: it does not): see IntraParams::chain.
// scan_split: CTAs per unit of a recompute pass's scan beside which the backward's runs (ScanPair::fwd), 0 where it runs alone.
struct ChainArgs {
  float *beta_c_w, *a_chain, *sa, *AT;
};
int run_forward_stages(const pkda_problem& p, const Geo& geo, const float* beta_c, bf16* u_ws, bf16* Aqk,
                       bf16* Akk, bf16* kt, float* gc, const float* a_start, bf16* w, bf16* kg, bf16* v_new,
                       bf16* h, bf16* qg, float* ST, bool recompute, int* status, int* cursor,
                       cudaStream_t st, bf16* o = nullptr, bool* o_done = nullptr, const ChainArgs* chain = nullptr,
                       int scan_split = 0);

}  // namespace pkda
