// Building blocks of the state scans for few (sequence, head) units (forward, and the state cotangent of
// the backward).
//
// A scan carries a 128 x 128 fp32 matrix X[k][v] through the chunks of one (sequence, head).  The
// value columns v never meet, so one WARP owns 16 of them with all 128 rows, transposed: X^T[v][k] is
// the accumulator of mma.sync m16n8k16, 16 column tiles = 64 registers per lane, for the whole
// sequence.  The accumulator layout of one product is the A-operand layout of the next (row = lane / 4,
// column pair = lane % 4), so rounding X to bf16 and multiplying it with a chunk tile needs no
// shared memory, no barrier and no other warp; the B operands are the chunk's W, kg, qg, P tiles, read
// by ldmatrix from the 128-byte-swizzled tiles that TMA wrote.
//
// Why not tensor memory here: a chunk step through TMEM is a chain of MMA -> commit -> wait -> TMEM read ->
// shared memory -> fence -> block barrier, three times, about 4,500 cycles however few columns a CTA
// has; here it is some 140 mma.sync at 8.2 cycles each and a few hundred cycles between them, and the eight
// warps of a unit spread over four or eight SMs.  Why not for many units: every warp reads whole B tiles from shared
// memory (448 KB per unit and step when all eight sit on one SM), which took 330 us against the 192 us of
// the tensor-memory kernel at 128 units, T = 4096.
//
// Both kinds multiply the same bf16 operands in the same order of 16-deep k steps into fp32 accumulators
// (U enters through an identity operand here as there), and their results are the same bits; the tests
// compare rows of large batches with the same rows alone.
#pragma once

#include "pkda_chunk.cuh"
#include "pkda_tc.cuh"

namespace pkda {
namespace scanw {

constexpr int kTile = 16384;   // [64 tok][128] bf16 tile: two swizzled 64-column blocks
constexpr int kBlk = 8192;     // one block, and the [64][64] P tile

// Per-lane address parts.  N form: tile rows are the n index of B, k contiguous (plain ldmatrix);
// T form: tile rows are the k index of B, n contiguous (transposing ldmatrix).
struct Lane {
  uint32_t n_row, n_x, t_row, t_x;
  int g, t;
  __device__ __forceinline__ explicit Lane(int lane) {
    const uint32_t r7 = lane & 7, b8 = (lane >> 3) & 1, b16 = lane >> 4;
    n_row = (r7 + (b16 << 3)) * 128;
    n_x = (b8 ^ r7) << 4;
    t_row = (r7 + (b8 << 3)) * 128;
    t_x = (b16 ^ r7) << 4;
    g = lane >> 2;
    t = lane & 3;
  }
};

// B fragments of two n tiles (16 np ..) and one 16-element k step.
__device__ __forceinline__ void ldb_n(uint32_t (&r)[4], uint32_t tile, const Lane& L, int ks, int np) {
  ldsm_x4(r, tile + L.n_row + np * 2048 + (ks >> 2) * kBlk + (L.n_x ^ ((ks & 3) << 5)));
}
__device__ __forceinline__ void ldb_t(uint32_t (&r)[4], uint32_t tile, const Lane& L, int ks, int np) {
  ldsm_x4_t(r, tile + L.t_row + ks * 2048 + (np >> 2) * kBlk + (L.t_x ^ ((np & 3) << 5)));
}

// The warp's 16 columns of a [tok][v] tile, tokens 16 j .. + 15, transposed: an A operand [v][tok], and at
// the same time the pairs of accumulator tiles 2 j (r[0], r[1]: rows g, g + 8) and 2 j + 1 (r[2], r[3]).
// `piece`: 16-byte piece of the warp's first column inside its 64-column block.
__device__ __forceinline__ void ld_cols(uint32_t (&r)[4], uint32_t block, const Lane& L, int j, int piece) {
  ldsm_x4_t(r, block + L.n_row + j * 2048 + (L.n_x ^ (piece << 4)));
}

// A operand (k step ks): bf16 of accumulator tiles 2 ks and 2 ks + 1.
template <int N>
__device__ __forceinline__ void pack_a(uint32_t (&a)[4], const float (&x)[N][4], int ks) {
  a[0] = pack_bf16(x[2 * ks][0], x[2 * ks][1]);
  a[1] = pack_bf16(x[2 * ks][2], x[2 * ks][3]);
  a[2] = pack_bf16(x[2 * ks + 1][0], x[2 * ks + 1][1]);
  a[3] = pack_bf16(x[2 * ks + 1][2], x[2 * ks + 1][3]);
}

__device__ __forceinline__ uint32_t movmatrix(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// N pairs of 8x8 tiles (columns v0 .. +7 and v0 + 8 .. +15 of the destination, transposed in registers: the
// rows of tile pair i are destination rows first + 8 i + 0 .. 7) to global memory.  Lane (g, t) writes 8 bytes
// of row g, so that the four lanes of a row fill one 32-byte sector.  The pairs go through each of the three
// dependent steps together: one after the other they cost about 90 cycles each.
template <int N>
__device__ __forceinline__ void store_pairs(bf16* row, size_t stride8, int first, int valid, uint32_t (&lo)[N],
                                            uint32_t (&hi)[N], int t) {
  const bool odd = t & 1;
  uint32_t got[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    lo[i] = movmatrix(lo[i]);
    hi[i] = movmatrix(hi[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) got[i] = __shfl_xor_sync(0xffffffffu, odd ? lo[i] : hi[i], 1);
  row += odd ? 6 + 2 * t : 2 * t;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (first + 8 * i < valid)
      *reinterpret_cast<uint2*>(row + i * stride8) = odd ? make_uint2(got[i], hi[i]) : make_uint2(lo[i], got[i]);
}
// Two A operands (32 destination rows).
__device__ __forceinline__ void store_a2(bf16* row, size_t stride8, int first, int valid, const uint32_t (&a)[4],
                                         const uint32_t (&b)[4], int t) {
  uint32_t lo[4] = {a[0], a[2], b[0], b[2]}, hi[4] = {a[1], a[3], b[1], b[3]};
  store_pairs<4>(row, stride8, first, valid, lo, hi, t);
}

// Plain shared-memory accesses at a byte offset (compiler-visible, so that they can be scheduled).
__device__ __forceinline__ void put4(unsigned char* s, const uint32_t (&a)[4]) {
  *reinterpret_cast<uint4*>(s) = make_uint4(a[0], a[1], a[2], a[3]);
}
__device__ __forceinline__ void get4(const unsigned char* s, uint32_t (&a)[4]) {
  const uint4 x = *reinterpret_cast<const uint4*>(s);
  a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
}
__device__ __forceinline__ float2 get2f(const unsigned char* s) { return *reinterpret_cast<const float2*>(s); }

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One poll of each of two barriers, both in flight together.  A poll takes about a hundred cycles even when
// its phase is complete, so it is issued well before its answer is needed.
__device__ __forceinline__ bool mbar_try2(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1) {
  uint32_t d0, d1;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%2], %3;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 q, [%4], %5;\n\t"
      "selp.u32 %0, 1, 0, p;\n\tselp.u32 %1, 1, 0, q;\n\t}"
      : "=r"(d0), "=r"(d1) : "r"(bar0), "r"(parity0), "r"(bar1), "r"(parity1) : "memory");
  return d0 & d1;
}
// The same with a bounded wait behind it; the answer is the warp's.
__device__ __forceinline__ bool mbar_wait2(bool tried, uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1) {
  if (__all_sync(0xffffffffu, tried)) return true;
  const bool ok = tc::mbar_wait(bar0, parity0) && tc::mbar_wait(bar1, parity1);
  return __all_sync(0xffffffffu, ok);
}
// One arrival for the warp, after all its lanes are done.
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// Product of a bf16 pair with two fp32 factors, rounded back.
__device__ __forceinline__ uint32_t scale_pair(uint32_t x, float2 s) {
  const float2 v = unpack_bf16(x);
  return pack_bf16(s.x * v.x, s.y * v.y);
}

// B fragment half of the identity: nonzero where k = n inside an 8 x 8 block.
__device__ __forceinline__ uint32_t identity_b(const Lane& L) {
  return L.g == 2 * L.t ? 0x00003F80u : L.g == 2 * L.t + 1 ? 0x3F800000u : 0u;
}

// The four fragment pairs of a k step (N form), and of half a k step of a state update (T form, eight of the
// sixteen column tiles).
struct Frags { uint32_t r[4][4]; };
__device__ __forceinline__ void load_n(Frags& b, uint32_t tile, const Lane& L, int ks) {
#pragma unroll
  for (int np = 0; np < 4; ++np) ldb_n(b.r[np], tile, L, ks, np);
}
__device__ __forceinline__ void load_t(Frags& b, uint32_t tile, const Lane& L, int half) {
#pragma unroll
  for (int x = 0; x < 4; ++x) ldb_t(b.r[x], tile, L, half >> 1, 4 * (half & 1) + x);
}
__device__ __forceinline__ void mma4(float (*acc)[4], const uint32_t (&a)[4], const Frags& b) {
#pragma unroll
  for (int np = 0; np < 4; ++np) {
    mma_bf16(acc[2 * np], a, b.r[np][0], b.r[np][1]);
    mma_bf16(acc[2 * np + 1], a, b.r[np][2], b.r[np][3]);
  }
}

// X^T += f x tile: k steps of 16 tokens (tile rows), all 16 column tiles.  The fragments of the next half
// step are asked for before the products of the current one (the assembler keeps this order; loads behind
// the products cost their latency, about 50 cycles, every time); b: those of the first half, loaded before.
__device__ __forceinline__ void update_state(float (&X)[16][4], const uint32_t (&f)[4][4], uint32_t tile, const Lane& L,
                                             const Frags& first) {
  Frags b[2];
  b[0] = first;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i < 7) load_t(b[(i + 1) & 1], tile, L, i + 1);
    mma4(&X[8 * (i & 1)], f[i >> 1], b[i & 1]);
  }
}

// [64 tok][128] tile of an activation [tokens][H][128] in one TMA: dims {64, tokens, 2, H}.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// blocks: 2 = whole rows, 1 = one 64-column block per copy.
inline bool rows_map(CUtensorMap* map, const bf16* x, uint64_t heads, uint64_t tokens, uint32_t blocks) {
  const uint64_t dims[4] = {64, tokens, 2, heads}, str[3] = {heads * kD * 2, 128, kD * 2};
  const uint32_t box[4] = {64, 64, blocks, 1};
  return encode_bf16_map(map, x, 4, dims, str, box);
}
inline bool pairs_map(CUtensorMap* map, const bf16* x, uint64_t heads, uint64_t tokens) {  // [tokens][H][64]
  const uint64_t dims[3] = {kChunk, heads, tokens}, str[2] = {kChunk * 2, heads * kChunk * 2};
  const uint32_t box[3] = {64, 1, 64};
  return encode_bf16_map(map, x, 3, dims, str, box);
}

}  // namespace scanw
}  // namespace pkda
