// Intra-chunk stage of the chunked forward on tcgen05 / tensor memory (D = 128, chunk 64).
//
// Persistent CTAs of 256 threads, two per SM (112 KB of shared memory and 256 tensor-memory
// columns each), walk the (chunk, head) items.  What the stage computes is described at the top of
// pkda_chunk_fwd.cu.  A chunk whose decay lets it be ONE direct block (pkda_chunk.cuh) has one set of gated
// operands for all its pairs, k 2^G, q 2^G and kt 2^-G with G the cumulative log2-decay from the chunk
// start, and its pair products are tcgen05.mma.  A chunk that turns out (once its cumulative decay is known)
// to decay by more than kDirectLimit takes its pair products strip by strip on mma.sync (pairs_of_strip
// below) and rejoins the others at the inverse.  The decision depends on the inputs only, so the
// recompute pass of a lean backward decides the same way.  (Such chunks used to go on a list for a kernel of
// their own, 198 KB of staged operands and one CTA per SM: 2,048 of them 303 us with the pass that listed them, 164 here.)
//
//  * Elementwise work runs on registers in a "strip" layout: warp w owns rows 8w..8w+7 of the
//    chunk, lane l owns channels 4l..4l+3, so a warp reads or writes whole 256-byte token rows.
//    The two sequential passes over the rows (cumulative log-decay, the preconditioner
//    recurrence A_t) are blocked scans: eight rows in registers, one exchange of (block total,
//    block decay) through shared memory, then each block continues from the prefix it is owed.
//  * q, k and the raw gate arrive by TMA straight in the places of the operand tiles their
//    gated values will take (128-byte-swizzled canonical layout); the gating happens in
//    place, each thread touching only its own 8-byte pieces.  (24 eight-byte cp.async a thread
//    instead cost 100 instructions of address arithmetic: 475 -> 467 us for 8 x 4,096 tokens of
//    16 heads, 1,865 -> 1,795 us for 65,536 packed tokens of 32.)  The rows of k and q are stacked
//    to one 128-row A operand, the write keys are the B operand: eight tcgen05.mma (M = 128,
//    N = 64, K = 16) give M = k kt^T in accumulator rows 0..63 and P = q kt^T in rows 64..127.
//    All eight warps read the accumulator back (one tensor-memory lane = one row per thread)
//    and write L = tril(M, -1) diag(beta) in fp32 and scale tril(P) in bf16.
//  * T = (I + L)^-1 stays on the CUDA cores and 3xTF32 mma.sync (pkda_chunk.cuh): it needs
//    fp32-level accuracy and its products are at most 32 x 32.
//  * W = T Kd and U = T V are two more accumulators (M = 64 tokens, N = 128 channels, K = 64
//    tokens): a thread reads back channel pairs of two tokens, which it rounds and stores by stmatrix (with channels as rows a
//    thread held one channel of 32 tokens, 64 two-byte stores: 414 -> 406 us at 8 x 4,096 tokens of 16 heads).  V and the
//    outputs of full chunks move by TMA.
//
// Every mbarrier wait is bounded; a CTA whose wait gives up sets the status word.
#include "pkda_chunk.cuh"
#include "pkda_tc.cuh"


namespace pkda {

namespace intratc {
constexpr int kThreads = 256;
constexpr int kLdL = 68;                    // row stride of L and T: float4 rows, and conflict-free MMA fragments
constexpr int oA = 0;                       // 2 blocks [128 rows][64 ch]: rows 0..63 k 2^G (= Kd, the MN-major B of
                                            // W = T Kd), rows 64..127 q 2^G (together the K-major A of the pair products)
constexpr int oY = oA + 32768;              // 2 blocks [64 rows][64 ch]: kt 2^-G (K-major B); + 1 KB so that T fits
constexpr int oV = oY + 16384 + 1024;       // 2 blocks [64 tok][64 ch]: V (MN-major B of U = T V)
constexpr int oTm = oV + 16384;             // [64 i][64 j] bf16 T (K-major A)
constexpr int oX = oTm + 8192;              // the last quarter of oG; with oP the place U leaves from (W: from oV)
constexpr int oG = oV;                      // f32 [64][128], while a chunk is paired by strips: kt 2^(z - G), or G; V, T and 8 KB more
constexpr int oP = oX + 8192;               // [64 i][64 j] bf16 scale * P
constexpr int oL = oP + 8192;               // f32 [64][68] L; before the products: the scan exchange arrays; when recomputing the
                                            // write keys, 2 blocks [64 tok][64 ch] by TMA
constexpr int oBeta = oL + 64 * kLdL * 4;   // f32 [64]
constexpr int oDiag = oBeta + 256;          // f32 [64] q_i . kt_i
constexpr int oStep = oDiag + 256;          // f32 [8][128] factors between the strips (pairs_of_strip)
constexpr int oBar = oStep + 4096;          // TMA barrier, MMA barrier, tensor-memory base address
constexpr int kSmem = oBar + 64 + 1024;     // + slack to align the tiles to 1024 bytes
// inside the L region before the products
constexpr int oTot = oL;                    // f32 [8][128] per-strip decay totals
constexpr int oEnd = oL + 4096;             // f32 [8][128] per-strip end value of the zero-start A scan
constexpr int oDec = oL + 8192;             // f32 [8] per-strip product of preconditioner decays
constexpr int oSum = oDec + 32;             // f32 [8] per-strip sum of the preconditioner's log-decays
constexpr int oA0 = oSum + 32;              // f32 [128] the chunk-entry preconditioner state (chained mode)
constexpr int oZin = oL + 9216;             // f32 [8][128] G of the fifth row of every strip
// between those and the products, the strip's own factors where its rows of P come later: strip w, 2 x f32 [128]
constexpr int oD0 = oP, oD1 = oP + 512;     // + 1024 w
// while the inverse runs: T in the (dead) write-key operand, its scratch in the (dead) q rows of block 0
constexpr int oT = oY;                      // f32 [64][68]
constexpr int oY2 = oA + 8192;              // f32 [1280]
static_assert(oG + 32768 == oP && oBar % 8 == 0, "the decays fill what lies between the write keys and P");
static_assert(oL % 1024 == 0 && oL + 16384 <= oBeta, "the write keys arrive in swizzled blocks");
static_assert(oA0 + 512 <= oZin && oZin + 4096 <= oBeta && oT + 64 * kLdL * 4 <= oV && oY2 + 5120 <= oA + 16384, "aliases must fit");
static_assert(2 * (kSmem + 1024) <= 233472, "two CTAs per SM");
constexpr uint32_t kCols = 256;             // pair accumulator 0..63; later W 0..127, U 128..255
}  // namespace intratc

__device__ __forceinline__ void unpack4(uint2 r, float (&f)[4]) {
  const float2 a = unpack_bf16(r.x), b = unpack_bf16(r.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ uint2 scale4(uint2 r, const float (&f)[4]) {
  float x[4];
  unpack4(r, x);
  return make_uint2(pack_bf16(x[0] * f[0], x[1] * f[1]), pack_bf16(x[2] * f[2], x[3] * f[3]));
}

// The hand-over of the preconditioner state between items: one 32-bit word per channel that is either kNotYet or the
// value, so that nothing has to be ordered (no arithmetic result has this bit pattern: a NaN comes out as 0x7fffffff).
constexpr uint32_t kNotYet = 0xffffffffu;
__device__ __forceinline__ uint32_t ld_relaxed(const float* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(__float_as_uint(v)) : "memory");
}
__device__ __forceinline__ uint32_t ld_u16(const bf16* p) {
  uint32_t v;
  asm volatile("ld.global.nc.u16 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
// Before a chained launch: every word of the hand-over to kNotYet, the status word and the cursors to zero.
// (By single words: the caller's a_chain need not start on a 16-byte boundary.)
__global__ void __launch_bounds__(256) pkda_chain_init_kernel(uint32_t* a_chain, size_t n, int* zero) {
  after_previous();
  if (blockIdx.x == 0 && threadIdx.x < 8) zero[threadIdx.x] = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) a_chain[i] = kNotYet;
}

// ---- Pair products of a chunk that decays too much for one reference row.
//
// The unit is a strip of 8 rows, one per warp.  Its k rows and its q rows together are the 16-row A operand of
// mma.sync m16n8k16, the 8 write keys of strip J <= I the B operand, so one product gives both M and P of
// a strip pair.  With a reference row x(I) for the rows of strip I and z(J) for the columns of strip J,
//   2^(G_i - G_j) = 2^(G_i - x(I)) 2^(x(I) - z(J)) 2^(z(J) - G_j):
// the first factor is in the A operand, staged once per strip; kt times the third is kept in fp32, and a warp
// multiplies it with the second, one number per channel and strip pair, and rounds the product to the B operand.
// x(I) is the strip's first row and z(J) its last, so every factor of two strips is <= 1; inside a strip the second one is
// 2^(decay of 7 tokens), which kDirectLimit bounds.  Strips that decay by more go by halves: x is the first row of the row's
// own half, z the strip's fifth row, and a strip pair takes one product per half (the other half's rows of the A operand are zero),
// with the factors 2^(x - z) of either.  The factors of the rows behind z are > 1; strip_decays bounds them, so nothing
// inside a strip is lost, and of two strips nothing above 2^(2 kOuterLimit - 126).  (One row in the middle as the reference of all
// eight needs no second product, but then two of eight neighbours keep an operand as it is, not four, and neighbours are
// what the gradient of such gates is made of: its error against 64 bits was 1.5 % larger on average.  The second product
// costs 538 -> 546 us here and 1,386 -> 1,416 in the backward at 8 x 4,096 tokens of 16 heads, exp(A_log) from 1 to 16.)  Chunks beyond that go
// through pair_exact.  A strip pair costs 11 instructions per 16 channels and no exponential;
// gating both fragments from G by exponentials took 66, and with them the pairs were 10,000 of the 34,000 cycles of an
// item alone on its SM instead of 4,500 (2,048 chunks: 182 us instead of 164).
struct PairLane {
  uint32_t a_row, s_row, s_blk, a_x, b_row, b_x, g_x;
  int g, t;
  __device__ __forceinline__ explicit PairLane(int lane) {
    using namespace intratc;
    const uint32_t m = lane >> 3, r = lane & 7;
    a_row = oA + (m & 1) * 8192 + r * 128;    // matrices: k rows, q rows (channels 0..7 of the step), k rows, q rows (8..15)
    s_row = ((m & 1) ? oA + 8192 : oY) + r * 128;  // the same of the staged operand: its k rows are where the write keys
    s_blk = (m & 1) ? 16384 : 8192;                // of other chunks are (Kd has the place of k)
    a_x = ((m >> 1) ^ r) << 4;
    b_row = r * 128;                          // matrices: write keys (channels 0..7, 8..15), twice
    b_x = ((m & 1) ^ r) << 4;
    g = lane >> 2;
    t = lane & 3;
    g_x = row_x(g);
  }
  // Byte offset of this lane's channel pair 2 t inside an fp32 row whose index is r (mod 4): the 16-byte pieces of a
  // row are permuted by 2 (r mod 4), so that the 4 rows x 2 pieces of half a warp lie in different banks.  A step
  // of 16 channels flips bits from 64 up, the pair 8 channels on is 32 bytes away (both by exclusive or).
  __device__ __forceinline__ uint32_t row_x(int r) const { return (((t >> 1) ^ ((r & 3) << 1)) << 4) + ((t & 1) << 3); }
};
__device__ __forceinline__ float2 ld_f2(const unsigned char* s) { return *reinterpret_cast<const float2*>(s); }
// L = tril(M, -1) diag(beta) and scale * tril(P) (its diagonal is ungated) of strip pair (I, J).
__device__ __forceinline__ void put_pair(unsigned char* tiles, const PairLane& L, int I, int J, const float (&acc)[4], float scale) {
  using namespace intratc;
  const int i = 8 * I + L.g, j = 8 * J + 2 * L.t;
  const float2 be = ld_f2(tiles + oBeta + 4 * j);
  const float dv = *reinterpret_cast<const float*>(tiles + oDiag + 4 * i);
  *reinterpret_cast<float2*>(tiles + oL + (i * kLdL + j) * 4) =
      make_float2(j < i ? acc[0] * be.x : 0.f, j + 1 < i ? acc[1] * be.y : 0.f);
  const float p0 = j < i ? acc[2] : j == i ? dv : 0.f, p1 = j + 1 < i ? acc[3] : j + 1 == i ? dv : 0.f;
  *reinterpret_cast<uint32_t*>(tiles + oP + i * 128 + ((J ^ L.g) << 4) + 4 * L.t) = pack_bf16(p0 * scale, p1 * scale);
}
// All pairs of strip I (the warp's), with the factors 2^(x(I) - z(I)) at oD0, 2^(x(I) - z(I - 1)) at oD1 and
// 2^(z(J) - z(J - 1)) at oStep; by halves x(I) is the first half's there, and the second half's is z(I).
template <bool kHalves>
__device__ __forceinline__ void pairs_of_strip(unsigned char* tiles, uint32_t base, int I, int lane, float scale) {
  using namespace intratc;
  const PairLane L(lane);
  // Strips whose factor is zero (below the smallest normal number) in all channels are left out.
  int n = 1;
  {
    float4 d = *reinterpret_cast<const float4*>(tiles + oD1 + I * 1024 + (lane << 4));
    while (n <= I && __any_sync(0xffffffffu, fmaxf(fmaxf(d.x, d.y), fmaxf(d.z, d.w)) > 0.f)) {
      ++n;
      const float4 f = *reinterpret_cast<const float4*>(tiles + oStep + (I - n + 1) * 512 + (lane << 4));
      d.x *= f.x; d.y *= f.y; d.z *= f.z; d.w *= f.w;
    }
  }
  float acc[8][4];  // [d]: strip I - d
#pragma unroll
  for (int d = 0; d < 8; ++d) acc[d][0] = acc[d][1] = acc[d][2] = acc[d][3] = 0.f;
  const uint32_t ra = base + L.s_row + I * 1024, tx = L.row_x(0);
  const unsigned char *y = tiles + oG + (8 * I + L.g) * 512, *d0 = tiles + oD0 + I * 1024, *d1 = tiles + oD1 + I * 1024,
                      *step = tiles + oStep + I * 512;
  uint32_t a[4];
  ldsm_x4(a, ra + L.a_x);
#pragma unroll 1
  for (int ks = 0; ks < 8; ++ks) {
    const uint32_t yo = L.g_x ^ (ks << 6), to = tx + (ks << 6);
    uint32_t an[4] = {0u, 0u, 0u, 0u};
    if (ks < 7) ldsm_x4(an, ra + ((ks + 1) >> 2) * L.s_blk + (L.a_x ^ (((ks + 1) & 3) << 5)));
    float2 f0 = ld_f2(d0 + to), f1 = ld_f2(d0 + to + 32);
    const float2 c0 = make_float2(__fdividef(1.f, f0.x), __fdividef(1.f, f0.y));  // from the first half's factor to the second's
    const float2 c1 = make_float2(__fdividef(1.f, f1.x), __fdividef(1.f, f1.y));
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      // in twos: a strip too many (before the chunk's first, or one that has vanished) is computed and dropped
      if (!(d & 1) && d >= n) break;
      if (d == 1) {
        f0 = ld_f2(d1 + to);
        f1 = ld_f2(d1 + to + 32);
      } else if (d > 1) {
        const float2 s0 = ld_f2(step + to - (d - 1) * 512), s1 = ld_f2(step + to + 32 - (d - 1) * 512);
        f0.x *= s0.x; f0.y *= s0.y; f1.x *= s1.x; f1.y *= s1.y;
      }
      const float2 y0 = ld_f2(y + yo - d * 4096), y1 = ld_f2(y + (yo ^ 32) - d * 4096);
      uint32_t b0 = pack_bf16(y0.x * f0.x, y0.y * f0.y), b1 = pack_bf16(y1.x * f1.x, y1.y * f1.y);
      if (!kHalves) {
        mma_bf16(acc[d], a, b0, b1);
      } else {
        const bool lo = L.g < kHalfRow;
        const uint32_t al[4] = {lo ? a[0] : 0u, lo ? a[1] : 0u, lo ? a[2] : 0u, lo ? a[3] : 0u};
        const uint32_t ah[4] = {lo ? 0u : a[0], lo ? 0u : a[1], lo ? 0u : a[2], lo ? 0u : a[3]};
        if (d == 0 && !lo) b0 = b1 = 0u;  // (columns of the second half have no rows in the first, and their factor no bound)
        mma_bf16(acc[d], al, b0, b1);
        if (d == 0) mma_bf16(acc[d], ah, pack_bf16(y0.x, y0.y), pack_bf16(y1.x, y1.y));
        else mma_bf16(acc[d], ah, pack_bf16(y0.x * (f0.x * c0.x), y0.y * (f0.y * c0.y)), pack_bf16(y1.x * (f1.x * c1.x), y1.y * (f1.y * c1.y)));
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = an[e];
  }
  __syncwarp();  // (P takes the place of the strip's factors)
#pragma unroll
  for (int d = 0; d < 8; ++d) {
    if (d >= n) acc[d][0] = acc[d][1] = acc[d][2] = acc[d][3] = 0.f;
    if (d <= I) put_pair(tiles, L, I, I - d, acc[d], scale);
  }
}
// Strip pair (I, J) at any decay, from the raw rows and G.  J < I: relative to the first row of I.  J = I: the pairs of
// level lvl = 4, 2, 1 (rows with that bit set against rows without, relative to the first row of the upper half; every row
// has its own reference); acc keeps the others.
__device__ __forceinline__ void pair_exact(float (&acc)[4], const unsigned char* tiles, uint32_t base, const PairLane& L, int I,
                                           int J, int lvl) {
  using namespace intratc;
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  const int rr = J < I ? 0 : (L.g & ~(2 * lvl - 1)) + lvl;
  const unsigned char *gi = tiles + oG + (8 * I + L.g) * 512, *gj = tiles + oG + (8 * J + L.g) * 512, *gr = tiles + oG + (8 * I + rr) * 512;
  const uint32_t r_x = L.row_x(rr);
#pragma unroll 1
  for (int ks = 0; ks < 8; ++ks) {
    const uint32_t go = L.g_x ^ (ks << 6), ro = r_x ^ (ks << 6), blk = ks >> 2, kx = (ks & 3) << 5;
    uint32_t a[4], y[4];
    ldsm_x4(a, base + L.a_row + I * 1024 + blk * 16384 + (L.a_x ^ kx));
    ldsm_x4(y, base + oY + L.b_row + J * 1024 + blk * 8192 + (L.b_x ^ kx));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float2 r = ld_f2(gr + (ro ^ (32 * u))), x = ld_f2(gi + (go ^ (32 * u))), z = ld_f2(gj + (go ^ (32 * u)));
      const float fx = ex2(-fabsf(x.x - r.x)), fy = ex2(-fabsf(x.y - r.y));
      const float2 k2 = unpack_bf16(a[2 * u]), q2 = unpack_bf16(a[2 * u + 1]), y2 = unpack_bf16(y[u]);
      a[2 * u] = pack_bf16(k2.x * fx, k2.y * fy);
      a[2 * u + 1] = pack_bf16(q2.x * fx, q2.y * fy);
      y[u] = pack_bf16(y2.x * ex2(-fabsf(z.x - r.x)), y2.y * ex2(-fabsf(z.y - r.y)));
    }
    mma_bf16(d, a, y[0], y[1]);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (J < I || level_pair_ok(L.g, 2 * L.t + (e & 1), lvl)) acc[e] = d[e];
}
__device__ __forceinline__ void pairs_of_strip_exact(unsigned char* tiles, uint32_t base, int I, int lane, float scale) {
  const PairLane L(lane);
#pragma unroll 1
  for (int J = 0; J <= I; ++J) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int lvl = 4; lvl; lvl = J < I ? 0 : lvl >> 1) pair_exact(acc, tiles, base, L, I, J, lvl);
    put_pair(tiles, L, I, J, acc, scale);
  }
}

template <bool kRecompute>
__global__ void __launch_bounds__(intratc::kThreads, 2)
pkda_intra_fwd_tc_kernel(const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_akk,
                         const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_w,
                         const __grid_constant__ CUtensorMap tm_u, const __grid_constant__ CUtensorMap tm_g,
                         const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_q,
                         const IntraParams p) {
  wait_prerequisites();
  using namespace intratc;
  extern __shared__ unsigned char smem_raw[];
  const int H = p.geo.heads;
  const int n_items = p.geo.total_chunks * H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long gld = (long)H * kD;

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* tiles = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar_tma = base + oBar, bar_mma = base + oBar + 8, tmem_slot = base + oBar + 16, bar_in = base + oBar + 24;
  float* sL = reinterpret_cast<float*>(tiles + oL);
  float* sBeta = reinterpret_cast<float*>(tiles + oBeta);
  float* sDiag = reinterpret_cast<float*>(tiles + oDiag);
  float* sTot = reinterpret_cast<float*>(tiles + (kRecompute ? oStep : oTot));  // (when recomputing, the write keys arrive in oL)
  float* sEnd = reinterpret_cast<float*>(tiles + oEnd);
  float* sDec = reinterpret_cast<float*>(tiles + oDec);
  float* sSum = reinterpret_cast<float*>(tiles + oSum);
  float* sA0 = reinterpret_cast<float*>(tiles + oA0);
  const bool chain = !kRecompute && p.chain;
  const int units = p.geo.n_seqs * H;  // (chained mode: items are drawn level by level over all units)

  // strip layout: this thread's rows r0..r0+7, channels c4..c4+3
  const int r0 = warp * 8, c4 = lane << 2;
  // byte offset of the thread's 8-byte half piece inside a swizzled row is ((piece ^ row%8) << 4) + half * 8
  const int blk = lane >> 4, piece = (lane & 15) >> 1, half8 = (lane & 1) << 3;
  // The slot of strip row i is the very place its gated value goes later: row r0 + i of the
  // stacked operand for k (rows 0..63) and q (rows 64..127), of the write-key operand for g (and,
  // once g is consumed, for the write key kt).  A thread only ever touches its own 8-byte pieces
  // there until the operands are complete, so the in-place updates need no barrier.
  unsigned char* aBase = tiles + oA + blk * 16384 + half8;  // + slot_off(i): k; + 8192: q
  unsigned char* yBase = tiles + oY + blk * 8192 + half8;   // + slot_off(i): g, then kt
  auto slot_off = [&](int i) { return (r0 + i) * 128 + ((piece ^ i) << 4); };
  auto ld_k = [&](int i) { return *reinterpret_cast<const uint2*>(aBase + slot_off(i)); };
  auto ld_q = [&](int i) { return *reinterpret_cast<const uint2*>(aBase + 8192 + slot_off(i)); };
  auto ld_y = [&](int i) { return *reinterpret_cast<const uint2*>(yBase + slot_off(i)); };

  if (tid == 0) {
    tc::mbar_init(bar_tma, 1);
    tc::mbar_init(bar_mma, 1);
    tc::mbar_init(bar_in, 1);
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, kCols);
  tc::tc_fence_before();
  __syncthreads();
  launch_dependents();
  tc::tc_fence_after();
  const uint32_t tmem = tc::uniform(*reinterpret_cast<volatile uint32_t*>(tiles + oBar + 16));
  const int warp_u = (int)tc::uniform(warp);
  bool ok = true;
  uint32_t ph = 0;  // bit 0: bar_mma, 1: bar_tma, 2: bar_in

  // Items differ in cost (one whose pairs go strip by strip takes longer), so
  // the CTAs draw them one at a time from a cursor instead of striding through them.  One thread draws the
  // next item and looks its chunk up while the current one waits for its products, and the item's rows are
  // asked into L2 from then on: drawn at the end of an item, the cursor, the lookup and the rows were four
  // dependent memory round trips of every item.  (An item only ever waits for items drawn before it, also
  // for ones that are still next on their CTA, so the chained mode cannot lock up.)
  __shared__ int4 s_item[2];  // {item or -1, first token, valid tokens, sequence}: this item, the next one
  auto describe = [&](int draw) {
    int4 it = make_int4(-1, 0, 0, 0);
    if (draw < n_items) {
      // in chained mode chunk level draw / units of unit draw % units (a dense batch)
      const int level = chain ? draw / units : 0;
      it.x = chain ? ((draw % units) / H * p.geo.chunks_per_seq + level) * H + (draw % units) % H : draw;
      if (!chunk_lookup(p.geo, it.x / H, it.w, it.y, it.z)) it.x = -1;  // past the last real chunk of a packed batch (items ascend)
    }
    return it;
  };
  // The strips of an item by TMA: g as soon as the item before it no longer needs the write-key operand (the inverse is
  // over), k and q once its last products have read the stacked operand; their epilogue and stores go on meanwhile.
  // With the scalars below, the hand-over in one word and the rows of pass 3 read ahead: 8 x 4,096 tokens of 16 heads
  // 466 -> 436 us; asked for at the top of an item, strips and scalars were 4,000 of its 30,000 cycles, and the stores 1,400.
  auto request_g = [&](const int4& it) {  // one thread; also arms the barrier for k and q
    tc::mbar_expect_tx(bar_in, (kRecompute ? 8 : 6) * 8192);
    if (kRecompute) {
      tc::tma_load_3d(base + oL, &tm_p, bar_in, 0, it.x % H, it.y);
      tc::tma_load_3d(base + oL + 8192, &tm_p, bar_in, 64, it.x % H, it.y);
    }
    tc::tma_load_3d(base + oY, &tm_g, bar_in, 0, it.x % H, it.y);
    tc::tma_load_3d(base + oY + 8192, &tm_g, bar_in, 64, it.x % H, it.y);
  };
  auto request_kq = [&](const int4& it) {  // all warps
    if (lane != 0 || warp < 2 || warp >= 6) return;
    const int b = warp & 1;
    if (warp < 4) tc::tma_load_3d(base + oA + b * 16384, &tm_k, bar_in, 64 * b, it.x % H, it.y);
    else tc::tma_load_3d(base + oA + 8192 + b * 16384, &tm_q, bar_in, 64 * b, it.x % H, it.y);
  };
  // The scalars of an item, asked for with its strips, and not used, not even converted, before they are needed.
  uint32_t n_beta = 0, n_bp = 0, n_chain = 0;  // lane i < 8: of row r0 + i; thread < 128: the entry state of its channel
  float n_pd = 0.f, n_alog = 0.f, n_centre = 0.f;
  float4 n_bias = make_float4(0.f, 0.f, 0.f, 0.f);
  auto request_scalars = [&](const int4& it) {
    const int h = it.x % H, r = r0 + (lane & 7);
    const size_t chh = it.x, s = (size_t)(it.y + min(r, it.z - 1)) * H + h;  // (rows past the end are masked where they are used)
    n_beta = chain ? ld_u16(p.beta + s) : __float_as_uint(p.beta_c[chh * kChunk + r]);
    if (!kRecompute) {
      n_pd = p.g_atk[s];
      n_bp = ld_u16(p.beta_atk + s);
      n_centre = p.log_atk_scale[h];
      if (tid < kD) {  // (chained: normally published long ago by the item of the chunk before)
        if (!chain) n_chain = __float_as_uint(p.a_start[chh * kD + tid]);
        else if (it.y > it.w * p.geo.seq_len) n_chain = ld_relaxed(p.a_chain + chh * kD + tid);
        else n_chain = p.A0 ? __float_as_uint(p.A0[((size_t)it.w * H + h) * kD + tid]) : 0u;
      }
    }
    n_bias = *reinterpret_cast<const float4*>(p.dt_bias + h * kD + c4);
    n_alog = p.A_log[h];
  };
  if (tid == 32) {
    s_item[0] = describe(atomicAdd(p.cursor, 1));
    if (s_item[0].x >= 0) request_g(s_item[0]);
  }
  __syncthreads();
  if (s_item[0].x >= 0) {
    request_kq(s_item[0]);
    request_scalars(s_item[0]);
  }
  int slot = 0;
#pragma unroll 1
  for (;; slot ^= 1) {
  const int4 cur = s_item[slot];
  const int item = cur.x, tok0 = cur.y, valid = cur.z, n = cur.w;
  if (item < 0) break;
  const int h = item % H;
  const size_t chh = (size_t)item;
  const size_t row0 = ((size_t)tok0 * H + h) * kD;
  const bool full = valid == kChunk;
  // The operand descriptors depend on the tile base only; keeping the base opaque per item stops the
  // compiler from computing all of them ahead of the loop and holding them in registers.
  const uint32_t dbase = tc::uniform(base);

  // ---- 0. V (and T when recomputing) by TMA; the strips of g, k and q are on their way into their operand slots
  auto request_v = [&]() {  // thread 0, when its stores from there are done
    tc::mbar_expect_tx(bar_tma, kRecompute ? 16384 + 8192 : 16384);
    tc::tma_load_3d(base + oV, &tm_v, bar_tma, 0, h, tok0);
    tc::tma_load_3d(base + oV + 8192, &tm_v, bar_tma, 64, h, tok0);
    if (kRecompute) tc::tma_load_3d(base + oTm, &tm_akk, bar_tma, 0, h, tok0);
  };
  if (kRecompute && tid == 0) {
    tc::bulk_wait_read();
    request_v();
  }  // (the forward asks for V once it knows whether the decays need its place first)
  // (opaque, so that nothing is computed from them, and waits for them, where they were asked for)
  asm volatile("" : "+r"(n_beta), "+r"(n_bp), "+r"(n_chain), "+f"(n_pd), "+f"(n_alog), "+f"(n_centre), "+f"(n_bias.x), "+f"(n_bias.y),
               "+f"(n_bias.z), "+f"(n_bias.w));
  const bool row_in = lane < 8 && r0 + lane < valid;  // lane i < 8: scalars of row r0 + i
  const float sc_beta = !chain || row_in ? __uint_as_float(chain ? n_beta << 16 : n_beta) : 0.f;
  const float sc_bp = row_in ? __uint_as_float(n_bp << 16) : 0.f;
  float sc_pd = row_in ? n_pd : 0.f;
  if (chain && lane < 8) p.beta_c_w[chh * kChunk + r0 + lane] = sc_beta;  // packed chunk-major on the way, for the later stages
  const float4 bias4 = n_bias;
  const float ea2 = __expf(n_alog) * kLog2e, centre = n_centre;
  uint32_t chain_a0 = n_chain;
  int drawn = 0;
  if (kRecompute && tid == 32) drawn = atomicAdd(p.cursor, 1);
  ok = tc::mbar_wait(bar_in, ph >> 2) && ok;
  ph ^= 4;
  if (!full) {  // rows past the sequence end read as zero, whatever lies there
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (r0 + i >= valid) {
        *reinterpret_cast<uint2*>(yBase + slot_off(i)) = make_uint2(0, 0);
        *reinterpret_cast<uint2*>(aBase + slot_off(i)) = make_uint2(0, 0);
        *reinterpret_cast<uint2*>(aBase + 8192 + slot_off(i)) = make_uint2(0, 0);
      }
  }

  // ---- 1. decay gate, strip-local cumulative sum; strip-local preconditioner scan from zero
  // (The row loops of passes 1 and 3 take four rows a turn, their rows of G moved down in between: unrolled by eight, the
  // passes were some 40 KB of instructions that two CTAs in different phases kept evicting, and the first stall was
  // the fetch.  2,048 items: 131 -> 125 us, strongly decaying ones 161 -> 154; issue slots in use 48 -> 55 %.)
  float G[8][4];
  {
    const float bias[4] = {bias4.x, bias4.y, bias4.z, bias4.w};
    float run[4] = {0.f, 0.f, 0.f, 0.f}, a[4] = {0.f, 0.f, 0.f, 0.f}, dblk = 1.f, gsum = 0.f;
    const float lg = sc_pd;
    sc_pd = __expf(sc_pd);  // rows past the end: exp(0) = 1, beta 0
#pragma unroll 1
    for (int i0 = 0; i0 < 8; i0 += 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float x[4];
        unpack4(ld_y(i0 + i), x);
        const bool in = r0 + i0 + i < valid;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float gv = in ? -ea2 * softplus_fast(x[e] + bias[e]) : 0.f;
          run[e] += gv;
          G[i][e] = G[i + 4][e];
          G[i + 4][e] = run[e];
        }
        if (!kRecompute) {
          if (chain) gsum += __shfl_sync(0xffffffffu, lg, i0 + i);  // the strip's summed log-decay, added in row order
          const float pd = __shfl_sync(0xffffffffu, sc_pd, i0 + i), bp = __shfl_sync(0xffffffffu, sc_bp, i0 + i);
          float kc[4];
          unpack4(ld_k(i0 + i), kc);
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = pd * a[e] + bp * kc[e] * kc[e];
          dblk *= pd;
        }
      }
    }
    if (!kRecompute) {
      *reinterpret_cast<float4*>(sEnd + warp * kD + c4) = make_float4(a[0], a[1], a[2], a[3]);
      if (lane == 0) {
        sDec[warp] = dblk;
        if (chain) sSum[warp] = gsum;
      }
    }
  }
  *reinterpret_cast<float4*>(sTot + warp * kD + c4) = make_float4(G[7][0], G[7][1], G[7][2], G[7][3]);
  if (lane < 8) sBeta[r0 + lane] = sc_beta;
  __syncthreads();

  if (!kRecompute && !chain && tid < kD) sA0[tid] = __uint_as_float(chain_a0);
  // Chained mode: this chunk's entry state of the preconditioner comes from the item of the chunk
  // before it (or the initial state), the next chunk's goes out.  Four warps, one channel per thread, in front of everything that can
  // wait: few units are a chain of these hand-overs (behind the prefixes below: 1 x 8,191 tokens of 16 heads 166 -> 163.5 us,
  // 2 x 3,102 of 12 98 -> 94.7).
  if (chain && tid < kD) {
    const int level = (tok0 - n * p.geo.seq_len) / kChunk;
    float loc = 0.f, gs = 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      loc = sDec[b] * loc + sEnd[b * kD + tid];
      gs += sSum[b];
    }
    if (level == 0) {
      p.a_chain[chh * kD + tid] = __uint_as_float(chain_a0);
    } else {
      uint32_t it = 0;  // not there yet when it was asked for: poll (bounded)
      while (chain_a0 == kNotYet && ++it < tc::kSpinLimit) chain_a0 = ld_relaxed(p.a_chain + chh * kD + tid);
      ok = ok && chain_a0 != kNotYet;
    }
    const float a0 = __uint_as_float(chain_a0);
    sA0[tid] = a0;
    const float an = __expf(gs) * a0 + loc;
    if (level + 1 < p.geo.chunks_per_seq) st_relaxed(p.a_chain + (chh + H) * kD + tid, an);
    else if (p.AT) p.AT[((size_t)n * H + h) * kD + tid] = an;
    if (tid == 0) p.sa[chh] = gs;
  }
  // ---- 2. prefixes over the strips: cumulative decay of every row, and of the chunk's last row
  float Glast[4];
  {
    float P[4] = {0.f, 0.f, 0.f, 0.f}, pre[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int wp = 0; wp < 8; ++wp) {
      const float4 to = *reinterpret_cast<const float4*>(sTot + wp * kD + c4);
      if (wp == warp) {
#pragma unroll
        for (int e = 0; e < 4; ++e) pre[e] = P[e];
      }
      P[0] += to.x; P[1] += to.y; P[2] += to.z; P[3] += to.w;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) Glast[e] = P[e];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) G[i][e] += pre[e];
  }
  if (!kRecompute && tid == 0) tc::bulk_wait_read();  // the stores of the item before from the tiles that are written next
  // Does the chunk decay too much for one direct block?  (The same answer for all threads: every thread holds the
  // totals of its four channels, the CTA all 128.)  If so, which reference rows do its strips take?
  if (kRecompute && tid == 32) s_item[slot ^ 1] = describe(drawn);
  const bool by_strip =
      __syncthreads_or(-fminf(fminf(Glast[0], Glast[1]), fminf(Glast[2], Glast[3])) > kDirectLimit) || p.by_strip;
  // A recompute item is half as long and waits for memory first, so the next one is known here already: its scalars are asked for,
  // its tiles into L2 (behind the products as in the forward, with the write keys by plain loads at the top of the item, the
  // wait there was 6,000 of an item's 17,800 cycles; 8,192 items 296 -> 196 us, 1,536 strongly decaying ones 65 -> 47).
  auto prefetch = [&](const int4& it) {  // the item's tiles of g, k, q and v into L2; when recomputing the write keys and T too
    if (lane != 0 || it.x < 0) return;
    const CUtensorMap* m = warp < 2 ? &tm_g : warp < 4 ? &tm_k : warp < 6 ? &tm_q : &tm_v;
    tc::tma_prefetch_3d(m, 64 * (warp & 1), it.x % H, it.y);
    if (kRecompute && warp < 2) tc::tma_prefetch_3d(&tm_p, 64 * warp, it.x % H, it.y);
    if (kRecompute && warp == 2) tc::tma_prefetch_3d(&tm_akk, 0, it.x % H, it.y);
  };
  if (kRecompute) {
    prefetch(s_item[slot ^ 1]);
    if (s_item[slot ^ 1].x >= 0) request_scalars(s_item[slot ^ 1]);
  }
  int refs = 0;  // 0: first and last row, 1: by halves, 2: pair_exact
  if (!kRecompute) {
    if (!by_strip) {
      if (tid == 0) request_v();
    } else {
      float all = 0.f, mid = 0.f, outer = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        all = fmaxf(all, G[0][e] - G[7][e]);
        const float2 d = strip_decays(G[0][e], G[2][e], G[kHalfRow][e], G[5][e], G[7][e]);
        mid = fmaxf(mid, d.x);
        outer = fmaxf(outer, d.y);
      }
      constexpr int kz = kHalfRow;
      *reinterpret_cast<float4*>(tiles + oZin + warp * 512 + (lane << 4)) = make_float4(G[kz][0], G[kz][1], G[kz][2], G[kz][3]);
      if (__syncthreads_or(all > kDirectLimit)) refs = 1 + (__syncthreads_or(mid > kDirectLimit || outer > kOuterLimit) != 0);
      if (p.direct_cap < 8) refs = 2;
    }
  }

  // ---- 3. one pass over the strip: preconditioner states of its rows -> write keys kt = k * B(A_t)
  // (to global memory), kg = kt * decay to the chunk end, the diagonal q_i . kt_i, and the gated operands
  // in place: Kd = k 2^G (rows 0..63 of the stacked operand, later an operand of W), q 2^G (rows
  // 64..127), kt 2^-G (into the slots g has left); qg goes to global memory.  The decay to the chunk
  // end is 2^G_last times the 2^-G the operand needs anyway.  Nothing of the strip is needed afterwards.
  // A chunk that is paired by strips leaves its operands as pairs_of_strip or pair_exact reads them.
  {
    float A[4] = {0.f, 0.f, 0.f, 0.f};
    if (!kRecompute) {
      const float4 a0 = *reinterpret_cast<const float4*>(sA0 + c4);  // (written before the barrier of the decision)
      A[0] = a0.x; A[1] = a0.y; A[2] = a0.z; A[3] = a0.w;
      for (int b = 0; b < warp; ++b) {
        const float d = sDec[b];
        const float4 e4 = *reinterpret_cast<const float4*>(sEnd + b * kD + c4);
        A[0] = d * A[0] + e4.x; A[1] = d * A[1] + e4.y; A[2] = d * A[2] + e4.z; A[3] = d * A[3] + e4.w;
      }
    }
    if (!by_strip || (!kRecompute && warp == 0)) {
      const float glE[4] = {ex2(Glast[0]), ex2(Glast[1]), ex2(Glast[2]), ex2(Glast[3])};
      if (!kRecompute && warp == 0)
        *reinterpret_cast<float4*>(p.gc + chh * kD + c4) = make_float4(glE[0], glE[1], glE[2], glE[3]);
      if (!by_strip) {
#pragma unroll
        for (int c = 0; c < 4; ++c) Glast[c] = glE[c];  // from here on the decay itself (one set of registers for both kinds)
      }
    }
    float zr[4], xr[4];  // the strip's reference rows
    if (!kRecompute && by_strip && refs < 2) {
      float4 prev = make_float4(0.f, 0.f, 0.f, 0.f);  // z of the strip before
      if (refs) {
        if (warp) prev = *reinterpret_cast<const float4*>(tiles + oZin + (warp - 1) * 512 + (lane << 4));
      } else {
        for (int wp = 0; wp < warp; ++wp) {
          const float4 to = *reinterpret_cast<const float4*>(sTot + wp * kD + c4);
          prev.x += to.x; prev.y += to.y; prev.z += to.z; prev.w += to.w;
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        zr[c] = refs ? G[kHalfRow][c] : G[7][c];
        xr[c] = G[0][c];
      }
      unsigned char* at = tiles + warp * 1024 + (lane << 4);
      *reinterpret_cast<float4*>(at + oD0) = make_float4(ex2(xr[0] - zr[0]), ex2(xr[1] - zr[1]), ex2(xr[2] - zr[2]), ex2(xr[3] - zr[3]));
      *reinterpret_cast<float4*>(at + oD1) = make_float4(ex2(xr[0] - prev.x), ex2(xr[1] - prev.y), ex2(xr[2] - prev.z), ex2(xr[3] - prev.w));
      *reinterpret_cast<float4*>(tiles + oStep + warp * 512 + (lane << 4)) = make_float4(ex2(zr[0] - prev.x), ex2(zr[1] - prev.y), ex2(zr[2] - prev.z), ex2(zr[3] - prev.w));
    }
    float dg[4];
    // (the next row is read before this one is written: the compiler cannot tell their places apart and would start it after)
    uint2 k_next = ld_k(0), q_next = ld_q(0);
#pragma unroll 1
    for (int i0 = 0; i0 < 8; i0 += 4) {
    if (!kRecompute && refs == 1 && i0) {  // the second half's reference is its own first row
#pragma unroll
      for (int c = 0; c < 4; ++c) xr[c] = G[0][c];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = i0 + i, off = slot_off(row);
      const uint2 kr = k_next, qr = q_next;
      k_next = ld_k((row + 1) & 7);
      q_next = ld_q((row + 1) & 7);
      uint2 kt = make_uint2(0, 0);
      if (kRecompute) kt = *reinterpret_cast<const uint2*>(tiles + oL + blk * 8192 + half8 + off);
      if (!kRecompute) {
        const float pd = __shfl_sync(0xffffffffu, sc_pd, row), bp = __shfl_sync(0xffffffffu, sc_bp, row);
        float kc[4], f[4];
        unpack4(kr, kc);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          A[e] = pd * A[e] + bp * kc[e] * kc[e];
          const float dev = __logf(A[e] + p.eps) - centre;
          f[e] = __expf(-p.ln_x * __fdividef(dev, 1.f + fabsf(dev)));
        }
        kt = scale4(kr, f);
        if (r0 + row < valid) *reinterpret_cast<uint2*>(p.kt + row0 + (size_t)(r0 + row) * gld + c4) = kt;
        float kc2[4], qc[4];
        unpack4(kt, kc2);
        unpack4(qr, qc);
        dg[i] = qc[0] * kc2[0] + qc[1] * kc2[1] + qc[2] * kc2[2] + qc[3] * kc2[3];
      }
      float e[4], es[4], tl[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        e[c] = ex2(G[i][c]);
        es[c] = e[c] * p.scale;
      }
      if (!by_strip) {
        float fi[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          fi[c] = __fdividef(1.f, e[c]);
          tl[c] = Glast[c] * fi[c];
        }
        *reinterpret_cast<uint2*>(aBase + off) = scale4(kr, e);
        if (!kRecompute) {
          *reinterpret_cast<uint2*>(aBase + 8192 + off) = scale4(qr, e);
          *reinterpret_cast<uint2*>(yBase + off) = scale4(kt, fi);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) tl[c] = ex2(Glast[c] - G[i][c]);
        if (kRecompute) {
          *reinterpret_cast<uint2*>(aBase + off) = scale4(kr, e);
        } else {
          float y[4];
          if (refs < 2) {
            float x[4];
            unpack4(kt, y);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              x[c] = ex2(G[i][c] - xr[c]);
              y[c] *= ex2(zr[c] - G[i][c]);
            }
            *reinterpret_cast<uint2*>(aBase + off) = scale4(kr, e);
            *reinterpret_cast<uint2*>(yBase + off) = scale4(kr, x);
            *reinterpret_cast<uint2*>(aBase + 8192 + off) = scale4(qr, x);
          } else {
            *reinterpret_cast<uint2*>(yBase + off) = kt;
#pragma unroll
            for (int c = 0; c < 4; ++c) y[c] = G[i][c];
          }
          *reinterpret_cast<float4*>(tiles + oG + (r0 + row) * 512 + ((lane ^ ((i & 3) << 1)) << 4)) = make_float4(y[0], y[1], y[2], y[3]);
        }
      }
      if (r0 + row < valid) {
        *reinterpret_cast<uint2*>(p.kg + row0 + (size_t)(r0 + row) * gld + c4) = scale4(kt, tl);
        *reinterpret_cast<uint2*>(p.qg + row0 + (size_t)(r0 + row) * gld + c4) = scale4(qr, es);
      }
    }
    if (!kRecompute) {
      row_sums4(dg, lane);
      if ((lane & 7) == 0) sDiag[r0 + i0 + ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1)] = dg[0];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int c = 0; c < 4; ++c) G[i][c] = G[i + 4][c];
    }
    }
  }
  if (!kRecompute && tid == 32) drawn = atomicAdd(p.cursor, 1);  // (looked up while the pair products run)
  tc::fence_proxy_async();
  tc::tc_fence_before();
  __syncthreads();  // (the strip exchange arrays are dead from here on: L takes their place)
  if (!kRecompute && by_strip) {
    if (tid == 32) s_item[slot ^ 1] = describe(drawn);
    if (refs == 0) {
      pairs_of_strip<false>(tiles, base, warp, lane, p.scale);
    } else if (refs == 1) {
      pairs_of_strip<true>(tiles, base, warp, lane, p.scale);
    } else {
      pairs_of_strip_exact(tiles, base, warp, lane, p.scale);
      __syncwarp();  // (only this warp reads the k rows of its strip; they become Kd)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 g4 = *reinterpret_cast<const float4*>(tiles + oG + (r0 + i) * 512 + ((lane ^ ((i & 3) << 1)) << 4));
        const float e[4] = {ex2(g4.x), ex2(g4.y), ex2(g4.z), ex2(g4.w)};
        *reinterpret_cast<uint2*>(aBase + slot_off(i)) = scale4(ld_k(i), e);
      }
    }
    // what lies above the strip diagonal of P reads as zero
    for (int J = warp + 1 + (lane >> 3); J < 8; J += 4)
      *reinterpret_cast<uint4*>(tiles + oP + (r0 + (lane & 7)) * 128 + ((J ^ (lane & 7)) << 4)) = make_uint4(0, 0, 0, 0);
  } else if (!kRecompute) {
    if (warp_u == 0 && tc::elect_one()) {
      tc::tc_fence_after();
      constexpr uint32_t idesc_pair = tc::idesc_bf16(128, 64, false, false);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const uint64_t a = tc::desc_kmajor(dbase + oA + (kk >> 2) * 16384 + (kk & 3) * 32);
        const uint64_t b = tc::desc_kmajor(dbase + oY + (kk >> 2) * 8192 + (kk & 3) * 32);
        tc::umma_bf16(tmem, a, b, idesc_pair, kk > 0);
      }
      tc::umma_commit(bar_mma);
    }
    if (tid == 32) s_item[slot ^ 1] = describe(drawn);
    ok = tc::mbar_wait(bar_mma, ph & 1) && ok;
    ph ^= 1;
    tc::tc_fence_after();
    {
      int wl = tid;  // (opaque: what follows from it is formed here and not kept all along)
      asm volatile("" : "+r"(wl));
      const int wp = wl >> 5, ei = (32 * (wp & 3) + (wl & 31)) & 63, j0 = 32 * (wp >> 2);  // this thread's accumulator row and columns
      const bool isP = (wp & 3) >= 2;
      float acc[32];
      tc::tmem_ld32(tmem + ((uint32_t)(32 * (wp & 3)) << 16) + j0, acc);
      tc::tmem_ld_wait();
      if (!isP) {  // L = tril(M, -1) diag(beta)
#pragma unroll
        for (int t = 0; t < 32; t += 4) {
          float4 x;
          x.x = (j0 + t < ei) ? acc[t] * sBeta[j0 + t] : 0.f;
          x.y = (j0 + t + 1 < ei) ? acc[t + 1] * sBeta[j0 + t + 1] : 0.f;
          x.z = (j0 + t + 2 < ei) ? acc[t + 2] * sBeta[j0 + t + 2] : 0.f;
          x.w = (j0 + t + 3 < ei) ? acc[t + 3] * sBeta[j0 + t + 3] : 0.f;
          *reinterpret_cast<float4*>(sL + ei * kLdL + j0 + t) = x;
        }
      } else {     // scale * tril(P) with the ungated diagonal
        unsigned char* prow = tiles + oP + ei * 128;
        const float dv = sDiag[ei];
#pragma unroll
        for (int pc = 0; pc < 4; ++pc) {
          float x[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const int j = j0 + 8 * pc + t;
            x[t] = (j < ei ? acc[8 * pc + t] : (j == ei ? dv : 0.f)) * p.scale;
          }
          *reinterpret_cast<uint4*>(prow + ((((j0 >> 3) + pc) ^ (ei & 7)) << 4)) =
              make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
        }
      }
    }
    tc::tc_fence_before();
  }
  auto await_v = [&]() {
    ok = tc::mbar_wait(bar_tma, (ph >> 1) & 1) && ok;  // V (and T) landed long ago
    ph ^= 2;
    if (!full) {  // rows past the sequence end hold another sequence's data: they must not reach the product
      for (int idx = tid; idx < kChunk * 16; idx += kThreads) {
        const int r = idx >> 4, pc = idx & 15;
        if (r >= valid)
          *reinterpret_cast<uint4*>(tiles + oV + (pc >> 3) * 8192 + r * 128 + ((pc & 7) << 4)) = make_uint4(0, 0, 0, 0);
      }
    }
  };
  if (kRecompute) await_v();
  tc::fence_proxy_async();
  __syncthreads();
  if (!kRecompute && by_strip && tid == 0) request_v();  // (the decays have been read)
  const int4 nx = s_item[slot ^ 1];
  if (!kRecompute) prefetch(nx);

  if (!kRecompute) {
    // ---- 5. scaled P -> Aqk;  T = (I + L)^-1 -> bf16 operand tile and Akk
    if (full) {
      if (tid == 0) {
        tc::tma_store_3d(&tm_p, base + oP, 0, h, tok0);
        tc::bulk_commit();
      }
    } else {
      for (int idx = tid; idx < kChunk * 8; idx += kThreads) {
        const int r = idx >> 3, pc = idx & 7;
        if (r < valid)
          *reinterpret_cast<uint4*>(p.Aqk + ((size_t)(tok0 + r) * H + h) * kChunk + 8 * pc) =
              *reinterpret_cast<const uint4*>(tiles + oP + r * 128 + ((pc ^ (r & 7)) << 4));
      }
    }
    float* sT = reinterpret_cast<float*>(tiles + oT);
    unit_lower_inverse_64<8>(sL, sT, reinterpret_cast<float*>(tiles + oY2), kLdL, kLdL, tid, kThreads);  // ends with a barrier
    for (int idx = tid; idx < kChunk * 8; idx += kThreads) {
      const int r = idx >> 3, pc = idx & 7;
      const float4 s0 = *reinterpret_cast<const float4*>(sT + r * kLdL + 8 * pc);
      const float4 s1 = *reinterpret_cast<const float4*>(sT + r * kLdL + 8 * pc + 4);
      const uint4 pk = make_uint4(pack_bf16(s0.x, s0.y), pack_bf16(s0.z, s0.w), pack_bf16(s1.x, s1.y),
                                  pack_bf16(s1.z, s1.w));
      *reinterpret_cast<uint4*>(tiles + oTm + r * 128 + ((pc ^ (r & 7)) << 4)) = pk;
      if (!full && r < valid)
        *reinterpret_cast<uint4*>(p.Akk + ((size_t)(tok0 + r) * H + h) * kChunk + 8 * pc) = pk;
    }
    await_v();
    if (tid == 0) tc::bulk_wait_read();  // (scale P has left: U takes its place)
    tc::fence_proxy_async();
    tc::tc_fence_before();
    __syncthreads();
  }

  // ---- 6. W = T Kd, U = T V (64 rows: the tokens)
  if (nx.x >= 0) {
    if (tid == 32) request_g(nx);
  }
  if (!kRecompute && full && tid == 0) {
    tc::tma_store_3d(&tm_akk, base + oTm, 0, h, tok0);
    tc::bulk_commit();
  }
  if (warp_u == 2 && tc::elect_one()) {  // (warp 0 stores T, warp 1 asks for the next gate)
    tc::tc_fence_after();
    constexpr uint32_t idesc = tc::idesc_bf16(64, 128, /*a_mn_major=*/false, /*b_mn_major=*/true);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      tc::umma_bf16(tmem, tc::desc_kmajor(dbase + oTm + kk * 32), tc::desc_mnmajor(dbase + oA + kk * 2048, 16384), idesc, kk > 0);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      tc::umma_bf16(tmem + 128, tc::desc_kmajor(dbase + oTm + kk * 32), tc::desc_mnmajor(dbase + oV + kk * 2048, 8192), idesc,
                    kk > 0);
    tc::umma_commit(bar_mma);
  }
  ok = tc::mbar_wait(bar_mma, ph & 1) && ok;
  ph ^= 1;
  tc::tc_fence_after();
  if (nx.x >= 0) {
    request_kq(nx);
    if (!kRecompute) request_scalars(nx);
  }
  {
    const int q = warp & 3, m = warp >> 2;  // this warp's 16 tokens; W or U
    const int r = lane & 7, mat = lane >> 3;  // the row whose address this lane gives: row r of rows 8 (mat & 1) .., 8 columns (mat >> 1)
    const uint32_t row = base + (m ? oX : oV) + (16 * q + 8 * (mat & 1) + r) * 128, rx = ((mat >> 1) ^ r) << 4;
#pragma unroll 1
    for (int blk = 0; blk < 2; ++blk) {
      float acc[32];
      tc::tmem_ld_rows(tmem + ((uint32_t)(32 * q) << 16) + 128 * m + 64 * blk, acc);
      tc::tmem_ld_wait();
      uint32_t x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = pack_bf16(acc[2 * i], acc[2 * i + 1]);
      if (full) {  // a swizzled [token][channel] tile for the TMA store
#pragma unroll
        for (int i = 0; i < 4; ++i) stsm_x4(row + blk * 8192 + (rx ^ (i << 5)), &x[4 * i]);
      } else {
        bf16* dst = (m ? p.u : p.w) + row0 + (size_t)(16 * q + (lane >> 2)) * gld + 64 * blk + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (16 * q + (lane >> 2) + 8 * (i & 1) < valid)
            *reinterpret_cast<uint32_t*>(dst + (size_t)(8 * (i & 1)) * gld + 8 * (i >> 1)) = x[i];
      }
    }
  }
  tc::fence_proxy_async();
  tc::tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    if (full) {
      tc::tma_store_3d(&tm_w, base + oV, 0, h, tok0);
      tc::tma_store_3d(&tm_w, base + oV + 8192, 64, h, tok0);
      tc::tma_store_3d(&tm_u, base + oX, 0, h, tok0);
      tc::tma_store_3d(&tm_u, base + oX + 8192, 64, h, tok0);
      tc::bulk_commit();
    }
  }
  }  // item loop
  if (tid == 0) tc::bulk_wait_read();
  if (__syncthreads_or(!ok) && tid == 0) atomicExch(p.status, 1);
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, kCols);
}

// ------------------------------------------------------------------ host side
int launch_chain_init(float* a_chain, size_t items, int* zero, cudaStream_t st) {
  const size_t n = items * kD, most = 8 * (size_t)sm_count(), blocks = (n + 255) / 256;
  begin_stage(kStageChainInit, st);
  const int rc = launch_kernel(pkda_chain_init_kernel, (unsigned)(blocks < most ? blocks : most), 256, 0, st, reinterpret_cast<uint32_t*>(a_chain),
                n, zero);
  end_stage(st);
  return rc;
}

int launch_intra_fwd_tc(const IntraParams& ip, bool recompute, cudaStream_t st) {
  const uint64_t H = ip.geo.heads, tok = ip.geo.total_tokens;
  CUtensorMap tm_v, tm_akk, tm_p, tm_w, tm_u, tm_g, tm_k, tm_q;  // tm_p: scaled P, which leaves; when recomputing the write keys, which arrive
  {
    const uint64_t dims[3] = {kD, H, tok}, str[2] = {kD * 2, H * kD * 2};
    const uint32_t box[3] = {64, 1, 64};
    if (!encode_bf16_map(&tm_v, ip.v, 3, dims, str, box) || !encode_bf16_map(&tm_w, ip.w, 3, dims, str, box) ||
        !encode_bf16_map(&tm_u, ip.u, 3, dims, str, box) || !encode_bf16_map(&tm_g, ip.g, 3, dims, str, box) ||
        !encode_bf16_map(&tm_k, ip.k, 3, dims, str, box) || !encode_bf16_map(&tm_q, ip.q, 3, dims, str, box) ||
        (recompute && !encode_bf16_map(&tm_p, ip.kt, 3, dims, str, box)))
      return PKDA_ERR_LAUNCH;
  }
  {
    const uint64_t dims[3] = {kChunk, H, tok}, str[2] = {kChunk * 2, H * kChunk * 2};
    const uint32_t box[3] = {64, 1, 64};
    if (!encode_bf16_map(&tm_akk, ip.Akk, 3, dims, str, box) || (!recompute && !encode_bf16_map(&tm_p, ip.Aqk, 3, dims, str, box)))
      return PKDA_ERR_LAUNCH;
  }
  const int sms = sm_count();
  const int items = ip.geo.total_chunks * ip.geo.heads;
  const int grid = items < 2 * sms ? items : 2 * sms;  // persistent: two CTAs per SM
  // two CTAs per SM need the largest shared-memory carve-out
  if (recompute) {
    if (!ensure_dynamic_smem(pkda_intra_fwd_tc_kernel<true>, intratc::kSmem, 100))
      return PKDA_ERR_LAUNCH;
    return launch_kernel(false, pkda_intra_fwd_tc_kernel<true>, grid, intratc::kThreads, intratc::kSmem, st, tm_v, tm_akk, tm_p, tm_w, tm_u,
                  tm_g, tm_k, tm_q, ip);
  } else {
    if (!ensure_dynamic_smem(pkda_intra_fwd_tc_kernel<false>, intratc::kSmem, 100))
      return PKDA_ERR_LAUNCH;
    return launch_kernel(false, pkda_intra_fwd_tc_kernel<false>, grid, intratc::kThreads, intratc::kSmem, st, tm_v, tm_akk, tm_p, tm_w, tm_u,
                  tm_g, tm_k, tm_q, ip);
  }
}

}  // namespace pkda

