// Shared by the token-by-token kernels (forward, exact backward, decoding step).
#pragma once

#include "pkda_common.cuh"

namespace pkda {

// Decoding step: a CTA keeps a D x D fp32 matrix in registers, thread (kq, vq) owning rows
// [kq*R, kq*R + R) and the four columns [4 vq, 4 vq + 4).
template <int D> struct RecCfg {
  static constexpr int kThreads = D >= 32 ? 256 : (D == 16 ? 64 : 32);
  static constexpr int kVQ = D / 4;                                        // threads across v
  static constexpr int kKW = (kThreads / kVQ) < D ? (kThreads / kVQ) : D;  // row groups
  static constexpr int kActive = kVQ * kKW;
  static constexpr int kR = D / kKW;                                       // rows per thread
};

// Token-by-token scans (forward, and the state cotangent of the exact backward).  The value
// columns of the state never meet inside the recurrence, so every WARP owns a few columns of one
// (sequence, head) with all D rows: lane = column group * kRG + row group, kCPL adjacent columns per
// lane, rows of a lane interleaved in runs of kU so that one vector load per lane covers a contiguous
// stretch.  A sum over rows is a short chain in the lane plus shuffles; nothing else of the state
// leaves the warp, and the warps of one unit may sit on different SMs.
//   kCPL = 1: shortest chain, most warps (few units);
//   kCPL = 4: a row value read from shared memory serves four columns (many units: what bounds it
//   then is shared-memory wavefronts and issue slots, not the chain).
template <int D, int kCPL_> struct ScanLay {
  static constexpr int kCPL = kCPL_;
  static constexpr int kRG = D >= 16 ? 8 : 4;  // row groups = lanes per column group
  static constexpr int kR = D / kRG;                  // rows per lane
  static constexpr int kU = kR >= 4 ? 4 : 2;          // consecutive rows of a lane
  static constexpr int kCols = 32 / kRG * kCPL;       // columns per warp
  static constexpr int kWarps = D / kCols;            // warps per (sequence, head)
  static constexpr int kTB = 8;                       // tokens per staged block
  static constexpr int kTO = kCPL == 4 ? 2 : kTB;     // tokens whose outputs are summed up together
  static constexpr int kSums = kTO * kCPL / kRG;      // (token, column) totals a lane ends up with each time
  static constexpr int kGroups = kCPL == 4 ? 2 : 4;   // producer groups (each its share of a block's tokens)
  static constexpr int kTPG = kTB / kGroups;          // tokens of a producer group
  static constexpr int kProdPerGroup = D < 32 ? 32 : D;
  static constexpr int kProd = kGroups * kProdPerGroup;
  static constexpr int kMaxConsumers = 8;             // consumer warps per CTA, at most
  static constexpr int kVecs = 5;                     // row vectors per token
  static constexpr int kStage = kTB * kVecs * D;      // floats of one staged block
  static constexpr int kSmem = 2 * kStage * 4;
  // first row of run `b` of row group `rg`
  static __host__ __device__ constexpr int row(int b, int rg) { return (b * kRG + rg) * kU; }
};

constexpr int kCkpt = 32;  // tokens between two state checkpoints of the exact backward

// Checkpoints of all sequences lie on one axis; sequence n starts here (disjoint also when packed:
// floor((b + l) / 32) - floor(b / 32) + 1 >= ceil(l / 32)).
__host__ __device__ inline long ckpt_base(const Geo& g, int n, int bos) {
  return g.cu_seqlens ? (long)bos / kCkpt + n : (long)n * ((g.seq_len + kCkpt - 1) / kCkpt);
}
inline size_t ckpt_bound(const pkda_problem& p) {
  return p.cu_seqlens ? (size_t)p.total_tokens / kCkpt + p.n_seqs
                      : (size_t)p.n_seqs * ((p.seq_len + kCkpt - 1) / kCkpt);
}

// What the forward leaves for the exact backward, all fp32: per token exp(g), the write key beta * kw,
// the preconditioner state A and the residual e ([tokens][H][D] each), and the state S at the start of
// every 32-token block ([blocks][H][D][D]).
struct RecSaved {
  float *al, *w, *A, *e, *S;
};
RecSaved carve_rec_saved(const pkda_problem& p, void* base, size_t* bytes);

// A value as it lies in memory, in a register of its own: a 16-bit array element would be packed in
// pairs, which waits for the load, and so would a conversion.
template <typename T> struct Raw;
template <> struct Raw<float> {
  typedef float type;
  static __device__ __forceinline__ float load(const float* p) { return *p; }
  static __device__ __forceinline__ float value(float r) { return r; }
};
template <> struct Raw<bf16> {
  typedef uint32_t type;
  // (Widened by the load itself: the compiler moves a widening of its own behind the point where the checked and the unchecked loads of a
  // block meet, where it waits for them.  512 tokens, forward: 8 units at 64 rows 73 -> 66 us, 16 rows 70 -> 63, 8 rows 70 -> 63;
  // leaving what the backward needs, 300 units at 32 rows 233 -> 205.)
  static __device__ __forceinline__ uint32_t load(const bf16* p) {
    uint32_t x;
    asm volatile("ld.global.u16 %0, [%1];" : "=r"(x) : "l"(__cvta_generic_to_global(p)));
    return x;
  }
  static __device__ __forceinline__ float value(uint32_t r) { return __uint_as_float(r << 16); }
};

// Named barriers between the producer and the consumer warps of a scan CTA.
__device__ __forceinline__ void bar_sync_n(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive_n(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Shared-memory loads and shuffles of the scans (volatile: the compiler keeps their order; the assembler may still move a load in
// front of a shuffle).
template <int kU>
__device__ __forceinline__ void load_run(uint32_t s, float2* out) {
  if (kU == 4)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(out[0].x), "=f"(out[0].y), "=f"(out[1].x), "=f"(out[1].y) : "r"(s));
  else
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(out[0].x), "=f"(out[0].y) : "r"(s));
}
__device__ __forceinline__ float xor_lane(float x, int o) {
  float y;
  asm volatile("shfl.sync.bfly.b32 %0, %1, %2, 0x1f, 0xffffffff;" : "=f"(y) : "f"(x), "r"(o));
  return y;
}

// The kR values of one row vector (shared address) that belong to the lane.
template <typename L>
__device__ __forceinline__ void load_rows(uint32_t vec, int rg, float2 (&x)[L::kR / 2]) {
#pragma unroll
  for (int b = 0; b < L::kR / L::kU; ++b) load_run<L::kU>(vec + 4 * L::row(b, rg), &x[b * (L::kU / 2)]);
}

// kN per-lane partial sums: after the rounds o = kRG / 2, kRG / 4, .. 1 (n = kN / 2, kN / 4, ..) lane rg holds the totals of entries
// rg * (kN / kRG) ... in x[0 .. kN / kRG) (a transposing butterfly: about kN shuffles instead of kN * log2(kRG)).
template <int kN>
__device__ __forceinline__ void rg_sum_round(float (&x)[kN], int rg, int o, int n) {
  const bool upper = rg & o;
#pragma unroll
  for (int i = 0; i < kN / 2; ++i) {
    if (i < n) {
      const float keep = upper ? x[i + n] : x[i];
      const float send = upper ? x[i] : x[i + n];
      x[i] = keep + xor_lane(send, o);
    }
  }
}
template <int kRG, int kN>
__device__ __forceinline__ void rg_sum_transposed(float (&x)[kN], int rg) {
  int n = kN;
#pragma unroll
  for (int o = kRG / 2; o >= 1; o >>= 1) rg_sum_round(x, rg, o, n >>= 1);
}

// A scan may hold the row vectors of two tokens in registers and ask for a token's two tokens ahead: the loads of a token are 32
// cycles of the warp's way to shared memory per vector at 64 rows, and shuffles queue behind them.  It pays only where a chain warp
// has (nearly) a scheduler to itself, and the registers cost an SM its second CTA.  The most chain warps of a CTA with which it is
// done (0: never); 512 tokens, us, one token ahead -> two:
//   forward, 64 rows: 1 warp (8 units) 69 -> 64, leaving what the backward needs 74 -> 68; 2 (16 units) 72 -> 76; 8 (40 units)
//   110 -> 119; beyond 148 units, leaving it, 345 -> 374.  32 rows: 1 warp 57 -> 55; 4 (40 units) 57 -> 61; 150 units 125 -> 162.
//   state cotangent, 64 rows: 1, 2, 4 warps 71 -> 57, 76 -> 62, 82 -> 77; 8 106 -> 112, beyond 148 units 291 -> 333.  32 rows: up to
//   2 warps no difference, 4 53 -> 56, 8 66 -> 75.
// (8 and 16 rows: 3 to 10 % slower everywhere.  At 128 rows a lane has 16 of them and the registers are not there.)
template <int D> constexpr int two_ahead_forward() { return D == 32 || D == 64 ? 1 : 0; }
template <int D> constexpr int two_ahead_reverse() { return D == 64 ? 4 : 0; }

// Where the warps of a scan CTA stand.  A warp's scheduler is its index modulo 4: a lone chain warp has one to itself, the producers'
// warps lie on the other three (every fourth index stays empty).  With what stands between the shuffles of a token: 2 x 4 units,
// 512 tokens, D = 64, fp32, a chain warp's token in the forward 335 -> 295 cycles.
struct ScanWarps {
  int nw, spread;  // chain warps; whether the producers are spread
  __host__ __device__ int threads(int producers) const {
    const int n = producers / 32;
    return 32 * (spread ? 1 + n + (n - 1) / 3 : nw + n);
  }
  __device__ bool idle(int warp) const { return spread && warp > 0 && (warp & 3) == 0; }
  __device__ int producer(int warp) const { return spread ? warp - 1 - (warp >> 2) : warp - nw; }
};

// Only where the CTA has its SM to itself: the empty indexes of several CTAs crowd the other schedulers.  (One chain warp a CTA and more
// CTAs than SMs is 8 rows: 512 tokens of 300 units, leaving what the backward needs, spread 120 us, one after another 95.)
inline bool spread_producers(int nw, int ctas, int sms) { return nw == 1 && ctas <= sms; }

// Consumer warps per CTA: as few as possible while all CTAs run in one wave (a short chain wants
// its own SM), at most kMaxConsumers (the producers of a CTA redo the same row vectors, so with more
// units than SMs wide CTAs waste less).
inline int scan_consumers(int units, int warps_per_unit, int max_consumers, int sms) {
  int nw = 1;
  while (nw < max_consumers && nw < warps_per_unit && (long)units * warps_per_unit > (long)nw * sms) nw *= 2;
  return nw;
}

}  // namespace pkda
