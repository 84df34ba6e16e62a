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
  static __device__ __forceinline__ uint32_t load(const bf16* p) { return *reinterpret_cast<const unsigned short*>(p); }
  static __device__ __forceinline__ float value(uint32_t r) { return __uint_as_float(r << 16); }
};

// Named barriers between the producer and the consumer warps of a scan CTA.
__device__ __forceinline__ void bar_sync_n(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive_n(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Sums over the kRG lanes of a column group, one per column; every lane gets all of them.  Four columns
// trade halves first, so that the remaining steps run on one register.
template <int kRG>
__device__ __forceinline__ void rg_sum(float (&v)[1], int) {
#pragma unroll
  for (int o = kRG / 2; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}
template <int kRG>
__device__ __forceinline__ void rg_sum(float (&v)[4], int rg) {
  const bool hi = rg & (kRG / 2), hi2 = rg & (kRG / 4);
  const float a = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], kRG / 2);
  const float b = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], kRG / 2);
  float x = (hi2 ? b : a) + __shfl_xor_sync(0xffffffffu, hi2 ? a : b, kRG / 4);
#pragma unroll
  for (int o = kRG / 8; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  const float y = __shfl_xor_sync(0xffffffffu, x, kRG / 4);
  const float p = hi2 ? y : x, q = hi2 ? x : y;
  const float r = __shfl_xor_sync(0xffffffffu, p, kRG / 2), t = __shfl_xor_sync(0xffffffffu, q, kRG / 2);
  v[0] = hi ? r : p;
  v[1] = hi ? t : q;
  v[2] = hi ? p : r;
  v[3] = hi ? q : t;
}

// kN per-lane partial sums: afterwards lane rg holds the totals of entries rg * (kN / kRG) ... in
// x[0 .. kN / kRG) (a transposing butterfly: about kN shuffles instead of kN * log2(kRG)).
template <int kRG, int kN>
__device__ __forceinline__ void rg_sum_transposed(float (&x)[kN], int rg) {
  int n = kN;
#pragma unroll
  for (int o = kRG / 2; o >= 1; o >>= 1) {
    const bool upper = rg & o;
    n >>= 1;
#pragma unroll
    for (int i = 0; i < kN / 2; ++i) {
      if (i < n) {
        const float keep = upper ? x[i + n] : x[i];
        const float send = upper ? x[i] : x[i + n];
        x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
}

// One run of kU consecutive fp32 values from shared memory, as pairs.
template <int kU>
__device__ __forceinline__ void load_run(const float* s, float2* out) {
  if (kU == 4) {
    const float4 x = *reinterpret_cast<const float4*>(s);
    out[0] = make_float2(x.x, x.y);
    out[1] = make_float2(x.z, x.w);
  } else {
    out[0] = *reinterpret_cast<const float2*>(s);
  }
}

// The kR values of one row vector that belong to the lane.
template <typename L>
__device__ __forceinline__ void load_rows(const float* vec, int rg, float2 (&x)[L::kR / 2]) {
#pragma unroll
  for (int b = 0; b < L::kR / L::kU; ++b) load_run<L::kU>(vec + L::row(b, rg), &x[b * (L::kU / 2)]);
}

// Consumer warps per CTA: as few as possible while all CTAs run in one wave (a short chain wants
// its own SM), at most kMaxConsumers (the producers of a CTA redo the same row vectors, so with more
// units than SMs wide CTAs waste less).
inline int scan_consumers(int units, int warps_per_unit, int max_consumers, int sms) {
  int nw = 1;
  while (nw < max_consumers && nw < warps_per_unit && (long)units * warps_per_unit > (long)nw * sms) nw *= 2;
  return nw;
}

}  // namespace pkda
