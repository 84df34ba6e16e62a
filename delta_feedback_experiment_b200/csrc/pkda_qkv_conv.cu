// Fused Q|K|V short convolution of the PKDA layer, forward and backward:
//   y[t][c] = sum_j w[c][j] * x[t - (taps-1) + j][c]      (causal, depthwise, <= 4 taps)
//   s = silu(y)
//   out = s * rsqrt(sum over the head of s^2 + eps)        for c < norm_channels (Q and K)
//   out = s                                                otherwise (V)
// written as three slabs q, k, v.  Streaming work that is bound by instruction issue rather than by DRAM: a
// warp's pass over one token of 128 channels is 55 instructions forward and 115 backward.  So
//  * a warp walks a span of tokens of 128 channels (four adjacent ones per lane) by itself, without block
//    barriers; the filter's window and, in the backward, the gradients of the pre-activation that the next
//    tokens' dx needs stay in registers, so nothing but the three rows around a span is computed twice;
//  * its rows arrive through a ring in the warp's own shared memory (16-byte cp.async copies two or three
//    steps of four tokens ahead).  Prefetched into registers instead, one step ahead, the forward has half
//    the bytes in flight and waits for memory (227 us at 8 x 4096 tokens of 16 heads x 128, against 133);
//  * the per-head sums of the four tokens of a step are reduced together, transposed: 10 shuffles and one
//    rsqrt instead of 20 and 4 (backward: 18 instead of 24);
//  * the arithmetic is written on pairs of channels with the packed fp32x2 instructions of sm_100, on half
//    the filter taps, which is what the sigmoid's tanh wants; silu' shares the forward's terms.
// The backward recomputes the pre-activation instead of saving it.  The weight gradient is reduced in a
// fixed order (registers -> across the CTA's token groups -> one partial per CTA -> a small second kernel).
// At 8 x 4096 tokens of 16 heads x 128: forward 166 -> 133 us, backward 453 -> 292 us, against a version
// with block-wide double-buffered tiles and per-token reductions (the traffic alone: 125 and 187 us).
#include "pkda_common.cuh"
#include "pkda_launch.h"

namespace pkda {

namespace conv {
constexpr int kVec = 4;          // channels per thread
constexpr int kThreads = 256;
constexpr int kTileCh = 256;     // channels per CTA = 64 lanes
constexpr int kLanes = kTileCh / kVec;
constexpr int kGroups = kThreads / kLanes;  // token groups per CTA (4)
constexpr int kMaxTaps = 4;
constexpr int kHalo = kMaxTaps - 1;
constexpr int kStep = 4;         // tokens of one step of a walk
constexpr int kWarpCh = 32 * kVec;
constexpr int kRing = 4;         // steps in the ring
constexpr int kWarps = kThreads / 32;
// Tokens one warp walks.  The four tokens that a backward walk looks ahead cost 3% at 128 and 6% at 64
// (298 and 342 us at the size above); 256 leaves the last wave emptier and gains nothing.
constexpr int kMaxSpan = 128, kMinSpan = 16;
template <typename T> __host__ __device__ constexpr int fwd_smem() { return kWarps * kRing * kStep * kWarpCh * (int)sizeof(T); }
template <typename T> __host__ __device__ constexpr int bwd_smem() { return 2 * fwd_smem<T>(); }
}  // namespace conv

struct ConvParams {
  int batch, seq_len, channels, slab, taps, head_lanes, norm_channels, spans_per_row, span;
  float eps;
  const void* x;
  const float* w;
  void *q, *k, *v;
  const void *dq, *dk, *dv;
  void* dx;
  float* part;  // [gridDim.y][channels][taps]
};

// Four adjacent channels as two pairs.
template <typename T> struct Vec4;
template <> struct Vec4<bf16> {
  using Raw = uint2;
  static __device__ __forceinline__ Raw fetch(const bf16* p) { return *reinterpret_cast<const uint2*>(p); }
  static __device__ __forceinline__ Raw zero() { return make_uint2(0u, 0u); }
  static __device__ __forceinline__ void unpack(const Raw& u, float2 (&f)[2]) {
    f[0] = unpack_bf16(u.x);
    f[1] = unpack_bf16(u.y);
  }
  static __device__ __forceinline__ void store(bf16* p, const float2 (&f)[2]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(f[0].x, f[0].y), pack_bf16(f[1].x, f[1].y));
  }
  // 2 sigmoid(2 h) = 1 + tanh(h) with the single-instruction tanh: relative error 2^-11,
  // below the bf16 rounding of the result.
  static __device__ __forceinline__ float2 two_sigmoid(float2 h) {
    float2 t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(h.x));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(h.y));
    return add2(t, f2(1.f, 1.f));
  }
};
template <> struct Vec4<float> {
  using Raw = float4;
  static __device__ __forceinline__ Raw fetch(const float* p) { return *reinterpret_cast<const float4*>(p); }
  static __device__ __forceinline__ Raw zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  static __device__ __forceinline__ void unpack(const Raw& u, float2 (&f)[2]) {
    f[0] = f2(u.x, u.y);
    f[1] = f2(u.z, u.w);
  }
  static __device__ __forceinline__ void store(float* p, const float2 (&f)[2]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
  }
  static __device__ __forceinline__ float2 two_sigmoid(float2 h) {
    return f2(2.f / (1.f + expf(-2.f * h.x)), 2.f / (1.f + expf(-2.f * h.y)));
  }
};

// Sum over the kHeadLanes adjacent lanes of one head (a power of two <= 32; a
// template parameter so that the token loops around it unroll without control flow).
template <int kHeadLanes>
__device__ __forceinline__ float head_sum(float v) {
#pragma unroll
  for (int o = kHeadLanes >> 1; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Two sums at once: the two halves of the head first trade one value each, so the
// butterfly runs on a single register (log2(L) + 1 shuffles instead of 2 log2(L)).
template <int kHeadLanes>
__device__ __forceinline__ void head_sum2(float& a, float& b, int lane) {
  if (kHeadLanes == 1) return;
  constexpr int kHalf = kHeadLanes / 2;
  const bool upper = lane & kHalf;
  float keep = upper ? b : a;
  const float send = upper ? a : b;
  keep += __shfl_xor_sync(0xffffffffu, send, kHalf);
#pragma unroll
  for (int o = kHalf >> 1; o >= 1; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
  const float other = __shfl_xor_sync(0xffffffffu, keep, kHalf);
  a = upper ? other : keep;
  b = upper ? keep : other;
}

// Half the filter taps of the thread's four channels as pairs: w[pair][tap], padded to four taps.  With them
// the convolution gives y / 2 exactly, which is what the sigmoid's tanh wants.
__device__ __forceinline__ void load_half_taps(const ConvParams& p, int c, bool active, float2 (&w)[2][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int jj = j - (conv::kMaxTaps - p.taps);  // tap j of the filter padded to four taps
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = (active && jj >= 0) ? 0.5f * p.w[(size_t)(c + i) * p.taps + jj] : 0.f;
    w[0][j] = f2(v[0], v[1]);
    w[1][j] = f2(v[2], v[3]);
  }
}

// Half the pre-activation of one token for the thread's two channel pairs.
__device__ __forceinline__ void conv4(float2 (&y)[2], const float2 (&w)[2][4], const float2 (&w0)[2],
                                      const float2 (&w1)[2], const float2 (&w2)[2], const float2 (&x)[2]) {
#pragma unroll
  for (int pr = 0; pr < 2; ++pr) {
    float2 a = mul2(w[pr][0], w0[pr]);
    a = fma2(w[pr][1], w1[pr], a);
    a = fma2(w[pr][2], w2[pr], a);
    y[pr] = fma2(w[pr][3], x[pr], a);
  }
}

// The rows of one walk on their way in: a ring of kRing steps in the warp's own shared memory, filled by
// 16-byte cp.async copies some steps ahead and read by all lanes behind a warp barrier.
template <typename T>
struct Feed {
  static constexpr int kPiece = 16 / (int)sizeof(T), kPerRow = conv::kWarpCh / kPiece, kRowsPerCopy = 32 / kPerRow;
  const T* src;  // the lane's 16-byte column piece in the row that it copies next
  T* dst;        // its place in slot 0
  int stride;

  // column: first element of the piece's column, in row 0 of the sequence; t: first row to copy
  __device__ __forceinline__ Feed(const T* column, int row_stride, int t, T* ring, int lane)
      : src(column + (long)(t + lane / kPerRow) * row_stride),
        dst(ring + (lane / kPerRow) * conv::kWarpCh + (lane % kPerRow) * kPiece), stride(row_stride) {}

  // Copies the next step's rows into `slot`.  row: the lane's first row; rows outside [0, end) read as zero
  // (end = 0 for a piece past the last channel); `valid` is any address that may be named.
  __device__ __forceinline__ void step(int slot, int row, int end, const T* valid) {
#pragma unroll
    for (int r = 0; r < conv::kStep; r += kRowsPerCopy) {
      const bool in = (unsigned)(row + r) < (unsigned)end;
      cp_async16(dst + slot * (conv::kStep * conv::kWarpCh) + r * conv::kWarpCh, in ? src : valid, in);
      src += kRowsPerCopy * stride;
    }
  }
};

// Sum of v[0..n-1] over the lanes of a head, n = 4 or 8, transposed: at every step the two halves of the
// head trade half of their values, so the butterfly costs n - 1 shuffles until each lane is left with one
// value and one more per remaining lane bit, instead of n log2(L).  Lane l ends with value l / (L / n)
// (its index inside the head).
template <int kHeadLanes, int n>
__device__ __forceinline__ float head_sums(float (&v)[n], int lane) {
  static_assert(kHeadLanes >= n, "a head narrower than the values to sum");
  int o = kHeadLanes >> 1;
#pragma unroll
  for (int k = n >> 1; k >= 1; k >>= 1, o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int j = 0; j < k; ++j) {
      const float send = upper ? v[j] : v[j + k];
      v[j] = (upper ? v[j + k] : v[j]) + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// 1 / |s| of the four tokens of a step.
template <int kHeadLanes>
__device__ __forceinline__ void head_norms(const float (&ss)[conv::kStep], float (&r)[conv::kStep], bool normed, float eps, int lane) {
  if constexpr (kHeadLanes >= conv::kStep) {
    float v[conv::kStep];
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) v[u] = ss[u];
    const float total = head_sums<kHeadLanes, conv::kStep>(v, lane);
    const float mine = normed ? rsqrtf(total + eps) : 1.f;
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) r[u] = __shfl_sync(0xffffffffu, mine, u * (kHeadLanes / conv::kStep), kHeadLanes);
  } else {
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) {
      const float total = head_sum<kHeadLanes>(ss[u]);  // (every lane takes part in the shuffles)
      r[u] = normed ? rsqrtf(total + eps) : 1.f;
    }
  }
}

// 1 / |s| and -<s, d> / |s|^3 of the four tokens of a step.
template <int kHeadLanes>
__device__ __forceinline__ void head_norms_back(const float (&ss)[conv::kStep], const float (&sd)[conv::kStep], float (&r)[conv::kStep],
                                                float (&back)[conv::kStep], bool normed, float eps, int lane) {
  if constexpr (kHeadLanes >= 2 * conv::kStep) {
    float v[2 * conv::kStep];
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) {
      v[u] = ss[u];
      v[u + conv::kStep] = sd[u];
    }
    const float total = head_sums<kHeadLanes, 2 * conv::kStep>(v, lane);
    const float other = __shfl_xor_sync(0xffffffffu, total, kHeadLanes / 2);
    const bool upper = lane & (kHeadLanes / 2);
    const float r1 = normed ? rsqrtf((upper ? other : total) + eps) : 1.f;
    const float b1 = normed ? -r1 * r1 * r1 * (upper ? total : other) : 0.f;
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) {
      r[u] = __shfl_sync(0xffffffffu, r1, u * (kHeadLanes / (2 * conv::kStep)), kHeadLanes);
      back[u] = __shfl_sync(0xffffffffu, b1, u * (kHeadLanes / (2 * conv::kStep)), kHeadLanes);
    }
  } else {
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) {
      float a = ss[u], d = sd[u];
      head_sum2<kHeadLanes>(a, d, lane);
      r[u] = normed ? rsqrtf(a + eps) : 1.f;
      back[u] = normed ? -r[u] * r[u] * r[u] * d : 0.f;
    }
  }
}

// Rows t0-3 .. t0-1 of the thread's column (zero before the sequence).
template <typename T>
__device__ __forceinline__ void load_window(typename Vec4<T>::Raw (&win)[conv::kHalo], const T* col, int stride, int t0,
                                            bool active) {
#pragma unroll
  for (int j = 0; j < conv::kHalo; ++j) {
    const int t = t0 - conv::kHalo + j;
    win[j] = active && t >= 0 ? Vec4<T>::fetch(col + (long)t * stride) : Vec4<T>::zero();
  }
}

// One warp's walk over `own` tokens from t0 (forward).  kNorm: some channel of the warp is normalised.
template <typename T, int kHeadLanes, bool kNorm>
__device__ __forceinline__ void conv_fwd_walk(const T* col, int xs, Feed<T> feed, int row, int end, const T* valid,
                                              const T* ring, T* out, int os, const float2 (&w)[2][4], int t0, int own,
                                              bool active, bool normed, float eps) {
  using namespace conv;
  constexpr int kSlot = kStep * kWarpCh;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kRing - 1; ++i) {
    if (kStep * i < own) feed.step(i, row, end, valid);
    row += kStep;
    cp_async_commit();
  }
  float2 x[kHalo + kStep][2];  // the filter's window, then the step's rows
  {
    typename Vec4<T>::Raw win[kHalo];
    load_window<T>(win, col, xs, t0, active);
#pragma unroll
    for (int j = 0; j < kHalo; ++j) Vec4<T>::unpack(win[j], x[kStep + j]);
  }
  T* orow = out + (long)t0 * os;
  int slot = 0;
#pragma unroll 1
  for (int t = 0; t < own; t += kStep) {
    cp_async_wait<kRing - 2>();
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kHalo; ++j) {
      x[j][0] = x[kStep + j][0];
      x[j][1] = x[kStep + j][1];
    }
#pragma unroll
    for (int u = 0; u < kStep; ++u) Vec4<T>::unpack(Vec4<T>::fetch(ring + slot * kSlot + u * kWarpCh), x[kHalo + u]);
    if (t + (kRing - 1) * kStep < own) feed.step((slot + kRing - 1) % kRing, row, end, valid);
    row += kStep;
    cp_async_commit();
    slot = (slot + 1) % kRing;
    float2 s[kStep][2];
    float ss[kStep], r[kStep];
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      conv4(s[u], w, x[u], x[u + 1], x[u + 2], x[u + 3]);
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) s[u][pr] = mul2(s[u][pr], Vec4<T>::two_sigmoid(s[u][pr]));
      const float2 sq = fma2(s[u][1], s[u][1], mul2(s[u][0], s[u][0]));
      ss[u] = sq.x + sq.y;
    }
    if (kNorm) head_norms<kHeadLanes>(ss, r, normed, eps, lane);
#pragma unroll
    for (int u = 0; u < kStep; ++u) {
      if (kNorm) {
        s[u][0] = mul2(s[u][0], f2(r[u], r[u]));
        s[u][1] = mul2(s[u][1], f2(r[u], r[u]));
      }
      if (active && t + u < own) Vec4<T>::store(orow + u * os, s[u]);
    }
    orow += kStep * os;
  }
}

// One warp's walk (backward): dx of `own` tokens from t0 and their rows' part of the weight gradient.  dx of a
// token needs the pre-activation gradients of the three tokens after it, so the walk goes one step further
// than its own tokens; those gradients stay in registers.  w holds half the taps: the doubled
// pre-activation gradients make up for it in dx, and dwacc comes out doubled.
template <typename T, int kHeadLanes, bool kNorm>
__device__ __forceinline__ void conv_bwd_walk(Feed<T> fx, Feed<T> fd, int row, int end, const T* valid, const T* xring,
                                              const T* dring, T* drow, int xs, const float2 (&w)[2][4],
                                              float2 (&dwacc)[2][4], int own, bool active, bool normed, float eps) {
  constexpr int kSlot = conv::kStep * conv::kWarpCh;
  const int walk = own + conv::kHalo;
  const int lane = threadIdx.x & 31;
  // Step i lies in slot i % kRing of both rings; the three rows before the walk count as step -1.  The step
  // before the current one is still read (the filter's window), so the copies run kAhead = kRing - 2 ahead.
  constexpr int kAhead = conv::kRing - 2;
  fx.step(conv::kRing - 1, row - conv::kStep, end, valid);
#pragma unroll
  for (int i = 0; i < kAhead; ++i) {
    if (conv::kStep * i < walk) {
      fx.step(i, row, end, valid);
      fd.step(i, row, end, valid);
    }
    row += conv::kStep;
    cp_async_commit();
  }
  float2 dy[conv::kHalo + conv::kStep][2];
#pragma unroll
  for (int j = 0; j < conv::kHalo; ++j) dy[conv::kStep + j][0] = dy[conv::kStep + j][1] = f2(0.f, 0.f);
  int slot = 0;
#pragma unroll 1
  for (int t = 0; t < walk; t += conv::kStep) {
    cp_async_wait<kAhead - 1>();
    __syncwarp();
    if (t + kAhead * conv::kStep < walk) {
      fx.step((slot + kAhead) % conv::kRing, row, end, valid);
      fd.step((slot + kAhead) % conv::kRing, row, end, valid);
    }
    row += conv::kStep;
    cp_async_commit();
    const T* xc = xring + slot * kSlot;
    const T* xp = xring + (slot + conv::kRing - 1) % conv::kRing * kSlot + (conv::kStep - conv::kHalo) * conv::kWarpCh;
    float2 sc[conv::kStep][2], dc[conv::kStep][2];  // s silu'(y) and d silu'(y), doubled
    float ss[conv::kStep], sd[conv::kStep], r[conv::kStep], back[conv::kStep];
#pragma unroll
    for (int j = 0; j < conv::kHalo; ++j) {
      dy[j][0] = dy[conv::kStep + j][0];
      dy[j][1] = dy[conv::kStep + j][1];
    }
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) {
      Vec4<T>::unpack(Vec4<T>::fetch(dring + slot * kSlot + u * conv::kWarpCh), dc[u]);
    }
    {
      float2 x[conv::kHalo + conv::kStep][2];
#pragma unroll
      for (int j = 0; j < conv::kHalo + conv::kStep; ++j)
        Vec4<T>::unpack(Vec4<T>::fetch(j < conv::kHalo ? xp + j * conv::kWarpCh : xc + (j - conv::kHalo) * conv::kWarpCh), x[j]);
#pragma unroll
      for (int u = 0; u < conv::kStep; ++u) {
        float2 h[2], s[2], c[2];
        conv4(h, w, x[u], x[u + 1], x[u + 2], x[u + 3]);
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) {  // with g = 2 sigmoid(y): s = h g and 2 silu'(y) = g + s (2 - g)
          const float2 g = Vec4<T>::two_sigmoid(h[pr]);
          s[pr] = mul2(h[pr], g);
          c[pr] = fma2(s[pr], fma2(g, f2(-1.f, -1.f), f2(2.f, 2.f)), g);
        }
        if (kNorm) {
          const float2 sq = fma2(s[1], s[1], mul2(s[0], s[0]));
          const float2 sv = fma2(s[1], dc[u][1], mul2(s[0], dc[u][0]));
          ss[u] = sq.x + sq.y;
          sd[u] = sv.x + sv.y;
        }
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) {
          if (kNorm) sc[u][pr] = mul2(s[pr], c[pr]);
          dc[u][pr] = mul2(dc[u][pr], c[pr]);
        }
      }
    }
    // Four rows are read a second time for the weight gradient: kept in between, they would be registers that the
    // walk does not have.  (Its three oldest rows kept unpacked for the next step instead: 291.6 -> 294.5 us.)
    asm volatile("" ::: "memory");
    if (kNorm) head_norms_back<kHeadLanes>(ss, sd, r, back, normed, eps, lane);
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u)
#pragma unroll
      for (int pr = 0; pr < 2; ++pr)  // (r d - s r^3 <s, d>) silu'(y)
        dy[conv::kHalo + u][pr] = kNorm ? fma2(sc[u][pr], f2(back[u], back[u]), mul2(dc[u][pr], f2(r[u], r[u]))) : dc[u][pr];
    // dx of the rows t - 3 .. t, and with the same four gradients of the pre-activation each row's part of the weight gradient.
    // (A walk's weight gradient by the rows of x that it owns, not by their outputs, needs four rows a step instead of seven:
    // 296.5 -> 291.6 us at 8 x 4,096 tokens of 16 heads.)
#pragma unroll
    for (int u = 0; u < conv::kStep; ++u) {
      const int e = t + u - conv::kHalo;
      float2 o[2], x[2];
      Vec4<T>::unpack(Vec4<T>::fetch(u < conv::kHalo ? xp + u * conv::kWarpCh : xc), x);
      const bool mine = e >= 0 && e < own;  // (rows before the walk are the neighbour's, rows behind it too)
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) {
        float2 a = mul2(w[pr][3], dy[u][pr]);
        a = fma2(w[pr][2], dy[u + 1][pr], a);
        a = fma2(w[pr][1], dy[u + 2][pr], a);
        o[pr] = fma2(w[pr][0], dy[u + 3][pr], a);
        if (mine) {
#pragma unroll
          for (int j = 0; j < 4; ++j) dwacc[pr][j] = fma2(dy[u + 3 - j][pr], x[pr], dwacc[pr][j]);
        }
      }
      if (active && mine) Vec4<T>::store(drow + u * xs, o);
    }
    drow += conv::kStep * xs;
    slot = (slot + 1) % conv::kRing;
  }
}

template <typename T, int kHeadLanes>
__global__ void __launch_bounds__(conv::kThreads, sizeof(T) == 2 ? 3 : 2)
pkda_qkv_conv_fwd_kernel(const ConvParams p) {
  after_previous();
  using namespace conv;
  const int b = blockIdx.y / p.spans_per_row;
  const int lane = threadIdx.x % kLanes, grp = threadIdx.x / kLanes;
  const int t0 = ((blockIdx.y - b * p.spans_per_row) * kGroups + grp) * p.span;
  const int own = min(p.span, p.seq_len - t0);
  const int c = blockIdx.x * kTileCh + kVec * lane;
  const bool active = c < p.channels;
  const bool normed = active && c < p.norm_channels;
  if (own <= 0) return;
  float2 w[2][4];
  load_half_taps(p, c, active, w);
  const int cc = active ? c : 0;
  const int slab_id = cc / p.slab, cs = cc - slab_id * p.slab;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kWarpRing = kRing * kStep * kWarpCh;
  const int wl = threadIdx.x & 31;
  T* ring = reinterpret_cast<T*>(smem_raw) + (threadIdx.x >> 5) * kWarpRing;
  const T* x = static_cast<const T*>(p.x) + (size_t)b * p.seq_len * p.channels;
  T* out = static_cast<T*>(slab_id == 0 ? p.q : slab_id == 1 ? p.k : p.v) + (size_t)b * p.seq_len * p.slab + cs;
  const int pc = c - kVec * wl + (wl % Feed<T>::kPerRow) * Feed<T>::kPiece;  // channel of the lane's copy piece
  const bool pok = pc < p.channels;
  const int row = t0 + wl / Feed<T>::kPerRow, end = pok ? p.seq_len : 0;
  const Feed<T> feed(x + (pok ? pc : 0), p.channels, t0, ring, wl);
  const T* valid = static_cast<const T*>(p.x);
  if (__any_sync(0xffffffffu, normed))
    conv_fwd_walk<T, kHeadLanes, true>(x + cc, p.channels, feed, row, end, valid, ring + kVec * wl, out, p.slab, w, t0,
                                       own, active, normed, p.eps);
  else
    conv_fwd_walk<T, kHeadLanes, false>(x + cc, p.channels, feed, row, end, valid, ring + kVec * wl, out, p.slab, w, t0,
                                        own, active, normed, p.eps);
}

template <typename T, int kHeadLanes>
__global__ void __launch_bounds__(conv::kThreads, sizeof(T) == 2 ? 2 : 1)
pkda_qkv_conv_bwd_kernel(const ConvParams p) {
  after_previous();
  using namespace conv;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sPart = reinterpret_cast<float*>(smem_raw);  // [kGroups][kLanes][16]; entry 4 * channel + padded tap
  const int b = blockIdx.y / p.spans_per_row;
  const int lane = threadIdx.x % kLanes, grp = threadIdx.x / kLanes;
  const int t0 = ((blockIdx.y - b * p.spans_per_row) * kGroups + grp) * p.span;
  const int own = min(p.span, p.seq_len - t0);
  const int c = blockIdx.x * kTileCh + kVec * lane;
  const bool active = c < p.channels;
  const bool normed = active && c < p.norm_channels;
  float2 w[2][4], dwacc[2][4];
  load_half_taps(p, c, active, w);
#pragma unroll
  for (int pr = 0; pr < 2; ++pr)
#pragma unroll
    for (int j = 0; j < 4; ++j) dwacc[pr][j] = f2(0.f, 0.f);
  if (own > 0) {
    constexpr int kWarpRing = kRing * kStep * kWarpCh;
    const int cc = active ? c : 0, wl = threadIdx.x & 31;
    T* xring = reinterpret_cast<T*>(smem_raw) + (threadIdx.x >> 5) * 2 * kWarpRing;
    T* dring = xring + kWarpRing;
    const size_t row = (size_t)b * p.seq_len;
    const T* x = static_cast<const T*>(p.x) + row * p.channels;
    // the lane's copy piece; a 16-byte piece never straddles slabs because the slab width is a multiple of 8
    const int pc = c - kVec * wl + (wl % Feed<T>::kPerRow) * Feed<T>::kPiece;
    const bool pok = pc < p.channels;
    const int ps = pok ? pc / p.slab : 0;
    const T* d = static_cast<const T*>(ps == 0 ? p.dq : ps == 1 ? p.dk : p.dv) + row * p.slab + (pok ? pc - ps * p.slab : 0);
    const int wrow = t0 + wl / Feed<T>::kPerRow, end = pok ? p.seq_len : 0;
    const Feed<T> fx(x + (pok ? pc : 0), p.channels, t0 - kStep, xring, wl);
    const Feed<T> fd(d, p.slab, t0, dring, wl);
    const T* valid = static_cast<const T*>(p.x);
    T* drow = static_cast<T*>(p.dx) + row * p.channels + cc + (long)(t0 - kHalo) * p.channels;
    if (__any_sync(0xffffffffu, normed))
      conv_bwd_walk<T, kHeadLanes, true>(fx, fd, wrow, end, valid, xring + kVec * wl, dring + kVec * wl, drow,
                                         p.channels, w, dwacc, own, active, normed, p.eps);
    else
      conv_bwd_walk<T, kHeadLanes, false>(fx, fd, wrow, end, valid, xring + kVec * wl, dring + kVec * wl, drow,
                                          p.channels, w, dwacc, own, active, normed, p.eps);
  }
  cp_async_wait<0>();
  __syncthreads();  // the partials take the place of the rings
  // ---- weight gradient: the token groups in a fixed order, one partial per CTA
#pragma unroll
  for (int pr = 0; pr < 2; ++pr)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sPart[(grp * kLanes + lane) * 16 + 4 * (2 * pr) + j] = 0.5f * dwacc[pr][j].x;
      sPart[(grp * kLanes + lane) * 16 + 4 * (2 * pr + 1) + j] = 0.5f * dwacc[pr][j].y;
    }
  __syncthreads();
  if (grp == 0 && active) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      for (int j = 0; j < p.taps; ++j) {
        const int e = 4 * i + j + (kMaxTaps - p.taps);
        float a = 0.f;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) a += sPart[(g * kLanes + lane) * 16 + e];
        p.part[((size_t)blockIdx.y * p.channels + c + i) * p.taps + j] = a;
      }
  }
}

// Sums the per-CTA partials in a fixed order: a warp takes every eighth partial of 32 entries.  (A thread that walks all
// partials of its entry waits for memory once per four of them; forward + backward at 8 x 4,096 tokens of 16 heads: 0.6 % less.)
__global__ void __launch_bounds__(256) pkda_qkv_conv_dw_kernel(const float* part, float* dw, int n, int groups) {
  after_previous();
  __shared__ float s[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, idx = blockIdx.x * 32 + lane;
  float a = 0.f;
  if (idx < n) {
#pragma unroll 8
    for (int g = warp; g < groups; g += 8) a += part[(size_t)g * n + idx];
  }
  s[warp][lane] = a;
  __syncthreads();
  if (warp == 0 && idx < n) {
#pragma unroll
    for (int w = 1; w < 8; ++w) a += s[w][lane];
    dw[idx] = a;
  }
}

// ------------------------------------------------------------------ host side
static int conv_check(const pkda_qkv_conv_args& a, ConvParams& p) {
  if (a.batch < 0 || a.seq_len < 0 || a.channels <= 0 || a.channels % 3) return PKDA_ERR_SHAPE;
  if (a.taps < 1 || a.taps > conv::kMaxTaps) return PKDA_ERR_SHAPE;
  const int slab = a.channels / 3, hd = a.head_dim;
  if (hd < 8 || hd > 128 || (hd & (hd - 1)) || slab % hd) return PKDA_ERR_SHAPE;
  if (a.norm_channels < 0 || a.norm_channels > a.channels || a.norm_channels % hd) return PKDA_ERR_SHAPE;
  if (a.dtype != PKDA_BF16 && a.dtype != PKDA_F32) return PKDA_ERR_DTYPE;
  p.batch = a.batch; p.seq_len = a.seq_len; p.channels = a.channels; p.slab = slab; p.taps = a.taps;
  p.head_lanes = hd / conv::kVec; p.norm_channels = a.norm_channels; p.eps = a.eps;
  p.spans_per_row = 0;
  p.x = a.x; p.w = a.weight; p.q = a.q; p.k = a.k; p.v = a.v;
  p.dq = a.dq; p.dk = a.dk; p.dv = a.dv; p.dx = a.dx; p.part = nullptr;
  return PKDA_OK;
}

// Grid of both directions, and the tokens one warp walks (p.span): the longest span that still gives every SM
// four CTAs (two waves of the backward's two), so that short inputs spread over the chip instead.
static dim3 conv_grid(ConvParams& p) {
  const unsigned cols = (unsigned)((p.channels + conv::kTileCh - 1) / conv::kTileCh);
  const long wanted = 4L * sm_count();
  p.span = conv::kMaxSpan;
  for (;; p.span /= 2) {
    const int tokens = p.span * conv::kGroups;
    p.spans_per_row = (p.seq_len + tokens - 1) / tokens;
    const dim3 grid(cols, (unsigned)(p.batch * p.spans_per_row));
    if (p.span == conv::kMinSpan || (long)grid.x * grid.y >= wanted) return grid;
  }
}

static bool aligned16(const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; }

template <typename T, int kHeadLanes>
static int launch_conv_fwd(const ConvParams& p, dim3 grid, cudaStream_t st) {
  if (!ensure_dynamic_smem(pkda_qkv_conv_fwd_kernel<T, kHeadLanes>, conv::fwd_smem<T>())) return PKDA_ERR_LAUNCH;
  begin_stage(kStageConvFwd, st);
  const int rc = launch_kernel(pkda_qkv_conv_fwd_kernel<T, kHeadLanes>, grid, conv::kThreads, conv::fwd_smem<T>(), st, p);
  end_stage(st);
  return rc;
}

template <typename T, int kHeadLanes>
static int launch_conv_bwd(const ConvParams& p, dim3 grid, cudaStream_t st) {
  if (!ensure_dynamic_smem(pkda_qkv_conv_bwd_kernel<T, kHeadLanes>, conv::bwd_smem<T>())) return PKDA_ERR_LAUNCH;
  begin_stage(kStageConvBwd, st);
  const int rc = launch_kernel(pkda_qkv_conv_bwd_kernel<T, kHeadLanes>, grid, conv::kThreads, conv::bwd_smem<T>(), st, p);
  end_stage(st);
  return rc;
}

// Picks the instantiation for the activation type and the lanes per head.
#define PKDA_CONV_DISPATCH(FN, T)                                   \
  switch (p.head_lanes) {                                           \
    case 2: rc = FN<T, 2>(p, grid, st); break;                      \
    case 4: rc = FN<T, 4>(p, grid, st); break;                      \
    case 8: rc = FN<T, 8>(p, grid, st); break;                      \
    case 16: rc = FN<T, 16>(p, grid, st); break;                    \
    default: rc = FN<T, 32>(p, grid, st); break;                    \
  }

int qkv_conv_fwd(const pkda_qkv_conv_args* a, cudaStream_t st) {
  ConvParams p;
  if (int rc = conv_check(*a, p)) return rc;
  if (a->batch == 0 || a->seq_len == 0) return PKDA_OK;
  if (!a->x || !a->weight || !a->q || !a->k || !a->v) return PKDA_ERR_NULL;
  if (!aligned16(a->x) || !aligned16(a->q) || !aligned16(a->k) || !aligned16(a->v)) return PKDA_ERR_ALIGN;
  const dim3 grid = conv_grid(p);
  int rc = PKDA_OK;
  if (a->dtype == PKDA_BF16) { PKDA_CONV_DISPATCH(launch_conv_fwd, bf16) } else { PKDA_CONV_DISPATCH(launch_conv_fwd, float) }
  return rc;
}

size_t qkv_conv_bwd_workspace(const pkda_qkv_conv_args& a) {
  ConvParams p;
  if (conv_check(a, p) != PKDA_OK) return 0;
  const dim3 grid = conv_grid(p);
  return align_up((size_t)grid.y * a.channels * a.taps * sizeof(float));
}

int qkv_conv_bwd(const pkda_qkv_conv_args* a, cudaStream_t st) {
  ConvParams p;
  if (int rc = conv_check(*a, p)) return rc;
  if (!a->dweight) return PKDA_ERR_NULL;
  const int n = a->channels * a->taps;
  if (a->batch == 0 || a->seq_len == 0) {
    return cudaMemsetAsync(a->dweight, 0, (size_t)n * sizeof(float), st) == cudaSuccess ? PKDA_OK : PKDA_ERR_LAUNCH;
  }
  if (!a->x || !a->weight || !a->dq || !a->dk || !a->dv || !a->dx) return PKDA_ERR_NULL;
  if (!aligned16(a->x) || !aligned16(a->dq) || !aligned16(a->dk) || !aligned16(a->dv) || !aligned16(a->dx))
    return PKDA_ERR_ALIGN;
  if (!a->workspace || a->workspace_bytes < qkv_conv_bwd_workspace(*a)) return PKDA_ERR_WORKSPACE;
  p.part = static_cast<float*>(a->workspace);
  const dim3 grid = conv_grid(p);
  int rc = PKDA_OK;
  if (a->dtype == PKDA_BF16) { PKDA_CONV_DISPATCH(launch_conv_bwd, bf16) } else { PKDA_CONV_DISPATCH(launch_conv_bwd, float) }
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageConvDw, st);
  rc = launch_kernel(pkda_qkv_conv_dw_kernel, (n + 31) / 32, 256, 0, st, p.part, a->dweight, n, (int)grid.y);
  end_stage(st);
  return rc;
}

}  // namespace pkda
