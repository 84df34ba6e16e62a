// Control epilogue of the PKDA layer.  The layer projects its input once to a packed
// row  [decay hidden (D) | beta logits (H) | precond decay logits (H) | precond beta
// logits (H) | output-gate hidden (D)]  (delta_feedback_experiment/pkda.py:318-353);
// the two hidden slices go on to further projections unchanged and the three
// per-head slices become
//   beta     = sigmoid(logits)
//   g_atk    = -exp(A_log_precond) * softplus(logits + dt_bias_precond)      (fp32)
//   beta_atk = sigmoid(logits).
// Forward: one pass over the 3H logits of every row.  Backward: ONE pass that applies
// the three activations' derivatives and writes the packed gradient row directly,
// hidden slices included -- what the reference does with separate pointwise kernels
// plus pack_control_gradients (delta_feedback_experiment/cuda_kernels.py:1081-1172) --
// and reduces the two per-head parameter gradients in a fixed order.
// pkda_pack_control_gradients is that packer alone (five slices -> one row).
#include "pkda_common.cuh"
#include "pkda_launch.h"

namespace pkda {

struct CtrlParams {
  long long rows;
  int heads, hidden, total;
  const void* packed;
  const float *A_log, *dt_bias;
  void *beta, *beta_atk;
  float* g_atk;
  const void *d_hidden0, *d_beta, *d_beta_atk, *d_hidden1;
  const float* d_g_atk;
  void* d_packed;
  float* part;  // [gridDim.x][2][heads]
  int pairs;    // the hidden slices can be moved two elements at a time
};

constexpr int kCtrlThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kCtrlThreads)
pkda_controls_fwd_kernel(const CtrlParams p) {
  after_previous();
  const long long n = p.rows * p.heads;
  const T* packed = static_cast<const T*>(p.packed);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / p.heads;
    const int h = (int)(i - r * p.heads);
    const T* row = packed + r * p.total + p.hidden;
    const float lb = to_f(row[h]), ld = to_f(row[p.heads + h]), lp = to_f(row[2 * p.heads + h]);
    static_cast<T*>(p.beta)[i] = from_f<T>(1.f / (1.f + expf(-lb)));
    p.g_atk[i] = -expf(p.A_log[h]) * softplus_acc(ld + p.dt_bias[h]);
    static_cast<T*>(p.beta_atk)[i] = from_f<T>(1.f / (1.f + expf(-lp)));
  }
}

// Backward: the packed gradient row and the per-head parameter gradients.  A CTA owns a contiguous range of
// rows and takes ctrl_rows(H) of them at a time: the two hidden slices are copied and the three activations,
// formed again from the packed row, differentiated with one element (or pair) per thread; the contributions to the per-head sums go through
// shared memory and are added rows ascending, so that the sums have a fixed order.  (Row after row with one
// thread per column took a memory round trip per row: 45 us for 2,000 rows of 280, now 5.)
__host__ __device__ inline int ctrl_rows(int heads) { return heads >= 512 ? 1 : heads >= 256 ? 4 : 8; }

template <typename T>
__global__ void __launch_bounds__(kCtrlThreads)
pkda_controls_bwd_kernel(const CtrlParams p) {
  after_previous();
  extern __shared__ float sAcc[];  // [2][H] sums of the CTA, then [2][rows][H] contributions
  const int H = p.heads, D = p.hidden, total = p.total, tid = threadIdx.x;
  const int R = ctrl_rows(H);
  float* sPart = sAcc + 2 * H;
  for (int i = tid; i < 2 * H; i += kCtrlThreads) sAcc[i] = 0.f;
  __syncthreads();
  const T* packed = static_cast<const T*>(p.packed);
  T* out = static_cast<T*>(p.d_packed);
  const T *h0 = static_cast<const T*>(p.d_hidden0), *h1 = static_cast<const T*>(p.d_hidden1);
  const long long rows_per = (p.rows + gridDim.x - 1) / gridDim.x;
  const long long r_begin = (long long)blockIdx.x * rows_per;
  const long long r_end = r_begin + rows_per < p.rows ? r_begin + rows_per : p.rows;
  struct alignas(2 * sizeof(T)) Pair { T a, b; };
  for (long long r0 = r_begin; r0 < r_end; r0 += R) {
    const int nr = (int)(r_end - r0 < R ? r_end - r0 : R);
    if (p.pairs) {
      const int w = D >> 1;
      const Pair zero = {from_f<T>(0.f), from_f<T>(0.f)};
      for (int i = tid; i < nr * w; i += kCtrlThreads) {
        const int r = i / w, c = 2 * (i - r * w);
        const Pair x = h0 ? *reinterpret_cast<const Pair*>(h0 + (r0 + r) * D + c) : zero;
        const Pair y = h1 ? *reinterpret_cast<const Pair*>(h1 + (r0 + r) * D + c) : zero;
        T* row = out + (r0 + r) * total + c;
        *reinterpret_cast<Pair*>(row) = x;
        *reinterpret_cast<Pair*>(row + D + 3 * H) = y;
      }
    } else {
      for (int i = tid; i < nr * D; i += kCtrlThreads) {
        const int r = i / D, c = i - r * D;
        T* row = out + (r0 + r) * total + c;
        row[0] = h0 ? h0[(r0 + r) * D + c] : from_f<T>(0.f);
        row[D + 3 * H] = h1 ? h1[(r0 + r) * D + c] : from_f<T>(0.f);
      }
    }
    for (int i = tid; i < nr * H; i += kCtrlThreads) {
      const int r = i / H, h = i - r * H;
      const long long at = (r0 + r) * H + h;
      const T* in = packed + (r0 + r) * total + D + h;
      T* row = out + (r0 + r) * total + D + h;
      const float l0 = to_f(in[0]), l2 = to_f(in[2 * H]), z = to_f(in[H]) + p.dt_bias[h], ea = expf(p.A_log[h]);
      const float d0 = p.d_beta ? to_f(static_cast<const T*>(p.d_beta)[at]) : 0.f;
      const float d1 = p.d_g_atk ? p.d_g_atk[at] : 0.f;
      const float d2 = p.d_beta_atk ? to_f(static_cast<const T*>(p.d_beta_atk)[at]) : 0.f;
      const float s0 = 1.f / (1.f + expf(-l0)), s2 = 1.f / (1.f + expf(-l2));
      const float v = d1 * (-ea) / (1.f + expf(-z));   // d softplus = sigmoid
      row[0] = from_f<T>(d0 * s0 * (1.f - s0));
      row[H] = from_f<T>(v);
      row[2 * H] = from_f<T>(d2 * s2 * (1.f - s2));
      const float da = d1 * (-ea) * softplus_acc(z);   // d/dA_log = g_atk;  v = d/ddt_bias
      if (R == 1) {
        sAcc[i] += da;
        sAcc[H + i] += v;
      } else {
        sPart[i] = da;
        sPart[R * H + i] = v;
      }
    }
    if (R == 1) continue;  // (a head belongs to one thread)
    __syncthreads();
    for (int i = tid; i < 2 * H; i += kCtrlThreads) {
      const float* col = i < H ? sPart + i : sPart + R * H + (i - H);
      float acc = sAcc[i];
      for (int r = 0; r < nr; ++r) acc += col[r * H];
      sAcc[i] = acc;
    }
    __syncthreads();
  }
  __syncthreads();
  for (int i = tid; i < 2 * H; i += kCtrlThreads) p.part[(size_t)blockIdx.x * 2 * H + i] = sAcc[i];
}

// One CTA per sum: strided partial sums, then a tree (fixed order).
__global__ void __launch_bounds__(128)
pkda_controls_reduce_kernel(const float* part, float* dA_log, float* ddt_bias, int heads, int groups) {
  after_previous();
  __shared__ float s[128];
  const int i = blockIdx.x, tid = threadIdx.x;
  float a = 0.f;
  for (int g = tid; g < groups; g += 128) a += part[(size_t)g * 2 * heads + i];
  s[tid] = a;
  __syncthreads();
  for (int o = 64; o >= 1; o >>= 1) {
    if (tid < o) s[tid] += s[tid + o];
    __syncthreads();
  }
  if (tid == 0) (i < heads ? dA_log[i] : ddt_bias[i - heads]) = s[0];
}

// out[r][:] = concat of five slices
template <typename T>
__global__ void __launch_bounds__(kCtrlThreads)
pkda_pack_control_kernel(const T* g0, const T* g1, const T* g2, const T* g3, const T* g4, T* out, long long rows,
                         int s0, int s1, int s2, int s3, int s4) {
  after_previous();
  const int total = s0 + s1 + s2 + s3 + s4;
  const long long n = rows * total;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / total;
    int c = (int)(i - r * total);
    T v;
    if (c < s0) v = g0[r * s0 + c];
    else if ((c -= s0) < s1) v = g1[r * s1 + c];
    else if ((c -= s1) < s2) v = g2[r * s2 + c];
    else if ((c -= s2) < s3) v = g3[r * s3 + c];
    else v = g4[r * s4 + (c - s3)];
    out[i] = v;
  }
}

// ------------------------------------------------------------------ host side
static int ctrl_check(const pkda_controls_args& a, CtrlParams& p) {
  if (a.rows < 0 || a.heads <= 0 || a.hidden <= 0) return PKDA_ERR_SHAPE;
  if (a.dtype != PKDA_BF16 && a.dtype != PKDA_F32) return PKDA_ERR_DTYPE;
  p.rows = a.rows; p.heads = a.heads; p.hidden = a.hidden; p.total = 2 * a.hidden + 3 * a.heads;
  p.packed = a.packed; p.A_log = a.A_log_precond; p.dt_bias = a.dt_bias_precond;
  p.beta = a.beta; p.beta_atk = a.beta_atk; p.g_atk = a.g_atk;
  p.d_hidden0 = a.d_decay_hidden; p.d_beta = a.d_beta; p.d_beta_atk = a.d_beta_atk; p.d_hidden1 = a.d_gate_hidden;
  p.d_g_atk = a.d_g_atk; p.d_packed = a.d_packed; p.part = nullptr; p.pairs = 0;
  return PKDA_OK;
}

static int ctrl_bwd_grid(const pkda_controls_args& a) {
  const int r = ctrl_rows(a.heads);
  const long long want = (a.rows + r - 1) / r, most = 16LL * sm_count();  // one turn per CTA until the chip is full several times over
  return (int)(want < 1 ? 1 : (want < most ? want : most));
}

int controls_fwd(const pkda_controls_args* a, cudaStream_t st) {
  CtrlParams p;
  if (int rc = ctrl_check(*a, p)) return rc;
  if (a->rows == 0) return PKDA_OK;
  if (!a->packed || !a->A_log_precond || !a->dt_bias_precond || !a->beta || !a->g_atk || !a->beta_atk)
    return PKDA_ERR_NULL;
  const long long n = a->rows * a->heads;
  const long long blocks = (n + kCtrlThreads - 1) / kCtrlThreads, most = 16LL * sm_count();
  const int grid = (int)(blocks < most ? blocks : most);
  begin_stage(kStageControlsFwd, st);
  const int rc = a->dtype == PKDA_BF16 ? launch_kernel(pkda_controls_fwd_kernel<bf16>, grid, kCtrlThreads, 0, st, p)
                                       : launch_kernel(pkda_controls_fwd_kernel<float>, grid, kCtrlThreads, 0, st, p);
  end_stage(st);
  return rc;
}

size_t controls_bwd_workspace(const pkda_controls_args& a) {
  if (a.rows < 0 || a.heads <= 0) return 0;
  return align_up((size_t)ctrl_bwd_grid(a) * 2 * a.heads * sizeof(float));
}

int controls_bwd(const pkda_controls_args* a, cudaStream_t st) {
  CtrlParams p;
  if (int rc = ctrl_check(*a, p)) return rc;
  if (!a->dA_log_precond || !a->ddt_bias_precond) return PKDA_ERR_NULL;
  if (a->rows == 0) {
    const size_t nb = (size_t)a->heads * sizeof(float);
    return (cudaMemsetAsync(a->dA_log_precond, 0, nb, st) == cudaSuccess &&
            cudaMemsetAsync(a->ddt_bias_precond, 0, nb, st) == cudaSuccess) ? PKDA_OK : PKDA_ERR_LAUNCH;
  }
  if (!a->packed || !a->A_log_precond || !a->dt_bias_precond || !a->d_packed) return PKDA_ERR_NULL;
  if (!a->workspace || a->workspace_bytes < controls_bwd_workspace(*a)) return PKDA_ERR_WORKSPACE;
  p.part = static_cast<float*>(a->workspace);
  const int grid = ctrl_bwd_grid(*a);
  const int turn = ctrl_rows(a->heads);
  const size_t smem = (size_t)2 * a->heads * (turn == 1 ? 1 : 1 + turn) * sizeof(float);
  // pairs: every slice starts at an even column of an even row, and every tensor at a pair
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(a->d_decay_hidden) | reinterpret_cast<uintptr_t>(a->d_gate_hidden) |
                         reinterpret_cast<uintptr_t>(a->d_packed);
  p.pairs = !(a->heads & 1) && !(a->hidden & 1) && ptrs % (a->dtype == PKDA_BF16 ? 4 : 8) == 0;
  begin_stage(kStageControlsBwd, st);
  int rc = a->dtype == PKDA_BF16 ? launch_kernel(pkda_controls_bwd_kernel<bf16>, grid, kCtrlThreads, smem, st, p)
                                 : launch_kernel(pkda_controls_bwd_kernel<float>, grid, kCtrlThreads, smem, st, p);
  end_stage(st);
  if (rc != PKDA_OK) return rc;
  begin_stage(kStageControlsBwd, st);
  rc = launch_kernel(pkda_controls_reduce_kernel, 2 * a->heads, 128, 0, st, p.part, a->dA_log_precond, a->ddt_bias_precond, a->heads,
                grid);
  end_stage(st);
  return rc;
}

int pack_control_gradients(const pkda_pack_control_args* a, cudaStream_t st) {
  if (a->rows < 0) return PKDA_ERR_SHAPE;
  for (int i = 0; i < 5; ++i)
    if (a->sizes[i] < 0) return PKDA_ERR_SHAPE;
  if (a->dtype != PKDA_BF16 && a->dtype != PKDA_F32) return PKDA_ERR_DTYPE;
  const int total = a->sizes[0] + a->sizes[1] + a->sizes[2] + a->sizes[3] + a->sizes[4];
  const long long n = a->rows * total;
  if (n == 0) return PKDA_OK;
  if (!a->out) return PKDA_ERR_NULL;
  for (int i = 0; i < 5; ++i)
    if (a->sizes[i] > 0 && !a->grads[i]) return PKDA_ERR_NULL;
  const long long blocks = (n + kCtrlThreads - 1) / kCtrlThreads, most = 32LL * sm_count();
  const int grid = (int)(blocks < most ? blocks : most);
  begin_stage(kStagePackControl, st);
  int rc;
  if (a->dtype == PKDA_BF16)
    rc = launch_kernel(pkda_pack_control_kernel<bf16>, grid, kCtrlThreads, 0, st, static_cast<const bf16*>(a->grads[0]),
                  static_cast<const bf16*>(a->grads[1]), static_cast<const bf16*>(a->grads[2]), static_cast<const
                  bf16*>(a->grads[3]), static_cast<const bf16*>(a->grads[4]), static_cast<bf16*>(a->out), a->rows, a->sizes[0],
                  a->sizes[1], a->sizes[2], a->sizes[3], a->sizes[4]);
  else
    rc = launch_kernel(pkda_pack_control_kernel<float>, grid, kCtrlThreads, 0, st, static_cast<const float*>(a->grads[0]),
                  static_cast<const float*>(a->grads[1]), static_cast<const float*>(a->grads[2]), static_cast<const
                  float*>(a->grads[3]), static_cast<const float*>(a->grads[4]), static_cast<float*>(a->out), a->rows, a->sizes[0],
                  a->sizes[1], a->sizes[2], a->sizes[3], a->sizes[4]);
  end_stage(st);
  return rc;
}

}  // namespace pkda
