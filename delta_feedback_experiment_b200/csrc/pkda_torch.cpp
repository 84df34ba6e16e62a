// Host side of the operators: turns torch tensors into the C ABI's argument structs,
// allocates outputs and scratch, and registers the differentiable operators with
// torch's dispatcher.  Everything between a Python call and the kernel launches runs
// here, because at small sizes (one decoding step, a short row, a narrow layer) the
// kernels are shorter than the interpreter work that used to surround them: filling
// one struct through ctypes, entering the device guard and allocating tensors from
// Python cost 33 us per decoding step and 0.8 ms per small training step, against
// 4 us and 0.13 ms of kernels.
//
// Three kinds of entry:
//  * dispatcher operators (delta_feedback::pkda_recurrence, pkda_qkv_conv, pkda_norm_gate
//    and their backwards): schema, CUDA kernel and autograd kernel; the fake kernels are
//    registered from Python;
//  * differentiable functions without a dispatcher name (chunked and exact recurrence with
//    states, control epilogue), called from Python through the module `_native`;
//  * plain launchers (`_native.*`) for the non-differentiable calls.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <atomic>
#include <functional>
#include <mutex>

#include "pkda_b200.h"

namespace {

using at::Tensor;
using c10::SymInt;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------ bookkeeping
std::atomic<long long> g_launches{0};  // kernels enqueued (launch accounting)

// Optional copies of the chunked calls' device status words (a debugging aid).
std::atomic<bool> g_track{false};
std::mutex g_status_mutex;
Tensor g_fwd_status, g_bwd_status;

void finish(int status, const char* what) {
  TORCH_CHECK(status == 0, what, " failed: ", pkda_status_string(status), " (status ", status, ")");
  g_launches.fetch_add(pkda_last_launch_count(), std::memory_order_relaxed);
}

void track_status(Tensor& slot, const Tensor& workspace, size_t offset) {
  if (!g_track.load(std::memory_order_relaxed)) return;
  Tensor word = workspace.narrow(0, (int64_t)offset, 4).clone();
  // The word before goes after the lock: Python may own it, and letting go of it then takes the interpreter lock,
  // which a reader of the status holds while it waits for this one.
  std::lock_guard<std::mutex> lock(g_status_mutex);
  std::swap(slot, word);
}

// ---------------------------------------------------------------------- tensors
Tensor empty(at::IntArrayRef shape, const c10::Device& dev, at::ScalarType dtype) {
  return at::detail::empty_cuda(shape, dtype, dev, std::nullopt);
}

Tensor scratch(size_t nbytes, const c10::Device& dev) {
  return empty({(int64_t)std::max<size_t>(nbytes, 16)}, dev, at::kByte);
}

// Every given tensor must live on one and the same CUDA device (the kernels run on a
// single device and dereference every pointer there).
struct DeviceCheck {
  c10::Device dev{c10::kCPU};
  bool seen = false;
  void operator()(const Tensor& t) {
    if (!t.defined()) return;
    TORCH_CHECK(t.is_cuda(), "PKDA CUDA operators need CUDA tensors; there is no CPU path");
    if (!seen) {
      dev = t.device();
      seen = true;
    } else {
      TORCH_CHECK(t.device() == dev, "PKDA operator arguments live on different devices (", dev, " and ", t.device(), ")");
    }
  }
  void operator()(const OptTensor& t) {
    if (t) (*this)(*t);
  }
};

template <typename... Ts>
c10::Device one_device(const Ts&... ts) {
  DeviceCheck check;
  (check(ts), ...);
  return check.dev;
}

// Tensors whose storage must outlive the launches of one call (casts, contiguous copies).
struct Keep {
  c10::SmallVector<Tensor, 16> held;

  const void* as(const Tensor& t, at::ScalarType dtype) {
    if (t.scalar_type() == dtype && t.is_contiguous()) return t.const_data_ptr();
    held.push_back(t.detach().to(dtype).contiguous());
    return held.back().const_data_ptr();
  }
};

int act_code(const Tensor& t, const char* who) {
  if (t.scalar_type() == at::kBFloat16) return PKDA_BF16;
  TORCH_CHECK(t.scalar_type() == at::kFloat, who, t.scalar_type());
  return PKDA_F32;
}

// A gradient in the shape and dtype of the input it belongs to.
Tensor like_input(Tensor g, const Tensor& input) {
  if (g.sizes() != input.sizes()) g = g.reshape(input.sizes());
  return g.scalar_type() == input.scalar_type() ? g : g.to(input.scalar_type());
}

// ------------------------------------------------------------------- recurrence
// The ten inputs, optional initial states and optional packing of every recurrence call.
struct Inputs {
  const Tensor &q, &k, &v, &g, &g_atk, &beta_atk, &beta, &A_log, &dt_bias, &log_atk_scale;
  const OptTensor &S0, &A0, &cu;
  double scale, squash_x, squash_eps;
};

const OptTensor kNone = std::nullopt;

struct Problem {
  pkda_problem p{};
  Keep keep;
  c10::Device dev{c10::kCPU};
  int64_t B, T, H, D, N;
  at::ScalarType act;

  explicit Problem(const Inputs& in) {
    dev = one_device(in.q, in.k, in.v, in.g, in.g_atk, in.beta_atk, in.beta, in.A_log, in.dt_bias, in.log_atk_scale,
                     in.S0, in.A0);
    TORCH_CHECK(in.q.dim() == 4, "PKDA input has ", in.q.dim(), " dimensions, expected [B, T, H, D]");
    B = in.q.size(0); T = in.q.size(1); H = in.q.size(2); D = in.q.size(3);
    p.dtype = act_code(in.q, "PKDA supports bf16 and fp32 activations, not ");
    act = in.q.scalar_type();
    const int64_t full[4] = {B, T, H, D};
    const at::IntArrayRef rows(full, 4), scalars(full, 3);
    p.q = activation(in.q, rows); p.k = activation(in.k, rows);
    p.v = activation(in.v, rows); p.g = activation(in.g, rows);
    p.g_atk = parameter(in.g_atk, B * T * H);
    p.beta_atk = activation(in.beta_atk, scalars);
    p.beta = activation(in.beta, scalars);
    if (in.cu) {
      TORCH_CHECK(B == 1, "packed input (cu_seqlens) needs batch size 1");
      Tensor cu = *in.cu;
      if (cu.device() != dev || cu.scalar_type() != at::kInt || !cu.is_contiguous())
        cu = cu.to(at::TensorOptions().device(dev).dtype(at::kInt)).contiguous();
      N = cu.numel() - 1;
      p.cu_seqlens = static_cast<const int32_t*>(cu.const_data_ptr());
      keep.held.push_back(std::move(cu));
    } else {
      N = B;
      p.seq_len = (int32_t)T;
    }
    p.n_seqs = (int32_t)N;
    p.total_tokens = (int32_t)(B * T);
    p.heads = (int32_t)H; p.head_dim = (int32_t)D;
    p.scale = (float)in.scale; p.squash_x = (float)in.squash_x; p.squash_eps = (float)in.squash_eps;
    p.A_log = parameter(in.A_log, H);
    p.dt_bias = parameter(in.dt_bias, H * D);
    p.log_atk_scale = parameter(in.log_atk_scale, H);
    if (in.S0) p.initial_state = parameter(*in.S0, N * H * D * D);
    if (in.A0) p.initial_A_state = parameter(*in.A0, N * H * D);
  }

  // Length of the flat chunk axis (packed: an upper bound, the exact count would need a read-back).
  int64_t chunks() const { return p.cu_seqlens ? T / 64 + N : B * ((T + 63) / 64); }

 private:
  const void* activation(const Tensor& t, at::IntArrayRef shape) {
    TORCH_CHECK(t.sizes() == shape, "PKDA input has shape ", t.sizes(), ", expected ", shape);
    return keep.as(t, act);
  }
  const float* parameter(const Tensor& t, int64_t numel) {
    TORCH_CHECK(t.numel() == numel, "PKDA parameter has ", t.numel(), " elements, expected ", numel);
    return static_cast<const float*>(keep.as(t, at::kFloat));
  }
};

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

constexpr int kKept = 6, kSaved = 11;  // intermediates kept by a lean forward / in all

// Intermediates of the chunked forward, in the operator's order: Aqk, Akk, k_precond, ac_atk,
// a_atk, sa_atk, then w, kg, v_new, h, qg (fla_ops.PKDA_INTERMEDIATES + PKDA_RETAINED).
void alloc_saved(const Problem& P, std::vector<Tensor>& saved, int from, int to) {
  const int64_t B = P.B, T = P.T, H = P.H, D = P.D, NT = P.p.cu_seqlens ? P.chunks() : (T + 63) / 64;
  for (int i = from; i < to; ++i) {
    switch (i) {
      case 0: case 1: saved.push_back(empty({B, T, H, 64}, P.dev, P.act)); break;
      case 3: case 4: saved.push_back(empty({B, NT, H, D}, P.dev, at::kFloat)); break;
      case 5: saved.push_back(empty({B, NT, H}, P.dev, at::kFloat)); break;
      case 9: saved.push_back(empty({B, NT, H, D, D}, P.dev, P.act)); break;
      default: saved.push_back(empty({B, T, H, D}, P.dev, P.act)); break;
    }
  }
}

// The list that the operator hands back must be exactly what its fake implementation promises to a compiler
// (count, and per entry shape, dtype, device, contiguity): a mismatch would surface far away, as a stride or
// shape error inside a compiled graph.  Derived from the inputs, not from alloc_saved, and run on every call
// of the operator (under a microsecond).
void check_intermediates(at::TensorList got, const Tensor& q, const Tensor& v, bool lean) {
  static const char* const names[kSaved] = {"Aqk", "Akk", "k_precond", "ac_atk", "a_atk", "sa_atk",
                                            "w", "kg", "v_new", "h", "qg"};
  const size_t count = lean ? kKept : kSaved;
  TORCH_CHECK(got.size() == count, "the PKDA forward produced ", got.size(), " intermediates where ", count,
              " are promised");
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3), N = (T + 63) / 64;
  const int64_t pairs[] = {B, T, H, 64}, keys[] = {B, T, H, K}, values[] = {B, T, H, V}, chunk_keys[] = {B, N, H, K},
                chunk_heads[] = {B, N, H}, states[] = {B, N, H, K, V};
  const at::IntArrayRef shapes[kSaved] = {pairs, pairs, keys, chunk_keys, chunk_keys, chunk_heads,
                                          keys, keys, values, states, keys};
  for (size_t i = 0; i < count; ++i) {
    const Tensor& t = got[i];
    const at::ScalarType dtype = i >= 3 && i <= 5 ? at::kFloat : q.scalar_type();
    TORCH_CHECK(t.defined(), "PKDA intermediate ", names[i], ": missing from the forward's list");
    TORCH_CHECK(t.sizes() == shapes[i] && t.scalar_type() == dtype && t.device() == q.device() && t.is_contiguous(),
                "PKDA intermediate ", names[i], ": forward produced ", t.sizes(), " ", t.scalar_type(), " on ",
                t.device(), t.is_contiguous() ? "" : ", not contiguous", "; the fake implementation promises ",
                shapes[i], " ", dtype, " on ", q.device(), ", contiguous");
  }
}

struct Forward {
  Tensor o, S, A;
  std::vector<Tensor> saved;
};

Forward chunk_forward(const Inputs& in, bool final_state) {
  Problem P(in);
  c10::cuda::CUDAGuard guard(P.dev);
  Forward r;
  r.saved.reserve(kSaved);
  alloc_saved(P, r.saved, 0, kSaved);
  r.o = empty(in.q.sizes(), P.dev, P.act);
  pkda_chunk_fwd_args a{};
  a.p = P.p;
  a.o = r.o.data_ptr();
  if (final_state) {
    r.S = empty({P.N, P.H, P.D, P.D}, P.dev, at::kFloat);
    r.A = empty({P.N, P.H, P.D}, P.dev, at::kFloat);
    a.final_state = r.S.data_ptr<float>();
    a.final_A_state = r.A.data_ptr<float>();
  }
  a.Aqk = r.saved[0].data_ptr(); a.Akk = r.saved[1].data_ptr(); a.k_precond = r.saved[2].data_ptr();
  a.ac_atk = r.saved[3].data_ptr<float>(); a.a_atk = r.saved[4].data_ptr<float>(); a.sa_atk = r.saved[5].data_ptr<float>();
  a.w = r.saved[6].data_ptr(); a.kg = r.saved[7].data_ptr(); a.v_new = r.saved[8].data_ptr();
  a.h = r.saved[9].data_ptr(); a.qg = r.saved[10].data_ptr();
  a.workspace_bytes = pkda_chunk_fwd_workspace_bytes(&P.p);
  Tensor ws = scratch(a.workspace_bytes, P.dev);
  a.workspace = ws.data_ptr();
  finish(pkda_chunk_fwd(&a, stream()), "pkda_chunk_fwd");
  track_status(g_fwd_status, ws, pkda_chunk_fwd_status_offset(&P.p));
  return r;
}

// `save`: also leave what the exact backward needs (one byte tensor in `saved`).
Forward recurrent_forward(const Inputs& in, bool final_state, bool inplace, bool save = false) {
  Problem P(in);
  c10::cuda::CUDAGuard guard(P.dev);
  Forward r;
  r.o = empty(in.q.sizes(), P.dev, P.act);
  pkda_recurrent_args a{};
  a.p = P.p;
  a.o = r.o.data_ptr();
  if (final_state) {
    if (inplace) {
      for (const OptTensor* t : {&in.S0, &in.A0})
        TORCH_CHECK(*t && (*t)->scalar_type() == at::kFloat && (*t)->is_contiguous(),
                    "in-place decode needs contiguous fp32 initial states");
      r.S = *in.S0;
      r.A = *in.A0;
    } else {
      r.S = empty({P.N, P.H, P.D, P.D}, P.dev, at::kFloat);
      r.A = empty({P.N, P.H, P.D}, P.dev, at::kFloat);
    }
    a.final_state = r.S.data_ptr<float>();
    a.final_A_state = r.A.data_ptr<float>();
  }
  if (save) {
    r.saved.push_back(scratch(pkda_recurrent_saved_bytes(&P.p), P.dev));
    finish(pkda_recurrent_fwd_saving(&a, r.saved[0].data_ptr(), (size_t)r.saved[0].numel(), stream()),
           "pkda_recurrent_fwd_saving");
  } else {
    finish(pkda_recurrent_fwd(&a, stream()), "pkda_recurrent_fwd");
  }
  return r;
}

// Ten gradients (dq, dk, dv, dg, dg_atk, dbeta_atk, dbeta, dA_log, ddt_bias, dlog_atk_scale), then the
// two state gradients when `want_state`; shared layout of both backwards' argument structs.
template <typename Args>
std::vector<Tensor> alloc_grads(const Problem& P, Args& a, bool want_state) {
  std::vector<Tensor> g;
  g.reserve(12);
  for (int i = 0; i < 4; ++i) g.push_back(empty({P.B, P.T, P.H, P.D}, P.dev, P.act));
  g.push_back(empty({P.B, P.T, P.H}, P.dev, at::kFloat));
  for (int i = 0; i < 2; ++i) g.push_back(empty({P.B, P.T, P.H}, P.dev, P.act));
  g.push_back(empty({P.H}, P.dev, at::kFloat));
  g.push_back(empty({P.H * P.D}, P.dev, at::kFloat));
  g.push_back(empty({P.H}, P.dev, at::kFloat));
  a.dq = g[0].data_ptr(); a.dk = g[1].data_ptr(); a.dv = g[2].data_ptr(); a.dg = g[3].data_ptr();
  a.dg_atk = g[4].data_ptr<float>();
  a.dbeta_atk = g[5].data_ptr(); a.dbeta = g[6].data_ptr();
  a.dA_log = g[7].data_ptr<float>(); a.ddt_bias = g[8].data_ptr<float>(); a.dlog_atk_scale = g[9].data_ptr<float>();
  if (want_state) {
    g.push_back(empty({P.N, P.H, P.D, P.D}, P.dev, at::kFloat));
    g.push_back(empty({P.N, P.H, P.D}, P.dev, at::kFloat));
    a.d_initial_state = g[10].data_ptr<float>();
    a.d_initial_A_state = g[11].data_ptr<float>();
  }
  return g;
}

// Cotangent of the output (zero where autograd has none) and of the final state.
template <typename Args>
void cotangents(Problem& P, Args& a, const Tensor& d_o, const OptTensor& dS) {
  DeviceCheck check;
  check.dev = P.dev;
  check.seen = true;
  check(d_o);
  check(dS);
  if (d_o.defined()) {
    a.d_o = P.keep.as(d_o, P.act);
  } else {
    P.keep.held.push_back(at::zeros({P.B, P.T, P.H, P.D}, at::TensorOptions().device(P.dev).dtype(P.act)));
    a.d_o = P.keep.held.back().const_data_ptr();
  }
  if (dS && dS->defined()) a.d_final_state = static_cast<const float*>(P.keep.as(*dS, at::kFloat));
}

// `saved` holds the six always-kept intermediates and, unless `lean`, the five retained ones.
std::vector<Tensor> chunk_backward(const Inputs& in, std::vector<Tensor> saved, const Tensor& d_o, const OptTensor& dS,
                                   bool lean, bool want_state) {
  Problem P(in);
  c10::cuda::CUDAGuard guard(P.dev);
  if (lean) {
    saved.resize(kKept);
    alloc_saved(P, saved, kKept, kSaved);
  }
  TORCH_CHECK(saved.size() == kSaved, "PKDA backward got ", saved.size(), " intermediates, not ", kSaved);
  pkda_chunk_bwd_args a{};
  a.p = P.p;
  cotangents(P, a, d_o, dS);
  a.recompute = lean;
  a.Aqk = saved[0].data_ptr(); a.Akk = saved[1].data_ptr(); a.k_precond = saved[2].data_ptr();
  a.ac_atk = saved[3].data_ptr<float>(); a.a_atk = saved[4].data_ptr<float>(); a.sa_atk = saved[5].data_ptr<float>();
  a.w = saved[6].data_ptr(); a.kg = saved[7].data_ptr(); a.v_new = saved[8].data_ptr();
  a.h = saved[9].data_ptr(); a.qg = saved[10].data_ptr();
  std::vector<Tensor> grads = alloc_grads(P, a, want_state);
  a.workspace_bytes = pkda_chunk_bwd_workspace_bytes(&P.p);
  Tensor ws = scratch(a.workspace_bytes, P.dev);
  a.workspace = ws.data_ptr();
  finish(pkda_chunk_bwd(&a, stream()), "pkda_chunk_bwd");
  track_status(g_bwd_status, ws, pkda_chunk_bwd_status_offset(&P.p));
  return grads;
}

// Exact backward of the recurrence: any supported head width.  `saved`: what a saving forward left, or
// undefined (the forward runs again).
std::vector<Tensor> recurrent_backward(const Inputs& in, const Tensor& d_o, const OptTensor& dS, bool want_state,
                                       const Tensor& saved = Tensor()) {
  Problem P(in);
  c10::cuda::CUDAGuard guard(P.dev);
  pkda_recurrent_bwd_args a{};
  a.p = P.p;
  cotangents(P, a, d_o, dS);
  std::vector<Tensor> grads = alloc_grads(P, a, want_state);
  a.workspace_bytes = saved.defined() ? pkda_recurrent_bwd_saved_workspace_bytes(&P.p)
                                      : pkda_recurrent_bwd_workspace_bytes(&P.p);
  Tensor ws = scratch(a.workspace_bytes, P.dev);
  a.workspace = ws.data_ptr();
  if (saved.defined())
    finish(pkda_recurrent_bwd_saved(&a, saved.const_data_ptr(), (size_t)saved.numel(), stream()),
           "pkda_recurrent_bwd_saved");
  else
    finish(pkda_recurrent_bwd(&a, stream()), "pkda_recurrent_bwd");
  return grads;
}

// bf16 activations of 128-channel heads take the chunked kernels, everything else the exact ones.
bool chunk_capable(const Tensor& q) { return q.scalar_type() == at::kBFloat16 && q.size(-1) == 128; }

// ------------------------------------- recurrence with states / packing (no dispatcher name)
OptTensor some(Tensor t) { return t.defined() ? OptTensor(std::move(t)) : std::nullopt; }

struct StatefulRecurrence : torch::autograd::Function<StatefulRecurrence> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g,
                               const Tensor& g_atk, const Tensor& beta_atk, const Tensor& beta, const Tensor& A_log,
                               const Tensor& dt_bias, const Tensor& log_atk_scale, const OptTensor& S0,
                               const OptTensor& A0, const OptTensor& cu, double scale, double x, double eps,
                               bool final_state, bool lean) {
    const Inputs in{q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, S0, A0, cu, scale, x, eps};
    const bool chunked = chunk_capable(q);
    Forward f = chunked ? chunk_forward(in, final_state) : recurrent_forward(in, final_state, false, !lean);
    if (lean && chunked) f.saved.resize(kKept);
    variable_list keep{q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale,
                       S0.value_or(Tensor()), A0.value_or(Tensor()), cu.value_or(Tensor())};
    keep.insert(keep.end(), f.saved.begin(), f.saved.end());
    ctx->save_for_backward(std::move(keep));
    ctx->set_materialize_grads(false);
    ctx->saved_data["conf"] = c10::IValue(std::vector<double>{scale, x, eps, lean ? 1.0 : 0.0});
    if (!final_state) return {f.o};
    ctx->mark_non_differentiable({f.A});
    return {f.o, f.S, f.A};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list t = ctx->get_saved_variables();
    const std::vector<double> conf = ctx->saved_data["conf"].toDoubleVector();
    const OptTensor S0 = some(t[10]), A0 = some(t[11]), cu = some(t[12]);
    const OptTensor dS = grads.size() > 1 ? some(grads[1]) : std::nullopt;
    const Inputs in{t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], S0, A0, cu, conf[0], conf[1], conf[2]};
    const bool want = S0 || A0;
    std::vector<Tensor> got =
        chunk_capable(t[0])
            ? chunk_backward(in, std::vector<Tensor>(t.begin() + 13, t.end()), grads[0], dS, conf[3] != 0.0, want)
            : recurrent_backward(in, grads[0], dS, want, t.size() > 13 ? t[13] : Tensor());
    variable_list out(18);
    for (int i = 0; i < 10; ++i) out[i] = like_input(std::move(got[i]), t[i]);
    if (S0) out[10] = std::move(got[10]);
    if (A0) out[11] = std::move(got[11]);
    return out;
  }
};

// ------------------------------------------- operator delta_feedback::pkda_recurrence
std::tuple<Tensor, std::vector<Tensor>> recurrence_cuda(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& g_atk, const Tensor& beta_atk,
    const Tensor& beta, const Tensor& A_log, const Tensor& dt_bias, const Tensor& log_atk_scale, double scale,
    double squash_x, double squash_eps, bool lean) {
  const Inputs in{q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, kNone, kNone, kNone,
                  scale, squash_x, squash_eps};
  Forward f;
  if (chunk_capable(q)) {
    f = chunk_forward(in, false);
    if (lean) f.saved.resize(kKept);
  } else {
    // The exact backward needs none of the intermediates; the list only keeps the operator's
    // output contract (names, shapes, dtypes), so it is left unwritten.
    f = recurrent_forward(in, false, false);
    Problem P(in);
    alloc_saved(P, f.saved, 0, lean ? kKept : kSaved);
  }
  check_intermediates(f.saved, q, v, lean);
  return {std::move(f.o), std::move(f.saved)};
}

std::vector<Tensor> recurrence_backward_cuda(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& g_atk, const Tensor& beta_atk,
    const Tensor& beta, const Tensor& A_log, const Tensor& dt_bias, const Tensor& log_atk_scale,
    at::TensorList saved, const Tensor& d_o, double scale, double squash_x, double squash_eps,
    std::optional<at::ScalarType> /*autocast_dtype: the kernels fix their own arithmetic*/, bool lean) {
  const size_t expected = lean ? kKept : kSaved;
  TORCH_CHECK(saved.size() == expected, "PKDA backward received ", saved.size(), " intermediates, not ", expected);
  const Inputs in{q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, kNone, kNone, kNone,
                  scale, squash_x, squash_eps};
  std::vector<Tensor> got = chunk_capable(q) ? chunk_backward(in, saved.vec(), d_o, std::nullopt, lean, false)
                                             : recurrent_backward(in, d_o, std::nullopt, false);
  const Tensor* inputs[10] = {&q, &k, &v, &g, &g_atk, &beta_atk, &beta, &A_log, &dt_bias, &log_atk_scale};
  for (int i = 0; i < 10; ++i) got[i] = like_input(std::move(got[i]), *inputs[i]);
  return got;
}

template <typename F>
auto typed_op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<F>();
}

// A backward's call of its operator.  Where no graph is recorded (an ordinary backward) the operator's autograd
// kernel has nothing to do and is passed by.  (Called behind get_saved_variables: unpacking may run the forward
// again, which must not be below autograd.)
template <typename Op, typename... A>
auto call_backward(const Op& op, A&&... args) {
  if (at::GradMode::is_enabled()) return op.call(std::forward<A>(args)...);
  at::AutoDispatchBelowADInplaceOrView below;
  return op.call(std::forward<A>(args)...);
}

// The backward operators have no derivative of their own.  Where one could be asked for (a graph is being
// recorded, create_graph = True), their results hang on a node that raises: without it they would come out as
// constants and a second derivative would silently be missing.
struct NotTwice : torch::autograd::Function<NotTwice> {
  static variable_list forward(AutogradContext* ctx, at::TensorList, const std::function<variable_list()>& run,
                               const char* name) {
    ctx->saved_data["name"] = std::string(name);
    return run();
  }
  static variable_list backward(AutogradContext* ctx, variable_list) {
    TORCH_CHECK(false, ctx->saved_data["name"].toStringRef(), " has no derivative: the PKDA operators are differentiable once");
  }
};

// `run` calls the operator again, below autograd; `inputs` are its tensor arguments.
variable_list once_differentiable(const char* name, at::TensorList inputs, const std::function<variable_list()>& run) {
  at::AutoDispatchBelowADInplaceOrView below;
  if (at::GradMode::is_enabled())
    for (const Tensor& t : inputs)
      if (t.requires_grad()) return NotTwice::apply(inputs, run, name);
  return run();
}

using RecurrenceSig = std::tuple<Tensor, std::vector<Tensor>>(
    const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
    const Tensor&, const Tensor&, const Tensor&, double, double, double, bool);
using RecurrenceBackwardSig = std::vector<Tensor>(
    const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
    const Tensor&, const Tensor&, const Tensor&, at::TensorList, const Tensor&, double, double, double,
    std::optional<at::ScalarType>, bool);

struct Recurrence : torch::autograd::Function<Recurrence> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g,
                               const Tensor& g_atk, const Tensor& beta_atk, const Tensor& beta, const Tensor& A_log,
                               const Tensor& dt_bias, const Tensor& log_atk_scale, double scale, double x, double eps,
                               bool lean) {
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = typed_op<RecurrenceSig>("delta_feedback::pkda_recurrence");
    auto [o, saved] = op.call(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale, x, eps, lean);
    variable_list keep{q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale};
    keep.insert(keep.end(), saved.begin(), saved.end());
    ctx->save_for_backward(std::move(keep));
    // No cotangent ever comes for the intermediates: leaving the gradients of the outputs undefined
    // instead of zero-filled saves one fill kernel per intermediate in every backward.
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable(saved);
    ctx->saved_data["conf"] = c10::IValue(std::vector<double>{scale, x, eps, lean ? 1.0 : 0.0});
    if (at::autocast::is_autocast_enabled(at::kCUDA))
      ctx->saved_data["autocast"] = c10::IValue((int64_t)at::autocast::get_autocast_dtype(at::kCUDA));
    variable_list out{o};
    out.insert(out.end(), saved.begin(), saved.end());
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    static const auto op = typed_op<RecurrenceBackwardSig>("delta_feedback::pkda_recurrence_backward");
    variable_list t = ctx->get_saved_variables();  // unpacked exactly once (checkpoint replays allow no more)
    const std::vector<double> conf = ctx->saved_data["conf"].toDoubleVector();
    std::optional<at::ScalarType> autocast;
    const auto it = ctx->saved_data.find("autocast");
    if (it != ctx->saved_data.end()) autocast = (at::ScalarType)it->second.toInt();
    const Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(t[0], at::MemoryFormat::Contiguous);
    std::vector<Tensor> got = call_backward(op, t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9],
                                            at::TensorList(t).slice(10), d_o, conf[0], conf[1], conf[2], autocast,
                                            conf[3] != 0.0);
    variable_list out(14);
    std::move(got.begin(), got.end(), out.begin());
    return out;
  }
};

std::tuple<Tensor, std::vector<Tensor>> recurrence_autograd(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& g_atk, const Tensor& beta_atk,
    const Tensor& beta, const Tensor& A_log, const Tensor& dt_bias, const Tensor& log_atk_scale, double scale,
    double squash_x, double squash_eps, bool lean) {
  variable_list r = Recurrence::apply(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, scale,
                                      squash_x, squash_eps, lean);
  Tensor o = std::move(r[0]);
  r.erase(r.begin());
  return {std::move(o), std::move(r)};
}

std::vector<Tensor> recurrence_backward_autograd(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& g_atk, const Tensor& beta_atk,
    const Tensor& beta, const Tensor& A_log, const Tensor& dt_bias, const Tensor& log_atk_scale,
    at::TensorList saved, const Tensor& d_o, double scale, double squash_x, double squash_eps,
    std::optional<at::ScalarType> autocast_dtype, bool lean) {
  constexpr const char* name = "delta_feedback::pkda_recurrence_backward";
  static const auto op = typed_op<RecurrenceBackwardSig>(name);
  variable_list in{q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, d_o};
  in.insert(in.end(), saved.begin(), saved.end());
  return once_differentiable(name, in, [&]() -> variable_list {
    return op.call(q, k, v, g, g_atk, beta_atk, beta, A_log, dt_bias, log_atk_scale, saved, d_o, scale, squash_x,
                   squash_eps, autocast_dtype, lean);
  });
}

// ---------------------------------------------- operator delta_feedback::pkda_qkv_conv
pkda_qkv_conv_args conv_args(const Tensor& x, const Tensor& weight, int64_t head_dim, int64_t norm_channels,
                             double eps) {
  TORCH_CHECK(x.dim() == 3 && weight.dim() == 2 && weight.size(0) == x.size(-1) && x.size(-1) % 3 == 0,
              "pkda_qkv_conv expects x [B,T,3W] and weight [3W,taps]");
  pkda_qkv_conv_args a{};
  a.batch = (int)x.size(0); a.seq_len = (int)x.size(1); a.channels = (int)x.size(2);
  a.taps = (int)weight.size(1);
  a.head_dim = (int)head_dim; a.norm_channels = (int)norm_channels; a.eps = (float)eps;
  a.dtype = act_code(x, "PKDA layer operators take bf16 or fp32 activations, got ");
  return a;
}

std::tuple<Tensor, Tensor, Tensor> conv_cuda(const Tensor& x, const Tensor& weight, int64_t head_dim,
                                             int64_t norm_channels, double eps) {
  const c10::Device dev = one_device(x, weight);
  c10::cuda::CUDAGuard guard(dev);
  pkda_qkv_conv_args a = conv_args(x, weight, head_dim, norm_channels, eps);
  Keep keep;
  a.x = keep.as(x, x.scalar_type());
  a.weight = static_cast<const float*>(keep.as(weight, at::kFloat));
  Tensor out[3];
  for (Tensor& t : out) t = empty({x.size(0), x.size(1), x.size(2) / 3}, dev, x.scalar_type());
  a.q = out[0].data_ptr(); a.k = out[1].data_ptr(); a.v = out[2].data_ptr();
  finish(pkda_qkv_conv_fwd(&a, stream()), "pkda_qkv_conv_fwd");
  return {out[0], out[1], out[2]};
}

std::tuple<Tensor, Tensor> conv_backward_cuda(const Tensor& x, const Tensor& weight, const Tensor& dq,
                                              const Tensor& dk, const Tensor& dv, int64_t head_dim,
                                              int64_t norm_channels, double eps) {
  const c10::Device dev = one_device(x, weight, dq, dk, dv);
  c10::cuda::CUDAGuard guard(dev);
  pkda_qkv_conv_args a = conv_args(x, weight, head_dim, norm_channels, eps);
  const at::ScalarType act = x.scalar_type();
  Keep keep;
  a.x = keep.as(x, act);
  a.weight = static_cast<const float*>(keep.as(weight, at::kFloat));
  a.dq = keep.as(dq, act); a.dk = keep.as(dk, act); a.dv = keep.as(dv, act);
  Tensor dx = empty(x.sizes(), dev, act), dw = empty(weight.sizes(), dev, at::kFloat);
  a.dx = dx.data_ptr();
  a.dweight = dw.data_ptr<float>();
  a.workspace_bytes = pkda_qkv_conv_bwd_workspace_bytes(&a);
  Tensor ws = scratch(a.workspace_bytes, dev);
  a.workspace = ws.data_ptr();
  finish(pkda_qkv_conv_bwd(&a, stream()), "pkda_qkv_conv_bwd");
  return {dx, like_input(dw, weight)};
}

Tensor zeros_if_undefined(const Tensor& g, const Tensor& like) {
  return g.defined() ? g : at::zeros_like(like, at::MemoryFormat::Contiguous);
}

using ConvSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, SymInt, SymInt, double);
using ConvBackwardSig = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                   const Tensor&, SymInt, SymInt, double);

struct Conv : torch::autograd::Function<Conv> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, SymInt head_dim,
                               SymInt norm_channels, double eps) {
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = typed_op<ConvSig>("delta_feedback::pkda_qkv_conv");
    auto [q, k, v] = op.call(x, weight, head_dim, norm_channels, eps);
    ctx->save_for_backward({x, weight});
    ctx->saved_data["head_dim"] = head_dim;
    ctx->saved_data["norm_channels"] = norm_channels;
    ctx->saved_data["eps"] = eps;
    return {q, k, v};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    static const auto op = typed_op<ConvBackwardSig>("delta_feedback::pkda_qkv_conv_backward");
    variable_list t = ctx->get_saved_variables();
    auto [dx, dw] = call_backward(op, t[0], t[1], grads[0], grads[1], grads[2], ctx->saved_data["head_dim"].toSymInt(),
                                  ctx->saved_data["norm_channels"].toSymInt(), ctx->saved_data["eps"].toDouble());
    return {dx, dw, Tensor(), Tensor(), Tensor()};
  }
};

std::tuple<Tensor, Tensor, Tensor> conv_autograd(const Tensor& x, const Tensor& weight, SymInt head_dim,
                                                 SymInt norm_channels, double eps) {
  variable_list r = Conv::apply(x, weight, std::move(head_dim), std::move(norm_channels), eps);
  return {r[0], r[1], r[2]};
}

std::tuple<Tensor, Tensor> conv_backward_autograd(const Tensor& x, const Tensor& weight, const Tensor& dq,
                                                  const Tensor& dk, const Tensor& dv, SymInt head_dim,
                                                  SymInt norm_channels, double eps) {
  constexpr const char* name = "delta_feedback::pkda_qkv_conv_backward";
  static const auto op = typed_op<ConvBackwardSig>(name);
  variable_list r = once_differentiable(name, {x, weight, dq, dk, dv}, [&]() -> variable_list {
    auto [dx, dw] = op.call(x, weight, dq, dk, dv, head_dim, norm_channels, eps);
    return {dx, dw};
  });
  return {r[0], r[1]};
}

// --------------------------------------------- operator delta_feedback::pkda_norm_gate
pkda_norm_gate_args norm_gate_args(const Tensor& x, const Tensor& gate, const Tensor& weight, double eps) {
  TORCH_CHECK(gate.sizes() == x.sizes() && weight.dim() == 1 && weight.size(0) == x.size(-1) && weight.size(0) > 0,
              "pkda_norm_gate expects x, gate [..., D] and weight [D]");
  pkda_norm_gate_args a{};
  a.dim = (int)x.size(-1);
  a.rows = x.numel() / x.size(-1);
  a.dtype = act_code(x, "PKDA layer operators take bf16 or fp32 activations, got ");
  a.eps = (float)eps;
  return a;
}

std::tuple<Tensor, Tensor> norm_gate_cuda(const Tensor& x, const Tensor& gate, const Tensor& weight, double eps) {
  const c10::Device dev = one_device(x, gate, weight);
  c10::cuda::CUDAGuard guard(dev);
  pkda_norm_gate_args a = norm_gate_args(x, gate, weight, eps);
  Keep keep;
  a.x = keep.as(x, x.scalar_type());
  a.gate = keep.as(gate, x.scalar_type());
  a.weight = static_cast<const float*>(keep.as(weight, at::kFloat));
  Tensor y = empty(x.sizes(), dev, x.scalar_type()), rstd = empty({(int64_t)a.rows}, dev, at::kFloat);
  a.y = y.data_ptr();
  a.rstd = rstd.data_ptr<float>();
  finish(pkda_norm_gate_fwd(&a, stream()), "pkda_norm_gate_fwd");
  return {y, rstd};
}

std::tuple<Tensor, Tensor, Tensor> norm_gate_backward_cuda(const Tensor& x, const Tensor& gate, const Tensor& weight,
                                                           const Tensor& rstd, const Tensor& dy, double eps) {
  const c10::Device dev = one_device(x, gate, weight, rstd, dy);
  c10::cuda::CUDAGuard guard(dev);
  pkda_norm_gate_args a = norm_gate_args(x, gate, weight, eps);
  const at::ScalarType act = x.scalar_type();
  Keep keep;
  a.x = keep.as(x, act);
  a.gate = keep.as(gate, act);
  a.weight = static_cast<const float*>(keep.as(weight, at::kFloat));
  a.rstd = static_cast<float*>(const_cast<void*>(keep.as(rstd, at::kFloat)));
  a.dy = keep.as(dy, act);
  Tensor dx = empty(x.sizes(), dev, act), dg = empty(x.sizes(), dev, act), dw = empty(weight.sizes(), dev, at::kFloat);
  a.dx = dx.data_ptr();
  a.dgate = dg.data_ptr();
  a.dweight = dw.data_ptr<float>();
  a.workspace_bytes = pkda_norm_gate_bwd_workspace_bytes(&a);
  Tensor ws = scratch(a.workspace_bytes, dev);
  a.workspace = ws.data_ptr();
  finish(pkda_norm_gate_bwd(&a, stream()), "pkda_norm_gate_bwd");
  return {dx, like_input(dg, gate), like_input(dw, weight)};
}

using NormGateSig = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, double);
using NormGateBackwardSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&,
                                                               const Tensor&, const Tensor&, double);

struct NormGate : torch::autograd::Function<NormGate> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& weight,
                               double eps) {
    at::AutoDispatchBelowADInplaceOrView below;
    static const auto op = typed_op<NormGateSig>("delta_feedback::pkda_norm_gate");
    auto [y, rstd] = op.call(x, gate, weight, eps);
    ctx->save_for_backward({x, gate, weight, rstd});
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({rstd});
    ctx->saved_data["eps"] = eps;
    return {y, rstd};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    static const auto op = typed_op<NormGateBackwardSig>("delta_feedback::pkda_norm_gate_backward");
    variable_list t = ctx->get_saved_variables();
    auto [dx, dg, dw] = call_backward(op, t[0], t[1], t[2], t[3], zeros_if_undefined(grads[0], t[0]),
                                      ctx->saved_data["eps"].toDouble());
    return {dx, dg, dw, Tensor()};
  }
};

std::tuple<Tensor, Tensor> norm_gate_autograd(const Tensor& x, const Tensor& gate, const Tensor& weight, double eps) {
  variable_list r = NormGate::apply(x, gate, weight, eps);
  return {r[0], r[1]};
}

std::tuple<Tensor, Tensor, Tensor> norm_gate_backward_autograd(const Tensor& x, const Tensor& gate,
                                                               const Tensor& weight, const Tensor& rstd,
                                                               const Tensor& dy, double eps) {
  constexpr const char* name = "delta_feedback::pkda_norm_gate_backward";
  static const auto op = typed_op<NormGateBackwardSig>(name);
  variable_list r = once_differentiable(name, {x, gate, weight, rstd, dy}, [&]() -> variable_list {
    auto [dx, dg, dw] = op.call(x, gate, weight, rstd, dy, eps);
    return {dx, dg, dw};
  });
  return {r[0], r[1], r[2]};
}

// ------------------------------------------------------------------ control epilogue
pkda_controls_args controls_args(const Tensor& packed, const Tensor& A_log_precond, int64_t hidden) {
  const int64_t H = A_log_precond.size(0), row = 2 * hidden + 3 * H;
  TORCH_CHECK(packed.size(-1) == row && row > 0, "packed control row must be [hidden | H | H | H | hidden]");
  pkda_controls_args a{};
  a.rows = packed.numel() / row;
  a.heads = (int)H;
  a.hidden = (int)hidden;
  a.dtype = act_code(packed, "PKDA layer operators take bf16 or fp32 activations, got ");
  return a;
}

// Split of the packed control projection with the three per-head activations fused in (forward) and
// the packed gradient written in one pass (backward).
struct Controls : torch::autograd::Function<Controls> {
  static variable_list forward(AutogradContext* ctx, const Tensor& packed_in, const Tensor& A_log_precond,
                               const Tensor& dt_bias_precond, int64_t hidden) {
    const c10::Device dev = one_device(packed_in, A_log_precond, dt_bias_precond);
    c10::cuda::CUDAGuard guard(dev);
    const Tensor packed = packed_in.contiguous();
    pkda_controls_args a = controls_args(packed, A_log_precond, hidden);
    const int64_t H = a.heads;
    Keep keep;
    a.packed = packed.const_data_ptr();
    a.A_log_precond = static_cast<const float*>(keep.as(A_log_precond, at::kFloat));
    a.dt_bias_precond = static_cast<const float*>(keep.as(dt_bias_precond, at::kFloat));
    std::vector<int64_t> shape = packed.sizes().vec();
    shape.back() = H;
    Tensor beta = empty(shape, dev, packed.scalar_type()), beta_atk = empty(shape, dev, packed.scalar_type());
    Tensor g_atk = empty(shape, dev, at::kFloat);
    a.beta = beta.data_ptr();
    a.g_atk = g_atk.data_ptr<float>();
    a.beta_atk = beta_atk.data_ptr();
    finish(pkda_controls_fwd(&a, stream()), "pkda_controls_fwd");
    ctx->save_for_backward({packed, A_log_precond, dt_bias_precond});
    ctx->set_materialize_grads(false);
    ctx->saved_data["hidden"] = hidden;
    return {packed.narrow(-1, 0, hidden), beta, g_atk, beta_atk, packed.narrow(-1, hidden + 3 * H, hidden)};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list t = ctx->get_saved_variables();  // unpacked exactly once (checkpoint replays allow no more)
    const Tensor &packed = t[0], &A_log = t[1], &dt_bias = t[2];
    const c10::Device dev = packed.device();
    c10::cuda::CUDAGuard guard(dev);
    const at::ScalarType act = packed.scalar_type();
    pkda_controls_args a = controls_args(packed, A_log, ctx->saved_data["hidden"].toInt());
    Keep keep;
    a.packed = packed.const_data_ptr();
    a.A_log_precond = static_cast<const float*>(keep.as(A_log, at::kFloat));
    a.dt_bias_precond = static_cast<const float*>(keep.as(dt_bias, at::kFloat));
    const void* in[5];
    for (int i = 0; i < 5; ++i) in[i] = grads[i].defined() ? keep.as(grads[i], i == 2 ? at::kFloat : act) : nullptr;
    a.d_decay_hidden = in[0];
    a.d_beta = in[1];
    a.d_g_atk = static_cast<const float*>(in[2]);
    a.d_beta_atk = in[3];
    a.d_gate_hidden = in[4];
    Tensor d_packed = empty(packed.sizes(), dev, act);
    Tensor dA = empty(A_log.sizes(), dev, at::kFloat), db = empty(dt_bias.sizes(), dev, at::kFloat);
    a.d_packed = d_packed.data_ptr();
    a.dA_log_precond = dA.data_ptr<float>();
    a.ddt_bias_precond = db.data_ptr<float>();
    a.workspace_bytes = pkda_controls_bwd_workspace_bytes(&a);
    Tensor ws = scratch(a.workspace_bytes, dev);
    a.workspace = ws.data_ptr();
    finish(pkda_controls_bwd(&a, stream()), "pkda_controls_bwd");
    return {d_packed, like_input(dA, A_log), like_input(db, dt_bias), Tensor()};
  }
};

// ----------------------------------------------------------------------- decode step
struct DecodeInputs {
  const Tensor &qkv, &conv_q, &conv_k, &conv_v, &conv_weight, &g, &g_atk, &beta_atk, &beta, &A_log, &dt_bias,
      &log_atk_scale, &state, &a_state;
  const OptTensor &gate, &norm_weight;
  int64_t head_dim;
  std::optional<double> scale;
  double squash_x, squash_eps, qk_eps, norm_eps;
};

Tensor decode_step(const DecodeInputs& in) {
  const c10::Device dev = one_device(in.qkv, in.conv_weight, in.g, in.g_atk, in.beta_atk, in.beta, in.state,
                                     in.a_state, in.conv_q, in.conv_k, in.conv_v, in.A_log, in.dt_bias,
                                     in.log_atk_scale, in.gate, in.norm_weight);
  c10::cuda::CUDAGuard guard(dev);
  TORCH_CHECK(in.qkv.dim() == 2 && in.conv_weight.dim() == 2 && in.head_dim > 0,
              "pkda_decode_step expects qkv [B,3W] and conv_weight [3W,taps]");
  const int64_t B = in.qkv.size(0), W = in.qkv.size(1) / 3, H = W / in.head_dim, taps = in.conv_weight.size(1);
  const at::ScalarType act = in.qkv.scalar_type();
  bool plain = in.state.scalar_type() == at::kFloat && in.a_state.scalar_type() == at::kFloat;
  for (const Tensor* c : {&in.state, &in.a_state, &in.conv_q, &in.conv_k, &in.conv_v}) plain = plain && c->is_contiguous();
  TORCH_CHECK(plain, "the decode cache (state, a_state fp32; conv histories) must be contiguous: it is updated in place");
  const int64_t hist[3] = {B, W, taps - 1};
  for (const Tensor* c : {&in.conv_q, &in.conv_k, &in.conv_v})
    TORCH_CHECK(c->scalar_type() == act && c->sizes() == at::IntArrayRef(hist, 3),
                "conv_state must be three [B, W, taps-1] tensors of the activation dtype");
  pkda_decode_step_args a{};
  a.batch = (int)B; a.heads = (int)H; a.head_dim = (int)in.head_dim; a.taps = (int)taps;
  a.dtype = act_code(in.qkv, "PKDA layer operators take bf16 or fp32 activations, got ");
  a.scale = (float)in.scale.value_or(std::pow((double)in.head_dim, -0.5));
  a.squash_x = (float)in.squash_x; a.squash_eps = (float)in.squash_eps;
  a.qk_eps = (float)in.qk_eps; a.norm_eps = (float)in.norm_eps;
  Keep keep;
  auto f32 = [&](const Tensor& t) { return static_cast<const float*>(keep.as(t, at::kFloat)); };
  a.qkv = keep.as(in.qkv, act);
  a.conv_weight = f32(in.conv_weight);
  a.g = keep.as(in.g, act);
  a.g_atk = f32(in.g_atk);
  a.beta_atk = keep.as(in.beta_atk, act);
  a.beta = keep.as(in.beta, act);
  a.A_log = f32(in.A_log); a.dt_bias = f32(in.dt_bias); a.log_atk_scale = f32(in.log_atk_scale);
  a.conv_q = in.conv_q.data_ptr(); a.conv_k = in.conv_k.data_ptr(); a.conv_v = in.conv_v.data_ptr();
  a.state = in.state.data_ptr<float>();
  a.a_state = in.a_state.data_ptr<float>();
  Tensor out = empty({B, H, in.head_dim}, dev, act);
  if (in.gate) {
    TORCH_CHECK(in.norm_weight, "the output gate needs the norm weight");
    a.gate = keep.as(*in.gate, act);
    a.norm_weight = f32(*in.norm_weight);
  }
  a.out = out.data_ptr();
  finish(pkda_decode_step(&a, stream()), "pkda_decode_step");
  return out;
}

TORCH_LIBRARY_FRAGMENT(delta_feedback, m) {
  const std::vector<at::Tag> tags{at::Tag::pt2_compliant_tag};
  m.def("pkda_recurrence(Tensor q, Tensor k, Tensor v, Tensor g, Tensor g_atk, Tensor beta_atk, Tensor beta, "
        "Tensor A_log, Tensor dt_bias, Tensor log_atk_scale, float scale, float squash_x, float squash_eps, bool lean) "
        "-> (Tensor, Tensor[])", tags);
  m.def("pkda_recurrence_backward(Tensor q, Tensor k, Tensor v, Tensor g, Tensor g_atk, Tensor beta_atk, Tensor beta, "
        "Tensor A_log, Tensor dt_bias, Tensor log_atk_scale, Tensor[] saved, Tensor do, float scale, float squash_x, "
        "float squash_eps, ScalarType? autocast_dtype, bool lean) -> Tensor[]", tags);
  m.def("pkda_qkv_conv(Tensor x, Tensor weight, SymInt head_dim, SymInt norm_channels, float eps) "
        "-> (Tensor, Tensor, Tensor)", tags);
  m.def("pkda_qkv_conv_backward(Tensor x, Tensor weight, Tensor dq, Tensor dk, Tensor dv, SymInt head_dim, "
        "SymInt norm_channels, float eps) -> (Tensor, Tensor)", tags);
  m.def("pkda_norm_gate(Tensor x, Tensor gate, Tensor weight, float eps) -> (Tensor, Tensor)", tags);
  m.def("pkda_norm_gate_backward(Tensor x, Tensor gate, Tensor weight, Tensor rstd, Tensor dy, float eps) "
        "-> (Tensor, Tensor, Tensor)", tags);
}

TORCH_LIBRARY_IMPL(delta_feedback, CUDA, m) {
  m.impl("pkda_recurrence", recurrence_cuda);
  m.impl("pkda_recurrence_backward", recurrence_backward_cuda);
  m.impl("pkda_qkv_conv", conv_cuda);
  m.impl("pkda_qkv_conv_backward", conv_backward_cuda);
  m.impl("pkda_norm_gate", norm_gate_cuda);
  m.impl("pkda_norm_gate_backward", norm_gate_backward_cuda);
}

TORCH_LIBRARY_IMPL(delta_feedback, Autograd, m) {
  m.impl("pkda_recurrence", recurrence_autograd);
  m.impl("pkda_recurrence_backward", recurrence_backward_autograd);
  m.impl("pkda_qkv_conv", conv_autograd);
  m.impl("pkda_qkv_conv_backward", conv_backward_autograd);
  m.impl("pkda_norm_gate", norm_gate_autograd);
  m.impl("pkda_norm_gate_backward", norm_gate_backward_autograd);
}

// ----------------------------------------------------------------- Python entry points
// Positional calls only (METH_FASTCALL); keyword handling and defaults live in the Python wrappers.
struct Args {
  PyObject* const* a;
  Py_ssize_t n;

  Args(PyObject* const* args, Py_ssize_t count, Py_ssize_t want, const char* who) : a(args), n(count) {
    if (n != want) throw torch::TypeError(c10::str(who, " takes ", want, " arguments, got ", n));
  }
  const Tensor& tensor(int i) const {
    if (!THPVariable_Check(a[i])) throw torch::TypeError(c10::str("argument ", i, " must be a Tensor, not ", Py_TYPE(a[i])->tp_name));
    return THPVariable_Unpack(a[i]);
  }
  // A sequence of tensors; None becomes an undefined one.
  std::vector<Tensor> tensors(int i) const {
    THPObjectPtr seq(PySequence_Fast(a[i], "expected a sequence of tensors"));
    if (!seq) throw python_error();
    std::vector<Tensor> list;
    for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(seq.get()); ++k) {
      PyObject* t = PySequence_Fast_GET_ITEM(seq.get(), k);
      if (t != Py_None && !THPVariable_Check(t)) throw torch::TypeError("expected a sequence of tensors");
      list.push_back(t == Py_None ? Tensor() : THPVariable_Unpack(t));
    }
    return list;
  }
  OptTensor opt(int i) const { return a[i] == Py_None ? std::nullopt : OptTensor(tensor(i)); }
  double num(int i) const {
    const double v = PyFloat_AsDouble(a[i]);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
  }
  std::optional<double> opt_num(int i) const { return a[i] == Py_None ? std::nullopt : std::optional<double>(num(i)); }
  int64_t whole(int i) const {
    const long long v = PyLong_AsLongLong(a[i]);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  bool flag(int i) const { return PyObject_IsTrue(a[i]) == 1; }
};

PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}

PyObject* wrap3(const Tensor& a, const Tensor& b, const Tensor& c) {
  PyObject* r = PyTuple_New(3);
  if (!r) throw python_error();
  PyTuple_SET_ITEM(r, 0, wrap(a));
  PyTuple_SET_ITEM(r, 1, wrap(b));
  PyTuple_SET_ITEM(r, 2, wrap(c));
  return r;
}

PyObject* wrap_list(const std::vector<Tensor>& v) {
  PyObject* r = PyList_New((Py_ssize_t)v.size());
  if (!r) throw python_error();
  for (size_t i = 0; i < v.size(); ++i) PyList_SET_ITEM(r, (Py_ssize_t)i, wrap(v[i]));
  return r;
}

// The sixteen leading arguments of every recurrence call: ten inputs, S0, A0, cu_seqlens, then
// scale (None: 1 / sqrt(D)), squash_x and squash_eps.
constexpr int kInputArgs = 16;
struct ParsedInputs {
  OptTensor S0, A0, cu;
  Inputs in;
  explicit ParsedInputs(const Args& A)
      : S0(A.opt(10)), A0(A.opt(11)), cu(A.opt(12)),
        in{A.tensor(0), A.tensor(1), A.tensor(2), A.tensor(3), A.tensor(4), A.tensor(5), A.tensor(6), A.tensor(7),
           A.tensor(8), A.tensor(9), S0, A0, cu, 0.0, A.num(14), A.num(15)} {
    const std::optional<double> s = A.opt_num(13);
    in.scale = s ? *s : std::pow((double)in.q.size(-1), -0.5);
  }
};

// Whether the call has to go through its autograd function: some input takes part in a recorded graph, or carries
// a forward-mode tangent (which that function refuses; past it the tangent would silently be dropped).
bool takes_autograd(const ParsedInputs& p) {
  const bool graph = at::GradMode::is_enabled();
  auto takes = [&](const Tensor& t) { return (graph && t.requires_grad()) || t._fw_grad(0).defined(); };
  for (const Tensor* t : {&p.in.q, &p.in.k, &p.in.v, &p.in.g, &p.in.g_atk, &p.in.beta_atk, &p.in.beta, &p.in.A_log,
                          &p.in.dt_bias, &p.in.log_atk_scale})
    if (takes(*t)) return true;
  return (p.S0 && takes(*p.S0)) || (p.A0 && takes(*p.A0));
}

// recurrence(<inputs>, output_final_state, lean) -> (o, S | None, A | None), differentiable
PyObject* py_recurrence(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, kInputArgs + 2, "recurrence");
  const ParsedInputs P(A);
  const bool final_state = A.flag(16), lean = A.flag(17);
  Tensor o, S, AT;
  {
    pybind11::gil_scoped_release no_gil;
    if (takes_autograd(P)) {
      variable_list r = StatefulRecurrence::apply(P.in.q, P.in.k, P.in.v, P.in.g, P.in.g_atk, P.in.beta_atk, P.in.beta,
                                                  P.in.A_log, P.in.dt_bias, P.in.log_atk_scale, P.S0, P.A0, P.cu,
                                                  P.in.scale, P.in.squash_x, P.in.squash_eps, final_state, lean);
      o = r[0];
      if (final_state) { S = r[1]; AT = r[2]; }
    } else {
      Forward f = chunk_capable(P.in.q) ? chunk_forward(P.in, final_state) : recurrent_forward(P.in, final_state, false);
      o = f.o; S = f.S; AT = f.A;
    }
  }
  return wrap3(o, S, AT);
  END_HANDLE_TH_ERRORS
}

// recurrent_forward(<inputs>, output_final_state, inplace_state) -> (o, S | None, A | None)
PyObject* py_recurrent_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, kInputArgs + 2, "recurrent_forward");
  const ParsedInputs P(A);
  const bool final_state = A.flag(16), inplace = A.flag(17);
  Forward f;
  {
    pybind11::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    f = recurrent_forward(P.in, final_state, inplace);
  }
  return wrap3(f.o, f.S, f.A);
  END_HANDLE_TH_ERRORS
}

// chunk_forward(<inputs>, output_final_state) -> (o, S | None, A | None, [eleven intermediates])
PyObject* py_chunk_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, kInputArgs + 1, "chunk_forward");
  const ParsedInputs P(A);
  const bool final_state = A.flag(16);
  Forward f;
  {
    pybind11::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    f = chunk_forward(P.in, final_state);
  }
  PyObject* r = PyTuple_New(4);
  if (!r) throw python_error();
  PyTuple_SET_ITEM(r, 0, wrap(f.o));
  PyTuple_SET_ITEM(r, 1, wrap(f.S));
  PyTuple_SET_ITEM(r, 2, wrap(f.A));
  PyTuple_SET_ITEM(r, 3, wrap_list(f.saved));
  return r;
  END_HANDLE_TH_ERRORS
}

// backward(<inputs>, saved | None, do, dS | None, lean, want_state_grads) -> [gradients]; without
// `saved` the exact kernels run.
PyObject* py_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, kInputArgs + 5, "backward");
  const ParsedInputs P(A);
  const bool exact = A.a[16] == Py_None;
  std::vector<Tensor> saved;
  if (!exact) saved = A.tensors(16);
  for (const Tensor& t : saved)
    if (!t.defined()) throw torch::TypeError("saved must hold tensors");
  const Tensor& d_o = A.tensor(17);
  const OptTensor dS = A.opt(18);
  const bool lean = A.flag(19), want = A.flag(20);
  std::vector<Tensor> g;
  {
    pybind11::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    g = exact ? recurrent_backward(P.in, d_o, dS, want) : chunk_backward(P.in, std::move(saved), d_o, dS, lean, want);
  }
  return wrap_list(g);
  END_HANDLE_TH_ERRORS
}

// decode_step(qkv, conv_q, conv_k, conv_v, conv_weight, g, g_atk, beta_atk, beta, A_log, dt_bias,
//             log_atk_scale, state, a_state, gate | None, norm_weight | None, head_dim, scale | None,
//             squash_x, squash_eps, qk_eps, norm_eps) -> out
PyObject* py_decode_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, 22, "decode_step");
  const OptTensor gate = A.opt(14), norm_weight = A.opt(15);
  const DecodeInputs in{A.tensor(0), A.tensor(1), A.tensor(2), A.tensor(3), A.tensor(4), A.tensor(5), A.tensor(6),
                        A.tensor(7), A.tensor(8), A.tensor(9), A.tensor(10), A.tensor(11), A.tensor(12), A.tensor(13),
                        gate, norm_weight, A.whole(16), A.opt_num(17), A.num(18), A.num(19), A.num(20), A.num(21)};
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    out = decode_step(in);
  }
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// controls(packed, A_log_precond, dt_bias_precond, hidden) -> (h0, beta, g_atk, beta_atk, h1)
PyObject* py_controls(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, 4, "controls");
  const Tensor &packed = A.tensor(0), &A_log = A.tensor(1), &dt_bias = A.tensor(2);
  const int64_t hidden = A.whole(3);
  variable_list r;
  {
    pybind11::gil_scoped_release no_gil;
    r = Controls::apply(packed, A_log, dt_bias, hidden);
  }
  PyObject* out = PyTuple_New(5);
  if (!out) throw python_error();
  for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(out, i, wrap(r[i]));
  return out;
  END_HANDLE_TH_ERRORS
}

// Eager kernels of the layer operators for callers that want them without autograd.
PyObject* py_conv(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n == 5) {
    const Args A(args, n, 5, "conv");
    auto [q, k, v] = conv_cuda(A.tensor(0), A.tensor(1), A.whole(2), A.whole(3), A.num(4));
    return wrap3(q, k, v);
  }
  const Args A(args, n, 8, "conv");
  auto [dx, dw] = conv_backward_cuda(A.tensor(0), A.tensor(1), A.tensor(2), A.tensor(3), A.tensor(4), A.whole(5),
                                     A.whole(6), A.num(7));
  return wrap_list({dx, dw});
  END_HANDLE_TH_ERRORS
}

PyObject* py_norm_gate(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n == 4) {
    const Args A(args, n, 4, "norm_gate");
    auto [y, rstd] = norm_gate_cuda(A.tensor(0), A.tensor(1), A.tensor(2), A.num(3));
    return wrap_list({y, rstd});
  }
  const Args A(args, n, 6, "norm_gate");
  auto [dx, dg, dw] = norm_gate_backward_cuda(A.tensor(0), A.tensor(1), A.tensor(2), A.tensor(3), A.tensor(4), A.num(5));
  return wrap3(dx, dg, dw);
  END_HANDLE_TH_ERRORS
}

// check_intermediates([tensors | None], q, v, lean): the check of the operator's intermediates alone.
PyObject* py_check_intermediates(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Args A(args, n, 4, "check_intermediates");
  const std::vector<Tensor> list = A.tensors(0);
  check_intermediates(list, A.tensor(1), A.tensor(2), A.flag(3));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches.load()); }

PyObject* py_track_status(PyObject*, PyObject* enable) {
  g_track = PyObject_IsTrue(enable) == 1;
  std::lock_guard<std::mutex> lock(g_status_mutex);
  g_fwd_status = g_bwd_status = Tensor();
  Py_RETURN_NONE;
}

PyObject* py_tracking(PyObject*, PyObject*) { return PyBool_FromLong(g_track.load()); }

// last_status(which): the 4 status bytes of the last chunked forward (0) / backward (1), or None.
PyObject* py_last_status(PyObject*, PyObject* which) {
  HANDLE_TH_ERRORS
  Tensor t;
  {
    std::lock_guard<std::mutex> lock(g_status_mutex);
    t = PyObject_IsTrue(which) == 1 ? g_bwd_status : g_fwd_status;
  }
  return wrap(t);
  END_HANDLE_TH_ERRORS
}

// Forgets the forward's status word (another entry point ran last).
PyObject* py_drop_forward_status(PyObject*, PyObject*) {
  std::lock_guard<std::mutex> lock(g_status_mutex);
  g_fwd_status = Tensor();
  Py_RETURN_NONE;
}

#define PKDA_FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    PKDA_FAST("recurrence", py_recurrence),
    PKDA_FAST("recurrent_forward", py_recurrent_forward),
    PKDA_FAST("chunk_forward", py_chunk_forward),
    PKDA_FAST("backward", py_backward),
    PKDA_FAST("decode_step", py_decode_step),
    PKDA_FAST("controls", py_controls),
    PKDA_FAST("conv", py_conv),
    PKDA_FAST("norm_gate", py_norm_gate),
    PKDA_FAST("check_intermediates", py_check_intermediates),
    {"launches", py_launches, METH_NOARGS, nullptr},
    {"track_status", py_track_status, METH_O, nullptr},
    {"tracking", py_tracking, METH_NOARGS, nullptr},
    {"last_status", py_last_status, METH_O, nullptr},
    {"drop_forward_status", py_drop_forward_status, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// (The marker is what tells a library built for another torch from a current one without loading it.)
PyMODINIT_FUNC PyInit__native() {
  PyObject* m = PyModule_Create(&kModule);
  if (m && PyModule_AddStringConstant(m, "built_for", PKDA_NATIVE_MARKER) < 0) Py_CLEAR(m);
  return m;
}
