// The Python module _host: the public operators' host path in native code.  Argument checks, the choice of the
// blocking, allocation through torch's caching allocator, autograd nodes and the calls into the C ABI
// (include/pr_b200.h) all happen here, because the small cases are bound by them: a forward + backward of 1024
// tokens x 4 heads is 52 us of kernels, and driven from Python (autograd.Function, ctypes, one tensor
// method at a time) it took 208 us a pass; it takes 97 here.  A decode step of one sequence (8 + 5 us of kernels that
// overlap): 30 us, and 10 here.
//
// Everything runs on torch's current stream of the tensors' device.  Workspaces come from the caching allocator on
// every call: they are tied to the stream, so calls from several threads and streams do not share any.
#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <limits>
#include <optional>
#include <string>
#include <tuple>
#include <variant>

#include "../../include/pr_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

std::atomic<long long> g_launches{0};  // kernels launched through this module
PyObject* g_error = nullptr;           // the package's PRError

// Messages of the three kinds of failure a caller can see.  c10::Error would reach Python as RuntimeError too, but
// PRError and AssertionError are what the package promises.  The module's exception translator turns them into those for
// a call from Python; a backward pass is called by the autograd engine, which knows torch's own carrier of a Python
// exception (in_engine).
struct PrError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct AssertError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
void pr_require(bool ok, const char* msg) {
  if (!ok) throw PrError(msg);
}
void require(bool ok, const char* msg) {
  if (!ok) throw AssertError(msg);
}
void check(int rc, const char* what, int kernels) {
  if (rc != PR_OK)
    throw PrError(std::string(what) + " failed with code " + std::to_string(rc) + ": " + pr_last_error());
  g_launches.fetch_add(kernels, std::memory_order_relaxed);
}

template <typename F>
auto in_engine(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (const PrError& e) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(g_error ? g_error : PyExc_RuntimeError, e.what());
    python_error carried;
    carried.persist();
    throw carried;
  }
}

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return PR_BF16;
  if (t.scalar_type() == at::kHalf) return PR_FP16;
  throw PrError(std::string("dtype ") + c10::toString(t.scalar_type()) + " unsupported: use bfloat16 or float16");
}
const void* cptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* mptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* fptr(const Tensor& t) { return t.defined() ? static_cast<const float*>(t.const_data_ptr()) : nullptr; }
float* fmptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }

// Device of a call: its index, its current stream, and a guard (the C ABI sets the device and leaves it set).
struct On {
  c10::cuda::CUDAGuard guard;
  int device;
  void* stream;
  explicit On(const Tensor& t)
      : guard(t.device()), device(t.get_device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device()).stream()) {}
};

Tensor empty_f32(at::IntArrayRef size, const Tensor& like) { return at::empty(size, like.options().dtype(at::kFloat)); }
Tensor empty_bytes(size_t n, const Tensor& like) {
  return at::empty({(int64_t)std::max<size_t>(n, 16)}, like.options().dtype(at::kByte));
}
Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
// dense, and on the 16-byte boundary that TMA and 128-bit accesses want (a view may start anywhere)
Tensor aligned(const Tensor& t) {
  if (!t.defined()) return t;
  Tensor d = dense(t);
  return (reinterpret_cast<uintptr_t>(d.const_data_ptr()) & 15u) ? d.clone() : d;
}
Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

// ------------------------------------------------------------------------------------------------- training
pr_problem problem_of(const Tensor& Q, int64_t h, int64_t c, double scale) {
  return pr_problem{dtype_code(Q), (int)Q.size(0), (int)Q.size(1), (int)h, (int)Q.size(2), (int)Q.size(3), (int)c, (float)scale};
}
int64_t state_rows(int64_t d) { return 128 * (d / 16) * (d / 16 + 1); }

struct FwdOut {
  Tensor O, saved, Fs, Fg;
};

// c = 0: the state-free branch
FwdOut run_forward(const Tensor& Q, const Tensor& K, const Tensor& V, const Tensor& G, int64_t c, int64_t deg, double scale,
                   const Tensor& Cs, const Tensor& Cg, bool want_final) {
  const On on(Q);
  const int64_t h = K.size(2), d = Q.size(3), b = Q.size(0);
  const pr_problem p = problem_of(Q, h, c, scale);
  FwdOut r;
  size_t n = 0;
  r.O = at::empty_like(Q);
  if (c == 0) {
    check(pr_attention_workspace_bytes(&p, PR_WS_SAVED, &n), "pr_attention_workspace_bytes", 0);
    r.saved = empty_bytes(n, Q);
    check(pr_attention_fwd(&p, (int)deg, cptr(Q), cptr(K), cptr(V), fptr(G), mptr(r.O), mptr(r.saved), on.device, on.stream),
          "pr_attention_fwd", G.defined() ? 2 : 1);
    return r;
  }
  check(pr_workspace_bytes(&p, PR_WS_SAVED, &n), "pr_workspace_bytes", 0);
  r.saved = empty_bytes(n, Q);
  check(pr_workspace_bytes(&p, PR_WS_FWD_SCRATCH, &n), "pr_workspace_bytes", 0);
  const Tensor scratch = empty_bytes(n, Q);
  if (want_final) {
    r.Fs = empty_f32({b, h, state_rows(d) * d}, Q);
    r.Fg = empty_f32({b, h, d * d}, Q);
  }
  check(pr_retention_fwd(&p, cptr(Q), cptr(K), cptr(V), fptr(G), fptr(Cs), fptr(Cg), mptr(r.O), mptr(r.saved), mptr(scratch),
                         fmptr(r.Fs), fmptr(r.Fg), on.device, on.stream),
        "pr_retention_fwd", G.defined() ? 5 : 4);
  return r;
}

class Retention : public torch::autograd::Function<Retention> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& Q, const Tensor& K, const Tensor& V,
                               const OptTensor& gates, int64_t c, int64_t deg, double scale, const OptTensor& carry_state,
                               const OptTensor& carry_gram, bool want_final) {
    const Tensor G = opt(gates), Cs = opt(carry_state), Cg = opt(carry_gram);
    FwdOut r = run_forward(Q, K, V, G, c, deg, scale, Cs, Cg, want_final);
    ctx->save_for_backward({Q, K, V, G, r.O, r.saved});
    ctx->saved_data["c"] = c;
    ctx->saved_data["deg"] = deg;
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["carry"] = Cs.defined();
    if (!want_final) return {r.O};
    ctx->mark_non_differentiable({r.Fs, r.Fg});
    return {r.O, r.Fs, r.Fg};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return in_engine([&] { return run_backward(ctx, grads); });
  }
  static variable_list run_backward(AutogradContext* ctx, const variable_list& grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &Q = s[0], &K = s[1], &V = s[2], &G = s[3], &O = s[4], &saved = s[5];
    variable_list out(10);
    if (!grads[0].defined()) return out;
    const int64_t c = ctx->saved_data["c"].toInt(), deg = ctx->saved_data["deg"].toInt();
    const On on(Q);
    const Tensor dO = aligned(grads[0]);
    const pr_problem p = problem_of(Q, K.size(2), c, ctx->saved_data["scale"].toDouble());
    const Tensor dQ = at::empty_like(Q), dK = at::empty_like(K), dV = at::empty_like(V);
    const Tensor dG = G.defined() ? at::empty_like(G) : Tensor();
    size_t n = 0;
    if (c == 0) {
      check(pr_attention_workspace_bytes(&p, PR_WS_BWD_SCRATCH, &n), "pr_attention_workspace_bytes", 0);
      const Tensor scratch = empty_bytes(n, Q);
      check(pr_attention_bwd(&p, (int)deg, cptr(Q), cptr(K), cptr(V), fptr(G), cptr(O), cptr(dO), mptr(saved), mptr(scratch),
                             mptr(dQ), mptr(dK), mptr(dV), fmptr(dG), on.device, on.stream),
            "pr_attention_bwd", G.defined() ? 4 : 3);
    } else {
      check(pr_workspace_bytes(&p, PR_WS_BWD_SCRATCH, &n), "pr_workspace_bytes", 0);
      const Tensor scratch = empty_bytes(n, Q);
      check(pr_retention_bwd(&p, cptr(Q), cptr(K), cptr(V), fptr(G), cptr(O), cptr(dO), ctx->saved_data["carry"].toBool(),
                             mptr(saved), mptr(scratch), mptr(dQ), mptr(dK), mptr(dV), fmptr(dG), on.device, on.stream),
            "pr_retention_bwd", G.defined() ? 11 : 10);
    }
    out[0] = dQ;
    out[1] = dK;
    out[2] = dV;
    out[3] = dG;
    return out;
  }
};

// A state pair in the exact layout, on the device of `like`.
void check_state(const Tensor& state, const Tensor& sok, int64_t b, int64_t h, int64_t d, const Tensor& like) {
  const int64_t D = d * (d + 1) / 2;
  require(state.dim() == 4 && state.size(0) == b && state.size(1) == h && state.size(2) == D && state.size(3) == d,
          "state must be [b,h,d(d+1)/2,d] (exact layout)");
  require(sok.dim() == 3 && sok.size(0) == b && sok.size(1) == h && sok.size(2) == D && sok.scalar_type() == at::kFloat,
          "sum_of_keys must be [b,h,d(d+1)/2] float32");
  pr_require(state.is_cuda() && sok.is_cuda(), "the state must live on a CUDA device: this package has no CPU path");
  require(state.device() == like.device() && sok.device() == like.device(), "tensors must live on one device");
}

using StatePair = std::tuple<Tensor, Tensor>;

// The pair after the last token in the exact layout, from the scans' carries.
StatePair final_state(const Tensor& S, const Tensor& gram, int64_t b, int64_t h, int64_t d, const On& on) {
  const int64_t D = d * (d + 1) / 2;
  const Tensor ns = at::empty({b, h, D, d}, S.options()), nk = empty_f32({b, h, D}, S);
  check(pr_state_merge(dtype_code(S), (int)b, (int)h, (int)d, nullptr, nullptr, cptr(S), fptr(gram), nullptr, mptr(ns),
                       fmptr(nk), on.device, on.stream),
        "pr_state_merge", 1);
  return {ns, nk};
}

// torch.jit.trace records torch's own operators.  Of a call made here it would see the allocations of the results and
// none of the kernels, and the trace would give back memory that nothing has written.  The Python callers have an
// autograd.Function for this case, which the tracer records as one node: the entry points answer None.
bool being_traced() { return at::tracer::impl::is_dispatch_enabled(); }

using Retained = std::variant<Tensor, std::tuple<Tensor, StatePair>>;  // with a final state: (output, pair)

// power_retention with the blocking chosen here.  Returns None for the head dims that the caller has to widen first, and
// where the caller's own path has to run.  switch_over is a double because callers say "never" with infinity.
std::optional<Retained> power_retention(Tensor Q, Tensor K, Tensor V, const OptTensor& log_G, const OptTensor& state,
                                        const OptTensor& sok, bool want_final, int64_t deg, double scale,
                                        std::optional<int64_t> chunk_size, std::optional<double> switch_over,
                                        bool auto_chunk, int64_t quadratic_tokens) {
  if (being_traced()) return std::nullopt;
  require(deg % 2 == 0, "deg must be even");
  pr_require(!chunk_size.has_value() || *chunk_size > 0, "chunk_size must be positive");
  pr_require(state.has_value() == sok.has_value(), "initial_state is the pair (state, sum_of_keys)");
  const int64_t chunk = chunk_size.value_or(0);  // 0: not given
  require(Q.dim() == 4 && K.dim() == 4 && V.dim() == 4, "Q, K, V must be [batch, seq_len, heads, dim]");
  const int64_t b = Q.size(0), t = Q.size(1), hq = Q.size(2), d = Q.size(3), h = K.size(2);
  const bool with_state = state.has_value() || want_final;
  if ((d == 16 || d == 32) && with_state)
    throw PrError("states are kept for head dim 64 only (got " + std::to_string(d) + ")");
  if (d == 48) return std::nullopt;
  int64_t c = (auto_chunk && deg == 2) ? pr_fast_chunk(t, (int)std::min<int64_t>(chunk, std::numeric_limits<int>::max())) : chunk;
  if (c != chunk || !switch_over.has_value()) {
    // the blocking is this function's own choice: one chunk is the quadratic form, and so is what the caller says is short
    switch_over = c ? std::optional<double>((double)c) : std::nullopt;
    if (auto_chunk && deg == 2 && !with_state && t <= quadratic_tokens) c = 0;
  }
  const bool quadratic = !switch_over.has_value() || c == 0 || (double)((t + c - 1) / c * c) <= *switch_over;
  if (deg != 2 && !(deg == 4 && quadratic && !with_state))
    throw PrError("deg=" + std::to_string(deg) +
                  ": the state kernels implement deg=2 (as the reference's state operators do); "
                  "deg=4 runs on the state-free branch only (chunk_size=None or t <= switch_over_seq_len)");
  pr_require(Q.is_cuda() && K.is_cuda() && V.is_cuda(), "Q, K, V must be CUDA tensors: this package has no CPU path");
  require(Q.scalar_type() == K.scalar_type() && Q.scalar_type() == V.scalar_type(), "dtypes of inputs must match");
  dtype_code(Q);
  require(h > 0 && hq % h == 0, "Q heads must be a multiple of KV heads");
  if (d != 16 && d != 32 && d != 64)
    throw PrError("head dim " + std::to_string(d) + " unsupported by this build (supported: 16, 32, 48, 64)");
  require(K.sizes() == V.sizes() && K.size(0) == b && K.size(1) == t && K.size(3) == d, "K and V must be [b, t, h, d]");
  require(K.device() == Q.device() && V.device() == Q.device(), "tensors must live on one device");
  Tensor G = opt(log_G);
  if (G.defined()) {
    require(G.dim() == 3 && G.size(0) == b && G.size(1) == t && G.size(2) == h, "log_G must be [batch, seq_len, kv_heads]");
    require(G.device() == Q.device(), "tensors must live on one device");
    G = dense(G.scalar_type() == at::kFloat ? G : G.to(at::kFloat));
  }
  Q = aligned(Q);
  K = aligned(K);
  V = aligned(V);
  if (scale == 0) scale = 1.0 / std::sqrt((double)d);
  if (quadratic) c = with_state ? t : 0;  // a short sequence that carries a state is one chunk of the chunked form
  // the autograd node also where an input carries a tangent: forward mode is not implemented, and the node says so
  auto any_of = [&](auto f) { return f(Q) || f(K) || f(V) || (G.defined() && f(G)); };
  const bool grad = (at::GradMode::is_enabled() && any_of([](const Tensor& t) { return t.requires_grad(); })) ||
                    any_of([](const Tensor& t) { return t._fw_grad(0).defined(); });
  Tensor Cs, Cg;
  if (state.has_value()) {
    check_state(*state, *sok, b, h, d, Q);
    const On on(Q);
    const Tensor s = aligned(state->detach().to(Q.scalar_type())), k = aligned(sok->detach());
    Cs = empty_f32({b, h, state_rows(d) * d}, Q);
    Cg = empty_f32({b, h, d * d}, Q);
    check(pr_state_to_chunk_layout(dtype_code(Q), (int)b, (int)h, (int)d, cptr(s), fptr(k), nullptr, fmptr(Cs), fmptr(Cg),
                                   nullptr, nullptr, on.device, on.stream),
          "pr_state_to_chunk_layout", 1);
  }
  Tensor O, Fs, Fg;
  if (grad) {
    auto given = [](const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; };
    const variable_list out = Retention::apply(Q, K, V, given(G), c, deg, scale, given(Cs), given(Cg), want_final);
    O = out[0];
    if (want_final) {
      Fs = out[1];
      Fg = out[2];
    }
  } else {
    const FwdOut r = run_forward(Q, K, V, G, c, deg, scale, Cs, Cg, want_final);
    O = r.O;
    Fs = r.Fs;
    Fg = r.Fg;
  }
  if (!want_final) return Retained(O);
  const On on(Q);
  return Retained(std::make_tuple(O, final_state(Fs.detach().to(Q.scalar_type()), Fg.detach(), b, h, d, on)));
}

// ------------------------------------------------------------------------------------------------ inference
// The tensor as it is when everything inside a batch entry is dense (a slice [:, :n] of a longer preallocated cache
// is), its start is 16-byte aligned and its batch stride a multiple of `unit` elements; a dense copy otherwise.
Tensor batch_strided(const Tensor& t, int64_t unit, int64_t* stride) {
  int64_t inner = 1;
  bool ok = true;
  for (int64_t i = t.dim() - 1; i >= 1 && ok; --i) {
    ok = t.size(i) == 1 || t.stride(i) == inner;
    inner *= t.size(i);
  }
  *stride = t.size(0) > 1 ? t.stride(0) : inner;
  ok = ok && *stride >= inner && *stride % unit == 0 &&
       (unit == 1 || (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0);
  if (ok) return t;
  *stride = inner;
  return aligned(t);
}

struct Partials {
  Tensor both;  // one allocation: rows of d, then their sums
  float *y = nullptr, *l = nullptr;
  int kernels = 1;
  // workspace of a decode step that is split over several CTAs per (batch, head); none when it is not
  Partials(int64_t b, int64_t h, int64_t hq, int64_t d, const Tensor& like) {
    if (pr_decode_split((int)b, (int)h, (int)hq) <= 1) return;
    const int64_t ns = pr_decode_nsplit();
    both = empty_f32({b * hq * ns * (d + 1)}, like);
    y = fmptr(both);
    l = y + b * hq * ns * d;
    kernels = 2;
  }
};

Tensor decode_step(const Tensor& Q0, const Tensor& K0, const Tensor& V0, const Tensor& G0, const Tensor& state,
                   const Tensor& sok, double scale, int64_t h) {
  const On on(Q0);
  const int64_t b = Q0.size(0), hq = Q0.size(2), d = Q0.size(3), tk = K0.defined() ? K0.size(1) : 0;
  int64_t qs = 0, ks = 0, vs = 0, gs = 0;
  const Tensor Q = batch_strided(Q0, 8, &qs);
  Tensor K, V, G;
  if (tk > 0) {
    K = batch_strided(K0, 8, &ks);
    V = batch_strided(V0, 8, &vs);
    if (ks != vs) {
      K = aligned(K);
      V = aligned(V);
      ks = tk * h * d;
    }
    if (G0.defined()) G = batch_strided(G0, 1, &gs);
  }
  const Tensor O = at::empty({b, 1, hq, d}, Q.options());
  const Partials part(b, h, hq, d, Q);
  check(pr_decode_step_strided(dtype_code(Q), (int)b, (int)tk, (int)h, (int)hq, (int)d, cptr(Q), qs, cptr(K), cptr(V), ks,
                               fptr(G), gs, cptr(state), fptr(sok), (float)scale, nullptr, part.y, part.l,
                               mptr(O), on.device, on.stream),
        "pr_decode_step_strided", part.kernels);
  return O;
}

// gated, transposed keys and / or the gate sums of one chunk that is the whole cache
void gate_sums(const Tensor& K, const Tensor& G, const Tensor& a, const Tensor& total, const Tensor& xt, const On& on) {
  const int64_t b = K.size(0), tk = K.size(1), h = K.size(2), d = K.size(3);
  if (!xt.defined() && tk > 16384) {  // longer than the chunk-local scan holds in shared memory
    check(pr_gate_cumsum((int)b, (int)tk, (int)h, fptr(G), tk * h, fmptr(a), on.device, on.stream), "pr_gate_cumsum", 1);
    return;
  }
  check(pr_gate_prep(dtype_code(K), (int)b, (int)tk, (int)h, (int)h, (int)d, (int)tk, fptr(G), cptr(K), fmptr(a), fmptr(total),
                     mptr(xt), nullptr, nullptr, 0, 1.f, a.defined(), on.device, on.stream),
        "pr_gate_prep", a.defined() && xt.defined() ? 2 : 1);
}

std::tuple<Tensor, OptTensor, OptTensor> inference(const Tensor& Q0, const OptTensor& K_, const OptTensor& V_,
                                                   const OptTensor& log_G, const OptTensor& state_,
                                                   const OptTensor& sok_, std::optional<double> scale_,
                                                   std::optional<double> switch_over) {
  const at::NoGradGuard no_grad;
  const bool has_cache = K_.has_value() && V_.has_value(), has_state = state_.has_value();
  require(has_cache || has_state, "initial_state or cache must be provided for inference");
  require(has_state == sok_.has_value(), "initial_state and sum_of_keys come together");
  require(Q0.dim() == 4, "Q must be [batch, tokens, heads, dim]");
  pr_require(Q0.is_cuda(), "tensors must be CUDA tensors: this package has no CPU path");
  const int64_t b = Q0.size(0), tq = Q0.size(1), hq = Q0.size(2), d = Q0.size(3);
  if (d != 64) throw PrError("head dim " + std::to_string(d) + " unsupported by this build (supported: 64)");
  int64_t tk = 0, h = 0;
  Tensor K, V, G;
  if (has_cache) {
    K = *K_;
    V = *V_;
    require(Q0.scalar_type() == K.scalar_type() && Q0.scalar_type() == V.scalar_type(), "dtypes of inputs must match");
    require(K.dim() == 4 && V.dim() == 4 && K.sizes() == V.sizes(), "key and value must have the same seq_len");
    require(K.size(0) == b && K.size(3) == d, "K and V must be [b, t, h, d]");
    require(K.device() == Q0.device() && V.device() == Q0.device(), "tensors must live on one device");
    tk = K.size(1);
    h = K.size(2);
  } else {
    require(state_->dim() == 4, "state must be [b,h,d(d+1)/2,d] (exact layout)");
    h = state_->size(1);
  }
  require(h > 0 && hq % h == 0, "Q heads must be a multiple of KV heads");
  dtype_code(Q0);
  Tensor state, sok;
  if (has_state) {
    check_state(*state_, *sok_, b, h, d, Q0);
    pr_require(state_->scalar_type() == Q0.scalar_type(), "the state's dtype must be the query's");
    state = aligned(*state_);
    sok = aligned(*sok_);
  }
  const double scale = scale_.has_value() ? *scale_ : 1.0 / std::sqrt((double)d);
  if (has_cache && log_G.has_value()) {
    G = *log_G;
    require(G.dim() == 3 && G.size(0) == b && G.size(1) == tk && G.size(2) == h, "log_G must be [batch, seq_len, kv_heads]");
    require(G.device() == Q0.device(), "tensors must live on one device");
    if (G.scalar_type() != at::kFloat) G = G.to(at::kFloat);
  }
  const bool compress = switch_over.has_value() && (double)tk >= *switch_over;

  Tensor Y;
  if (tq == 1 && has_state && !compress) {
    Y = decode_step(Q0, K, V, G, state, sok, scale, h);
    return {Y, state_, sok_};
  }
  const On on(Q0);
  const Tensor Q = aligned(Q0);
  const int dt = dtype_code(Q);
  if (has_cache) {
    K = aligned(K);
    V = aligned(V);
    if (G.defined()) G = dense(G);
  }
  // The gate sums serve the read-out and the compression; the compression's pass makes them on its way.
  Tensor a, total, xt;
  if (compress) xt = at::empty({b, 1, h, d, (tk + 63) / 64 * 64}, Q.options());
  if (G.defined()) a = empty_f32({b, tk, h}, Q);
  if (G.defined() && compress) total = empty_f32({b, h}, Q);
  if (xt.defined() || (a.defined() && !(tq == 1 && has_state))) gate_sums(K, G, a, total, xt, on);

  // ---- read-out
  if (tq == 1 && has_state) {
    Y = decode_step(Q, K, V, G, state, sok, scale, h);
  } else {
    Y = at::empty_like(Q);
    Tensor z, ghi, glo;
    if (has_state) {
      z = at::empty({b, h, state_rows(d), d}, Q.options());
      ghi = at::empty({b, h, d, d}, Q.options());
      glo = at::empty({b, h, d, d}, Q.options());
      check(pr_state_to_chunk_layout(dt, (int)b, (int)h, (int)d, cptr(state), fptr(sok), mptr(z), nullptr, nullptr, mptr(ghi),
                                     mptr(glo), on.device, on.stream),
            "pr_state_to_chunk_layout", 1);
    }
    const bool attn = tk > 0;
    check(pr_chunk_out(dt, (int)b, 1, (int)tq, (int)(attn ? tk : tq), (int)hq, (int)h, (int)d, cptr(Q), attn ? cptr(K) : nullptr,
                       attn ? cptr(V) : nullptr, attn ? fptr(a) : nullptr, cptr(z), cptr(ghi), cptr(glo), has_state ? 0 : 1,
                       has_state && attn, 1, (float)scale, 2, mptr(Y), nullptr, on.device, on.stream),
          "pr_chunk_out", 1);
  }
  if (!compress) return {Y, state_, sok_};

  // ---- the cache becomes a new state
  const int64_t D = d * (d + 1) / 2;
  const Tensor ns = at::empty({b, h, D, d}, Q.options()), nk = empty_f32({b, h, D}, Q);
  check(pr_compress_cache(dt, (int)b, (int)tk, (int)h, (int)d, cptr(xt), cptr(V), cptr(state), fptr(sok), fptr(total),
                          mptr(ns), fmptr(nk), on.device, on.stream),
        "pr_compress_cache", 1);
  return {Y, ns, nk};
}

Tensor decode_recurrent(const Tensor& q0, const Tensor& k0, const Tensor& v0, const OptTensor& log_g, const Tensor& state,
                        const Tensor& sok, const Tensor& new_state, const Tensor& new_sok, double scale) {
  const at::NoGradGuard no_grad;
  require(q0.dim() == 4 && k0.dim() == 4 && v0.dim() == 4 && q0.size(1) == 1 && k0.size(1) == 1 && k0.sizes() == v0.sizes() &&
              k0.size(0) == q0.size(0) && k0.size(3) == q0.size(3),
          "q, k, v must be [batch, 1, heads, dim]");
  const int64_t b = q0.size(0), hq = q0.size(2), d = q0.size(3), h = k0.size(2);
  require(h > 0 && hq % h == 0, "Q heads must be a multiple of KV heads");
  require(!log_g.has_value() || (log_g->dim() >= 1 && log_g->size(0) == b && log_g->numel() == b * h),
          "log_g must be [batch, 1, kv_heads]");
  require(q0.scalar_type() == k0.scalar_type() && q0.scalar_type() == v0.scalar_type(), "dtypes of inputs must match");
  dtype_code(q0);
  pr_require(state.scalar_type() == q0.scalar_type() && new_state.scalar_type() == q0.scalar_type(),
             "the state's dtype must be the query's");
  pr_require(q0.is_cuda() && k0.is_cuda() && v0.is_cuda(), "tensors must be CUDA tensors: this package has no CPU path");
  require(k0.device() == q0.device() && v0.device() == q0.device() && (!log_g.has_value() || log_g->device() == q0.device()),
          "tensors must live on one device");
  check_state(state, sok, b, h, d, q0);
  check_state(new_state, new_sok, b, h, d, q0);
  const On on(q0);
  require(state.is_contiguous() && sok.is_contiguous() && new_state.is_contiguous() && new_sok.is_contiguous(),
          "states must be contiguous");
  int64_t qs = 0, ks = 0, vs = 0, gs = 0;
  const Tensor q = batch_strided(q0, 8, &qs);
  Tensor k = batch_strided(k0, 8, &ks), v = batch_strided(v0, 8, &vs), g;
  if (ks != vs) {
    k = aligned(k);
    v = aligned(v);
    ks = h * d;
  }
  if (log_g.has_value()) {
    g = log_g->scalar_type() == at::kFloat ? *log_g : log_g->to(at::kFloat);
    g = batch_strided(g, 1, &gs);
  }
  const Tensor O = at::empty({b, 1, hq, d}, q.options());
  const Partials part(b, h, hq, d, q);
  check(pr_decode_recurrent(dtype_code(q), (int)b, (int)h, (int)hq, (int)d, cptr(q), qs, cptr(k), cptr(v), ks, fptr(g), gs,
                            cptr(state), fptr(sok), mptr(new_state), fmptr(new_sok), (float)scale, part.y,
                            part.l, mptr(O), on.device, on.stream),
        "pr_decode_recurrent", part.kernels);
  return O;
}

// ----------------------------------------------------------------------------------------- the callers' glue
class PrepareQKVG : public torch::autograd::Function<PrepareQKVG> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& sin, const Tensor& cos, int64_t h,
                               int64_t hq, int64_t d, bool gated, double bias, bool half_split) {
    const On on(x);
    const int64_t b = x.size(0), t = x.size(1);
    const Tensor Q = at::empty({b, t, hq, d}, x.options()), K = at::empty({b, t, h, d}, x.options()),
                 V = at::empty({b, t, h, d}, x.options());
    const Tensor G = gated ? empty_f32({b, t, h}, x) : Tensor();
    check(pr_caller_prep_fwd(dtype_code(x), (int)b, (int)t, (int)h, (int)hq, (int)d, cptr(x), x.size(2), fptr(cos), fptr(sin),
                             cos.dim() == 2 ? 0 : t * (d / 2), half_split, gated, (float)bias, mptr(Q), mptr(K), mptr(V),
                             fmptr(G), on.device, on.stream),
          "pr_caller_prep_fwd", 1);
    ctx->save_for_backward({x, sin, cos});
    ctx->saved_data["h"] = h;
    ctx->saved_data["hq"] = hq;
    ctx->saved_data["d"] = d;
    ctx->saved_data["gated"] = gated;
    ctx->saved_data["bias"] = bias;
    ctx->saved_data["half_split"] = half_split;
    if (gated) return {Q, K, V, G};
    return {Q, K, V};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return in_engine([&] { return run_backward(ctx, grads); });
  }
  static variable_list run_backward(AutogradContext* ctx, const variable_list& grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &sin = s[1], &cos = s[2];
    const On on(x);
    const int64_t b = x.size(0), t = x.size(1), W = x.size(2), h = ctx->saved_data["h"].toInt(),
                  hq = ctx->saved_data["hq"].toInt(), d = ctx->saved_data["d"].toInt();
    const bool gated = ctx->saved_data["gated"].toBool();
    // an output that nothing used has no gradient
    auto grad = [&](size_t i, int64_t heads) {
      return grads[i].defined() ? aligned(grads[i]) : at::zeros({b, t, heads, d}, x.options());
    };
    const Tensor dQ = grad(0, hq), dK = grad(1, h), dV = grad(2, h);
    Tensor dG;
    if (gated) dG = grads[3].defined() ? dense(grads[3].to(at::kFloat)) : at::zeros({b, t, h}, x.options().dtype(at::kFloat));
    const Tensor dx = W == (hq + 2 * h) * d + (gated ? h : 0) ? at::empty_like(x) : at::zeros_like(x);
    check(pr_caller_prep_bwd(dtype_code(x), (int)b, (int)t, (int)h, (int)hq, (int)d, cptr(x), W, fptr(cos), fptr(sin),
                             cos.dim() == 2 ? 0 : t * (d / 2), ctx->saved_data["half_split"].toBool(), gated,
                             (float)ctx->saved_data["bias"].toDouble(), cptr(dQ), cptr(dK), cptr(dV), fptr(dG), mptr(dx),
                             on.device, on.stream),
          "pr_caller_prep_bwd", 1);
    variable_list out(9);
    out[0] = dx;
    return out;
  }
};

using Prepared = std::tuple<Tensor, Tensor, Tensor, OptTensor>;

std::optional<Prepared> prepare_qkvg(Tensor x, Tensor sin, Tensor cos, int64_t h, int64_t hq, int64_t d, bool gated,
                                     double bias, bool half_split) {
  pr_require(x.is_cuda() && x.dim() == 3 && (x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kHalf),
             "prepare_qkvg wants a CUDA bf16/fp16 tensor [b, t, W]");
  const int64_t used = (hq + 2 * h) * d + (gated ? h : 0), t = x.size(1);
  if (x.size(2) < used)
    throw PrError("a row of " + std::to_string(x.size(2)) + " elements cannot hold " + std::to_string(used));
  if (d % 8 || (half_split && d % 16))
    throw PrError("head dim " + std::to_string(d) + ": a multiple of 8 (16 for half-split pairs)");
  // 16-byte rows; differentiable, the gradient is cut back
  if (x.size(2) % 8) x = at::constant_pad_nd(x, {0, 8 - x.size(2) % 8});
  x = aligned(x);
  sin = dense(sin.to(at::kFloat)).detach();
  cos = dense(cos.to(at::kFloat)).detach();
  pr_require(sin.dim() >= 2 && sin.size(-2) == t && sin.size(-1) == d / 2 && cos.sizes() == sin.sizes() &&
                 (sin.dim() == 2 || (sin.dim() == 3 && sin.size(0) == x.size(0))) && sin.device() == x.device() &&
                 cos.device() == x.device(),
             "sin / cos must be [t, d/2] (or [b, t, d/2]) for the tokens of the projection");
  if (being_traced()) return std::nullopt;
  const variable_list out = PrepareQKVG::apply(x, sin, cos, h, hq, d, gated, bias, half_split);
  return Prepared(out[0], out[1], out[2], gated ? OptTensor(out[3]) : std::nullopt);
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.doc() = "host path of power retention: see the wrappers in retention.py, cache.py and caller.py";
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const PrError& e) {
      PyErr_SetString(g_error ? g_error : PyExc_RuntimeError, e.what());
    } catch (const AssertError& e) {
      PyErr_SetString(PyExc_AssertionError, e.what());
    }
  });
  m.def("set_error_type", [](py::object cls) { g_error = cls.release().ptr(); });
  m.def("launches", [] { return g_launches.load(std::memory_order_relaxed); });
  // Without the interpreter lock: a launch into a full queue waits for the GPU, and other Python threads go on meanwhile.
  using no_gil = py::call_guard<py::gil_scoped_release>;
  m.def("power_retention", &power_retention, no_gil());
  m.def("inference", &inference, no_gil());
  m.def("decode_recurrent", &decode_recurrent, no_gil());
  m.def("prepare_qkvg", &prepare_qkvg, no_gil());
}
