// The torch operators of the package, in C++: argument checks and conversions, output and workspace allocation,
// autograd, and the calls into the C ABI (include/rwkv_ops_b200.h).  A training step of a small model launches a
// dozen kernels of a few microseconds each, so what the host does around them decides its time.  As Python
// functions registered with torch.library this layer took 45 us per forward call and 300 us per forward +
// backward on the host (B2 T371 H12: 323 us per step, of which 62 us were kernels).
//
// Every public function of the Python modules is one operator here:
//   generalized_delta_rule, rwkv7_varlen, rwkv7_fused, wkv6, wkv6_varlen   composite: checks, conversions, then
//   rwkv7_fwd / _bwd, rwkv7_fwd_varlen / _bwd_varlen, ...                  one C-ABI call each (CUDA), autograd
//   rwkv7_decode_step                                                      one C-ABI call, in place on the state
// The composite operators raise on every argument the Python layer documents as invalid; the Python layer then
// repeats its own checks to raise the documented exception type.  The shape functions of the CUDA operators
// (for tracing without a device) are registered from Python (_ops.py).
//
// The library is linked against torch only.  The rwkvb200_* symbols come from the C-ABI library that the Python
// layer has loaded before (RTLD_GLOBAL).
//
// The composite operators are traced with symbolic sizes, so they look at sizes as SymInt: comparing them leaves a guard,
// where asking for them as integers would make every length a program of its own.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/library.h>

#include <algorithm>
#include <cctype>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <strings.h>
#include <string>
#include <tuple>

#include "../../include/rwkv_ops_b200.h"

namespace {

using at::Tensor;
using c10::SymInt;
typedef std::optional<Tensor> OptTensor;
typedef torch::autograd::variable_list Vars;
typedef torch::autograd::AutogradContext Ctx;

// ---------------------------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------------------------
constexpr int HEAD = 64;      // head size of the tensor-core paths

void check(int rc, const char* what) {
  if (rc != RWKVB200_OK) {
    std::string msg = std::string("rwkv_ops_b200 ") + what + ": " + rwkvb200_strerror(rc) + " (code " +
                      std::to_string(rc) + ")";
    if (rc == RWKVB200_E_CUDA) msg += std::string(": ") + rwkvb200_last_cuda_error();
    const bool value = rc == RWKVB200_E_SHAPE || rc == RWKVB200_E_DTYPE || rc == RWKVB200_E_ALIGN ||
                       rc == RWKVB200_E_NULL || rc == RWKVB200_E_UNSUPPORTED || rc == RWKVB200_E_STATE_MAP ||
                       rc == RWKVB200_E_TOO_LARGE;
    TORCH_CHECK_VALUE(!value, msg);
    TORCH_CHECK(false, msg);
  }
  // RWKV_OPS_B200_CHECK_STATUS=1: synchronise and report a bounded wait that ran out inside a kernel
  const char* env = std::getenv("RWKV_OPS_B200_CHECK_STATUS");
  if (env && *env && std::strcmp(env, "0") != 0) {
    const int code = rwkvb200_device_status(1);
    TORCH_CHECK(code == 0, "rwkv_ops_b200 ", what, ": a bounded wait inside a tensor-core kernel ran out (code ", code,
                "); the results of this call are not valid");
  }
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return RWKVB200_F32;
    case at::kBFloat16: return RWKVB200_BF16;
    case at::kHalf: return RWKVB200_F16;
    default: TORCH_CHECK_VALUE(false, "unsupported token dtype ", t, "; use float32, bfloat16 or float16");
  }
}
// the dtype an operator computes in for tokens of dtype t
at::ScalarType compute_dtype(at::ScalarType t) {
  return t == at::kFloat || t == at::kBFloat16 || t == at::kHalf ? t : at::kFloat;
}

int algo_from_env(const char* name) {
  const char* env = std::getenv(name);
  if (!env || strcasecmp(env, "auto") == 0) return RWKVB200_ALGO_AUTO;
  if (strcasecmp(env, "recurrent") == 0) return RWKVB200_ALGO_RECURRENT;
  if (strcasecmp(env, "chunked") == 0) return RWKVB200_ALGO_CHUNKED;
  TORCH_CHECK_VALUE(false, name, " must be auto, recurrent or chunked");
}

// Largest per-call tile store that a training forward may hand to its backward: RWKV_OPS_B200_KEEP_LIMIT_MB when
// set, else a quarter of the device's memory.
size_t keep_limit_bytes(int device) {
  if (const char* env = std::getenv("RWKV_OPS_B200_KEEP_LIMIT_MB")) {
    char* end = nullptr;
    const long long mb = std::strtoll(env, &end, 10);
    while (std::isspace((unsigned char)*end)) ++end;
    TORCH_CHECK_VALUE(end != env && !*end, "RWKV_OPS_B200_KEEP_LIMIT_MB must be a whole number, got ", env);
    constexpr long long most = std::numeric_limits<long long>::max() >> 20;      // 8 exabytes
    return mb < 0 ? 0 : (size_t)std::min(mb, most) << 20;                        // (strtoll saturates)
  }
  if (c10::cuda::device_count() == 0) return std::numeric_limits<size_t>::max();      // traced where there is no device
  return (size_t)at::cuda::getDeviceProperties(device)->totalGlobalMem / 4;
}

Tensor dense(const Tensor& x, at::ScalarType t) { return x.to(t).contiguous(); }
OptTensor dense_state(const OptTensor& x) {
  if (!x.has_value() || !x->defined()) return std::nullopt;
  return x->to(at::kFloat).contiguous();
}
bool has(const OptTensor& x) { return x.has_value() && x->defined(); }
void* ptr(const Tensor& x) { return x.defined() ? x.data_ptr() : nullptr; }
void* ptr(const OptTensor& x) { return x.has_value() ? ptr(*x) : nullptr; }
float* fptr(const OptTensor& x) { return has(x) ? static_cast<float*>(x->data_ptr()) : nullptr; }
float* fptr(const Tensor& x) { return static_cast<float*>(ptr(x)); }
const int32_t* iptr(const OptTensor& x) { return has(x) ? x->data_ptr<int32_t>() : nullptr; }
int n_state_of(const OptTensor& x) { return has(x) ? (int)x->size(0) : 0; }

Tensor fresh(at::IntArrayRef size, at::ScalarType t, const Tensor& like) {
  return at::detail::empty_cuda(size, t, like.device(), std::nullopt);
}
Tensor fresh_like(const Tensor& x) { return fresh(x.sizes(), x.scalar_type(), x); }
Tensor bytes(size_t n, const Tensor& like) { return fresh({(int64_t)n}, at::kByte, like); }
// Memory that a call only runs faster with: an undefined tensor where it cannot be had.
Tensor bytes_if_any(size_t n, const Tensor& like) {
  try {
    return n ? bytes(n, like) : Tensor();
  } catch (const c10::OutOfMemoryError&) {
    return Tensor();
  }
}
size_t size_of(const Tensor& x) { return x.defined() ? (size_t)x.numel() : 0; }
void* stream_of(const Tensor& x) { return c10::cuda::getCurrentCUDAStream(x.device().index()).stream(); }

bool any_requires_grad(at::ArrayRef<const Tensor*> xs, const OptTensor& s) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* x : xs)
    if (x->requires_grad()) return true;
  return has(s) && s->requires_grad();
}

// gradient of the states a batch started from, summed where one state served every row
Tensor state_grad(const Tensor& rows, const OptTensor& s0) {
  if (s0->sym_size(0) == 1 && rows.sym_size(0) != 1) return rows.sum(at::IntArrayRef{0}, /*keepdim=*/true);
  return rows;
}
// gradients as the backward kernels take them
Tensor token_grad(const Tensor& g, const Tensor& like) {
  return g.defined() ? g.to(like.scalar_type()).contiguous() : at::zeros_like(like);
}
OptTensor final_state_grad(const Tensor& g) {
  if (!g.defined()) return std::nullopt;
  return g.to(at::kFloat).contiguous();
}

typedef std::tuple<Tensor, Tensor, Tensor> Three;
typedef std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> Six;
typedef std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> Seven;

// a dispatcher call of one of the operators below (looked up once per place of call)
#define RWKV_OP(fn, name, ...)                                                                          \
  [&] {                                                                                                 \
    static const auto op =                                                                              \
        c10::Dispatcher::singleton().findSchemaOrThrow("rwkv_ops_b200::" name, "").typed<decltype(fn)>(); \
    return op.call(__VA_ARGS__);                                                                        \
  }()

void check_tokens(const Tensor& r, at::ArrayRef<const Tensor*> rest, int dims) {
  TORCH_CHECK_VALUE(r.is_cuda() && r.dim() == dims, "expected CUDA token tensors with ", dims, " dimensions");
  for (const Tensor* x : rest)
    TORCH_CHECK_VALUE(x->is_cuda() && x->device() == r.device() && x->sym_sizes() == r.sym_sizes(),
                      "token tensors must agree in shape and device");
}
void check_state(const OptTensor& s, const Tensor& r, const SymInt& B, const SymInt& H, const SymInt& N) {
  if (!has(s)) return;
  TORCH_CHECK_VALUE(s->is_cuda() && s->device() == r.device() && s->dim() == 4 && s->sym_size(1) == H && s->sym_size(2) == N &&
                        s->sym_size(3) == N && (s->sym_size(0) == 1 || s->sym_size(0) == B),
                    "initial_state must be [", B, " or 1, ", H, ", ", N, ", ", N, "], got ", s->sym_sizes());
}

// ---------------------------------------------------------------------------------------------
// RWKV7, dense
// ---------------------------------------------------------------------------------------------
struct Dims { int B, T, H, K; };
Dims dims_of(const Tensor& r, bool head_first) {
  const int T = head_first ? 2 : 1, H = head_first ? 1 : 2;
  return {(int)r.size(0), (int)r.size(T), (int)r.size(H), (int)r.size(3)};
}

struct SymDims { SymInt B, T, H, K; };
SymDims sym_dims_of(const Tensor& r, bool head_first) {
  const int T = head_first ? 2 : 1, H = head_first ? 1 : 2;
  return {r.sym_size(0), r.sym_size(T), r.sym_size(H), r.sym_size(3)};
}
// whether the tiles that a training forward would leave for its backward stay within the limit
bool keep_fits(const SymDims& d, int algo, const Tensor& r) {
  const auto n = [](const SymInt& x) { return (int)x.guard_int(__FILE__, __LINE__); };
  return rwkvb200_rwkv7_fwd_workspace_bytes(n(d.B), n(d.T), n(d.H), n(d.K), RWKVB200_BF16, algo | RWKVB200_ALGO_KEEP) <=
         keep_limit_bytes(r.device().index());
}

// The same for the states of the float32 recurrence over blocks (rwkvb200_rwkv7_states_bytes; none up to 16 tokens).  Sizes
// that are symbols stay symbols, without a guard: a traced program serves every length, and keeps the states where they fit
// at every length that it is declared for.
bool states_fit(const SymDims& d, const Tensor& r) {
  const auto limit = (int64_t)std::min<size_t>(keep_limit_bytes(r.device().index()), std::numeric_limits<int64_t>::max());
  return !TORCH_STATICALLY_KNOWN_TRUE(d.T.sym_le(16)) &&
         TORCH_STATICALLY_KNOWN_TRUE((d.B * d.H * ((d.T + 15) / 16 - 1) * d.K * d.K * 4).sym_le(limit));
}
// whether rwkv7_fwd / _bwd take the chunked path, whose kept tensor holds tiles; elsewhere it holds states
bool chunked_rwkv7(const Dims& d, int code, int64_t algo) {
  return d.K == HEAD && code == RWKVB200_BF16 && (algo & 0xff) != RWKVB200_ALGO_RECURRENT;
}

Three rwkv7_fwd(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b,
                const OptTensor& h0, bool head_first, int64_t algo, bool keep) {
  const c10::cuda::CUDAGuard guard(r.device());
  const Dims d = dims_of(r, head_first);
  const int code = dtype_code(r.scalar_type()), flags = (int)algo | (keep ? RWKVB200_ALGO_KEEP : 0);
  Tensor o = fresh_like(r), ht = fresh({d.B, d.H, d.K, d.K}, at::kFloat, r), ws;
  if (d.T == 1 && !(keep && chunked_rwkv7(d, code, algo))) {
    check(rwkvb200_rwkv7_step(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), fptr(h0), n_state_of(h0), fptr(ht), ptr(o),
                              d.B, d.H, d.K, code, stream_of(r)), "rwkv7_step");
  } else if (keep && !chunked_rwkv7(d, code, algo)) {
    const size_t n = rwkvb200_rwkv7_states_bytes(d.B, d.T, d.H, d.K, code, (int)algo);
    ws = bytes_if_any(n, r);      // (without them the backward sweeps forward once more)
    const Tensor scratch = bytes_if_any(rwkvb200_rwkv7_fwd_workspace_bytes(d.B, d.T, d.H, d.K, code, (int)algo), r);
    check(size_of(ws) ? rwkvb200_rwkv7_fwd_states(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), fptr(h0), n_state_of(h0), ptr(o),
                                                  fptr(ht), fptr(ws), n, ptr(scratch), size_of(scratch), d.B, d.T, d.H, d.K, code,
                                                  head_first, (int)algo, stream_of(r))
                      : rwkvb200_rwkv7_fwd(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), fptr(h0), n_state_of(h0), ptr(o), fptr(ht),
                                           ptr(scratch), size_of(scratch), d.B, d.T, d.H, d.K, code, head_first, (int)algo, stream_of(r)),
          "rwkv7_fwd");
  } else {
    const size_t nws = rwkvb200_rwkv7_fwd_workspace_bytes(d.B, d.T, d.H, d.K, code, flags);
    if (chunked_rwkv7(d, code, algo)) ws = bytes(nws, r);
    else                              ws = bytes_if_any(nws, r);
    check(rwkvb200_rwkv7_fwd(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), fptr(h0), n_state_of(h0), ptr(o), fptr(ht),
                             ptr(ws), size_of(ws), d.B, d.T, d.H, d.K, code, head_first, flags, stream_of(r)), "rwkv7_fwd");
  }
  return {o, ht, keep && ws.defined() ? ws : bytes(0, r)};
}

// `kept` (may be empty): what a forward with keep left; the tiles of the chunked path also serve as scratch, but what the
// forward left in it is not changed, so a second backward through the same graph stays legal.
Seven rwkv7_bwd(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b,
                const OptTensor& h0, const Tensor& d_o, const OptTensor& d_ht, const Tensor& kept, bool head_first,
                int64_t algo) {
  const c10::cuda::CUDAGuard guard(r.device());
  const Dims d = dims_of(r, head_first);
  const int code = dtype_code(r.scalar_type());
  const bool have = kept.numel() > 0;
  Tensor dr = fresh_like(r), dw = fresh_like(r), dk = fresh_like(r), dv = fresh_like(r), da = fresh_like(r),
         db = fresh_like(r), dh0 = fresh({d.B, d.H, d.K, d.K}, at::kFloat, r);
  if (have && !chunked_rwkv7(d, code, algo)) {
    Tensor ws = bytes_if_any(rwkvb200_rwkv7_bwd_states_workspace_bytes(d.B, d.T, d.H, d.K, code, (int)algo), r);
    if (!ws.defined()) ws = bytes((size_t)kept.numel(), r);      // what is needed: as much as the forward left
    check(rwkvb200_rwkv7_bwd_states(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), fptr(h0), n_state_of(h0), ptr(d_o),
                                    fptr(d_ht), fptr(kept), (size_t)kept.numel(), ptr(dr), ptr(dw), ptr(dk), ptr(dv), ptr(da), ptr(db), fptr(dh0),
                                    ptr(ws), size_of(ws), d.B, d.T, d.H, d.K, code, head_first, (int)algo, stream_of(r)), "rwkv7_bwd");
    return {dr, dw, dk, dv, da, db, dh0};
  }
  const size_t nws = rwkvb200_rwkv7_bwd_workspace_bytes(d.B, d.T, d.H, d.K, code, (int)algo);
  Tensor ws = have ? kept : chunked_rwkv7(d, code, algo) ? bytes(nws, r) : bytes_if_any(nws, r);
  if (nws && !ws.defined()) ws = bytes((size_t)d.B * d.H * ((d.T + 7) / 8) * d.K * d.K * sizeof(float) + 255, r);      // what is needed
  check(rwkvb200_rwkv7_bwd(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), fptr(h0), n_state_of(h0), ptr(d_o), fptr(d_ht),
                           ptr(dr), ptr(dw), ptr(dk), ptr(dv), ptr(da), ptr(db), fptr(dh0), ptr(ws), size_of(ws), d.B, d.T, d.H,
                           d.K, code, head_first, (int)algo | (have ? RWKVB200_ALGO_KEEP : 0), stream_of(r)),
        "rwkv7_bwd");
  return {dr, dw, dk, dv, da, db, dh0};
}

struct Rwkv7Fn : torch::autograd::Function<Rwkv7Fn> {
  static Vars forward(Ctx* ctx, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                      const Tensor& b, const OptTensor& h0, bool head_first, int64_t algo, bool keep) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, ht, kept] = RWKV_OP(rwkv7_fwd, "rwkv7_fwd", r, w, k, v, a, b, h0, head_first, algo, keep);
    ctx->save_for_backward({r, w, k, v, a, b, has(h0) ? *h0 : Tensor(), kept});
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({kept});
    ctx->saved_data["head_first"] = head_first;
    ctx->saved_data["algo"] = algo;
    return {o, ht, kept};
  }
  static Vars backward(Ctx* ctx, Vars g) {
    const Vars s = ctx->get_saved_variables();
    const OptTensor h0 = s[6].defined() ? OptTensor(s[6]) : std::nullopt;
    auto [dr, dw, dk, dv, da, db, dh0] =
        RWKV_OP(rwkv7_bwd, "rwkv7_bwd", s[0], s[1], s[2], s[3], s[4], s[5], h0, token_grad(g[0], s[0]),
                final_state_grad(g[1]), s[7], ctx->saved_data["head_first"].toBool(), ctx->saved_data["algo"].toInt());
    const Tensor ds = has(h0) && ctx->needs_input_grad(6) ? state_grad(dh0, h0) : Tensor();
    return {dr, dw, dk, dv, da, db, ds, Tensor(), Tensor(), Tensor()};
  }
};

Three rwkv7_fwd_autograd(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                         const Tensor& b, const OptTensor& h0, bool head_first, int64_t algo, bool keep) {
  if (any_requires_grad({&r, &w, &k, &v, &a, &b}, h0)) {
    Vars out = Rwkv7Fn::apply(r, w, k, v, a, b, h0, head_first, algo, keep);
    return {out[0], out[1], out[2]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return RWKV_OP(rwkv7_fwd, "rwkv7_fwd", r, w, k, v, a, b, h0, head_first, algo, keep);
}

std::tuple<Tensor, Tensor> generalized_delta_rule(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v,
                                                  const Tensor& a, const Tensor& b, const OptTensor& initial_state,
                                                  bool head_first) {
  check_tokens(r, {&w, &k, &v, &a, &b}, 4);
  const SymDims d = sym_dims_of(r, head_first);
  TORCH_CHECK_VALUE(d.K == 64 || d.K == 128, "head size must be 64 or 128, got ", d.K);
  check_state(initial_state, r, d.B, d.H, d.K);
  const int algo = algo_from_env("RWKV_OPS_B200_RWKV7_ALGO");
  // RWKV_OPS_B200_RWKV7_ALGO=chunked sends float32 / float16 tokens through the tensor-core path as bfloat16
  const at::ScalarType t = d.K == HEAD && algo == RWKVB200_ALGO_CHUNKED ? at::kBFloat16 : compute_dtype(r.scalar_type());
  const Tensor r_ = dense(r, t), w_ = dense(w, t), k_ = dense(k, t), v_ = dense(v, t), a_ = dense(a, t), b_ = dense(b, t);
  const OptTensor h0 = dense_state(initial_state);
  bool keep = false;
  if (any_requires_grad({&r_, &w_, &k_, &v_, &a_, &b_}, h0)) {
    if (t == at::kBFloat16 && d.K == HEAD)
      keep = d.T > 1 && algo != RWKVB200_ALGO_RECURRENT && keep_fits(d, algo, r);
    else
      keep = algo != RWKVB200_ALGO_CHUNKED && states_fit(d, r);
  }
  auto [o, ht, kept] = RWKV_OP(rwkv7_fwd, "rwkv7_fwd", r_, w_, k_, v_, a_, b_, h0, head_first, algo, keep);
  return {o.to(r.scalar_type()), ht};
}

// ---------------------------------------------------------------------------------------------
// RWKV7, one token in place on a resident state
// ---------------------------------------------------------------------------------------------
Tensor rwkv7_decode_step(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                         const Tensor& b, Tensor state) {
  check_tokens(r, {&w, &k, &v, &a, &b}, (int)r.dim());
  const int64_t B = state.size(0), H = state.size(1);
  TORCH_CHECK_VALUE((r.dim() == 3 || (r.dim() == 4 && r.size(1) == 1)) && r.size(0) == B && r.size(r.dim() - 2) == H &&
                        r.size(-1) == HEAD && state.is_contiguous() && state.device() == r.device(),
                    "expected token tensors [", B, ", 1, ", H, ", 64] or [", B, ", ", H, ", 64], got ", r.sizes());
  const c10::cuda::CUDAGuard guard(r.device());
  const at::ScalarType t = compute_dtype(r.scalar_type());
  const Tensor r_ = dense(r, t), w_ = dense(w, t), k_ = dense(k, t), v_ = dense(v, t), a_ = dense(a, t), b_ = dense(b, t);
  Tensor o = fresh_like(r_);
  check(rwkvb200_rwkv7_decode_step(ptr(r_), ptr(w_), ptr(k_), ptr(v_), ptr(a_), ptr(b_), ptr(state),
                                   dtype_code(state.scalar_type()), ptr(o), (int)B, (int)H, HEAD, dtype_code(t),
                                   stream_of(r)), "rwkv7_decode_step");
  return o.to(r.scalar_type());
}
// decoding is never differentiated
Tensor rwkv7_decode_step_autograd(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                                  const Tensor& b, Tensor state) {
  Tensor o;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    o = RWKV_OP(rwkv7_decode_step, "rwkv7_decode_step", r, w, k, v, a, b, state);
  }
  if (!state.is_inference()) state.unsafeGetTensorImpl()->bump_version();
  return o;
}

// ---------------------------------------------------------------------------------------------
// RWKV7, sequences packed end to end
// ---------------------------------------------------------------------------------------------
Three rwkv7_fwd_varlen(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                       const Tensor& b, const Tensor& seq_start, const Tensor& seq_len, int64_t max_len,
                       const OptTensor& h0, bool keep) {
  const c10::cuda::CUDAGuard guard(r.device());
  const int T = (int)r.size(1), H = (int)r.size(2), n_seq = (int)seq_start.numel();
  Tensor o = fresh_like(r), ht = fresh({n_seq, H, HEAD, HEAD}, at::kFloat, r);
  const size_t nws = rwkvb200_rwkv7_varlen_workspace_bytes(n_seq, (int)max_len, H, HEAD, keep);
  Tensor ws = bytes(nws, r);
  check(rwkvb200_rwkv7_fwd_varlen(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), seq_start.data_ptr<int32_t>(),
                                  seq_len.data_ptr<int32_t>(), n_seq, (int)max_len, T, fptr(h0), n_state_of(h0), ptr(o),
                                  fptr(ht), ptr(ws), nws, H, HEAD, dtype_code(r.scalar_type()), keep, stream_of(r)),
        "rwkv7_fwd_varlen");
  return {o, ht, keep ? ws : bytes(0, r)};
}

Seven rwkv7_bwd_varlen(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                       const Tensor& b, const Tensor& seq_start, const Tensor& seq_len, int64_t max_len,
                       const OptTensor& h0, const Tensor& d_o, const OptTensor& d_ht, const Tensor& kept) {
  const c10::cuda::CUDAGuard guard(r.device());
  const int T = (int)r.size(1), H = (int)r.size(2), n_seq = (int)seq_start.numel();
  Tensor dr = fresh_like(r), dw = fresh_like(r), dk = fresh_like(r), dv = fresh_like(r), da = fresh_like(r),
         db = fresh_like(r), dh0 = fresh({n_seq, H, HEAD, HEAD}, at::kFloat, r);
  const size_t nws = rwkvb200_rwkv7_varlen_workspace_bytes(n_seq, (int)max_len, H, HEAD, 1);
  const bool have = (size_t)kept.numel() >= nws;
  const Tensor ws = have ? kept : bytes(nws, r);
  check(rwkvb200_rwkv7_bwd_varlen(ptr(r), ptr(w), ptr(k), ptr(v), ptr(a), ptr(b), seq_start.data_ptr<int32_t>(),
                                  seq_len.data_ptr<int32_t>(), n_seq, (int)max_len, T, fptr(h0), n_state_of(h0), ptr(d_o),
                                  fptr(d_ht), ptr(dr), ptr(dw), ptr(dk), ptr(dv), ptr(da), ptr(db), fptr(dh0), ptr(ws),
                                  nws, H, HEAD, dtype_code(r.scalar_type()), have, stream_of(r)),
        "rwkv7_bwd_varlen");
  return {dr, dw, dk, dv, da, db, dh0};
}

struct Rwkv7VarlenFn : torch::autograd::Function<Rwkv7VarlenFn> {
  static Vars forward(Ctx* ctx, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                      const Tensor& b, const Tensor& seq_start, const Tensor& seq_len, int64_t max_len,
                      const OptTensor& h0, bool keep) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, ht, kept] =
        RWKV_OP(rwkv7_fwd_varlen, "rwkv7_fwd_varlen", r, w, k, v, a, b, seq_start, seq_len, max_len, h0, keep);
    ctx->save_for_backward({r, w, k, v, a, b, seq_start, seq_len, has(h0) ? *h0 : Tensor(), kept});
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({kept});
    ctx->saved_data["max_len"] = max_len;
    return {o, ht, kept};
  }
  static Vars backward(Ctx* ctx, Vars g) {
    const Vars s = ctx->get_saved_variables();
    const OptTensor h0 = s[8].defined() ? OptTensor(s[8]) : std::nullopt;
    auto [dr, dw, dk, dv, da, db, dh0] =
        RWKV_OP(rwkv7_bwd_varlen, "rwkv7_bwd_varlen", s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7],
                ctx->saved_data["max_len"].toInt(), h0, token_grad(g[0], s[0]), final_state_grad(g[1]), s[9]);
    const Tensor ds = has(h0) && ctx->needs_input_grad(8) ? state_grad(dh0, h0) : Tensor();
    return {dr, dw, dk, dv, da, db, Tensor(), Tensor(), Tensor(), ds, Tensor()};
  }
};

Three rwkv7_fwd_varlen_autograd(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                                const Tensor& b, const Tensor& seq_start, const Tensor& seq_len, int64_t max_len,
                                const OptTensor& h0, bool keep) {
  if (any_requires_grad({&r, &w, &k, &v, &a, &b}, h0)) {
    Vars out = Rwkv7VarlenFn::apply(r, w, k, v, a, b, seq_start, seq_len, max_len, h0, keep);
    return {out[0], out[1], out[2]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return RWKV_OP(rwkv7_fwd_varlen, "rwkv7_fwd_varlen", r, w, k, v, a, b, seq_start, seq_len, max_len, h0, keep);
}

std::tuple<Tensor, Tensor> rwkv7_varlen(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v,
                                        const Tensor& a, const Tensor& b, const Tensor& seq_start, const Tensor& seq_len,
                                        int64_t max_len, const OptTensor& initial_state) {
  check_tokens(r, {&w, &k, &v, &a, &b}, 4);
  TORCH_CHECK_VALUE(r.sym_size(0) == 1 && r.sym_size(3) == HEAD && r.scalar_type() == at::kBFloat16,
                    "expected packed bfloat16 token tensors [1, total_len, H, 64], got ", r.sym_sizes());
  check_state(initial_state, r, seq_start.sym_numel(), r.sym_size(2), HEAD);
  const at::ScalarType t = at::kBFloat16;
  const Tensor r_ = dense(r, t), w_ = dense(w, t), k_ = dense(k, t), v_ = dense(v, t), a_ = dense(a, t), b_ = dense(b, t);
  const OptTensor h0 = dense_state(initial_state);
  const bool keep = any_requires_grad({&r_, &w_, &k_, &v_, &a_, &b_}, h0);
  auto [o, ht, kept] =
      RWKV_OP(rwkv7_fwd_varlen, "rwkv7_fwd_varlen", r_, w_, k_, v_, a_, b_, seq_start, seq_len, max_len, h0, keep);
  return {o, ht};
}

// ---------------------------------------------------------------------------------------------
// RWKV7 with the producers of w, a, b fused in
// ---------------------------------------------------------------------------------------------
Three rwkv7_fused_fwd(const Tensor& r, const Tensor& w_pre, const Tensor& k, const Tensor& v, const Tensor& kk_pre,
                      const Tensor& a_pre, const OptTensor& h0, bool keep) {
  const c10::cuda::CUDAGuard guard(r.device());
  const Dims d = dims_of(r, false);
  Tensor o = fresh_like(r), ht = fresh({d.B, d.H, d.K, d.K}, at::kFloat, r);
  const size_t nws = rwkvb200_rwkv7_fwd_workspace_bytes(d.B, d.T, d.H, d.K, RWKVB200_BF16,
                                                        RWKVB200_ALGO_CHUNKED | (keep ? RWKVB200_ALGO_KEEP : 0));
  Tensor ws = bytes(nws, r);
  check(rwkvb200_rwkv7_fused_fwd(ptr(r), ptr(w_pre), ptr(k), ptr(v), ptr(kk_pre), ptr(a_pre), fptr(h0), n_state_of(h0),
                                 ptr(o), fptr(ht), ptr(ws), nws, d.B, d.T, d.H, d.K, RWKVB200_BF16, keep, stream_of(r)),
        "rwkv7_fused_fwd");
  return {o, ht, keep ? ws : bytes(0, r)};
}

Seven rwkv7_fused_bwd(const Tensor& r, const Tensor& w_pre, const Tensor& k, const Tensor& v, const Tensor& kk_pre,
                      const Tensor& a_pre, const OptTensor& h0, const Tensor& d_o, const OptTensor& d_ht,
                      const Tensor& kept) {
  const c10::cuda::CUDAGuard guard(r.device());
  const Dims d = dims_of(r, false);
  Tensor dr = fresh_like(r), dw = fresh_like(r), dk = fresh_like(r), dv = fresh_like(r), du = fresh_like(r),
         dq = fresh_like(r), dh0 = fresh({d.B, d.H, d.K, d.K}, at::kFloat, r);
  const size_t nws = rwkvb200_rwkv7_bwd_workspace_bytes(d.B, d.T, d.H, d.K, RWKVB200_BF16, RWKVB200_ALGO_CHUNKED);
  const bool have = (size_t)kept.numel() >= nws;
  const Tensor ws = have ? kept : bytes(nws, r);
  check(rwkvb200_rwkv7_fused_bwd(ptr(r), ptr(w_pre), ptr(k), ptr(v), ptr(kk_pre), ptr(a_pre), fptr(h0), n_state_of(h0),
                                 ptr(d_o), fptr(d_ht), ptr(dr), ptr(dw), ptr(dk), ptr(dv), ptr(du), ptr(dq), fptr(dh0),
                                 ptr(ws), nws, d.B, d.T, d.H, d.K, RWKVB200_BF16, have, stream_of(r)),
        "rwkv7_fused_bwd");
  return {dr, dw, dk, dv, du, dq, dh0};
}

struct Rwkv7FusedFn : torch::autograd::Function<Rwkv7FusedFn> {
  static Vars forward(Ctx* ctx, const Tensor& r, const Tensor& w_pre, const Tensor& k, const Tensor& v,
                      const Tensor& kk_pre, const Tensor& a_pre, const OptTensor& h0, bool keep) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, ht, kept] = RWKV_OP(rwkv7_fused_fwd, "rwkv7_fused_fwd", r, w_pre, k, v, kk_pre, a_pre, h0, keep);
    ctx->save_for_backward({r, w_pre, k, v, kk_pre, a_pre, has(h0) ? *h0 : Tensor(), kept});
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({kept});
    return {o, ht, kept};
  }
  static Vars backward(Ctx* ctx, Vars g) {
    const Vars s = ctx->get_saved_variables();
    const OptTensor h0 = s[6].defined() ? OptTensor(s[6]) : std::nullopt;
    auto [dr, dw, dk, dv, du, dq, dh0] = RWKV_OP(rwkv7_fused_bwd, "rwkv7_fused_bwd", s[0], s[1], s[2], s[3], s[4], s[5], h0,
                                                 token_grad(g[0], s[0]), final_state_grad(g[1]), s[7]);
    const Tensor ds = has(h0) && ctx->needs_input_grad(6) ? state_grad(dh0, h0) : Tensor();
    return {dr, dw, dk, dv, du, dq, ds, Tensor()};
  }
};

Three rwkv7_fused_fwd_autograd(const Tensor& r, const Tensor& w_pre, const Tensor& k, const Tensor& v,
                               const Tensor& kk_pre, const Tensor& a_pre, const OptTensor& h0, bool keep) {
  if (any_requires_grad({&r, &w_pre, &k, &v, &kk_pre, &a_pre}, h0)) {
    Vars out = Rwkv7FusedFn::apply(r, w_pre, k, v, kk_pre, a_pre, h0, keep);
    return {out[0], out[1], out[2]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return RWKV_OP(rwkv7_fused_fwd, "rwkv7_fused_fwd", r, w_pre, k, v, kk_pre, a_pre, h0, keep);
}

std::tuple<Tensor, Tensor> rwkv7_fused(const Tensor& r, const Tensor& w_pre, const Tensor& k, const Tensor& v,
                                       const Tensor& kk_pre, const Tensor& a_pre, const OptTensor& initial_state) {
  check_tokens(r, {&w_pre, &k, &v, &kk_pre, &a_pre}, 4);
  const SymDims d = sym_dims_of(r, false);
  TORCH_CHECK_VALUE(d.K == HEAD, "head size must be 64, got ", d.K);
  check_state(initial_state, r, d.B, d.H, d.K);
  const Tensor r_ = r.contiguous(), w_ = w_pre.contiguous(), k_ = k.contiguous(), v_ = v.contiguous(),
               u_ = kk_pre.contiguous(), q_ = a_pre.contiguous();
  const OptTensor h0 = dense_state(initial_state);
  const bool keep = any_requires_grad({&r_, &w_, &k_, &v_, &u_, &q_}, h0) && keep_fits(d, RWKVB200_ALGO_CHUNKED, r);
  auto [o, ht, kept] = RWKV_OP(rwkv7_fused_fwd, "rwkv7_fused_fwd", r_, w_, k_, v_, u_, q_, h0, keep);
  return {o, ht};
}

// ---------------------------------------------------------------------------------------------
// RWKV6 wkv, dense
// ---------------------------------------------------------------------------------------------
// x itself if its first element is 16-byte aligned (what the C ABI asks for), else a copy
Tensor aligned(const Tensor& x) { return reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 ? x.clone() : x; }

Three wkv6_fwd(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u, const OptTensor& s0,
               const OptTensor& state_map, int64_t algo, bool keep) {
  const c10::cuda::CUDAGuard guard(r.device());
  const int B = (int)r.size(0), T = (int)r.size(1), H = (int)u.size(0), N = (int)u.size(1);
  const int code = dtype_code(r.scalar_type()), flags = (int)algo | (keep ? RWKVB200_ALGO_KEEP : 0);
  Tensor y = fresh_like(r), sT = fresh({B, H, N, N}, algo & RWKVB200_ALGO_TOKEN_STATES ? r.scalar_type() : at::kFloat, r);
  // states and u in the token dtype come as the caller holds them, e.g. as a view into a larger buffer
  const bool typed = algo & RWKVB200_ALGO_TOKEN_STATES;
  const Tensor u_ = typed ? aligned(u) : u;
  const OptTensor s0_ = typed && has(s0) ? OptTensor(aligned(*s0)) : s0;
  // a training forward of the chunked path leaves the chunk-boundary states for the backward
  const size_t nws = rwkvb200_wkv6_fwd_workspace_bytes(B, T, H, N, code, flags);
  Tensor ws = bytes(nws, r);
  check(rwkvb200_wkv6_fwd(ptr(r), ptr(k), ptr(v), ptr(w), ptr(u_), ptr(s0_), n_state_of(s0), iptr(state_map), ptr(y),
                          ptr(sT), nws ? ptr(ws) : nullptr, nws, B, T, H, N, code, flags, stream_of(r)), "wkv6_fwd");
  return {y, sT, keep ? ws : bytes(0, r)};
}

Six wkv6_bwd(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u, const OptTensor& s0,
             const OptTensor& state_map, const Tensor& d_y, const OptTensor& d_sT, const Tensor& kept, int64_t algo) {
  const c10::cuda::CUDAGuard guard(r.device());
  const int B = (int)r.size(0), T = (int)r.size(1), H = (int)u.size(0), N = (int)u.size(1);
  const int code = dtype_code(r.scalar_type());
  Tensor dr = fresh_like(r), dk = fresh_like(r), dv = fresh_like(r), dw = fresh_like(r), du = fresh_like(u),
         ds0 = fresh({B, H, N, N}, at::kFloat, r);
  const size_t nws = rwkvb200_wkv6_bwd_workspace_bytes(B, T, H, N, code, (int)algo);
  const bool have = kept.numel() > 0 && (size_t)kept.numel() >= nws;
  const Tensor ws = have ? kept : bytes(nws, r);
  check(rwkvb200_wkv6_bwd(ptr(r), ptr(k), ptr(v), ptr(w), fptr(u), fptr(s0), n_state_of(s0), iptr(state_map), ptr(d_y),
                          fptr(d_sT), ptr(dr), ptr(dk), ptr(dv), ptr(dw), fptr(du), fptr(ds0), ptr(ws), nws, B, T, H, N,
                          code, (int)algo | (have ? RWKVB200_ALGO_KEEP : 0), stream_of(r)), "wkv6_bwd");
  return {dr, dk, dv, dw, du, ds0};
}

// gradient of the state table: rows that started from the same table row add up
Tensor table_grad(const Tensor& rows, const Tensor& s0, const OptTensor& state_map) {
  if (has(state_map)) return at::zeros_like(s0).index_add_(0, state_map->to(at::kLong), rows);
  return state_grad(rows, s0);
}

struct Wkv6Fn : torch::autograd::Function<Wkv6Fn> {
  static Vars forward(Ctx* ctx, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                      const OptTensor& s0, const OptTensor& state_map, int64_t algo, bool keep) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [y, sT, kept] = RWKV_OP(wkv6_fwd, "wkv6_fwd", r, k, v, w, u, s0, state_map, algo, keep);
    ctx->save_for_backward({r, k, v, w, u, has(s0) ? *s0 : Tensor(), has(state_map) ? *state_map : Tensor(), kept});
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({kept});
    ctx->saved_data["algo"] = algo;
    return {y, sT, kept};
  }
  static Vars backward(Ctx* ctx, Vars g) {
    const Vars s = ctx->get_saved_variables();
    const OptTensor s0 = s[5].defined() ? OptTensor(s[5]) : std::nullopt,
                    map = s[6].defined() ? OptTensor(s[6]) : std::nullopt;
    auto [dr, dk, dv, dw, du, rows] =
        RWKV_OP(wkv6_bwd, "wkv6_bwd", s[0], s[1], s[2], s[3], s[4], s0, map, token_grad(g[0], s[0]),
                final_state_grad(g[1]), s[7], ctx->saved_data["algo"].toInt());
    const Tensor ds = has(s0) && ctx->needs_input_grad(5) ? table_grad(rows, *s0, map) : Tensor();
    return {dr, dk, dv, dw, du, ds, Tensor(), Tensor(), Tensor()};
  }
};

Three wkv6_fwd_autograd(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                        const OptTensor& s0, const OptTensor& state_map, int64_t algo, bool keep) {
  if (any_requires_grad({&r, &k, &v, &w, &u}, s0)) {
    Vars out = Wkv6Fn::apply(r, k, v, w, u, s0, state_map, algo, keep);
    return {out[0], out[1], out[2]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return RWKV_OP(wkv6_fwd, "wkv6_fwd", r, k, v, w, u, s0, state_map, algo, keep);
}

// what the two wkv6 operators check and convert alike; `rows` is the batch size or the number of sequences
struct Wkv6Args {
  Tensor r, k, v, w, u;
  OptTensor s0, map;
};
Wkv6Args wkv6_args(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u, int64_t N,
                   const SymInt& rows, const OptTensor& init_state, const OptTensor& state_map, bool typed = false) {
  check_tokens(r, {&k, &v, &w}, 3);
  const SymInt C = r.sym_size(2), H = C / N;
  const at::ScalarType dt = r.scalar_type(), t = compute_dtype(dt);
  TORCH_CHECK_VALUE(C % N == 0 && u.is_cuda() && u.device() == r.device() && u.sym_numel() == C && k.scalar_type() == dt &&
                        v.scalar_type() == dt && w.scalar_type() == dt, "r, k, v, w, u do not agree");
  Wkv6Args x;
  if (has(init_state)) {
    const Tensor s = init_state->dim() == 3 ? init_state->unsqueeze(0) : *init_state;
    TORCH_CHECK_VALUE(s.is_cuda() && s.device() == r.device() && s.dim() == 4 && s.sym_size(1) == H &&
                          s.sym_size(2) == N && s.sym_size(3) == N, "init_state must be [n_state, ", H, ", ", N, ", ", N, "]");
    if (has(state_map)) {
      TORCH_CHECK_VALUE(state_map->is_cuda() && state_map->sym_numel() == rows &&
                            (state_map->scalar_type() == at::kInt || state_map->scalar_type() == at::kLong),
                        "state_map must hold one int32 or int64 entry per row");
      x.map = state_map->to(r.device(), at::kInt).contiguous().view(-1);
    } else {
      TORCH_CHECK_VALUE(s.sym_size(0) == 1 || s.sym_size(0) == rows,
                        "state_map cannot be inferred from init_state; pass it explicitly");
    }
    x.s0 = typed ? s.contiguous() : s.to(at::kFloat).contiguous();
  } else {
    TORCH_CHECK_VALUE(!has(state_map), "state_map needs init_state");
  }
  x.r = dense(r, t); x.k = dense(k, t); x.v = dense(v, t); x.w = dense(w, t);
  x.u = u.reshape_symint({H, N});
  x.u = typed ? x.u.contiguous() : x.u.to(at::kFloat).contiguous();
  return x;
}
// the dtype of the states an operator hands to its caller
at::ScalarType state_dtype(at::ScalarType t) { return t == at::kHalf ? at::kFloat : t; }

std::tuple<Tensor, Tensor> wkv6(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                                int64_t head_size, const OptTensor& init_state, const OptTensor& state_map,
                                bool with_state) {
  TORCH_CHECK_VALUE(r.dim() == 3, "expected [B, T, C] tensors, got ", r.sym_sizes());
  // bfloat16 states outside training are read and written as they are: each conversion would be a launch of its own
  const bool typed = r.scalar_type() == at::kBFloat16 && u.scalar_type() == at::kBFloat16 &&
                     (!has(init_state) || init_state->scalar_type() == at::kBFloat16) &&
                     !any_requires_grad({&r, &k, &v, &w, &u}, init_state);
  const Wkv6Args x = wkv6_args(r, k, v, w, u, head_size, r.sym_size(0), init_state, state_map, typed);
  int algo = algo_from_env("RWKV_OPS_B200_WKV6_ALGO");
  if (head_size != HEAD) {
    TORCH_CHECK_VALUE(algo != RWKVB200_ALGO_CHUNKED, "the chunked wkv6 path is built for head size 64");
    algo = RWKVB200_ALGO_RECURRENT;
  }
  const bool keep = algo != RWKVB200_ALGO_RECURRENT && r.sym_size(1) > 1 &&
                    any_requires_grad({&x.r, &x.k, &x.v, &x.w, &x.u}, x.s0);
  if (typed) algo |= RWKVB200_ALGO_TOKEN_STATES;
  auto [y, sT, kept] = RWKV_OP(wkv6_fwd, "wkv6_fwd", x.r, x.k, x.v, x.w, x.u, x.s0, x.map, algo, keep);
  return {y.to(r.scalar_type()), with_state ? sT.to(state_dtype(r.scalar_type())) : sT};
}

// ---------------------------------------------------------------------------------------------
// RWKV6 wkv, sequences packed end to end
// ---------------------------------------------------------------------------------------------
Three wkv6_fwd_varlen(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                      const Tensor& seq_start, const Tensor& seq_len, int64_t max_len, const OptTensor& s0,
                      const OptTensor& state_map, bool keep) {
  const c10::cuda::CUDAGuard guard(r.device());
  const int T = (int)r.size(1), H = (int)u.size(0), N = (int)u.size(1), n_seq = (int)seq_start.numel();
  const int code = dtype_code(r.scalar_type());
  Tensor y = fresh_like(r), sT = fresh({n_seq, H, N, N}, at::kFloat, r);
  const size_t nws = rwkvb200_wkv6_varlen_workspace_bytes(n_seq, (int)max_len, H, N, code, keep);
  Tensor ws = bytes(nws, r);
  check(rwkvb200_wkv6_fwd_varlen(ptr(r), ptr(k), ptr(v), ptr(w), fptr(u), seq_start.data_ptr<int32_t>(),
                                 seq_len.data_ptr<int32_t>(), n_seq, (int)max_len, T, fptr(s0), n_state_of(s0),
                                 iptr(state_map), ptr(y), fptr(sT), ptr(ws), nws, H, N, code, keep, stream_of(r)),
        "wkv6_fwd_varlen");
  return {y, sT, keep ? ws : bytes(0, r)};
}

Six wkv6_bwd_varlen(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                    const Tensor& seq_start, const Tensor& seq_len, int64_t max_len, const OptTensor& s0,
                    const OptTensor& state_map, const Tensor& d_y, const OptTensor& d_sT, const Tensor& kept) {
  const c10::cuda::CUDAGuard guard(r.device());
  const int T = (int)r.size(1), H = (int)u.size(0), N = (int)u.size(1), n_seq = (int)seq_start.numel();
  const int code = dtype_code(r.scalar_type());
  Tensor dr = fresh_like(r), dk = fresh_like(r), dv = fresh_like(r), dw = fresh_like(r), du = fresh_like(u),
         ds0 = fresh({n_seq, H, N, N}, at::kFloat, r);
  const size_t nws = rwkvb200_wkv6_varlen_workspace_bytes(n_seq, (int)max_len, H, N, code, 1);
  const bool have = (size_t)kept.numel() >= nws;
  const Tensor ws = have ? kept : bytes(nws, r);
  check(rwkvb200_wkv6_bwd_varlen(ptr(r), ptr(k), ptr(v), ptr(w), fptr(u), seq_start.data_ptr<int32_t>(),
                                 seq_len.data_ptr<int32_t>(), n_seq, (int)max_len, T, fptr(s0), n_state_of(s0),
                                 iptr(state_map), ptr(d_y), fptr(d_sT), ptr(dr), ptr(dk), ptr(dv), ptr(dw), fptr(du),
                                 fptr(ds0), ptr(ws), nws, H, N, code, have, stream_of(r)), "wkv6_bwd_varlen");
  return {dr, dk, dv, dw, du, ds0};
}

struct Wkv6VarlenFn : torch::autograd::Function<Wkv6VarlenFn> {
  static Vars forward(Ctx* ctx, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                      const Tensor& seq_start, const Tensor& seq_len, int64_t max_len, const OptTensor& s0,
                      const OptTensor& state_map, bool keep) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [y, sT, kept] =
        RWKV_OP(wkv6_fwd_varlen, "wkv6_fwd_varlen", r, k, v, w, u, seq_start, seq_len, max_len, s0, state_map, keep);
    ctx->save_for_backward({r, k, v, w, u, seq_start, seq_len, has(s0) ? *s0 : Tensor(),
                            has(state_map) ? *state_map : Tensor(), kept});
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({kept});
    ctx->saved_data["max_len"] = max_len;
    return {y, sT, kept};
  }
  static Vars backward(Ctx* ctx, Vars g) {
    const Vars s = ctx->get_saved_variables();
    const OptTensor s0 = s[7].defined() ? OptTensor(s[7]) : std::nullopt,
                    map = s[8].defined() ? OptTensor(s[8]) : std::nullopt;
    auto [dr, dk, dv, dw, du, rows] =
        RWKV_OP(wkv6_bwd_varlen, "wkv6_bwd_varlen", s[0], s[1], s[2], s[3], s[4], s[5], s[6],
                ctx->saved_data["max_len"].toInt(), s0, map, token_grad(g[0], s[0]), final_state_grad(g[1]), s[9]);
    const Tensor ds = has(s0) && ctx->needs_input_grad(7) ? table_grad(rows, *s0, map) : Tensor();
    return {dr, dk, dv, dw, du, Tensor(), Tensor(), Tensor(), ds, Tensor(), Tensor()};
  }
};

Three wkv6_fwd_varlen_autograd(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                               const Tensor& seq_start, const Tensor& seq_len, int64_t max_len, const OptTensor& s0,
                               const OptTensor& state_map, bool keep) {
  if (any_requires_grad({&r, &k, &v, &w, &u}, s0)) {
    Vars out = Wkv6VarlenFn::apply(r, k, v, w, u, seq_start, seq_len, max_len, s0, state_map, keep);
    return {out[0], out[1], out[2]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return RWKV_OP(wkv6_fwd_varlen, "wkv6_fwd_varlen", r, k, v, w, u, seq_start, seq_len, max_len, s0, state_map, keep);
}

std::tuple<Tensor, Tensor> wkv6_varlen(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w,
                                       const Tensor& u, const Tensor& seq_start, const Tensor& seq_len, int64_t max_len,
                                       const OptTensor& init_state, const OptTensor& state_map) {
  TORCH_CHECK_VALUE(r.dim() == 3 && r.sym_size(0) == 1, "expected packed token tensors [1, total_len, H*64], got ", r.sym_sizes());
  const Wkv6Args x = wkv6_args(r, k, v, w, u, HEAD, seq_start.sym_numel(), init_state, state_map);
  const bool keep = any_requires_grad({&x.r, &x.k, &x.v, &x.w, &x.u}, x.s0);
  auto [y, sT, kept] = RWKV_OP(wkv6_fwd_varlen, "wkv6_fwd_varlen", x.r, x.k, x.v, x.w, x.u, seq_start, seq_len, max_len,
                               x.s0, x.map, keep);
  return {y.to(r.scalar_type()), sT.to(state_dtype(r.scalar_type()))};
}

// ---------------------------------------------------------------------------------------------
// the backward operators under autograd: a gradient can be asked for with create_graph, but differentiating it again is an
// error, not a silent zero
// ---------------------------------------------------------------------------------------------
constexpr char RWKV7_BWD[] = "rwkv_ops_b200::rwkv7_bwd", RWKV7_BWD_VARLEN[] = "rwkv_ops_b200::rwkv7_bwd_varlen",
               RWKV7_FUSED_BWD[] = "rwkv_ops_b200::rwkv7_fused_bwd", WKV6_BWD[] = "rwkv_ops_b200::wkv6_bwd",
               WKV6_BWD_VARLEN[] = "rwkv_ops_b200::wkv6_bwd_varlen";

void differentiable_inputs(Vars& to, const Tensor& x) { if (x.defined() && x.requires_grad()) to.push_back(x); }
void differentiable_inputs(Vars& to, const OptTensor& x) { if (has(x)) differentiable_inputs(to, *x); }
template <typename X> void differentiable_inputs(Vars&, const X&) {}

template <const char* NAME, auto F> struct Gradient;
template <const char* NAME, typename R, typename... A, R (*F)(A...)>
struct Gradient<NAME, F> {
  static R call(A... args) {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow(NAME, "").template typed<R(A...)>();
    Vars from;
    if (at::GradMode::is_enabled()) (differentiable_inputs(from, args), ...);
    R out = [&] {
      at::AutoDispatchBelowADInplaceOrView below;
      return op.call(args...);
    }();
    if (!from.empty()) {
      auto node = std::make_shared<torch::autograd::NotImplemented>(NAME);
      node->set_next_edges(torch::autograd::collect_next_edges(from));
      std::apply([&](auto&... x) { (torch::autograd::set_history(x, node), ...); }, out);
    }
    return out;
  }
};

}  // namespace

TORCH_LIBRARY(rwkv_ops_b200, m) {
#define SIX "Tensor r, Tensor w, Tensor k, Tensor v, Tensor a, Tensor b"
#define FUSED_SIX "Tensor r, Tensor w_pre, Tensor k, Tensor v, Tensor kk_pre, Tensor a_pre"
#define FIVE "Tensor r, Tensor k, Tensor v, Tensor w, Tensor u"
#define SEQS "Tensor seq_start, Tensor seq_len, int max_len"
#define OUT6 "(Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)"
#define OUT7 "(Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)"
  m.def("generalized_delta_rule(" SIX ", Tensor? initial_state, bool head_first) -> (Tensor, Tensor)", generalized_delta_rule);
  m.def("rwkv7_fwd(" SIX ", Tensor? h0, bool head_first, int algo, bool keep) -> (Tensor, Tensor, Tensor)");
  m.def("rwkv7_bwd(" SIX ", Tensor? h0, Tensor d_o, Tensor? d_ht, Tensor kept, bool head_first, int algo) -> " OUT7);
  m.def("rwkv7_decode_step(" SIX ", Tensor(a!) state) -> Tensor");
  m.def("rwkv7_varlen(" SIX ", " SEQS ", Tensor? initial_state) -> (Tensor, Tensor)", rwkv7_varlen);
  m.def("rwkv7_fwd_varlen(" SIX ", " SEQS ", Tensor? h0, bool keep) -> (Tensor, Tensor, Tensor)");
  m.def("rwkv7_bwd_varlen(" SIX ", " SEQS ", Tensor? h0, Tensor d_o, Tensor? d_ht, Tensor kept) -> " OUT7);
  m.def("rwkv7_fused(" FUSED_SIX ", Tensor? initial_state) -> (Tensor, Tensor)", rwkv7_fused);
  m.def("rwkv7_fused_fwd(" FUSED_SIX ", Tensor? h0, bool keep) -> (Tensor, Tensor, Tensor)");
  m.def("rwkv7_fused_bwd(" FUSED_SIX ", Tensor? h0, Tensor d_o, Tensor? d_ht, Tensor kept) -> " OUT7);
  m.def("wkv6(" FIVE ", int head_size, Tensor? init_state, Tensor? state_map, bool with_state) -> (Tensor, Tensor)", wkv6);
  m.def("wkv6_fwd(" FIVE ", Tensor? s0, Tensor? state_map, int algo, bool keep) -> (Tensor, Tensor, Tensor)");
  m.def("wkv6_bwd(" FIVE ", Tensor? s0, Tensor? state_map, Tensor d_y, Tensor? d_sT, Tensor kept, int algo) -> " OUT6);
  m.def("wkv6_varlen(" FIVE ", " SEQS ", Tensor? init_state, Tensor? state_map) -> (Tensor, Tensor)", wkv6_varlen);
  m.def("wkv6_fwd_varlen(" FIVE ", " SEQS ", Tensor? s0, Tensor? state_map, bool keep) -> (Tensor, Tensor, Tensor)");
  m.def("wkv6_bwd_varlen(" FIVE ", " SEQS ", Tensor? s0, Tensor? state_map, Tensor d_y, Tensor? d_sT, Tensor kept) -> " OUT6);
}

TORCH_LIBRARY_IMPL(rwkv_ops_b200, CUDA, m) {
  m.impl("rwkv7_fwd", rwkv7_fwd);
  m.impl("rwkv7_bwd", rwkv7_bwd);
  m.impl("rwkv7_decode_step", rwkv7_decode_step);
  m.impl("rwkv7_fwd_varlen", rwkv7_fwd_varlen);
  m.impl("rwkv7_bwd_varlen", rwkv7_bwd_varlen);
  m.impl("rwkv7_fused_fwd", rwkv7_fused_fwd);
  m.impl("rwkv7_fused_bwd", rwkv7_fused_bwd);
  m.impl("wkv6_fwd", wkv6_fwd);
  m.impl("wkv6_bwd", wkv6_bwd);
  m.impl("wkv6_fwd_varlen", wkv6_fwd_varlen);
  m.impl("wkv6_bwd_varlen", wkv6_bwd_varlen);
}

TORCH_LIBRARY_IMPL(rwkv_ops_b200, Autograd, m) {
  m.impl("rwkv7_fwd", rwkv7_fwd_autograd);
  m.impl("rwkv7_decode_step", rwkv7_decode_step_autograd);
  m.impl("rwkv7_fwd_varlen", rwkv7_fwd_varlen_autograd);
  m.impl("rwkv7_fused_fwd", rwkv7_fused_fwd_autograd);
  m.impl("wkv6_fwd", wkv6_fwd_autograd);
  m.impl("wkv6_fwd_varlen", wkv6_fwd_varlen_autograd);
  m.impl("rwkv7_bwd", Gradient<RWKV7_BWD, rwkv7_bwd>::call);
  m.impl("rwkv7_bwd_varlen", Gradient<RWKV7_BWD_VARLEN, rwkv7_bwd_varlen>::call);
  m.impl("rwkv7_fused_bwd", Gradient<RWKV7_FUSED_BWD, rwkv7_fused_bwd>::call);
  m.impl("wkv6_bwd", Gradient<WKV6_BWD, wkv6_bwd>::call);
  m.impl("wkv6_bwd_varlen", Gradient<WKV6_BWD_VARLEN, wkv6_bwd_varlen>::call);
}
