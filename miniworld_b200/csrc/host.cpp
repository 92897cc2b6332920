// Host side of the module calls in native code: argument checks, workspace and output allocation, the call of the C ABI on
// the current stream, and the autograd nodes of the training path.
//
// What bounds a small call is the host: at N = 64 the kernels of a forward take 22 us, and checking and collecting its
// arguments in Python took 59; a training step at N = 384 took 450 us of host time beside 370 us of kernels, 64 of them in
// the C ABI. Here one call does it all (and a backward runs on the autograd thread without the interpreter).
// Results and scratch come from the allocator without the dispatcher, and a module's registered parameters are looked up here:
// a training step of a small pair 174 -> 163 us of host time, a Transition 17.2 -> 14.6.
//
// Every function first looks whether the call is an ordinary one (plain dense CUDA tensors of the expected types and shapes
// on one device, boolean masks). If it is not, it answers None and changes nothing: the caller then takes the general
// Python path, which converts what can be converted and says what is wrong with the rest.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <array>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/b200_trimul.h"

// The parameters of a call, in Python a list of tensors or a pair (a module's _modules, ((child, name), ...)) that names the
// registered parameters `child.name`. One that is not there under its name (its child was wrapped or re-parametrised) leaves the
// list empty, which no ordinary call has.
struct CallParams {
  std::vector<at::Tensor> list;
};

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

void check(int rc, const char* what) {
  if (rc == B200_TRIMUL_OK) return;
  std::string s = std::string(what) + ": " + b200_trimul_strerror(rc) + " [" + std::to_string(rc) + "]";
  if (rc == B200_TRIMUL_E_CUDA) s += " (cuda error " + std::to_string(b200_trimul_last_cuda_error()) + ")";
  throw std::runtime_error(s);
}

// a dense CUDA tensor with storage of its own that no transform or dispatch mode wraps
bool plain(const Tensor& t) {
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.is_conj() || t.is_neg()) return false;
  const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                     c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize});
  return !t.key_set().has_any(wrapped) && t.is_contiguous();
}
bool plain_on(const Tensor& t, const Tensor& like, c10::ScalarType type, at::IntArrayRef shape) {
  return plain(t) && t.device() == like.device() && t.scalar_type() == type && t.sizes() == shape;
}
bool aligned16(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

// Memory for a result or scratch on the device of `like`, from the caching allocator without the dispatcher (0.7 instead of 1.5
// us each; a forward allocates one tensor, a backward twelve). All of it is overwritten. A dispatch mode sees its allocations: under
// one that hands out tensors without memory (fake tensors) a call has to fail at the C entry and not run for real.
Tensor empty_on(at::IntArrayRef shape, c10::ScalarType type, const Tensor& like) {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return at::empty(shape, at::device(like.device()).dtype(type));
  return Tensor(at::detail::empty_cuda(shape, type, like.device(), std::nullopt));
}
Tensor aligned_empty(size_t bytes, const Tensor& like) {
  const Tensor raw = empty_on({static_cast<int64_t>(bytes) + 1024}, at::kByte, like);
  const int64_t off = (1024 - reinterpret_cast<uintptr_t>(raw.data_ptr()) % 1024) % 1024;
  return raw.narrow(0, off, static_cast<int64_t>(bytes));
}
// scratch of one call: memory that holds `bytes` bytes from a 1024-byte boundary on
uint8_t* aligned_start(const Tensor& raw) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw.data_ptr()) + 1023) / 1024 * 1024);
}
Tensor scratch_for(size_t bytes, const Tensor& like) { return empty_on({static_cast<int64_t>(bytes) + 1024}, at::kByte, like); }
size_t scratch_bytes(const Tensor& raw) { return static_cast<size_t>(raw.numel()) - 1024; }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
const void* ptr(const OptTensor& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }

// ------------------------------------------------------------------------------------------ triangle update
// parameters in the order of the module's state: ln_pair weight, bias, to_left, to_left_gate, to_right, to_right_gate,
// ln_out weight, bias, to_gate, to_out
enum { kLnInW, kLnInB, kLeft, kLeftGate, kRight, kRightGate, kLnOutW, kLnOutB, kGate, kOut, kTriParams };

struct TriCall {
  int B, N, d_pair, d_hidden, direction;
  int wide;  // contracted channels in total
  float eps_in, eps_out;
  bool residual, any_n;
  int dtype;
  // The C entry points below are the ones whose intermediates have rows of whole lines, for every N; any_n says which lengths and
  // gradients are taken and which entry point of the general path refuses what they refuse.
  int sized_n() const { return (N + 7) / 8 * 8; }
};

bool fill_call(TriCall& c, const Tensor& z, at::TensorList p, const OptTensor& token_mask,
               const OptTensor& pair_mask, const OptTensor& drop_scale, int64_t d_pair, int64_t direction, double eps_in,
               double eps_out, bool residual, bool any_n) {
  if (!plain(z) || z.scalar_type() != at::kBFloat16 || z.dim() != 4 || p.size() != kTriParams) return false;
  const int64_t B = z.size(0), N = z.size(1), C = z.size(3);
  if (z.size(2) != N || C != d_pair || (C != 128 && C != 64) || B < 1 || N < 1 || B * N > 0x7FFFFFFFll / 128) return false;
  if (!any_n && N % 8 != 0) return false;
  if (!aligned16(z)) return false;
  const bool bidir = direction == B200_TRIMUL_BIDIRECTIONAL;
  const int64_t wide = bidir && C == 128 ? 256 : 128;
  const c10::ScalarType dt = p[kLeft].defined() ? p[kLeft].scalar_type() : at::kHalf;
  if (dt != at::kBFloat16 && dt != at::kFloat) return false;
  const std::array<int64_t, 2> proj{wide, C}, gate{C, C}, out{C, wide};
  for (int i : {kLeft, kLeftGate, kRight, kRightGate})
    if (!plain_on(p[i], z, dt, proj)) return false;
  if (!plain_on(p[kGate], z, dt, gate) || !plain_on(p[kOut], z, dt, out)) return false;
  for (int i : {kLnInW, kLnInB})
    if (!plain_on(p[i], z, at::kFloat, at::IntArrayRef(C))) return false;
  for (int i : {kLnOutW, kLnOutB})
    if (!plain_on(p[i], z, at::kFloat, at::IntArrayRef(wide))) return false;
  if (token_mask.has_value() && !plain_on(*token_mask, z, at::kBool, {B, N})) return false;
  if (pair_mask.has_value() && !plain_on(*pair_mask, z, at::kBool, {B, N, N})) return false;
  if (drop_scale.has_value()) {
    const Tensor& d = *drop_scale;
    if (C != 128 || !plain(d) || d.device() != z.device() || d.scalar_type() != at::kBFloat16 || d.dim() < 2 ||
        d.numel() != B * N * 128 || d.size(-1) != 128 || d.size(0) != B || !aligned16(d) || d.requires_grad())
      return false;
  }
  c.B = static_cast<int>(B);
  c.N = static_cast<int>(N);
  c.d_pair = static_cast<int>(C);
  c.wide = static_cast<int>(wide);
  c.d_hidden = C == 128 || !bidir ? 128 : 64;
  c.direction = static_cast<int>(direction);
  c.eps_in = static_cast<float>(eps_in);
  c.eps_out = static_cast<float>(eps_out);
  c.residual = residual;
  c.any_n = any_n;
  c.dtype = dt == at::kBFloat16 ? B200_TRIMUL_DTYPE_BF16 : B200_TRIMUL_DTYPE_F32;
  return true;
}

size_t forward_bytes(const TriCall& c) {
  size_t need = 0;
  check(b200_trimul_workspace_bytes(c.B, c.sized_n(), c.d_pair, c.d_hidden, c.direction, &need), "b200_trimul_workspace_bytes");
  return need;
}

void launch_forward(const TriCall& c, const Tensor& z, at::TensorList p, const OptTensor& token_mask,
                    const OptTensor& pair_mask, const OptTensor& drop_scale, const Tensor& y, void* ws, size_t ws_bytes) {
  const c10::cuda::CUDAGuard guard(z.device());
  auto fp = [&](int i) { return static_cast<const float*>(p[i].data_ptr()); };
  check(b200_trimul_forward_lines(z.data_ptr(), p[kLeft].data_ptr(), p[kLeftGate].data_ptr(), p[kRight].data_ptr(), p[kRightGate].data_ptr(),
          p[kGate].data_ptr(), p[kOut].data_ptr(), c.dtype, fp(kLnInW), fp(kLnInB), fp(kLnOutW), fp(kLnOutB), nullptr,
          static_cast<const uint8_t*>(ptr(token_mask)), static_cast<const uint8_t*>(ptr(pair_mask)), ptr(drop_scale),
          y.data_ptr(), ws, ws_bytes, c.B, c.N, c.d_pair, c.d_hidden, c.direction, c.eps_in,
          c.eps_out, c.residual ? 1 : 0, stream_of(z)),
        c.any_n ? "b200_trimul_forward_lines, for b200_trimul_forward_any" : "b200_trimul_forward_lines, for b200_trimul_forward_ex");
}

// Scratch memory that a module keeps from one call to the next, with the stream that it may be used on again: the memory of a
// call belongs to that call's launches, so only a later call on the same stream can take it. A call that is being captured
// neither takes kept memory (a graph would go on using it after the module has let it go) nor leaves any to be taken: what it
// allocates belongs to the graph's pool, and kNoStream marks it.
constexpr int64_t kNoStream = -1;
using Kept = std::tuple<int64_t, Tensor>;
int64_t stream_key(const Tensor& like) {
  const c10::cuda::CUDAGuard guard(like.device());
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return kNoStream;
  return static_cast<int64_t>(reinterpret_cast<intptr_t>(stream_of(like)));
}
bool usable(const Tensor& kept, int64_t kept_stream, int64_t stream, const Tensor& like) {
  return stream != kNoStream && kept_stream == stream && kept.device() == like.device();
}

// Forward without a graph: (y, (stream, workspace used)) or None. `kept`: what an earlier call returned, which no other call is
// using now.
std::optional<std::tuple<Tensor, Kept>> trimul_forward(const Tensor& z, const CallParams& call,
                                                       const OptTensor& token_mask, const OptTensor& pair_mask,
                                                       const std::optional<Kept>& kept, int64_t d_pair, int64_t direction,
                                                       double eps_in, double eps_out, bool residual, bool any_n) {
  const std::vector<Tensor>& params = call.list;
  TriCall c;
  if (!fill_call(c, z, params, token_mask, pair_mask, std::nullopt, d_pair, direction, eps_in, eps_out, residual, any_n))
    return std::nullopt;
  const at::NoGradGuard no_grad;
  const size_t need = forward_bytes(c);
  const int64_t stream = stream_key(z);
  Tensor ws;
  if (kept.has_value() && usable(std::get<1>(*kept), std::get<0>(*kept), stream, z) &&
      static_cast<size_t>(std::get<1>(*kept).numel()) >= need) {
    ws = std::get<1>(*kept);
  } else {
    ws = aligned_empty(need, z);
  }
  Tensor y = empty_on(z.sizes(), at::kBFloat16, z);
  launch_forward(c, z, params, token_mask, pair_mask, std::nullopt, y, ws.data_ptr(), static_cast<size_t>(ws.numel()));
  return std::make_tuple(y, Kept(stream, ws));
}

// Saved for the backward: the input and the parameters (as autograd saves them), the masks, the dropout scale and the
// forward's workspace, which holds the stage tensors and is let go by the first backward.
// (the parameters are passed as a TensorList: the graph only sees tensors that are arguments themselves or in such a list)
struct TriMul : public torch::autograd::Function<TriMul> {
  static Tensor forward(AutogradContext* ctx, const Tensor& z, at::TensorList params, TriCall c,
                        OptTensor token_mask, OptTensor pair_mask, OptTensor drop_scale) {
    Tensor ws = scratch_for(forward_bytes(c), z);
    Tensor y = empty_on(z.sizes(), at::kBFloat16, z);
    launch_forward(c, z, params, token_mask, pair_mask, drop_scale, y, aligned_start(ws), scratch_bytes(ws));
    variable_list save;
    save.reserve(1 + params.size());
    save.push_back(z);
    save.insert(save.end(), params.begin(), params.end());
    ctx->save_for_backward(std::move(save));
    auto& d = ctx->saved_data;
    d["ws"] = ws;
    if (token_mask.has_value()) d["token_mask"] = *token_mask;
    if (pair_mask.has_value()) d["pair_mask"] = *pair_mask;
    if (drop_scale.has_value()) d["drop_scale"] = *drop_scale;
    d["call"] = c10::IValue(std::vector<int64_t>{c.B, c.N, c.d_pair, c.d_hidden, c.direction, c.wide, c.residual, c.any_n, c.dtype});
    d["eps"] = c10::IValue(std::vector<double>{c.eps_in, c.eps_out});
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const at::NoGradGuard no_grad;
    const variable_list saved = ctx->get_saved_variables();
    auto& d = ctx->saved_data;
    TORCH_CHECK(d.count("ws") != 0,
                "the forward's stage tensors were released by the first backward of this call (a second backward through the "
                "same forward is not supported)");
    const Tensor ws = d["ws"].toTensor();
    const Tensor& z = saved[0];
    const std::vector<Tensor> p(saved.begin() + 1, saved.end());
    auto opt = [&](const char* k) { return d.count(k) != 0 ? OptTensor(d[k].toTensor()) : OptTensor(); };
    const OptTensor token_mask = opt("token_mask"), pair_mask = opt("pair_mask"), drop_scale = opt("drop_scale");
    const std::vector<int64_t> n = d["call"].toIntVector();
    const std::vector<double> eps = d["eps"].toDoubleVector();
    TriCall c;
    // (saved-tensor hooks may have brought the tensors back somewhere else: they are checked as in the forward)
    TORCH_CHECK(fill_call(c, z, p, token_mask, pair_mask, drop_scale, n[2], n[4], eps[0], eps[1], n[6] != 0, n[7] != 0) &&
                    c.B == n[0] && c.N == n[1] && c.dtype == n[8],
                "the tensors saved for the backward came back with another type, shape, layout or device");
    Tensor dy = grads[0].to(at::kBFloat16).contiguous();
    if (dy.sizes() != z.sizes())
      throw std::runtime_error("dy must be bf16 of the input's shape");
    if (c.any_n && !aligned16(dy)) dy = dy.clone();  // (a gradient that is a slice of a larger tensor)

    const c10::cuda::CUDAGuard guard(z.device());
    size_t need = 0;
    check(b200_trimul_backward_workspace_bytes(c.B, c.sized_n(), c.direction, &need), "b200_trimul_backward_workspace_bytes");
    const Tensor bws = scratch_for(need, z);
    Tensor dz = empty_on(z.sizes(), at::kBFloat16, z);
    variable_list g(kTriParams);
    for (int i = 0; i < kTriParams; ++i) g[i] = empty_on(p[i].sizes(), at::kFloat, z);
    void* dw[6] = {g[kLeft].data_ptr(), g[kLeftGate].data_ptr(), g[kRight].data_ptr(), g[kRightGate].data_ptr(),
                   g[kGate].data_ptr(), g[kOut].data_ptr()};
    auto fp = [&](int i) { return static_cast<const float*>(p[i].data_ptr()); };
    auto gp = [&](int i) { return static_cast<float*>(g[i].data_ptr()); };
    check(b200_trimul_backward_lines(dy.data_ptr(), z.data_ptr(), p[kLeft].data_ptr(), p[kLeftGate].data_ptr(), p[kRight].data_ptr(),
            p[kRightGate].data_ptr(), p[kGate].data_ptr(), p[kOut].data_ptr(), c.dtype, fp(kLnInW), fp(kLnInB), fp(kLnOutW),
            fp(kLnOutB), nullptr, static_cast<const uint8_t*>(ptr(token_mask)), static_cast<const uint8_t*>(ptr(pair_mask)),
            ptr(drop_scale), aligned_start(ws), dz.data_ptr(), dw, gp(kLnInW), gp(kLnInB), gp(kLnOutW), gp(kLnOutB),
            aligned_start(bws), scratch_bytes(bws), c.B, c.N, c.d_pair, c.d_hidden, c.direction, c.eps_in, c.eps_out,
            c.residual ? 1 : 0, stream_of(z)),
          c.any_n ? "b200_trimul_backward_lines, for b200_trimul_backward_any" : "b200_trimul_backward_lines, for b200_trimul_backward");
    d.erase("ws");

    variable_list out(1 + kTriParams + 4);  // z, the parameters; call, masks and scale have no gradient
    if (ctx->needs_input_grad(0)) out[0] = dz;
    for (int i = 0; i < kTriParams; ++i)
      if (ctx->needs_input_grad(1 + i)) out[1 + i] = g[i].to(p[i].scalar_type());
    return out;
  }
};

// Differentiable forward, or None.
OptTensor trimul_train(const Tensor& z, const CallParams& call, const OptTensor& token_mask,
                       const OptTensor& pair_mask, const OptTensor& drop_scale, int64_t d_pair, int64_t direction,
                       double eps_in, double eps_out, bool residual, bool any_n) {
  const std::vector<Tensor>& params = call.list;
  TriCall c;
  if (!fill_call(c, z, params, token_mask, pair_mask, drop_scale, d_pair, direction, eps_in, eps_out, residual, any_n))
    return std::nullopt;
  return TriMul::apply(z, at::TensorList(params), c, token_mask, pair_mask, drop_scale);
}

// ------------------------------------------------------------------------------------------ pair Transition
enum { kTrLnW, kTrLnB, kTrA, kTrB, kTrS, kTrParams };  // ln_in weight, bias, expand_a, expand_b, squeeze

bool transition_plain(const Tensor& x, at::TensorList p) {
  if (!plain(x) || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || x.size(-1) != 128 || x.numel() == 0 || !aligned16(x) ||
      p.size() != kTrParams)
    return false;
  const c10::ScalarType dt = p[kTrA].defined() ? p[kTrA].scalar_type() : at::kHalf;
  if (dt != at::kBFloat16 && dt != at::kFloat) return false;
  return plain_on(p[kTrA], x, dt, {512, 128}) && plain_on(p[kTrB], x, dt, {512, 128}) && plain_on(p[kTrS], x, dt, {128, 512}) &&
         plain_on(p[kTrLnW], x, at::kFloat, {128}) && plain_on(p[kTrLnB], x, at::kFloat, {128});
}
int dtype_code(const Tensor& w) { return w.scalar_type() == at::kBFloat16 ? B200_TRIMUL_DTYPE_BF16 : B200_TRIMUL_DTYPE_F32; }

void launch_transition(const Tensor& x, at::TensorList p, double eps, bool residual, void* packed, int* status,
                       bool clear_status, const Tensor& y) {
  check(b200_transition_pack_forward(x.data_ptr(), p[kTrA].data_ptr(), p[kTrB].data_ptr(), p[kTrS].data_ptr(), dtype_code(p[kTrA]),
                        static_cast<const float*>(p[kTrLnW].data_ptr()), static_cast<const float*>(p[kTrLnB].data_ptr()), packed,
                        y.data_ptr(), x.numel() / 128, 128, 4, static_cast<float>(eps), residual ? 1 : 0, status,
                        clear_status ? 1 : 0, stream_of(x)),
        "b200_transition_pack_forward");
}

// Forward without a graph: (y, (stream, scratch used)) or None. The scratch holds the packed weights, then 16 status words, which
// are cleared when it is allocated. `kept` as in trimul_forward.
std::optional<std::tuple<Tensor, Kept>> transition_forward(const Tensor& x, const CallParams& call,
                                                           const std::optional<Kept>& kept, double eps, bool residual) {
  const std::vector<Tensor>& params = call.list;
  if (!transition_plain(x, params)) return std::nullopt;
  const at::NoGradGuard no_grad;
  const c10::cuda::CUDAGuard guard(x.device());
  const size_t bytes = b200_transition_packed_bytes();
  const int64_t stream = stream_key(x);
  const bool keep = kept.has_value() && usable(std::get<1>(*kept), std::get<0>(*kept), stream, x);
  const Tensor scratch = keep ? std::get<1>(*kept) : aligned_empty(bytes + 64, x);
  uint8_t* base = static_cast<uint8_t*>(scratch.data_ptr());
  Tensor y = empty_on(x.sizes(), at::kBFloat16, x);
  launch_transition(x, params, eps, residual, base, reinterpret_cast<int*>(base + bytes), !keep, y);
  return std::make_tuple(y, Kept(stream, scratch));
}

struct TransitionNode : public torch::autograd::Function<TransitionNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, at::TensorList params, double eps, bool residual) {
    const c10::cuda::CUDAGuard guard(x.device());
    const size_t bytes = b200_transition_packed_bytes();
    const Tensor scratch = scratch_for(bytes + 64, x);  // packed weights, then the status words
    uint8_t* base = aligned_start(scratch);
    int* status = reinterpret_cast<int*>(base + bytes);
    Tensor y = empty_on(x.sizes(), at::kBFloat16, x);
    launch_transition(x, params, eps, residual, base, status, true, y);
    variable_list save;
    save.push_back(x);
    save.insert(save.end(), params.begin(), params.end());
    ctx->save_for_backward(std::move(save));
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["residual"] = residual;
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const at::NoGradGuard no_grad;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    const std::vector<Tensor> p(saved.begin() + 1, saved.end());
    TORCH_CHECK(transition_plain(x, p), "the tensors saved for the backward came back with another type, shape, layout or device");
    const Tensor dy = grads[0].to(at::kBFloat16).contiguous();
    if (dy.sizes() != x.sizes()) throw std::runtime_error("dy must have the input's shape");
    const c10::cuda::CUDAGuard guard(x.device());
    const long long positions = x.numel() / 128;
    size_t need = 0;
    check(b200_transition_backward_workspace_bytes(positions, &need), "b200_transition_backward_workspace_bytes");
    const Tensor ws = scratch_for(need, x);
    Tensor dx = empty_on(x.sizes(), at::kBFloat16, x);
    variable_list g(kTrParams);
    for (int i = 0; i < kTrParams; ++i) g[i] = empty_on(p[i].sizes(), at::kFloat, x);
    auto gp = [&](int i) { return static_cast<float*>(g[i].data_ptr()); };
    check(b200_transition_backward(dy.data_ptr(), x.data_ptr(), p[kTrA].data_ptr(), p[kTrB].data_ptr(), p[kTrS].data_ptr(),
                                   dtype_code(p[kTrA]), static_cast<const float*>(p[kTrLnW].data_ptr()),
                                   static_cast<const float*>(p[kTrLnB].data_ptr()), dx.data_ptr(), gp(kTrA), gp(kTrB), gp(kTrS),
                                   gp(kTrLnW), gp(kTrLnB), aligned_start(ws), scratch_bytes(ws), positions, 128, 4,
                                   static_cast<float>(ctx->saved_data["eps"].toDouble()),
                                   ctx->saved_data["residual"].toBool() ? 1 : 0, stream_of(x)),
          "b200_transition_backward");
    variable_list out(1 + kTrParams + 2);
    if (ctx->needs_input_grad(0)) out[0] = dx;
    for (int i = 0; i < kTrParams; ++i)
      if (ctx->needs_input_grad(1 + i)) out[1 + i] = g[i].to(p[i].scalar_type());
    return out;
  }
};

OptTensor transition_train(const Tensor& x, const CallParams& call, double eps, bool residual) {
  const std::vector<Tensor>& params = call.list;
  if (!transition_plain(x, params)) return std::nullopt;
  return TransitionNode::apply(x, at::TensorList(params), eps, residual);
}

}  // namespace

namespace pybind11::detail {
template <>
struct type_caster<CallParams> {
  PYBIND11_TYPE_CASTER(CallParams, const_name("parameters"));
  bool load(handle src, bool) {
    if (PyList_Check(src.ptr())) {
      for (Py_ssize_t i = 0; i < PyList_GET_SIZE(src.ptr()); ++i) {
        PyObject* t = PyList_GET_ITEM(src.ptr(), i);
        if (!THPVariable_Check(t)) return false;
        value.list.push_back(THPVariable_Unpack(t));
      }
      return true;
    }
    if (!PyTuple_Check(src.ptr()) || PyTuple_GET_SIZE(src.ptr()) != 2) return false;
    PyObject *children = PyTuple_GET_ITEM(src.ptr(), 0), *names = PyTuple_GET_ITEM(src.ptr(), 1);
    if (!PyDict_Check(children) || !PyTuple_Check(names)) return false;
    value.list.reserve(static_cast<size_t>(PyTuple_GET_SIZE(names)));
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(names); ++i) {
      PyObject* key = PyTuple_GET_ITEM(names, i);
      PyObject* child = PyDict_GetItem(children, PyTuple_GET_ITEM(key, 0));
      const object own = child != nullptr ? reinterpret_steal<object>(PyObject_GetAttrString(child, "_parameters")) : object();
      if (!own) PyErr_Clear();
      PyObject* t = own && PyDict_Check(own.ptr()) ? PyDict_GetItem(own.ptr(), PyTuple_GET_ITEM(key, 1)) : nullptr;
      if (t == nullptr || !THPVariable_Check(t)) {
        value.list.clear();
        return true;
      }
      value.list.push_back(THPVariable_Unpack(t));
    }
    return true;
  }
};
}  // namespace pybind11::detail

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("trimul_forward", torch::wrap_pybind_function_no_gil(trimul_forward));
  m.def("trimul_train", torch::wrap_pybind_function_no_gil(trimul_train));
  m.def("transition_forward", torch::wrap_pybind_function_no_gil(transition_forward));
  m.def("transition_train", torch::wrap_pybind_function_no_gil(transition_train));
}
