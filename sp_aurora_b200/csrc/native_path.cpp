// One-rank attention as a C++ autograd node: argument checks, allocation, the C-ABI calls and the
// backward without the interpreter.
//
// Through Python a small forward + backward (B=2, S=1024, 8 heads, D=64) spends 213 us of host
// time on some 60 us of kernels: the autograd.Function glue, the ctypes argument blocks and their
// checks, and the engine's trips through the interpreter lock. Through this node it takes 83 us; a
// forward of 512 rows 42 -> 16 us, four packed sequences forward + backward 275 -> 109. Packed
// gradients (kv, qkv) are written in place: slice by slice autograd fills, copies and adds them
// (2 x 3001 rows, 32 / 8 heads, kv packed: 847 -> 788 us).
//
// Calls this file does not take (several ranks, an unusual argument, a tensor subclass, a
// functorch transform, a tangent, a trace) answer None and go the Python way, which also words
// the errors. The kernels are reached through the function table of the library that _lib.py
// loaded; nothing is kept between calls.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <cmath>
#include <cstdlib>
#include <cstring>

#include "../../include/spa.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Api {
  decltype(&spa_attn_fwd) fwd;
  decltype(&spa_attn_fwd_workspace) fwd_workspace;
  decltype(&spa_attn_fwd_ws) fwd_ws;
  decltype(&spa_attn_bwd) bwd;
  decltype(&spa_attn_varlen_fwd) varlen_fwd;
  decltype(&spa_attn_varlen_bwd) varlen_bwd;
  decltype(&spa_bwd_delta) delta;
  decltype(&spa_rope_rows) rope_rows;
  decltype(&spa_check_status) check_status;
  decltype(&spa_last_error) last_error;
} api;
PyObject* spa_error = nullptr;   // _lib.SpaError, alive as long as the module

void check(int rc, const char* what) {
  if (rc == SPA_OK) return;
  const std::string msg = std::string(what) + " failed with status " + std::to_string(rc) + ": " + api.last_error();
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(spa_error, msg.c_str());
  python_error err;
  err.persist();
  throw std::move(err);
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SPA_DTYPE_F32;
    case at::kBFloat16: return SPA_DTYPE_BF16;
    case at::kHalf: return SPA_DTYPE_F16;
    default: return -1;
  }
}

// A plain CUDA tensor: no subclass, no functorch wrapper, no forward-mode tangent, no conj / neg view.
bool plain(const Tensor& t) {
  using c10::DispatchKey;
  static const c10::DispatchKeySet special({DispatchKey::Python, DispatchKey::FuncTorchBatched,
                                            DispatchKey::FuncTorchGradWrapper, DispatchKey::Functionalize,
                                            DispatchKey::Conjugate, DispatchKey::Negative, DispatchKey::ZeroTensor});
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(special) &&
         !t._fw_grad(0).defined();
}

// No functorch transform, no Python dispatch mode, no trace is active.
bool quiet_context() {
  return !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Python) && !torch::jit::tracer::isTracing();
}

bool takes_head_dim(int64_t D) { return D == 32 || D == 64 || D == 128; }

// What local_attn.check_qkv accepts, for tensors of `dim` dimensions that end in [H, D].
bool takes(const Tensor& q, const Tensor& k, const Tensor& v, int64_t dim) {
  for (const Tensor* t : {&q, &k, &v})
    if (t->dim() != dim || t->stride(dim - 1) != 1 || t->scalar_type() != q.scalar_type() || t->device() != q.device())
      return false;
  const int64_t D = q.size(dim - 1), Hkv = k.size(dim - 2);
  return dtype_code(q.scalar_type()) >= 0 && k.sizes() == v.sizes() && k.size(dim - 1) == D && takes_head_dim(D) &&
         (dim == 3 || k.size(0) == q.size(0)) && Hkv > 0 && q.size(dim - 2) % Hkv == 0;
}

template <typename A>
void fill_qkv(A& a, const Tensor& q, const Tensor& k, const Tensor& v) {
  a.q = q.data_ptr(); a.q_sb = q.stride(0); a.q_ss = q.stride(1); a.q_sh = q.stride(2);
  a.k = k.data_ptr(); a.k_sb = k.stride(0); a.k_ss = k.stride(1); a.k_sh = k.stride(2);
  a.v = v.data_ptr(); a.v_sb = v.stride(0); a.v_ss = v.stride(1); a.v_sh = v.stride(2);
  a.B = q.size(0); a.Sq = q.size(1); a.Sk = k.size(1); a.Hq = q.size(2); a.Hkv = k.size(2); a.D = q.size(3);
  a.dtype = dtype_code(q.scalar_type());
  a.stream = at::cuda::getCurrentCUDAStream(q.device().index()).stream();
}

struct Options {
  double scale;
  bool causal, deterministic;
  std::vector<spa_seq> seqs;   // packed sequences; empty: the tensors are one batch
};

void run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                 const Options& o) {
  spa_fwd_args a;
  std::memset(&a, 0, sizeof(a));
  fill_qkv(a, q, k, v);
  a.out = out.data_ptr(); a.o_sb = out.stride(0); a.o_ss = out.stride(1); a.o_sh = out.stride(2);
  a.lse = lse.data_ptr<float>(); a.lse_sb = lse.stride(0); a.lse_sh = lse.stride(1);
  a.causal = o.causal;
  a.scale = static_cast<float>(o.scale);
  if (!o.seqs.empty()) {
    check(api.varlen_fwd(&a, o.seqs.data(), (int32_t)o.seqs.size()), "spa_attn_varlen_fwd");
    return;
  }
  const int64_t need = api.fwd_workspace(&a);
  if (need > 0) {
    Tensor ws = at::empty({need}, q.options().dtype(at::kByte));
    check(api.fwd_ws(&a, ws.data_ptr(), need), "spa_attn_fwd");
  } else {
    check(api.fwd(&a), "spa_attn_fwd");
  }
}

std::pair<Tensor, Tensor> run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Options& o) {
  Tensor out = at::empty(q.sizes(), q.options());
  Tensor lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
  run_forward(q, k, v, out, lse, o);
  return {out, lse};
}

// Gradients into dq, dk, dv (any strides with a contiguous last dimension).
void run_backward(Tensor dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                  const Tensor& dq, const Tensor& dk, const Tensor& dv, const Options& o) {
  if (dout.stride(3) != 1) dout = dout.contiguous();
  TORCH_CHECK(dout.sizes() == out.sizes() && dout.scalar_type() == q.scalar_type() && dout.device() == q.device(),
              "dout does not match the attention output");
  Tensor delta = at::empty(lse.sizes(), lse.options());
  spa_bwd_args a;
  std::memset(&a, 0, sizeof(a));
  fill_qkv(a, q, k, v);
  a.dout = dout.data_ptr(); a.do_sb = dout.stride(0); a.do_ss = dout.stride(1); a.do_sh = dout.stride(2);
  check(api.delta(out.data_ptr(), out.stride(0), out.stride(1), out.stride(2), a.dout, a.do_sb, a.do_ss, a.do_sh,
                  delta.data_ptr<float>(), a.B, a.Sq, a.Hq, a.D, a.dtype, a.stream),
        "spa_bwd_delta");
  a.lse = lse.data_ptr<float>(); a.delta = delta.data_ptr<float>();
  a.lse_sb = (int64_t)a.Hq * a.Sq; a.lse_sh = a.Sq;
  a.dq = dq.data_ptr(); a.dq_sb = dq.stride(0); a.dq_ss = dq.stride(1); a.dq_sh = dq.stride(2);
  a.dq_overwrite = 1;
  a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
  a.dkv_sb = dk.stride(0); a.dkv_ss = dk.stride(1); a.dkv_sh = dk.stride(2);
  a.deterministic = o.deterministic;
  a.passes = SPA_BWD_BOTH;
  a.causal = o.causal;
  a.scale = static_cast<float>(o.scale);
  if (o.seqs.empty())
    check(api.bwd(&a), "spa_attn_bwd");
  else
    check(api.varlen_bwd(&a, o.seqs.data(), (int32_t)o.seqs.size()), "spa_attn_varlen_bwd");
}

void end_of_backward() {
  const char* e = std::getenv("SPA_CHECK_STATUS");
  if (e && std::strcmp(e, "1") == 0) check(api.check_status(), "spa_check_status");
}

void save_options(AutogradContext* ctx, const Options& o) {
  ctx->saved_data["scale"] = o.scale;
  ctx->saved_data["flags"] = static_cast<int64_t>(o.causal) + 2 * static_cast<int64_t>(o.deterministic);
  if (o.seqs.empty()) return;
  std::vector<int64_t> flat;
  flat.reserve(o.seqs.size() * 5);
  for (const spa_seq& s : o.seqs) flat.insert(flat.end(), {s.q0, s.sq, s.k0, s.sk, s.causal_off});
  ctx->saved_data["seqs"] = flat;
}

Options load_options(AutogradContext* ctx) {
  Options o;
  o.scale = ctx->saved_data["scale"].toDouble();
  const int64_t f = ctx->saved_data["flags"].toInt();
  o.causal = f & 1;
  o.deterministic = f & 2;
  const auto it = ctx->saved_data.find("seqs");
  if (it != ctx->saved_data.end()) {
    const auto flat = it->second.toIntVector();
    for (size_t i = 0; i < flat.size(); i += 5)
      o.seqs.push_back(spa_seq{(int32_t)flat[i], (int32_t)flat[i + 1], (int32_t)flat[i + 2], (int32_t)flat[i + 3],
                               (int32_t)flat[i + 4]});
  }
  return o;
}

variable_list finish_forward(AutogradContext* ctx, variable_list saved, std::pair<Tensor, Tensor> res, const Options& o,
                             bool lse_const) {
  saved.push_back(res.first);
  saved.push_back(res.second);
  ctx->save_for_backward(saved);
  ctx->set_materialize_grads(false);   // the lse gradient is ignored, as on the Python path
  if (lse_const) ctx->mark_non_differentiable({res.second});
  save_options(ctx, o);
  return {res.first, res.second};
}

Tensor grad_or_zeros(const variable_list& g, const Tensor& out) { return g[0].defined() ? g[0] : at::zeros_like(out); }

// q, k, v apart: [B,S,H,D], or [tokens,H,D] with packed sequences.
struct SplitAttn : torch::autograd::Function<SplitAttn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Options& o,
                               bool lse_const) {
    if (o.seqs.empty()) return finish_forward(ctx, {q, k, v}, run_forward(q, k, v, o), o, lse_const);
    Tensor out = at::empty(q.sizes(), q.options());
    Tensor lse = at::empty({q.size(1), q.size(0)}, q.options().dtype(at::kFloat));
    run_forward(q.unsqueeze(0), k.unsqueeze(0), v.unsqueeze(0), out.unsqueeze(0), lse.unsqueeze(0), o);
    return finish_forward(ctx, {q, k, v}, {out, lse}, o, lse_const);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Options o = load_options(ctx);
    const Tensor &q = s[0], &k = s[1], &v = s[2], &out = s[3], &lse = s[4];
    Tensor dout = grad_or_zeros(grads, out);
    Tensor dq = at::empty(q.sizes(), q.options());
    if (o.seqs.empty()) {
      Tensor dk = at::empty(k.sizes(), k.options()), dv = at::empty(k.sizes(), k.options());
      run_backward(dout, q, k, v, out, lse, dq, dk, dv, o);
      end_of_backward();
      return {dq, dk, dv, Tensor(), Tensor()};
    }
    int64_t keys = 0;
    for (const spa_seq& x : o.seqs) keys += x.sk;
    const bool all = keys == k.size(0);   // rows that no sequence uses have zero gradients
    Tensor dk = all ? at::empty(k.sizes(), k.options()) : at::zeros(k.sizes(), k.options());
    Tensor dv = all ? at::empty(k.sizes(), k.options()) : at::zeros(k.sizes(), k.options());
    run_backward(dout.unsqueeze(0), q.unsqueeze(0), k.unsqueeze(0), v.unsqueeze(0), out.unsqueeze(0), lse.unsqueeze(0),
                 dq.unsqueeze(0), dk.unsqueeze(0), dv.unsqueeze(0), o);
    end_of_backward();
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

// kv [B,S,2,H,D]: dK and dV are written straight into the packed gradient.
struct KvPackedAttn : torch::autograd::Function<KvPackedAttn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& kv, const Options& o) {
    return finish_forward(ctx, {q, kv}, run_forward(q, kv.select(2, 0), kv.select(2, 1), o), o, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Options o = load_options(ctx);
    const Tensor &q = s[0], &kv = s[1];
    Tensor dq = at::empty(q.sizes(), q.options()), dkv = at::empty(kv.sizes(), kv.options());
    run_backward(grad_or_zeros(grads, s[2]), q, kv.select(2, 0), kv.select(2, 1), s[2], s[3], dq, dkv.select(2, 0),
                 dkv.select(2, 1), o);
    end_of_backward();
    return {dq, dkv, Tensor()};
  }
};

// qkv [B,S,3,H,D]: all three gradients are written straight into the packed one.
struct QkvPackedAttn : torch::autograd::Function<QkvPackedAttn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Options& o) {
    return finish_forward(ctx, {x}, run_forward(x.select(2, 0), x.select(2, 1), x.select(2, 2), o), o, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Options o = load_options(ctx);
    const Tensor& x = s[0];
    Tensor dx = at::empty(x.sizes(), x.options());
    run_backward(grad_or_zeros(grads, s[1]), x.select(2, 0), x.select(2, 1), x.select(2, 2), s[1], s[2],
                 dx.select(2, 0), dx.select(2, 1), dx.select(2, 2), o);
    end_of_backward();
    return {dx, Tensor()};
  }
};

// dst = rotated src, both [B,S,H,D] with a contiguous last dimension; dst may be src.
void rope(const Tensor& src, const Tensor& dst, const Tensor& cos, const Tensor& sin, bool inverse) {
  const int64_t n[4] = {1, src.size(0), src.size(1), src.size(2)};
  const int64_t ss[4] = {0, src.stride(0), src.stride(1), src.stride(2)};
  const int64_t ds[4] = {0, dst.stride(0), dst.stride(1), dst.stride(2)};
  check(api.rope_rows(src.data_ptr(), dst.data_ptr(), n, ss, ds, src.size(3), dtype_code(src.scalar_type()),
                      cos.data_ptr<float>(), sin.data_ptr<float>(), cos.size(0), 2, 0, inverse,
                      at::cuda::getCurrentCUDAStream(src.device().index()).stream()),
        "spa_rope_rows");
}

// A projection's output x [B,S,Hq+2*Hkv,D] whose head slices are q, k and v, q and k rotated first
// when cos / sin are given. The kernels write the three gradients into the slices of one dx and
// the rotation is undone there in place: slice by slice, autograd would fill a zero tensor per
// slice, copy the slice in and add the tensors up (B=1, S=8192, 32/8 heads, D=128, rotated:
// 4360 -> 4030 us with both projections).
struct HeadsPackedAttn : torch::autograd::Function<HeadsPackedAttn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Options& o, int64_t hq, int64_t hkv,
                               const std::optional<Tensor>& cos, const std::optional<Tensor>& sin) {
    Tensor q = x.narrow(2, 0, hq), k = x.narrow(2, hq, hkv), v = x.narrow(2, hq + hkv, hkv);
    ctx->saved_data["hq"] = hq;
    ctx->saved_data["hkv"] = hkv;
    if (!cos) return finish_forward(ctx, {x}, run_forward(q, k, v, o), o, false);
    Tensor qk = at::empty({x.size(0), x.size(1), hq + hkv, x.size(3)}, x.options());
    rope(x.narrow(2, 0, hq + hkv), qk, *cos, *sin, false);
    return finish_forward(ctx, {x, qk, *cos, *sin},
                          run_forward(qk.narrow(2, 0, hq), qk.narrow(2, hq, hkv), v, o), o, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Options o = load_options(ctx);
    const int64_t hq = ctx->saved_data["hq"].toInt(), hkv = ctx->saved_data["hkv"].toInt();
    const bool rotated = s.size() == 6;
    const Tensor &x = s[0], &qk = rotated ? s[1] : s[0], &out = s[s.size() - 2], &lse = s[s.size() - 1];
    Tensor dx = at::empty(x.sizes(), x.options());
    run_backward(grad_or_zeros(grads, out), qk.narrow(2, 0, hq), qk.narrow(2, hq, hkv), x.narrow(2, hq + hkv, hkv), out,
                 lse, dx.narrow(2, 0, hq), dx.narrow(2, hq, hkv), dx.narrow(2, hq + hkv, hkv), o);
    if (rotated) {
      const Tensor dqk = dx.narrow(2, 0, hq + hkv);
      rope(dqk, dqk, s[2], s[3], true);
    }
    end_of_backward();
    return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

using Result = std::optional<std::tuple<Tensor, Tensor>>;

// Runs f without the interpreter lock, with the tensors' device current.
template <typename F>
Result released(const Tensor& on, F f) {
  try {
    pybind11::gil_scoped_release no_gil;
    const c10::cuda::CUDAGuard guard(on.device());
    variable_list r = f();
    return std::make_tuple(r[0], r[1]);
  } catch (python_error& e) {
    e.restore();
    throw pybind11::error_already_set();
  }
}

Options options(std::optional<double> scale, int64_t D, bool causal, bool deterministic) {
  return Options{scale ? *scale : 1.0 / std::sqrt(static_cast<double>(D)), causal, deterministic, {}};
}

Result attention(const Tensor& q, const Tensor& k, const Tensor& v, std::optional<double> scale, bool causal,
                 bool deterministic, bool lse_const) {
  if (!quiet_context() || !plain(q) || !plain(k) || !plain(v) || !takes(q, k, v, 4)) return std::nullopt;
  const Options o = options(scale, q.size(3), causal, deterministic);
  return released(q, [&] { return SplitAttn::apply(q, k, v, o, lse_const); });
}

Result attention_kvpacked(const Tensor& q, const Tensor& kv, std::optional<double> scale, bool causal,
                          bool deterministic) {
  if (!quiet_context() || !plain(q) || !plain(kv) || kv.dim() != 5 || kv.size(2) != 2) return std::nullopt;
  {
    at::NoGradGuard views_only;
    const Tensor k = kv.select(2, 0);
    if (!takes(q, k, k, 4)) return std::nullopt;
  }
  const Options o = options(scale, q.size(3), causal, deterministic);
  return released(q, [&] { return KvPackedAttn::apply(q, kv, o); });
}

Result attention_qkvpacked(const Tensor& x, std::optional<double> scale, bool causal, bool deterministic) {
  if (!quiet_context() || !plain(x) || x.dim() != 5 || x.size(2) != 3 || x.stride(4) != 1 || x.size(3) == 0 ||
      dtype_code(x.scalar_type()) < 0 || !takes_head_dim(x.size(4)))
    return std::nullopt;
  const Options o = options(scale, x.size(4), causal, deterministic);
  return released(x, [&] { return QkvPackedAttn::apply(x, o); });
}

Result attention_heads_packed(const Tensor& x, int64_t hq, int64_t hkv, const std::optional<Tensor>& cos,
                              const std::optional<Tensor>& sin, bool causal) {
  if (!quiet_context() || !plain(x) || x.dim() != 4 || x.stride(3) != 1 || x.numel() == 0 || hkv <= 0 || hq % hkv ||
      x.size(2) != hq + 2 * hkv || dtype_code(x.scalar_type()) < 0 || !takes_head_dim(x.size(3)) ||
      cos.has_value() != sin.has_value())
    return std::nullopt;
  for (const auto* t : {&cos, &sin})
    if (t->has_value() && (!plain(**t) || (*t)->scalar_type() != at::kFloat || (*t)->dim() != 2 ||
                           (*t)->size(1) != x.size(3) / 2 || !(*t)->is_contiguous() || (*t)->requires_grad() ||
                           (*t)->device() != x.device()))
      return std::nullopt;
  const Options o = options(std::nullopt, x.size(3), causal, false);
  return released(x, [&] { return HeadsPackedAttn::apply(x, o, hq, hkv, cos, sin); });
}

Result attention_packed(const Tensor& q, const Tensor& k, const Tensor& v,
                        const std::vector<std::tuple<int, int, int, int, int>>& seqs, std::optional<double> scale,
                        bool causal, bool deterministic) {
  if (seqs.empty() || !quiet_context() || !plain(q) || !plain(k) || !plain(v) || !takes(q, k, v, 3))
    return std::nullopt;
  Options o = options(scale, q.size(2), causal, deterministic);
  for (const auto& [q0, sq, k0, sk, off] : seqs) o.seqs.push_back(spa_seq{q0, sq, k0, sk, off});
  return released(q, [&] { return SplitAttn::apply(q, k, v, o, false); });
}

void set_api(const std::vector<uintptr_t>& f, pybind11::object error) {
  TORCH_CHECK(f.size() == 10, "ten entry points expected");
  api.fwd = reinterpret_cast<decltype(api.fwd)>(f[0]);
  api.fwd_workspace = reinterpret_cast<decltype(api.fwd_workspace)>(f[1]);
  api.fwd_ws = reinterpret_cast<decltype(api.fwd_ws)>(f[2]);
  api.bwd = reinterpret_cast<decltype(api.bwd)>(f[3]);
  api.varlen_fwd = reinterpret_cast<decltype(api.varlen_fwd)>(f[4]);
  api.varlen_bwd = reinterpret_cast<decltype(api.varlen_bwd)>(f[5]);
  api.delta = reinterpret_cast<decltype(api.delta)>(f[6]);
  api.check_status = reinterpret_cast<decltype(api.check_status)>(f[7]);
  api.last_error = reinterpret_cast<decltype(api.last_error)>(f[8]);
  api.rope_rows = reinterpret_cast<decltype(api.rope_rows)>(f[9]);
  spa_error = error.release().ptr();
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("set_api", &set_api);
  m.def("attention", &attention);
  m.def("attention_kvpacked", &attention_kvpacked);
  m.def("attention_qkvpacked", &attention_qkvpacked);
  m.def("attention_packed", &attention_packed);
  m.def("attention_heads_packed", &attention_heads_packed);
}
