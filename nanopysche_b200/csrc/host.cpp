// Native host path of the ops that run many times per layer: checks, output tensors, argument structures, the launch and the autograd
// nodes. Same operands, refusals and saved tensors as the Python statements in ops/; those stay for CPU tensors and, for
// the expert layer, the forms with peers or e4m3 operands. A call through ctypes from a Python autograd function took 20 us of host time forward and as much again backward (one
// RMSNorm 105 us with its backward, of which the kernels are 10), more than most kernels of a small layer.
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <cmath>
#include <sstream>

#include "args.h"

extern "C" {
int np_gemm_bf16(const NpGemmArgs*, void*);
int np_gemm_bf16_two(const NpGemmArgs*, const NpGemmArgs*, void*);
int np_attn_fwd(const NpAttnFwdArgs*, void*);
int np_attn_bwd(const NpAttnBwdArgs*, void*);
int np_decode_attn(const NpDecodeArgs*, void*);
int np_rmsnorm_fwd(const void*, const void*, const float*, void*, void*, float*, int, int, float, void*);
int np_rmsnorm_bwd_parts(int);
int np_rmsnorm_bwd(const void*, const void*, const float*, const float*, const void*, void*, float*, float*, int, int, int, void*);
int np_rope(const void*, void*, const float*, const float*, const int*, long long, int, int, int, int, int, long long, long long, float,
            void*);
int np_qkv_rope(const void*, long long, long long, int, const void*, long long, long long, int, const void*, long long, long long, int,
                void*, const float*, const float*, const int*, long long, int, int, int, int, int, float, void*);
int np_qkv_norm_rope_fwd(const void*, long long, int, int, const float*, const float*, const float*, const float*, float, void*, void*,
                         const float*, const float*, const int*, long long, int, int, void*);
int np_qkv_norm_rope_parts(long long);
int np_qkv_norm_rope_bwd(const void*, long long, long long, const void*, long long, long long, const void*, long long, long long,
                         const void*, long long, int, int, const float*, const float*, const void*, void*, float*, float*, const float*,
                         const float*, const int*, long long, int, int, int, void*);
int np_router_logits(const void*, const float*, const float*, float*, int, int, int, int*, int, void*);
int np_router_topk(const float*, const float*, float*, int*, int*, float*, float*, int, int, int, int, void*);
int np_router_aux(const int*, const float*, const float*, float, float*, float*, int, int, void*);
int np_router_bwd(const float*, const float*, const float*, const int*, const float*, const float*, const float*, float, float, float*,
                  int, int, int, int, void*);
long long np_router_dgate_scratch(int, int, int);
int np_router_dgate(const float*, const void*, float*, float*, float*, int, int, int, int, void*);
int np_router_dx(const float*, const float*, void*, int, int, int, void*);
int np_capacity_plan(const int*, int, int, int, int, int*, int*, int*, int*, int*, int*, int, long long*, void*);
int np_ep_dispatch(const NpDispatchArgs*, void*);
int np_ep_combine(const NpCombineArgs*, void*);
int np_slot_dot(const void*, const void*, const int*, float*, int, int, int, void*);
}

namespace {
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

std::atomic<long long> g_launches{0};
PyObject* g_kernel_error = nullptr;   // ops._lib.KernelError
PyObject* g_gemm_dict = nullptr;      // namespace of ops.gemm: _DEFER, _main_grad_done, _wgrad_into
PyObject *s_main_grad, *s_dirty, *s_defer, *s_done, *s_wgrad_into, *s_tp_partial;

[[noreturn]] void fail(PyObject* type, const std::string& msg) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(type, msg.c_str());
  python_error e;
  e.persist();
  throw e;
}
void require(bool ok, const char* msg) {
  if (!ok) fail(PyExc_AssertionError, msg);
}
void launched(int rc, const char* name) {
  if (rc != 0) fail(g_kernel_error, std::string(name) + " failed with code " + std::to_string(rc));
  g_launches.fetch_add(1, std::memory_order_relaxed);
}
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
template <class T = void>
T* ptr(const Tensor& t) {
  return t.defined() ? (T*)t.data_ptr() : nullptr;
}
Tensor empty_like_of(const Tensor& t, at::IntArrayRef shape, at::ScalarType dtype) { return at::empty(shape, t.options().dtype(dtype)); }

// An attribute of a tensor's Python object, or nothing (the caller holds the GIL)
py::object attr(const Tensor& t, PyObject* name) {
  py::object o = py::reinterpret_steal<py::object>(THPVariable_Wrap(t));
  PyObject* v = PyObject_GetAttr(o.ptr(), name);
  if (!v) PyErr_Clear();
  return py::reinterpret_steal<py::object>(v);
}
bool truthy(const py::object& o) { return o.ptr() && o.ptr() != Py_None && PyObject_IsTrue(o.ptr()) == 1; }
bool some(const py::object& o) { return o.ptr() && o.ptr() != Py_None; }
PyObject* gemm_global(PyObject* name) { return PyDict_GetItem(g_gemm_dict, name); }   // borrowed

// --------------------------------------------------------------------------------------------------------- products
NpGemmArgs product(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Tensor& out, bool accumulate, double alpha) {
  NpGemmArgs g{};
  g.A = a.data_ptr(); g.B = b.data_ptr(); g.C = out.data_ptr();
  g.lda = a.stride(0); g.ldb = b.stride(0); g.ldc = out.stride(0);
  g.a_rows = a.size(0); g.b_rows = b.size(0);
  g.M = (int)(a_mn ? a.size(1) : a.size(0)); g.K = (int)(a_mn ? a.size(0) : a.size(1));
  g.N = (int)(b_mn ? b.size(1) : b.size(0));
  g.a_mn = a_mn; g.b_mn = b_mn; g.out_f32 = out.scalar_type() == at::kFloat;
  g.accumulate = accumulate; g.alpha = (float)alpha;
  return g;
}
Tensor check_product(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const OptTensor& out, std::optional<at::ScalarType> dtype) {
  require(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "kernel path is bf16");
  require(a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1, "two-dimensional operands with contiguous rows");
  const int64_t M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0), Kb = b.size(b_mn ? 0 : 1);
  if (K != Kb) fail(PyExc_AssertionError, "contraction mismatch " + std::to_string(K) + " vs " + std::to_string(Kb));
  Tensor o = out ? *out : empty_like_of(a, {M, N}, dtype.value_or(at::kBFloat16));
  require(o.dim() == 2 && o.size(0) == M && o.size(1) == N && o.stride(1) == 1, "output shape");
  require(o.scalar_type() == at::kFloat || o.scalar_type() == at::kBFloat16, "output dtype");
  return o;
}
std::string describe(const char* what, int rc, const Tensor& a, const Tensor& b, const Tensor& out) {
  std::ostringstream s;
  s << what << " failed with code " << rc << ": a=" << a.sizes() << "/" << a.strides() << " b=" << b.sizes() << "/" << b.strides()
    << " out=" << out.sizes() << "/" << out.strides() << " " << out.scalar_type() << " ptrs=" << (uintptr_t)a.data_ptr() % 256 << ","
    << (uintptr_t)b.data_ptr() % 256 << "," << (uintptr_t)out.data_ptr() % 256;
  return s.str();
}
Tensor gemm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const OptTensor& out, std::optional<at::ScalarType> dtype,
            bool accumulate, double alpha, int bn, int max_ctas, const OptTensor& bias, const OptTensor& residual, int mt, int split,
            int pair_bn) {
  Tensor o = check_product(a, b, a_mn, b_mn, out, dtype);
  NpGemmArgs g = product(a, b, a_mn, b_mn, o, accumulate, alpha);
  g.bn = bn; g.max_ctas = max_ctas; g.mt = mt; g.split = split; g.pair_bn = pair_bn;
  if (bias) {
    require(bias->scalar_type() == at::kFloat && bias->numel() == g.N && bias->is_contiguous(), "bias: fp32, one per output column");
    g.bias = ptr<float>(*bias);
  }
  if (residual) {
    const Tensor& r = *residual;
    require(!accumulate && r.dim() == 2 && r.size(0) == g.M && r.size(1) == g.N && r.scalar_type() == o.scalar_type() && r.stride(1) == 1,
            "residual: shape and dtype of the output");
    g.accumulate = 1; g.Cin = r.data_ptr(); g.ldcin = r.stride(0);
  }
  const int rc = np_gemm_bf16(&g, stream());
  if (rc) fail(g_kernel_error, describe("gemm_bf16", rc, a, b, o));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return o;
}
Tensor mm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const OptTensor& out, std::optional<at::ScalarType> dtype,
          bool accumulate) {
  return gemm(a, b, a_mn, b_mn, out, dtype, accumulate, 1.0, 0, 0, std::nullopt, std::nullopt, 0, 0, 0);
}
// the two gradients of a linear layer; dw goes to `out` (added with `accumulate`)
std::pair<Tensor, Tensor> dgrad_wgrad(const Tensor& dy, const Tensor& w, const Tensor& x, const OptTensor& out, bool accumulate) {
  Tensor dx = check_product(dy, w, false, true, std::nullopt, std::nullopt), dw = check_product(dy, x, true, true, out, w.scalar_type());
  const NpGemmArgs a = product(dy, w, false, true, dx, false, 1.0), b = product(dy, x, true, true, dw, accumulate, 1.0);
  const int rc = np_gemm_bf16_two(&a, &b, stream());
  if (rc) fail(g_kernel_error, describe("gemm_bf16_two", rc, dy, w, dw));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return {dx, dw};
}

// ----------------------------------------------------------------------------------------------------- linear layer
struct Linear : torch::autograd::Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w) {
    ctx->save_for_backward({x, w});
    ctx->set_materialize_grads(false);
    const int64_t K = x.size(-1);
    Tensor y = mm(x.dim() == 2 ? x : x.reshape({-1, K}), w, false, false, std::nullopt, std::nullopt, false);
    if (x.dim() == 2) return y;
    auto shape = x.sizes().vec();
    shape.back() = w.size(0);
    return y.view(shape);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    at::AutoGradMode no_grad(false);   // nothing here is differentiated a second time
    Tensor dy2 = grads[0].dim() == 2 ? grads[0] : grads[0].reshape({-1, grads[0].size(-1)});
    if (!dy2.is_contiguous()) dy2 = dy2.contiguous();
    const Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    const bool want_dx = ctx->needs_input_grad(0);
    py::gil_scoped_acquire gil;
    const py::object mg = attr(w, s_main_grad);
    const bool want_dw = ctx->needs_input_grad(1) || mg.ptr();
    Tensor dx, dw;
    PyObject* defer = gemm_global(s_defer);
    if (want_dw && defer && defer != Py_None) {   // zero-bubble schedules: the weight gradient is queued
      if (want_dx) dx = mm(dy2, w, false, true, std::nullopt, std::nullopt, false);
      py::object r = py::reinterpret_borrow<py::object>(gemm_global(s_wgrad_into))(w, dy2, x2);
      if (some(r)) dw = r.cast<Tensor>();
    } else if (want_dw && some(mg)) {
      const Tensor out = mg.cast<Tensor>();
      const bool add = truthy(attr(w, s_dirty));
      if (want_dx) dx = dgrad_wgrad(dy2, w, x2, out, add).first;
      else mm(dy2, x2, true, true, out, std::nullopt, add);
      py::reinterpret_borrow<py::object>(gemm_global(s_done))(w);
    } else if (want_dw && want_dx) {
      std::tie(dx, dw) = dgrad_wgrad(dy2, w, x2, std::nullopt, false);
    } else if (want_dw) {
      dw = mm(dy2, x2, true, true, std::nullopt, w.scalar_type(), false);
    } else if (want_dx) {
      dx = mm(dy2, w, false, true, std::nullopt, std::nullopt, false);
    }
    return {dx.defined() && x.dim() != 2 ? dx.view(x.sizes()) : dx, dw};
  }
};

// ---------------------------------------------------------------------------------------------------------- RMSNorm
struct RmsNorm : torch::autograd::Function<RmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& residual, double eps) {
    const int64_t D = x.size(-1);
    const Tensor x2 = x.reshape({-1, D}).contiguous();
    const Tensor r2 = residual ? residual->reshape({-1, D}).contiguous() : Tensor();
    const int rows = (int)x2.size(0);
    Tensor y = at::empty_like(x2), h = residual ? at::empty_like(x2) : Tensor();
    Tensor rstd = empty_like_of(x, {rows}, at::kFloat);
    launched(np_rmsnorm_fwd(ptr(x2), ptr(r2), ptr<float>(w), ptr(y), ptr(h), ptr<float>(rstd), rows, (int)D, (float)eps, stream()),
             "rmsnorm_fwd");
    y = y.view(x.sizes());
    if (residual) h = h.view(x.sizes());
    ctx->save_for_backward({residual ? h : x2, w, rstd});
    ctx->saved_data["residual"] = (bool)residual;
    ctx->set_materialize_grads(false);
    if (residual) return {y, h};
    return {y};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const bool has_res = ctx->saved_data["residual"].toBool();
    const Tensor dh = has_res ? grads[1] : Tensor();
    if (!grads[0].defined() && !dh.defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const auto saved = ctx->get_saved_variables();
    const Tensor &xin = saved[0], &w = saved[1], &rstd = saved[2];
    at::AutoGradMode no_grad(false);
    const Tensor shaped = grads[0].defined() ? grads[0] : dh;
    const int64_t D = xin.size(-1), rows = xin.numel() / (D > 0 ? D : 1);
    const Tensor dy2 = grads[0].defined() ? grads[0].reshape({rows, D}).contiguous() : at::zeros({rows, D}, xin.options());
    const Tensor dres = dh.defined() ? dh.reshape({rows, D}).contiguous() : Tensor();
    Tensor dx = empty_like_of(xin, {rows, D}, xin.scalar_type());
    Tensor scratch = empty_like_of(xin, {np_rmsnorm_bwd_parts((int)rows), D}, at::kFloat), dw;
    py::gil_scoped_acquire gil;
    // weights whose gradient is partial per TP rank go through autograd so their reduce hook runs
    const py::object mg = truthy(attr(w, s_tp_partial)) ? py::object() : attr(w, s_main_grad);
    const bool into = some(mg), add = into && truthy(attr(w, s_dirty));
    if (!into) dw = empty_like_of(xin, {D}, at::kFloat);
    const Tensor out = into ? mg.cast<Tensor>() : dw;
    launched(np_rmsnorm_bwd(ptr(dy2), ptr(xin), ptr<float>(w), ptr<float>(rstd), ptr(dres), ptr(dx), ptr<float>(out), ptr<float>(scratch),
                            (int)rows, (int)D, add, stream()), "rmsnorm_bwd");
    if (into) py::reinterpret_steal<py::object>(THPVariable_Wrap(w)).attr(py::handle(s_dirty)) = true;
    dx = dx.view(shaped.sizes());
    return {dx, dw, has_res ? dx : Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------------- attention
bool rows_aligned(const Tensor& t) {
  return t.stride(3) == 1 && (uintptr_t)t.data_ptr() % 16 == 0 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 &&
         t.stride(0) != 0 && t.stride(1) != 0 && t.stride(2) != 0;
}
struct Heads {   // [B, S, H, hd] inside a packed [B, S, (hq + 2 hkv) hd] buffer, heads from h0 on
  char* p;
  long long sb, ss, sh;
};
Heads heads(const Tensor& buf, int64_t h0, int64_t hd) {
  return {(char*)buf.data_ptr() + h0 * hd * buf.element_size(), (long long)buf.stride(0), (long long)buf.stride(1), (long long)hd};
}

// Rotation (and per-head LayerNorm) of the q and k heads of a fused projection, and causal or full attention of the result:
// qkv [B, S, (hq + 2 hkv) hd] -> [B, S, hq hd].
struct QkvAttention : torch::autograd::Function<QkvAttention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const OptTensor& gq, const OptTensor& bq, const OptTensor& gk,
                        const OptTensor& bk, double eps, const Tensor& cos, const Tensor& sin, int64_t hq, int64_t hkv, int64_t hd,
                        int64_t pos, const OptTensor& pos_ids, bool causal, double scale) {
    const int64_t B = qkv.size(0), S = qkv.size(1), H = hq + 2 * hkv;
    require(qkv.dim() == 3 && qkv.size(2) == H * hd && qkv.stride(2) == 1 && qkv.stride(0) == S * qkv.stride(1), "packed projection");
    Tensor buf = empty_like_of(qkv, {B, S, H * hd}, at::kBFloat16), stats;
    const int* ids = pos_ids ? ptr<int>(*pos_ids) : nullptr;
    const float *c = ptr<float>(cos), *s = ptr<float>(sin);
    Tensor f[4];
    const Heads q0 = heads(qkv, 0, hd), k0 = heads(qkv, hq, hd), v0 = heads(qkv, hq + hkv, hd);
    if (gq) {
      const OptTensor* par[4] = {&gq, &bq, &gk, &bk};
      for (int i = 0; i < 4; ++i) f[i] = (*par[i])->detach().to(at::kFloat).contiguous();
      stats = empty_like_of(qkv, {B * S, hq + hkv, 2}, at::kFloat);
      launched(np_qkv_norm_rope_fwd(ptr(qkv), qkv.stride(1), (int)hq, (int)hkv, ptr<float>(f[0]), ptr<float>(f[1]), ptr<float>(f[2]),
                                    ptr<float>(f[3]), (float)eps, ptr(buf), ptr(stats), c, s, ids, B * S, (int)S, (int)pos, stream()),
               "qkv_norm_rope_fwd");
    } else {
      launched(np_qkv_rope(q0.p, q0.ss, hd, (int)hq, k0.p, k0.ss, hd, (int)hkv, v0.p, v0.ss, hd, (int)hkv, ptr(buf), c, s, ids, B * S,
                           (int)S, (int)pos, (int)hd, (int)(2 * cos.size(1)), (int)(hq + hkv), 1.f, stream()), "qkv_rope");
    }
    Tensor o = empty_like_of(qkv, {B, S, hq * hd}, at::kBFloat16), lse = empty_like_of(qkv, {B, hq, S}, at::kFloat);
    const Heads q = heads(buf, 0, hd), k = heads(buf, hq, hd), v = heads(buf, hq + hkv, hd), oh = heads(o, 0, hd);
    const void *kp[1] = {k.p}, *vp[1] = {v.p};
    NpAttnFwdArgs a{};
    a.q = q.p; a.q_sb = q.sb; a.q_ss = q.ss; a.q_sh = q.sh;
    a.k_ptrs = kp; a.v_ptrs = vp; a.k_sb = k.sb; a.k_ss = k.ss; a.k_sh = k.sh;
    a.o = oh.p; a.o_sb = oh.sb; a.o_ss = oh.ss; a.o_sh = oh.sh; a.lse = ptr<float>(lse);
    a.B = (int)B; a.Sq = (int)S; a.Hq = (int)hq; a.Hkv = (int)hkv; a.causal = causal; a.n_src = 1; a.src_len = (int)S;
    a.scale = (float)scale; a.head_dim = (int)hd;
    launched(np_attn_fwd(&a, stream()), "attn_fwd");
    const Tensor none;
    ctx->save_for_backward({gq ? qkv : none, buf, o, lse, stats, gq ? f[0] : none, gq ? f[2] : none, cos, sin, pos_ids ? *pos_ids : none});
    ctx->saved_data["cfg"] = std::vector<int64_t>{hq, hkv, hd, pos, (int64_t)causal, (int64_t)(bool)gq};
    ctx->saved_data["scale"] = scale;
    if (gq) {
      const OptTensor* par[4] = {&gq, &bq, &gk, &bk};
      std::vector<int64_t> types;
      for (int i = 0; i < 4; ++i) types.push_back((int64_t)(*par[i])->scalar_type());
      ctx->saved_data["types"] = types;
    }
    ctx->set_materialize_grads(false);
    return o;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list res(15);
    if (!grads[0].defined()) return res;
    const auto saved = ctx->get_saved_variables();
    const Tensor &qkv = saved[0], &buf = saved[1], &o = saved[2], &lse = saved[3], &stats = saved[4], &cos = saved[7], &sin = saved[8];
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    const int64_t hq = cfg[0], hkv = cfg[1], hd = cfg[2], pos = cfg[3];
    const bool norm = cfg[5] != 0;
    at::AutoGradMode no_grad(false);
    const int64_t B = buf.size(0), S = buf.size(1);
    const int* ids = ptr<int>(saved[9]);
    // dO is read through a tensor map: a strided view of 16-byte aligned rows, no broadcast dimension
    Tensor d_o = grads[0].reshape({B, S, hq, hd});
    if (!rows_aligned(d_o)) d_o = d_o.clone(at::MemoryFormat::Contiguous);
    Tensor delta = at::empty_like(lse), dq = empty_like_of(buf, {B, S, hq, hd}, at::kBFloat16),
           dk = empty_like_of(buf, {B, S, hkv, hd}, at::kBFloat16), dv = at::empty_like(dk);
    const Heads q = heads(buf, 0, hd), k = heads(buf, hq, hd), v = heads(buf, hq + hkv, hd), oh = heads(o, 0, hd);
    const void *ks[1] = {k.p}, *vs[1] = {v.p}, *qs[1] = {q.p}, *dos[1] = {d_o.data_ptr()};
    const float *ls[1] = {ptr<float>(lse)}, *ds[1] = {ptr<float>(delta)};
    NpAttnBwdArgs a{};
    a.q = q.p; a.q_sb = q.sb; a.q_ss = q.ss; a.q_sh = q.sh;
    a.k = k.p; a.v = v.p; a.k_sb = k.sb; a.k_ss = k.ss; a.k_sh = k.sh;
    a.o = oh.p; a.o_sb = oh.sb; a.o_ss = oh.ss; a.o_sh = oh.sh;
    a.d_o = d_o.data_ptr(); a.do_sb = d_o.stride(0); a.do_ss = d_o.stride(1); a.do_sh = d_o.stride(2);
    a.lse = ls[0]; a.delta = ptr<float>(delta);
    a.dq = dq.data_ptr(); a.dq_sb = dq.stride(0); a.dq_ss = dq.stride(1); a.dq_sh = dq.stride(2);
    a.dk = dk.data_ptr(); a.dv = dv.data_ptr(); a.dk_sb = dk.stride(0); a.dk_ss = dk.stride(1); a.dk_sh = dk.stride(2);
    a.k_src = ks; a.v_src = vs; a.q_src = qs; a.do_src = dos; a.lse_src = ls; a.delta_src = ds;
    a.B = (int)B; a.Sq = (int)S; a.Sk = (int)S; a.Hq = (int)hq; a.Hkv = (int)hkv; a.causal = (int)cfg[4]; a.n_src = 1; a.phase = 3;
    a.scale = (float)ctx->saved_data["scale"].toDouble(); a.head_dim = (int)hd;
    launched(np_attn_bwd(&a, stream()), "attn_bwd");
    Tensor dqkv = empty_like_of(buf, {B, S, (hq + 2 * hkv) * hd}, at::kBFloat16);
    if (norm) {
      Tensor dpar = empty_like_of(buf, {4, hd}, at::kFloat),
             scratch = empty_like_of(buf, {np_qkv_norm_rope_parts(B * S), 4 * hd}, at::kFloat);
      launched(np_qkv_norm_rope_bwd(ptr(dq), dq.stride(1), dq.stride(2), ptr(dk), dk.stride(1), dk.stride(2), ptr(dv), dv.stride(1),
                                    dv.stride(2), ptr(qkv), qkv.stride(1), (int)hq, (int)hkv, ptr<float>(saved[5]), ptr<float>(saved[6]),
                                    ptr(stats), ptr(dqkv), ptr<float>(dpar), ptr<float>(scratch), ptr<float>(cos), ptr<float>(sin), ids,
                                    B * S, (int)S, (int)pos, 0, stream()), "qkv_norm_rope_bwd");
      const auto types = ctx->saved_data["types"].toIntVector();
      for (int i = 0; i < 4; ++i) res[1 + i] = dpar[i].to((at::ScalarType)types[i]);
    } else {
      launched(np_qkv_rope(ptr(dq), dq.stride(1), dq.stride(2), (int)hq, ptr(dk), dk.stride(1), dk.stride(2), (int)hkv, ptr(dv),
                           dv.stride(1), dv.stride(2), (int)hkv, ptr(dqkv), ptr<float>(cos), ptr<float>(sin), ids, B * S, (int)S, (int)pos,
                           (int)hd, (int)(2 * cos.size(1)), (int)(hq + hkv), -1.f, stream()), "qkv_rope_bwd");
    }
    res[0] = dqkv;
    return res;
  }
};

// Rotation of x [B, S, H, hd] (contiguous heads, rows of any stride)
struct Rope : torch::autograd::Function<Rope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& cos, const Tensor& sin, int64_t pos,
                        const OptTensor& pos_ids) {
    const int64_t B = x.size(0), S = x.size(1), H = x.size(2), hd = x.size(3);
    require(x.stride(3) == 1 && x.stride(2) == hd && x.stride(0) == S * x.stride(1), "contiguous heads");
    Tensor out = empty_like_of(x, {B, S, H, hd}, x.scalar_type());
    launched(np_rope(ptr(x), ptr(out), ptr<float>(cos), ptr<float>(sin), pos_ids ? ptr<int>(*pos_ids) : nullptr, B * S, (int)S, (int)pos,
                     (int)H, (int)hd, (int)(2 * cos.size(1)), x.stride(1), out.stride(1), 1.f, stream()), "rope");
    ctx->save_for_backward({cos, sin, pos_ids ? *pos_ids : Tensor()});
    ctx->saved_data["pos"] = pos;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto saved = ctx->get_saved_variables();
    at::AutoGradMode no_grad(false);
    Tensor dy = grads[0];
    const int64_t B = dy.size(0), S = dy.size(1), H = dy.size(2), hd = dy.size(3);
    if (!(dy.stride(3) == 1 && dy.stride(2) == hd && dy.stride(0) == S * dy.stride(1))) dy = dy.contiguous();
    Tensor dx = empty_like_of(dy, {B, S, H, hd}, dy.scalar_type());
    launched(np_rope(ptr(dy), ptr(dx), ptr<float>(saved[0]), ptr<float>(saved[1]), ptr<int>(saved[2]), B * S, (int)S,
                     (int)ctx->saved_data["pos"].toInt(), (int)H, (int)hd, (int)(2 * saved[0].size(1)), dy.stride(1), dx.stride(1), -1.f,
                     stream()), "rope");
    return {dx, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// Attention of a few new positions behind a KV cache (no gradients): out and the concatenated keys and values
std::tuple<Tensor, Tensor, Tensor> decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k_new, const Tensor& v_new,
                                          bool causal, double scale) {
  const int64_t B = q.size(0), Sq = q.size(1), Hq = q.size(2), hd = q.size(3), P = k.size(1), Hkv = k.size(2), n = k_new.size(1);
  Tensor o = empty_like_of(q, {B, Sq, Hq, hd}, at::kBFloat16), ko = empty_like_of(q, {B, P + n, Hkv, hd}, at::kBFloat16),
         vo = at::empty_like(ko);
  NpDecodeArgs a{};
  a.q = q.data_ptr(); a.q_sb = q.stride(0); a.q_ss = q.stride(1); a.q_sh = q.stride(2);
  a.kc = k.data_ptr(); a.kc_sb = k.stride(0); a.kc_ss = k.stride(1); a.kc_sh = k.stride(2);
  a.vc = v.data_ptr(); a.vc_sb = v.stride(0); a.vc_ss = v.stride(1); a.vc_sh = v.stride(2);
  a.kn = k_new.data_ptr(); a.kn_sb = k_new.stride(0); a.kn_ss = k_new.stride(1); a.kn_sh = k_new.stride(2);
  a.vn = v_new.data_ptr(); a.vn_sb = v_new.stride(0); a.vn_ss = v_new.stride(1); a.vn_sh = v_new.stride(2);
  a.ko = ko.data_ptr(); a.vo = vo.data_ptr(); a.o = o.data_ptr();
  a.B = (int)B; a.Sq = (int)Sq; a.Hq = (int)Hq; a.Hkv = (int)Hkv; a.past = (int)P; a.fresh = (int)n; a.causal = causal;
  a.head_dim = (int)hd;
  a.scale = (float)scale;
  launched(np_decode_attn(&a, stream()), "decode_attn");
  return {o, ko, vo};
}

// ------------------------------------------------------------------------------------------------ mixture of experts
// logits -> top-k -> gating weights, with the load-balance and z-loss statistics: weights, indices, aux, counts
struct Router : torch::autograd::Function<Router> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x2, const Tensor& gate_w, const OptTensor& gate_b,
                               const OptTensor& score_bias, int64_t K, int64_t gating, double coef_z) {
    const int T = (int)x2.size(0), D = (int)x2.size(1), E = (int)gate_w.size(0);
    const auto i32 = x2.options().dtype(at::kInt), f32 = x2.options().dtype(at::kFloat);
    Tensor logits = at::empty({T, E}, f32), weights = at::empty({T, K}, f32), indices = at::empty({T, K}, i32);
    // token counts; probability sums, sum of lse^2 (set to zero by the first kernel, if it runs)
    Tensor counts_all = T > 0 ? at::empty({2 * E + 1}, i32) : at::zeros({2 * E + 1}, i32);
    Tensor counts = counts_all.narrow(0, 0, E);
    int* c = ptr<int>(counts_all);
    float *psum = (float*)(c + E), *zsum = psum + E;
    const float* sb = score_bias ? ptr<float>(*score_bias) : nullptr;
    launched(np_router_logits(ptr(x2), ptr<float>(gate_w), gate_b ? ptr<float>(*gate_b) : nullptr, ptr<float>(logits), T, D, E, c,
                              2 * E + 1, stream()), "router_logits");
    launched(np_router_topk(ptr<float>(logits), sb, ptr<float>(weights), ptr<int>(indices), c, psum, zsum, T, E, (int)K, (int)gating,
                            stream()), "router_topk");
    // tensors of their own: an output that is a view beside another differentiable output may not be changed in place,
    // and the saved load fractions must not share the loss's version counter
    Tensor f = at::empty({E}, f32), aux = at::empty({}, f32);
    launched(np_router_aux(c, psum, zsum, (float)coef_z, ptr<float>(f), ptr<float>(aux), T, E, stream()), "router_aux");
    ctx->save_for_backward({x2, gate_w, logits, weights, indices, f, score_bias ? *score_bias : Tensor()});
    ctx->saved_data["cfg"] = std::vector<int64_t>{K, gating};
    ctx->saved_data["z"] = coef_z;
    ctx->mark_non_differentiable({indices, counts});
    ctx->set_materialize_grads(false);
    return {weights, indices, aux, counts};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list res(7);
    if (!grads[0].defined() && !grads[2].defined()) return res;
    const auto saved = ctx->get_saved_variables();
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    const Tensor &x2 = saved[0], &gate_w = saved[1], &logits = saved[2], &sb = saved[6];
    at::AutoGradMode no_grad(false);
    const int T = (int)logits.size(0), E = (int)logits.size(1), D = (int)x2.size(1);
    const Tensor dw = grads[0].defined() ? grads[0].contiguous() : Tensor();
    const Tensor da = grads[2].defined() ? grads[2].reshape({1}).to(at::kFloat).contiguous() : Tensor();
    Tensor dl = at::empty_like(logits);
    launched(np_router_bwd(ptr<float>(logits), ptr<float>(sb), ptr<float>(saved[3]), ptr<int>(saved[4]), ptr<float>(dw),
                           ptr<float>(saved[5]), ptr<float>(da), 1.f, (float)ctx->saved_data["z"].toDouble(), ptr<float>(dl), T, E,
                           (int)cfg[0], (int)cfg[1], stream()), "router_bwd");
    const auto f32 = x2.options().dtype(at::kFloat);
    Tensor scratch = at::empty({np_router_dgate_scratch(T, D, E)}, f32);
    Tensor dgw = empty_like_of(x2, gate_w.sizes(), gate_w.scalar_type()), dgb = at::empty({E}, f32);
    if (T <= 0) {   // no tokens: the kernels below do nothing
      dgw.zero_();
      dgb.zero_();
    }
    launched(np_router_dgate(ptr<float>(dl), ptr(x2), ptr<float>(dgw), ptr<float>(dgb), ptr<float>(scratch), T, D, E, 0, stream()),
             "router_dgate");
    Tensor dx;
    if (x2.scalar_type() == at::kBFloat16 && gate_w.scalar_type() == at::kFloat && gate_w.is_contiguous()) {
      dx = at::empty_like(x2);
      launched(np_router_dx(ptr<float>(dl), ptr<float>(gate_w), ptr(dx), T, D, E, stream()), "router_dx");
    } else {
      dx = at::matmul(dl, gate_w.to(at::kFloat)).to(x2.scalar_type());
    }
    res[0] = dx; res[1] = dgw; res[2] = dgb;
    return res;
  }
};

// What the launches of FusedMoERuntime (ops/moe.py) take from it: sizes, buffers and tables that it keeps for its whole life. One rank:
// the form with peers is the Python one.
struct MoeRuntime : torch::CustomClassHolder {
  int64_t T, D, H, E, K, N, rank, E_local, R, bpr, rows_total, blocks, capacity, max_ctas, wait_ns;
  std::vector<Tensor> recv_x, ret_y, p_recv_x, p_ret_y;
  Tensor recv_g, ret_g, row_dst, mblk_rows, src_blocks, dispatch_flags, combine_flags, p_recv_g, p_ret_g, p_row_dst, p_mblk_rows,
      p_src_blocks, p_dispatch_flags, p_done_flag, mblk_group, mblk_flag, done_counters, dispatch_ctr, epoch_base;
  py::object heap, owner;   // the symmetric heap (epochs); weak reference to the Python runtime

  MoeRuntime(py::object rt, int64_t wait_limit_ns) : wait_ns(wait_limit_ns) {
    auto num = [&](const char* n) { return rt.attr(n).cast<int64_t>(); };
    auto ten = [&](const char* n) { return rt.attr(n).cast<Tensor>(); };
    auto list = [&](const char* n) { return rt.attr(n).cast<std::vector<Tensor>>(); };
    T = num("T"); D = num("D"); H = num("H"); E = num("E"); K = num("K"); N = num("N"); rank = num("rank"); E_local = num("E_local");
    R = num("R"); bpr = num("bpr"); rows_total = num("rows_total"); blocks = num("blocks"); capacity = num("capacity");
    max_ctas = num("max_ctas_dispatch");
    recv_x = list("recv_x"); ret_y = list("ret_y"); p_recv_x = list("p_recv_x"); p_ret_y = list("p_ret_y");
    recv_g = ten("recv_g"); ret_g = ten("ret_g"); row_dst = ten("row_dst"); mblk_rows = ten("mblk_rows"); src_blocks = ten("src_blocks");
    dispatch_flags = ten("dispatch_flags"); combine_flags = ten("combine_flags"); p_recv_g = ten("p_recv_g"); p_ret_g = ten("p_ret_g");
    p_row_dst = ten("p_row_dst"); p_mblk_rows = ten("p_mblk_rows"); p_src_blocks = ten("p_src_blocks");
    p_dispatch_flags = ten("p_dispatch_flags"); p_done_flag = ten("p_done_flag"); mblk_group = ten("mblk_group");
    mblk_flag = ten("mblk_flag"); done_counters = ten("done_counters"); dispatch_ctr = ten("dispatch_ctr");
    require(N == 1, "the native form of the expert layer is that of one rank");
    heap = rt.attr("heap");
    epoch_base = heap.attr("epoch_base").cast<Tensor>();
    owner = py::module_::import("weakref").attr("ref")(rt);
  }
  ~MoeRuntime() override {
    py::gil_scoped_acquire gil;
    heap = py::object();
    owner = py::object();
  }
  int next_epoch() const {
    py::gil_scoped_acquire gil;
    return heap.attr("next_epoch")().cast<int>();
  }
  // the counters of a product that pushes its rows: once behind every dispatch, the runtime refuses more
  int* push_counters() const {
    py::gil_scoped_acquire gil;
    py::object rt = owner();
    return rt.is_none() ? ptr<int>(done_counters) : (int*)rt.attr("_push_counters")().cast<uintptr_t>();
  }
  void dispatch(const Tensor& x, const Tensor& idx, const Tensor& slot_pos, const Tensor& counts, const Tensor& scale, const Tensor& rows,
                int epoch) const {
    NpDispatchArgs a{};
    a.x = x.data_ptr(); a.indices = ptr<int>(idx); a.slot_pos = ptr<int>(slot_pos); a.counts_kept = ptr<int>(counts);
    a.slot_scale = ptr<float>(scale);
    a.T = (int)T; a.K = (int)K; a.D = (int)D; a.E = (int)E; a.E_local = (int)E_local; a.n_ranks = (int)N; a.my_rank = (int)rank;
    a.region_rows = (int)R;
    a.peer_rows = (void* const*)rows.data_ptr();
    a.peer_row_dst = (long long* const*)p_row_dst.data_ptr(); a.peer_mblk_rows = (int* const*)p_mblk_rows.data_ptr();
    a.peer_src_blocks = (int* const*)p_src_blocks.data_ptr(); a.peer_flags = (int* const*)p_dispatch_flags.data_ptr();
    a.done_ctr = ptr<int>(dispatch_ctr); a.epoch = epoch; a.write_meta = 1; a.max_ctas = (int)max_ctas;
    a.epoch_base = ptr<int>(epoch_base); a.zero_ctr = ptr<int>(done_counters);
    launched(np_ep_dispatch(&a, stream()), "ep_dispatch");
    py::gil_scoped_acquire gil;
    py::object rt = owner();
    if (!rt.is_none()) rt.attr("_may_push") = true;
  }
  void combine(const Tensor& rows, const Tensor& slot_pos, const Tensor& weights, const Tensor& add, const Tensor& out, const Tensor& sent,
               int epoch) const {
    NpCombineArgs a{};
    a.rows = rows.data_ptr(); a.slot_pos = ptr<int>(slot_pos); a.weights = ptr<float>(weights); a.add1 = ptr(add); a.out = out.data_ptr();
    a.T = (int)T; a.K = (int)K; a.D = (int)D; a.E = (int)E; a.flags = ptr<int>(combine_flags); a.sent_to_peer = ptr<int>(sent);
    a.n_ranks = (int)N; a.epoch = epoch; a.limit_ns = (unsigned long long)wait_ns; a.epoch_base = ptr<int>(epoch_base);
    launched(np_ep_combine(&a, stream()), "ep_combine");
  }
  // rows grouped by expert: A [rows_total, K] times the expert's rows of B
  NpGemmArgs by_rows(const Tensor& A, const Tensor& B, int64_t n, int64_t k, bool b_mn) const {
    NpGemmArgs g{};
    g.A = A.data_ptr(); g.B = B.data_ptr(); g.lda = A.stride(0); g.ldb = B.stride(0); g.a_rows = A.size(0); g.b_rows = B.size(0);
    g.M = (int)rows_total; g.N = (int)n; g.K = (int)k; g.b_mn = b_mn; g.mode = 1; g.alpha = 1.f; g.paired = bpr % 2 == 0;
    g.mblk_group = ptr<int>(mblk_group); g.mblk_rows = ptr<int>(mblk_rows); g.group_stride_b = H; g.mblk_flag = ptr<int>(mblk_flag);
    g.epoch_base = ptr<int>(epoch_base);
    return g;
  }
  void wait_for(NpGemmArgs& g, int epoch) const {   // tiles wait for the rows of the dispatch
    g.ready_flags = ptr<int>(dispatch_flags); g.epoch = epoch; g.flag_limit_ns = (unsigned long long)wait_ns;
  }
  void push_to(NpGemmArgs& g, const Tensor& peers, int epoch) const {   // output rows go back to their sources
    g.row_dst = (const long long*)row_dst.data_ptr(); g.peer_base = (void* const*)peers.data_ptr();
    g.done_counters = push_counters(); g.done_expected = ptr<int>(src_blocks);
    g.done_flag_ptr = (int* const*)p_done_flag.data_ptr(); g.epoch = epoch; g.ldc = g.N; g.local_push = 1;
  }
  // A [rows, M (x outputs)] and B [rows, N] contracted over the rows of every expert, into the fp32 outputs of M rows per expert
  NpGemmArgs by_expert(const Tensor& A, const Tensor& B, int64_t M, int64_t n, const std::vector<Tensor>& outs, bool add) const {
    NpGemmArgs g{};
    g.A = A.data_ptr(); g.B = B.data_ptr(); g.C = outs[0].data_ptr(); g.lda = A.stride(0); g.ldb = B.stride(0); g.ldc = n;
    g.a_rows = A.size(0); g.b_rows = B.size(0); g.M = (int)(M * (int64_t)outs.size()); g.N = (int)n; g.K = (int)rows_total;
    if (outs.size() > 1) { g.C2 = outs[1].data_ptr(); g.m_split = (int)M; }
    g.a_mn = g.b_mn = 1; g.mode = 2; g.alpha = 1.f; g.out_f32 = 1; g.accumulate = add; g.mblk_rows = ptr<int>(mblk_rows);
    g.num_groups = (int)E_local; g.blocks_per_group = (int)(N * bpr); g.group_stride_c = M * n;
    return g;
  }
  // A product over the dispatched rows and the weight gradient beside it, together: without peers the rows are there when the dispatch
  // kernel has ended. The six expert GEMMs, us, apart / paired: 4096 tokens, 8 experts of 2048 x 2816 606 / 525, 512 of 768 x 2048
  // 199 / 174, 2472, 16 of 1024 x 2816 417 / 382.
  void both(const NpGemmArgs& rows, const NpGemmArgs& experts) const {
    launched(np_gemm_bf16_two(&rows, &experts, stream()), "grouped_gemm and grouped_wgrad");
  }
};

// Weight gradients of one launch: into the weights' main_grad where they have one, else new tensors. `launch` gets the fp32
// outputs and whether to add.
struct ExpertGrads {
  std::vector<Tensor> outs, grads;   // where the kernel writes; what autograd gets (undefined: nothing)
  bool add = false, main = false;
};
ExpertGrads expert_outputs(const std::vector<Tensor>& ws, int64_t rows, int64_t cols) {
  ExpertGrads r;
  py::gil_scoped_acquire gil;
  const py::object mg = attr(ws[0], s_main_grad);
  r.main = some(mg);
  r.add = r.main && truthy(attr(ws[0], s_dirty));
  for (const Tensor& w : ws)
    r.outs.push_back(r.main ? attr(w, s_main_grad).cast<Tensor>() : empty_like_of(w, {rows, cols}, at::kFloat));
  return r;
}
void expert_done(ExpertGrads& r, const std::vector<Tensor>& ws) {
  if (r.main) {
    py::gil_scoped_acquire gil;
    for (const Tensor& w : ws) py::reinterpret_steal<py::object>(THPVariable_Wrap(w)).attr(py::handle(s_dirty)) = true;
    r.grads.resize(ws.size());
  } else {
    for (size_t i = 0; i < ws.size(); ++i) r.grads.push_back(r.outs[i].to(ws[i].scalar_type()));
  }
}
bool same_main_grad(const Tensor& a, const Tensor& b) {
  py::gil_scoped_acquire gil;
  return some(attr(a, s_main_grad)) == some(attr(b, s_main_grad)) && truthy(attr(a, s_dirty)) == truthy(attr(b, s_dirty));
}

// The bf16 form of ops.moe._FusedMoE on one rank: plan, dispatch, expert GEMMs, combine, and their mirror. Returns the output and the
// tokens that each expert dropped.
struct FusedMoE : torch::autograd::Function<FusedMoE> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weights, const Tensor& idx, const Tensor& w1,
                               const Tensor& w3, const Tensor& w2, c10::intrusive_ptr<MoeRuntime> rt, int64_t layer,
                               const OptTensor& stats, const OptTensor& shared) {
    const int64_t T = rt->T, D = rt->D, K = rt->K, H = rt->H;
    const Tensor x2 = x.reshape({T, D}).contiguous();
    const auto i32 = x.options().dtype(at::kInt), b16 = x.options().dtype(at::kBFloat16);
    Tensor slot_pos = at::empty({T, K}, i32), keep = at::empty({T}, i32), counts = at::empty({rt->E}, i32), drops = at::empty({rt->E}, i32),
           n_dropped = at::empty({1}, i32), sent = at::empty({rt->N}, i32);
    launched(np_capacity_plan(ptr<int>(idx), (int)T, (int)rt->E, (int)K, (int)rt->capacity, ptr<int>(slot_pos), ptr<int>(keep),
                              ptr<int>(counts), ptr<int>(drops), ptr<int>(n_dropped), ptr<int>(sent), (int)rt->N,
                              stats ? (long long*)stats->data_ptr() : nullptr, stream()), "capacity_plan");
    const int epoch = rt->next_epoch();
    Tensor gu = at::empty({rt->rows_total, 2 * H}, b16), h = at::empty({rt->rows_total, H}, b16);
    rt->dispatch(x2, idx, slot_pos, counts, Tensor(), rt->p_recv_x[layer], epoch);
    // [gate | up] GEMM with the SwiGLU epilogue, waits per block on the source's arrival flag
    NpGemmArgs g = rt->by_rows(rt->recv_x[layer], w1, H, D, false);
    g.B2 = w3.data_ptr(); g.epilogue = 1; g.C2 = gu.data_ptr(); g.ldc2 = gu.stride(0); g.C = h.data_ptr(); g.ldc = h.stride(0);
    rt->wait_for(g, epoch);
    launched(np_gemm_bf16(&g, stream()), "grouped_gemm");
    // down projection (w2 is stored [H, D] per expert: MN-major B), rows pushed back to their sources
    g = rt->by_rows(h, w2, D, H, true);
    rt->push_to(g, rt->p_ret_y[layer], epoch);
    launched(np_gemm_bf16(&g, stream()), "grouped_gemm");
    Tensor out = at::empty({T, D}, b16), add;
    // the shared expert's output joins in the combine pass; a token dropped by the capacity rule gets no MoE output at all,
    // shared expert included (reference: model/moe.py:1383-1390)
    if (shared) add = shared->reshape({T, D}) * keep.to(shared->scalar_type()).unsqueeze(1);
    rt->combine(rt->ret_y[layer], slot_pos, weights, add, out, sent, epoch);
    ctx->save_for_backward({x2, weights, idx, slot_pos, counts, sent, gu, w1, w3, w2, h, shared ? keep : Tensor()});
    ctx->saved_data["rt"] = c10::IValue::make_capsule(rt);
    ctx->saved_data["layer"] = layer;
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->mark_non_differentiable({drops});
    ctx->set_materialize_grads(false);
    return {out.view(x.sizes()), drops};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list res(10);
    if (!grads[0].defined()) return res;
    const auto saved = ctx->get_saved_variables();
    const Tensor &weights = saved[1], &idx = saved[2], &slot_pos = saved[3], &counts = saved[4], &sent = saved[5], &gu = saved[6],
                 &w1 = saved[7], &w3 = saved[8], &w2 = saved[9], &h = saved[10], &keep = saved[11];
    const auto rt = c10::static_intrusive_pointer_cast<MoeRuntime>(ctx->saved_data["rt"].toCapsule());
    const int64_t layer = ctx->saved_data["layer"].toInt();
    const auto shape = ctx->saved_data["shape"].toIntVector();
    at::AutoGradMode no_grad(false);
    const int64_t T = rt->T, D = rt->D, K = rt->K, H = rt->H;
    const Tensor do2 = grads[0].reshape({T, D}).contiguous();
    const auto b16 = do2.options().dtype(at::kBFloat16);
    // d(router weights)[t, k] = <dout[t], y[t, k]>
    Tensor dweights = at::empty({T, K}, do2.options().dtype(at::kFloat));
    launched(np_slot_dot(ptr(do2), ptr(rt->ret_y[layer]), ptr<int>(slot_pos), ptr<float>(dweights), (int)T, (int)K, (int)D, stream()),
             "slot_dot");
    // send w[t, k] * dout[t] to the experts (same slots as forward)
    const int epoch = rt->next_epoch();
    rt->dispatch(do2, idx, slot_pos, counts, weights, rt->p_recv_g, epoch);
    // dH = dY @ w2^T (w2 [H, D] per expert is K-major for this contraction), taken to [dG | dU] in the epilogue
    Tensor dgu = at::empty_like(gu);
    NpGemmArgs g = rt->by_rows(rt->recv_g, w2, H, D, false);
    g.epilogue = 2; g.C2 = gu.data_ptr(); g.ldc2 = gu.stride(0); g.C = dgu.data_ptr(); g.ldc = dgu.stride(0);
    rt->wait_for(g, epoch);
    ExpertGrads d2 = expert_outputs({w2}, rt->E_local * H, D);
    rt->both(g, rt->by_expert(h, rt->recv_g, H, D, d2.outs, d2.add));
    expert_done(d2, {w2});
    const Tensor& xr = rt->recv_x[layer];
    Tensor dw1, dw3;
    // dX = [dG | dU] @ [w1; w3], one contraction over both weights (no bf16 partial result in between), pushed back to the
    // sources. H is a multiple of 256 (MoEBase), the K steps of 64 never straddle the two.
    g = rt->by_rows(dgu, w1, D, 2 * H, true);
    g.B2 = w3.data_ptr(); g.k_split = (int)H;
    rt->push_to(g, rt->p_ret_g, epoch);
    if (H % 256 == 0 && same_main_grad(w1, w3)) {   // gate and up against the same rows in one product
      ExpertGrads d = expert_outputs({w1, w3}, rt->E_local * H, D);
      rt->both(g, rt->by_expert(dgu, xr, H, D, d.outs, d.add));
      expert_done(d, {w1, w3});
      dw1 = d.grads[0]; dw3 = d.grads[1];
    } else {
      launched(np_gemm_bf16(&g, stream()), "grouped_gemm");
      for (int i = 0; i < 2; ++i) {
        const Tensor& w = i ? w3 : w1;
        ExpertGrads d = expert_outputs({w}, rt->E_local * H, D);
        const NpGemmArgs e = rt->by_expert(dgu.narrow(1, i * H, H), xr, H, D, d.outs, d.add);
        launched(np_gemm_bf16(&e, stream()), "grouped_wgrad");
        expert_done(d, {w});
        (i ? dw3 : dw1) = d.grads[0];
      }
    }
    Tensor dx = at::empty({T, D}, b16);
    rt->combine(rt->ret_g, slot_pos, Tensor(), Tensor(), dx, sent, epoch);
    res[0] = dx.view(shape); res[1] = dweights; res[3] = dw1; res[4] = dw3; res[5] = d2.grads[0];
    if (keep.defined()) res[9] = (do2 * keep.to(do2.scalar_type()).unsqueeze(1)).view(shape);
    return res;
  }
};
variable_list router(const Tensor& x2, const Tensor& gate_w, const OptTensor& gate_b, const OptTensor& score_bias, int64_t K,
                     int64_t gating, double coef_z) {
  return Router::apply(x2, gate_w, gate_b, score_bias, K, gating, coef_z);
}
variable_list fused_moe(const Tensor& x, const Tensor& weights, const Tensor& idx, const Tensor& w1, const Tensor& w3, const Tensor& w2,
                        c10::intrusive_ptr<MoeRuntime> rt, int64_t layer, const OptTensor& stats, const OptTensor& shared) {
  return FusedMoE::apply(x, weights, idx, w1, w3, w2, rt, layer, stats, shared);
}

Tensor linear(const Tensor& x, const Tensor& w) { return Linear::apply(x, w); }
variable_list rms_norm(const Tensor& x, const Tensor& w, const OptTensor& residual, double eps) {
  return RmsNorm::apply(x, w, residual, eps);
}
Tensor rope(const Tensor& x, const Tensor& cos, const Tensor& sin, int64_t pos, const OptTensor& ids) {
  return Rope::apply(x, cos, sin, pos, ids);
}
Tensor qkv_attention(const Tensor& qkv, const OptTensor& gq, const OptTensor& bq, const OptTensor& gk, const OptTensor& bk, double eps,
                     const Tensor& cos, const Tensor& sin, int64_t hq, int64_t hkv, int64_t hd, int64_t pos, const OptTensor& pos_ids,
                     bool causal, double scale) {
  return QkvAttention::apply(qkv, gq, bq, gk, bk, eps, cos, sin, hq, hkv, hd, pos, pos_ids, causal, scale);
}

void setup(py::object kernel_error, py::dict gemm_namespace) {
  g_kernel_error = kernel_error.release().ptr();
  g_gemm_dict = gemm_namespace.release().ptr();
}
}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  s_main_grad = PyUnicode_InternFromString("main_grad");
  s_dirty = PyUnicode_InternFromString("_main_grad_dirty");
  s_defer = PyUnicode_InternFromString("_DEFER");
  s_done = PyUnicode_InternFromString("_main_grad_done");
  s_wgrad_into = PyUnicode_InternFromString("_wgrad_into");
  s_tp_partial = PyUnicode_InternFromString("_tp_partial");
  py::class_<MoeRuntime, c10::intrusive_ptr<MoeRuntime>>(m, "MoeRuntime").def(py::init<py::object, int64_t>());
  m.def("router", torch::wrap_pybind_function(router));
  m.def("fused_moe", torch::wrap_pybind_function(fused_moe));
  m.def("setup", &setup);
  m.def("launches", [] { return g_launches.load(); });
  m.def("gemm", torch::wrap_pybind_function(gemm));
  m.def("linear", torch::wrap_pybind_function(linear));
  m.def("rms_norm", torch::wrap_pybind_function(rms_norm));
  m.def("rope", torch::wrap_pybind_function(rope));
  m.def("qkv_attention", torch::wrap_pybind_function(qkv_attention));
  m.def("decode", torch::wrap_pybind_function(decode));
}
