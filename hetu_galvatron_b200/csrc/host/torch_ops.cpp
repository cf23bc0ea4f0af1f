// The autograd nodes of a training step's layers in C++: linear, norm, gated activation, residual add, rotation and packed
// flash attention, and the callbacks at the edges of a sharded unit; and the arguments of a cached decoder layer.
//
// They do what the Python classes of ops/gemm.py, ops/fused.py, ops/attention.py, models/modules.py and parallel/zero.py do,
// with the same kernels, saved tensors, gradients and errors.  What they save is the host: a short kernel takes the GPU a few
// microseconds, and a Python autograd function took the host 30 us for a forward and a backward that do nothing and 75 us
// for those of a linear layer, so that a two-layer step of hidden 512 (84 launches) took 2.5 ms of which the GPU worked 0.6;
// from here 1.75 ms, an attention block of 1531 x 3584 483 us instead of 598, and a decode step of four 4096-wide layers 516
// instead of 587, both now bound by the device.
//
// Every function here returns None when a call is not one of the plain ones (see `plain`), and the caller then takes the
// Python class, which raises what there is to raise.  The kernels' addresses come from the library that ops/_lib.py has
// loaded (bind), so that each build of it is served.
#include <ATen/FuncTorchTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>

#include "../sm100/attn_tensor.h"
#include "../sm100/decoder_step.h"
#include "../sm100/native_interface.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ---- the kernel library ---------------------------------------------------------------------------------------
using V = const void*;
using A = const HgAttnTensor*;
struct Kernels {
  int (*gemm)(V, V, void*, V, int, int, int, int, int, int, int, int, int, int, void*);
  int (*gemm2)(V, V, void*, V, int, int, int, int, int, int, int, int, int, int, void*, long long, void*);
  long long (*gemm2_scratch)(int, int, int);
  int (*gemm_skinny)(V, V, void*, V, int, int, int, int, int, int, int, int, int, void*);
  int (*colsum_parts)(int, int);
  int (*colsum)(V, long long, int, int, void*, int, void*, void*, int, void*);
  int (*norm_fwd)(V, V, V, V, void*, void*, void*, void*, int, int, float, int, void*);
  int (*norm_bwd)(V, V, V, V, V, V, void*, void*, void*, void*, int, int, int, int, int, void*);
  int (*glu_fwd)(V, void*, long long, int, int, void*);
  int (*glu_bwd)(V, V, void*, long long, int, int, void*);
  int (*add)(V, V, void*, long long, void*);
  int (*rope)(void*, V, int, int, int, int, int, V, int, V, V, int, int, void*);
  int (*flash_fwd)(A, A, A, A, void*, int, int, int, int, int, int, int, int, int, float, void*);
  int (*flash_bwd_wants)(int, int, int, int, int, int, int, int, int, long long*);
  int (*flash_bwd_has_room)(int);
  int (*flash_bwd_no_room)(int);
  int (*flash_bwd)(A, A, A, A, A, V, void*, long long, void* const*, int, long long, A, A, A, int, int, int, int, int, int, int, int, int, float, int*, void*);
  long long (*decoder_step_scratch)(const HgDecoderStep*);
  int (*decoder_step)(HgDecoderStep*, void*);
};
Kernels K{};
at::ScalarType g_lp = at::kBFloat16;       // the library's 16-bit type
int g_pair_mode = -1;                      // HG_GEMM_PAIR: -1 auto, 0 never, 1 always
std::atomic<bool> g_pair_ok{true};         // cleared once the device has refused to co-schedule a pair
PyObject* g_kernel_error = nullptr;        // ops._lib.KernelError
std::atomic<long long> g_launches{0};

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
void count(int n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

[[noreturn]] void raise(PyObject* type, const std::string& what) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(type, what.c_str());
  python_error e;
  e.persist();
  throw e;
}
void check(int rc, const char* what) {
  if (rc != 0) raise(g_kernel_error, std::string(what) + " failed with code " + std::to_string(rc));
}

// ---- which calls are taken ------------------------------------------------------------------------------------
// Nothing that wants to see the operations of a call one by one: tracing, functorch, dispatch modes.
bool plain_mode() {
  return !torch::jit::tracer::isTracing() && at::functorch::functorchTLSAccessor() == nullptr &&
         !c10::impl::TorchDispatchModeTLS::any_modes_set();
}
// A dense 16-bit tensor on a GPU that is nothing but that.
bool plain(const Tensor& t) {
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.scalar_type() == g_lp && !at::isTensorSubclassLike(t) &&
         !t._fw_grad(0).defined();
}
bool plain_vector(const Tensor& t, int64_t n, const Tensor& like) {
  return plain(t) && t.dim() == 1 && t.numel() == n && t.is_contiguous() && t.device() == like.device();
}
uintptr_t address(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()); }
bool aligned(const Tensor& t) { return address(t) % 16 == 0; }
Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const Tensor& like) {
  return at::empty(shape, like.options().dtype(dtype).requires_grad(false));
}

// ---- matrix products (ops/gemm.py) -----------------------------------------------------------------------------
enum { kOutLp = 0, kOutF32 = 1, kOutF32Acc = 2 };

Tensor rowmajor(const Tensor& t) { return t.stride(1) != 1 || t.stride(0) % 8 != 0 || !aligned(t) ? t.contiguous() : t; }
// 0: general kernel, 1: CTA pairs, 2: weight streaming.  The rules are those of ops/gemm.py (_use_skinny, _use_pair), which
// say why; a test holds the two against each other.
int route(int64_t M, int64_t N, int64_t Kd, bool a_mn, int mode, int pair_mode, bool pair_ok) {
  if (!a_mn && mode <= kOutF32 && pair_mode != 1) {
    if (M <= 64 ? N <= 65535 * 128 : M <= 128 && N <= 8192 && Kd >= (N <= 4096 ? 1536 : 3072)) return 2;
  }
  if (!pair_ok || pair_mode == 0) return 0;
  return pair_mode == 1 || (M >= 256 && N >= 256) ? 1 : 0;
}
void gemm(const Tensor& a_in, const Tensor& b_in, const Tensor& out, const void* bias, bool a_mn, bool b_mn, int mode) {
  const Tensor a = rowmajor(a_in), b = rowmajor(b_in);
  const int64_t M = a.size(a_mn), Kd = a.size(!a_mn), N = b.size(b_mn);
  const int m = int(M), n = int(N), k = int(Kd), lda = int(a.stride(0)), ldb = int(b.stride(0)), ldc = int(out.stride(0));
  void* st = stream();
  const int how = route(M, N, Kd, a_mn, mode, g_pair_mode, g_pair_ok);
  if (how == 2) {
    check(K.gemm_skinny(a.data_ptr(), b.data_ptr(), out.data_ptr(), bias, m, n, k, lda, ldb, ldc, b_mn, mode, 0, st),
          "hg_gemm_skinny_bf16");
    return count();
  }
  if (how == 1) {
    const long long need = K.gemm2_scratch(m, n, k);        // parts of tiles that several CTA pairs share
    const Tensor ws = need ? empty({need}, at::kByte, a) : Tensor();
    const int rc = K.gemm2(a.data_ptr(), b.data_ptr(), out.data_ptr(), bias, m, n, k, lda, ldb, ldc, a_mn, b_mn, mode, 0,
                           need ? ws.data_ptr() : nullptr, need, st);
    if (rc != -2) {
      check(rc, "hg_gemm2_bf16");
      return count();
    }
    g_pair_ok = false;
  }
  check(K.gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), bias, m, n, k, lda, ldb, ldc, a_mn, b_mn, mode, 0, st), "hg_gemm_bf16");
  count();
}
// The sums of the columns of x, in its type; or, where `into` is defined, written or added to that fp32 vector.
Tensor column_sums(const Tensor& x_in, const Tensor& into = Tensor(), bool accumulate = false) {
  const int64_t rows = x_in.size(0), cols = x_in.size(1);
  const bool graph = at::GradMode::is_enabled() && x_in.requires_grad();     // a graph of the gradient is wanted
  const Tensor x = graph || x_in.scalar_type() != g_lp ? x_in : rowmajor(x_in);
  if (graph || rows == 0 || cols == 0 || x.scalar_type() != g_lp || x.stride(0) % 8 || !aligned(x)) {
    const Tensor sums = x.to(at::kFloat).sum(0);
    if (!into.defined()) return sums.to(x.scalar_type());
    at::NoGradGuard no_grad;
    return accumulate ? into.add_(sums) : into.copy_(sums);
  }
  Tensor out = into.defined() ? into : empty({cols}, g_lp, x);
  const int parts = K.colsum_parts(int(rows), int(cols));
  const Tensor partial = parts > 1 ? empty({parts, cols}, at::kFloat, x) : Tensor();
  check(K.colsum(x.data_ptr(), x.stride(0), int(rows), int(cols), parts > 1 ? partial.data_ptr() : nullptr, parts,
                 into.defined() ? nullptr : out.data_ptr(), into.defined() ? out.data_ptr() : nullptr, accumulate, stream()),
        "hg_colsum");
  count(parts > 1 ? 2 : 1);
  return out;
}

// The fp32 gradient buffer that a sharded unit has bound to a parameter (``p.main_grad``), and whether it holds nothing yet
// (``p.mg_fresh``); read when the gradient is written, since a unit may bind another buffer until then.
struct MainGrad {
  Tensor buf;
  bool fresh = false;
  MainGrad() = default;
  explicit MainGrad(const Tensor& p) {
    pybind11::gil_scoped_acquire gil;
    py::object o = py::reinterpret_steal<py::object>(THPVariable_Wrap(p));
    py::object mg = py::getattr(o, "main_grad", py::none());
    if (mg.is_none()) return;
    if (!THPVariable_Check(mg.ptr())) raise(PyExc_TypeError, "main_grad is no tensor");
    buf = THPVariable_Unpack(mg.ptr());
    fresh = py::cast<bool>(py::bool_(py::getattr(o, "mg_fresh", py::bool_(false))));
  }
  static void written(const Tensor& p) {
    pybind11::gil_scoped_acquire gil;
    py::object o = py::reinterpret_steal<py::object>(THPVariable_Wrap(p));
    py::setattr(o, "mg_fresh", py::bool_(false));
  }
};

// Whether this node may write the gradient of a bias or norm bias to its buffer itself: a vector of `n` fp32 values, in a plain
// backward() into the leaves (autograd.grad, backward(inputs=...) and a graph of the gradient get it through autograd), and nobody on
// the way to the parameter who wants to see it (hooks of the tensor or behind its accumulation).
bool takes_vector(const MainGrad& mg, const Tensor& p, int64_t n) {
  const auto* asked = torch::autograd::get_current_graph_task_exec_info();
  if (at::GradMode::is_enabled() || asked == nullptr || !asked->empty()) return false;
  if (!mg.buf.defined() || mg.buf.scalar_type() != at::kFloat || !mg.buf.is_cuda() || mg.buf.numel() != n || !mg.buf.is_contiguous())
    return false;
  if (!p.is_leaf() || !torch::autograd::impl::hooks(p).empty() || torch::autograd::impl::post_acc_grad_hooks(p) != nullptr) return false;
  const auto node = torch::autograd::impl::try_get_grad_accumulator(p);
  return node == nullptr || (node->pre_hooks().empty() && node->post_hooks().empty() && node->tensor_pre_hooks().empty());
}

struct Linear : public Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias) {
    ctx->save_for_backward({x, w});
    if (bias) ctx->saved_data["bias"] = *bias;      // to find its buffer; its values are not needed and may change
    Tensor y = empty({x.size(0), w.size(0)}, g_lp, x);
    gemm(x, w, y, bias ? bias->data_ptr() : nullptr, false, false, kOutLp);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const Tensor dy = rowmajor(grads[0]);
    Tensor dx, dw, db;
    if (ctx->needs_input_grad(0)) {
      dx = empty({dy.size(0), w.size(1)}, g_lp, dy);
      gemm(dy, w, dx, nullptr, false, true, kOutLp);
    }
    if (ctx->needs_input_grad(1)) {
      const MainGrad mg(w);
      if (mg.buf.defined()) {
        if (mg.buf.dim() != 2 || mg.buf.size(0) != dy.size(1) || mg.buf.size(1) != x.size(1) || mg.buf.stride(1) != 1 ||
            mg.buf.scalar_type() != at::kFloat || !mg.buf.is_cuda())
          raise(PyExc_ValueError, "bad output tensor");
        gemm(dy, x, mg.buf, nullptr, true, true, mg.fresh ? kOutF32 : kOutF32Acc);
        MainGrad::written(w);
      } else {
        dw = empty({dy.size(1), x.size(1)}, g_lp, dy);
        gemm(dy, x, dw, nullptr, true, true, kOutLp);
      }
    }
    if (ctx->saved_data.count("bias") && ctx->needs_input_grad(2)) {
      const Tensor b = ctx->saved_data["bias"].toTensor();
      const MainGrad mg(b);
      if (takes_vector(mg, b, dy.size(1))) {
        column_sums(dy, mg.buf, !mg.fresh);
        MainGrad::written(b);
      } else {
        db = column_sums(dy);
      }
    }
    return {dx, dw, db};
  }
};

// ---- norm (ops/fused.py) ----------------------------------------------------------------------------------------
constexpr int kNormParts = 296;

struct Norm : public Function<Norm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& residual, const Tensor& w,
                               const OptTensor& b, double eps, bool rms) {
    const int64_t rows = x.size(0), H = x.size(1);
    Tensor y = at::empty_like(x), h = residual ? at::empty_like(x) : x;
    const Tensor rstd = empty({rows}, at::kFloat, x), mean = rms ? Tensor() : empty({rows}, at::kFloat, x);
    check(K.norm_fwd(x.data_ptr(), residual ? residual->data_ptr() : nullptr, w.data_ptr(), b ? b->data_ptr() : nullptr,
                     y.data_ptr(), residual ? h.data_ptr() : nullptr, rstd.data_ptr(), rms ? nullptr : mean.data_ptr(),
                     int(rows), int(H), float(eps), rms, stream()), "hg_norm_fwd");
    count();
    ctx->save_for_backward({h, w, rstd, rms ? rstd : mean});
    if (b) ctx->saved_data["bias"] = *b;            // as in Linear
    ctx->saved_data["rms"] = rms;
    ctx->saved_data["residual"] = residual.has_value();
    ctx->set_materialize_grads(false);
    return residual ? variable_list{y, h} : variable_list{y};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &h = saved[0], &w = saved[1], &rstd = saved[2], &mean = saved[3];
    const bool rms = ctx->saved_data["rms"].toBool(), residual = ctx->saved_data["residual"].toBool(),
               bias = ctx->saved_data.count("bias") != 0;
    const int64_t rows = h.size(0), H = h.size(1);
    const Tensor dy = grads[0].defined() ? grads[0].contiguous() : at::zeros_like(h);
    const Tensor dres = grads.size() > 1 && grads[1].defined() ? grads[1].contiguous() : Tensor();
    Tensor dx = at::empty_like(h);
    const Tensor partial = empty({(rms ? 1 : 2) * kNormParts * H}, at::kFloat, h);
    const MainGrad mg(w);
    if (mg.buf.defined() && (mg.buf.scalar_type() != at::kFloat || !mg.buf.is_cuda() || mg.buf.numel() != H || !mg.buf.is_contiguous()))
      raise(PyExc_ValueError, "bad output tensor");
    const Tensor dw = mg.buf.defined() ? mg.buf : empty({H}, at::kFloat, h);
    // The kernel's accumulate switch is shared with dw (which may add into main_grad): db goes the same way, or into zeros.
    const bool adds = mg.buf.defined() && !mg.fresh;
    const Tensor b = bias ? ctx->saved_data["bias"].toTensor() : Tensor();
    const MainGrad mg_b = bias ? MainGrad(b) : MainGrad();
    const bool b_direct = bias && ctx->needs_input_grad(residual ? 3 : 2) && takes_vector(mg_b, b, H) && !mg_b.fresh == adds;
    const Tensor db = b_direct ? mg_b.buf : bias ? at::zeros({H}, h.options().dtype(at::kFloat)) : Tensor();
    check(K.norm_bwd(dy.data_ptr(), h.data_ptr(), w.data_ptr(), rstd.data_ptr(), rms ? nullptr : mean.data_ptr(),
                     dres.defined() ? dres.data_ptr() : nullptr, dx.data_ptr(), dw.data_ptr(), bias ? db.data_ptr() : nullptr,
                     partial.data_ptr(), kNormParts, int(rows), int(H), rms, adds, stream()),
          "hg_norm_bwd");
    count(2);
    if (mg.buf.defined()) MainGrad::written(w);
    if (b_direct) MainGrad::written(b);
    // dx is the gradient of both x and the residual input (they are summed in the forward)
    return {dx, residual ? dx : Tensor(), mg.buf.defined() ? Tensor() : dw.to(w.scalar_type()),
            bias && !b_direct ? db.to(w.scalar_type()) : Tensor(), Tensor(), Tensor()};
  }
};

// ---- gated activations, residual add ----------------------------------------------------------------------------
struct Glu : public Function<Glu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& y, int64_t kind) {
    const int64_t rows = y.size(0), F = kind == 2 ? y.size(1) : y.size(1) / 2;
    Tensor out = empty({rows, F}, g_lp, y);
    check(K.glu_fwd(y.data_ptr(), out.data_ptr(), rows, int(F), int(kind), stream()), "hg_glu_fwd");
    count();
    ctx->save_for_backward({y});
    ctx->saved_data["kind"] = kind;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const Tensor y = ctx->get_saved_variables()[0], g = grads[0].contiguous();
    Tensor dy = at::empty_like(y);
    check(K.glu_bwd(g.data_ptr(), y.data_ptr(), dy.data_ptr(), y.size(0), int(g.size(1)), int(ctx->saved_data["kind"].toInt()),
                    stream()), "hg_glu_bwd");
    count();
    return {dy, Tensor()};
  }
};

struct Add : public Function<Add> {
  static Tensor forward(AutogradContext*, const Tensor& a, const Tensor& b) {
    Tensor out = at::empty_like(a);
    check(K.add(a.data_ptr(), b.data_ptr(), out.data_ptr(), a.numel(), stream()), "hg_add");
    count();
    return out;
  }
  static variable_list backward(AutogradContext*, const variable_list& grads) { return {grads[0], grads[0]}; }
};

// ---- rotation in place ------------------------------------------------------------------------------------------
struct Rope : public Function<Rope> {
  static void launch(const Tensor& buf, AutogradContext* ctx, bool backward) {
    auto& d = ctx->saved_data;
    const Tensor slots = d["slots"].toTensor(), cos = d["cos"].toTensor(), sin = d["sin"].toTensor();
    const bool has_pos = d["pos"].isTensor();
    const Tensor pos = has_pos ? d["pos"].toTensor() : Tensor();
    check(K.rope(buf.data_ptr(), slots.data_ptr(), int(d["width"].toInt()), int(slots.numel()), int(buf.size(1)), int(buf.size(0)),
                 int(d["batch"].toInt()), has_pos ? pos.data_ptr() : nullptr, int(d["offset"].toInt()), cos.data_ptr(),
                 sin.data_ptr(), int(2 * cos.size(1)), int(backward) | (d["interleaved"].toBool() ? 2 : 0), stream()), "hg_rope");
    count();
  }
  static Tensor forward(AutogradContext* ctx, Tensor buf, const Tensor& slots, int64_t width, const Tensor& cos,
                        const Tensor& sin, int64_t batch, const OptTensor& pos, int64_t offset, bool interleaved) {
    auto& d = ctx->saved_data;
    d["slots"] = slots; d["cos"] = cos; d["sin"] = sin;
    if (pos) d["pos"] = *pos;
    else d["pos"] = c10::IValue();
    d["width"] = width; d["batch"] = batch; d["offset"] = offset; d["interleaved"] = interleaved;
    launch(buf, ctx, false);
    ctx->mark_dirty({buf});
    return buf;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    // the gradient buffer is produced by the attention backward for this node alone: rotated back in place
    const Tensor g = grads[0].contiguous();
    launch(g, ctx, true);
    return {g, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- packed flash attention (ops/attention.py) --------------------------------------------------------------------
struct Packed {
  int S, B, nh, ng, hd;
  bool causal;
  float scale;
  // queries, keys and values inside the packed projection (or its gradient), heads of the context
  HgAttnTensor q(void* p) const { return at(p, 1, 0); }
  HgAttnTensor k(void* p) const { return at(p, 0, nh / ng); }
  HgAttnTensor v(void* p) const { return at(p, 0, nh / ng + 1); }
  HgAttnTensor o(void* p) const { return {p, (long long)B * nh * hd, (long long)nh * hd, nh, nh / ng, 1, 0}; }

 private:
  HgAttnTensor at(void* p, int hs, int off) const {
    const long long P = (long long)(nh + 2 * ng) * hd;
    return {p, B * P, P, nh + 2 * ng, nh / ng + 2, hs, off};
  }
};

struct FlashPacked : public Function<FlashPacked> {
  static Packed layout(AutogradContext* ctx) {
    const auto c = ctx->saved_data["cfg"].toIntVector();
    return {int(c[0]), int(c[1]), int(c[2]), int(c[3]), int(c[4]), c[5] != 0, float(ctx->saved_data["scale"].toDouble())};
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, int64_t S, int64_t B, int64_t nh, int64_t ng, int64_t hd,
                        bool causal, double scale) {
    ctx->saved_data["cfg"] = std::vector<int64_t>{S, B, nh, ng, hd, causal};
    ctx->saved_data["scale"] = scale;
    const Packed l = layout(ctx);
    Tensor out = empty({qkv.size(0), nh * hd}, g_lp, qkv);
    const Tensor lse = empty({B, nh, S}, at::kFloat, qkv);
    const HgAttnTensor q = l.q(qkv.data_ptr()), k = l.k(qkv.data_ptr()), v = l.v(qkv.data_ptr()), o = l.o(out.data_ptr());
    check(K.flash_fwd(&q, &k, &v, &o, lse.data_ptr(), l.S, l.S, l.B, l.nh, l.ng, l.hd, causal, 0, 0, l.scale, stream()),
          "hg_flash_fwd");
    count();
    ctx->save_for_backward({qkv, out, lse});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &qkv = saved[0], &out = saved[1], &lse = saved[2];
    const Packed l = layout(ctx);
    const Tensor dout = grads[0].contiguous();
    Tensor dqkv = at::empty_like(qkv);
    // Row sums and parts, and the pieces of dS; a single piece shares an allocation with the others.
    long long wants[3];
    K.flash_bwd_wants(l.S, l.S, l.B, l.nh, l.ng, l.hd, l.causal, 0, 0, wants);
    int n = wants[1] > 0 && K.flash_bwd_has_room(qkv.get_device()) ? int(wants[1]) : 0;
    Tensor ws;
    variable_list tiles;
    try {
      ws = empty({wants[0] + (n == 1 ? wants[2] : 0)}, at::kFloat, qkv);
      for (int i = 0; n > 1 && i < n; ++i) tiles.push_back(empty({wants[2]}, at::kFloat, qkv));
    } catch (const c10::OutOfMemoryError&) {           // no room for dS: the kernels do without
      if (n == 0) throw;
      K.flash_bwd_no_room(qkv.get_device());
      n = 0;
      tiles.clear();
      if (!ws.defined()) ws = empty({wants[0]}, at::kFloat, qkv);
    }
    void* tiles_at[kHgDsPieces];
    if (n == 1) tiles_at[0] = ws.data_ptr<float>() + wants[0];
    for (int i = 0; n > 1 && i < n; ++i) tiles_at[i] = tiles[i].data_ptr();
    int kernels = 0;
    const HgAttnTensor q = l.q(qkv.data_ptr()), k = l.k(qkv.data_ptr()), v = l.v(qkv.data_ptr()), o = l.o(out.data_ptr()),
                       d = l.o(dout.data_ptr()), dq = l.q(dqkv.data_ptr()), dk = l.k(dqkv.data_ptr()), dv = l.v(dqkv.data_ptr());
    check(K.flash_bwd(&q, &k, &v, &o, &d, lse.data_ptr(), ws.data_ptr(), wants[0], tiles_at, n, wants[2], &dq, &dk, &dv, l.S, l.S,
                      l.B, l.nh, l.ng, l.hd, l.causal, 0, 0, l.scale, &kernels, stream()), "hg_flash_bwd");
    count(kernels);
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- edge of a sharded unit (parallel/zero.py) --------------------------------------------------------------------
// Identity in the forward; calls back when the gradient passes in the backward.
struct Callback : public torch::CustomClassHolder {
  PyObject* fn;
  explicit Callback(PyObject* f) : fn(f) { Py_INCREF(fn); }
  ~Callback() override {
    pybind11::gil_scoped_acquire gil;
    Py_DECREF(fn);
  }
};

struct Boundary : public Function<Boundary> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const c10::intrusive_ptr<Callback>& cb) {
    ctx->saved_data["cb"] = c10::IValue::make_capsule(cb);
    return x.view_as(x);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    {
      pybind11::gil_scoped_acquire gil;
      const auto cb = c10::static_intrusive_pointer_cast<Callback>(ctx->saved_data["cb"].toCapsule());
      PyObject* r = PyObject_CallNoArgs(cb->fn);
      if (r == nullptr) {
        python_error e;
        e.persist();
        throw e;
      }
      Py_DECREF(r);
    }
    return {grads[0], Tensor()};
  }
};

// ---- Python entry points ------------------------------------------------------------------------------------------
const Tensor& arg(PyObject* o) { return THPVariable_Unpack(o); }
OptTensor opt(PyObject* o) { return o == Py_None ? OptTensor() : OptTensor(THPVariable_Unpack(o)); }
bool tensors(std::initializer_list<PyObject*> need, std::initializer_list<PyObject*> may = {}) {
  for (PyObject* o : need)
    if (!THPVariable_Check(o)) return false;
  for (PyObject* o : may)
    if (o != Py_None && !THPVariable_Check(o)) return false;
  return plain_mode();
}
long long whole(PyObject* o) { return THPUtils_unpackLong(o); }
std::vector<int64_t> with_last(const Tensor& t, int64_t n) {
  std::vector<int64_t> shape(t.sizes().begin(), t.sizes().end());
  shape.back() = n;
  return shape;
}

// linear(x, w, bias | None)
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !tensors({a[0], a[1]}, {a[2]})) Py_RETURN_NONE;
  const Tensor &x = arg(a[0]), &w = arg(a[1]);
  const OptTensor bias = opt(a[2]);
  if (!plain(x) || !plain(w) || x.dim() < 1 || w.dim() != 2 || x.size(-1) != w.size(1) || x.device() != w.device() ||
      x.numel() == 0 || w.numel() == 0 || (bias && !plain_vector(*bias, w.size(0), x)))
    Py_RETURN_NONE;
  Tensor y;
  {
    pybind11::gil_scoped_release no_gil;
    y = Linear::apply(x.reshape({-1, x.size(-1)}), w, bias);
    if (x.dim() != 2) y = y.view(with_last(x, w.size(0)));
  }
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// norm(x, residual | None, w, b | None, eps, rms): (y, h), h None without a residual
PyObject* py_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !tensors({a[0], a[2]}, {a[1], a[3]})) Py_RETURN_NONE;
  const Tensor &x = arg(a[0]), &w = arg(a[2]);
  const OptTensor residual = opt(a[1]), b = opt(a[3]);
  if (!plain(x) || x.dim() < 1 || x.numel() == 0) Py_RETURN_NONE;
  const int64_t H = x.size(-1);
  const bool rms = PyObject_IsTrue(a[5]);
  if (H % 8 || H > 16384 || !plain_vector(w, H, x) || (b && !plain_vector(*b, H, x)) ||
      (residual && !(plain(*residual) && residual->sizes() == x.sizes() && residual->device() == x.device())) || (!rms && !b))
    Py_RETURN_NONE;
  const double eps = THPUtils_unpackDouble(a[4]);
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    const Tensor x2 = x.reshape({-1, H}).contiguous();
    const OptTensor r2 = residual ? OptTensor(residual->reshape({-1, H}).contiguous()) : OptTensor();
    out = Norm::apply(x2, r2, w, b, eps, rms);
    for (Tensor& t : out) t = t.view(x.sizes());
  }
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) throw python_error();
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(out[0]));
  if (residual) {
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(out[1]));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(r, 1, Py_None);
  }
  return r;
  END_HANDLE_TH_ERRORS
}

// activation(y, kind)
PyObject* py_activation(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !tensors({a[0]})) Py_RETURN_NONE;
  const Tensor& y = arg(a[0]);
  const int64_t kind = whole(a[1]);
  if (!plain(y) || y.dim() < 1 || y.numel() == 0 || y.size(-1) % (kind == 2 ? 8 : 16)) Py_RETURN_NONE;
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = Glu::apply(y.reshape({-1, y.size(-1)}).contiguous(), kind);
    out = out.view(with_last(y, out.size(1)));
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// add(a, b)
PyObject* py_add(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !tensors({a[0], a[1]})) Py_RETURN_NONE;
  const Tensor &x = arg(a[0]), &y = arg(a[1]);
  if (!plain(x) || !plain(y) || !x.is_contiguous() || !y.is_contiguous() || x.sizes() != y.sizes() || x.device() != y.device())
    Py_RETURN_NONE;
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = Add::apply(x, y);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// rope_packed(qkv, slots, width, cos, sin, batch, pos | None, offset, interleaved): qkv, rotated in place
PyObject* py_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9 || !tensors({a[0], a[1], a[3], a[4]}, {a[6]})) Py_RETURN_NONE;
  const Tensor &buf = arg(a[0]), &slots = arg(a[1]), &cos = arg(a[3]), &sin = arg(a[4]);
  const OptTensor pos = opt(a[6]);
  auto table = [&](const Tensor& t) {
    return t.is_cuda() && t.dim() == 2 && t.scalar_type() == at::kFloat && t.is_contiguous() && !t.requires_grad() &&
           t.device() == buf.device();
  };
  auto numbers = [&](const Tensor& t) {
    return t.is_cuda() && t.scalar_type() == at::kInt && t.is_contiguous() && t.device() == buf.device();
  };
  if (!plain(buf) || (buf.requires_grad() && !at::GradMode::is_enabled()) || buf.dim() != 2 || !buf.is_contiguous() ||
      buf.numel() == 0 || !table(cos) || !table(sin) || !numbers(slots) || (pos && !numbers(*pos)))
    Py_RETURN_NONE;
  const long long width = whole(a[2]), batch = whole(a[5]), offset = whole(a[7]);
  const bool interleaved = PyObject_IsTrue(a[8]);
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = Rope::apply(buf, slots, int64_t(width), cos, sin, int64_t(batch), pos, int64_t(offset), interleaved);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// flash_packed(qkv, S, B, nh, ng, hd, causal, scale)
PyObject* py_flash_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !tensors({a[0]})) Py_RETURN_NONE;
  const Tensor& qkv = arg(a[0]);
  const long long S = whole(a[1]), B = whole(a[2]), nh = whole(a[3]), ng = whole(a[4]), hd = whole(a[5]);
  const bool causal = PyObject_IsTrue(a[6]);
  const double scale = THPUtils_unpackDouble(a[7]);
  if (!plain(qkv) || qkv.dim() != 2 || S < 1 || B < 1 || ng < 1 || nh < ng || nh % ng || qkv.size(0) != S * B ||
      qkv.size(1) != (nh + 2 * ng) * hd)
    Py_RETURN_NONE;
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = FlashPacked::apply(qkv.contiguous(), int64_t(S), int64_t(B), int64_t(nh), int64_t(ng), int64_t(hd), causal, scale);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

bool dense_like(const Tensor& t, const Tensor& x) {
  return plain(t) && t.device() == x.device() && t.is_contiguous() && aligned(t);
}

// Whether `list` holds the six (weight, bias | None) of a decoder layer, in the order of HgDecoderStep, as dense 16-bit
// tensors of the right shapes on x's GPU; their addresses go to `w`.
bool layer_weights(const Tensor& x, PyObject* list, int64_t nh, int64_t ng, int64_t hd, int64_t F, int64_t act, const void** w) {
  if (!PyList_Check(list) || PyList_GET_SIZE(list) != 12 || x.dim() != 3) return false;
  const int64_t H = x.size(2), F1 = act == 2 ? F : 2 * F;
  const int64_t shapes[6][2] = {{H, 0}, {(nh + 2 * ng) * hd, H}, {H, nh * hd}, {H, 0}, {F1, H}, {H, F}};
  for (int i = 0; i < 12; ++i) {
    PyObject* o = PyList_GET_ITEM(list, i);
    w[i] = nullptr;
    if (o == Py_None && i % 2 == 1) continue;
    if (!THPVariable_Check(o)) return false;
    const Tensor& t = arg(o);
    const int64_t* s = shapes[i / 2];
    const bool vector = i % 2 == 1 || s[1] == 0;
    if (!dense_like(t, x) || t.dim() != (vector ? 1 : 2) || t.size(0) != s[0] || (!vector && t.size(1) != s[1])) return false;
    w[i] = t.data_ptr();
  }
  return true;
}

// decoder_weights(x, weights, nh, ng, hd, ffn, act kind): see layer_weights; None where dispatch is watched
PyObject* py_decoder_weights(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 || !tensors({a[0]})) Py_RETURN_NONE;
  const void* w[12];
  if (layer_weights(arg(a[0]), a[1], whole(a[2]), whole(a[3]), whole(a[4]), whole(a[5]), whole(a[6]), w)) Py_RETURN_TRUE;
  Py_RETURN_FALSE;
  END_HANDLE_TH_ERRORS
}

// decoder_step(x, weights, k_cache, v_cache, cos | None, sin | None, past, first sequence, nh, ng, hd, ffn, rms, act kind,
// interleaved, eps): the output of one cached decoder layer whose kernels one native call launches (decoder_step.cu).
// None unless the weights are those of layer_weights and the caches two separate contiguous buffers with room for the tokens.
PyObject* py_decoder_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 16 || !tensors({a[0], a[2], a[3]}, {a[4], a[5]})) Py_RETURN_NONE;
  const Tensor &x = arg(a[0]), &kc = arg(a[2]), &vc = arg(a[3]);
  const OptTensor cos = opt(a[4]), sin = opt(a[5]);
  const long long past = whole(a[6]), b0 = whole(a[7]), nh = whole(a[8]), ng = whole(a[9]), hd = whole(a[10]), F = whole(a[11]),
                  act = whole(a[13]);
  const bool rms = PyObject_IsTrue(a[12]), interleaved = PyObject_IsTrue(a[14]);
  const double eps = THPUtils_unpackDouble(a[15]);
  const void* w[12];
  if (at::GradMode::is_enabled() || !plain(x) || !dense_like(x, x) || x.dim() != 3 || x.numel() == 0 ||
      !layer_weights(x, a[1], nh, ng, hd, F, act, w))
    Py_RETURN_NONE;
  const int64_t S = x.size(0), B = x.size(1), H = x.size(2);
  auto cache = [&](const Tensor& c) {
    return dense_like(c, x) && !c.requires_grad() && c.dim() == 4 && c.size(0) >= past + S && c.size(1) >= b0 + B &&
           c.size(2) == ng && c.size(3) == hd && (c10::InferenceMode::is_enabled() || !c.is_inference());
  };
  if (past < 0 || b0 < 0 || !cache(kc) || !cache(vc) || ng < 1 || (ng * hd) % 8 ||
      !(address(kc) + kc.nbytes() <= address(vc) || address(vc) + vc.nbytes() <= address(kc)))
    Py_RETURN_NONE;
  for (const OptTensor* t : {&cos, &sin})
    if (*t && !((*t)->is_cuda() && (*t)->scalar_type() == at::kFloat && (*t)->dim() == 2 && (*t)->is_contiguous() &&
                (*t)->size(0) >= past + S && (*t)->device() == x.device()))
      Py_RETURN_NONE;
  if (cos.has_value() != sin.has_value()) Py_RETURN_NONE;
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = at::empty_like(x);
    HgDecoderStep d{};
    d.S = int(S); d.B = int(B); d.H = int(H); d.nh = int(nh); d.ng = int(ng); d.hd = int(hd); d.F = int(F); d.past = int(past);
    d.rms = rms; d.act = int(act); d.rot_dim = cos ? int(2 * cos->size(1)) : 0; d.interleaved = interleaved;
    d.eps = float(eps); d.scale = float(1.0 / std::sqrt(double(hd)));
    d.w_norm1 = w[0]; d.b_norm1 = w[1]; d.w_qkv = w[2]; d.b_qkv = w[3]; d.w_proj = w[4]; d.b_proj = w[5];
    d.w_norm2 = w[6]; d.b_norm2 = w[7]; d.w_fc1 = w[8]; d.b_fc1 = w[9]; d.w_fc2 = w[10]; d.b_fc2 = w[11];
    d.cos_t = cos ? cos->data_ptr() : nullptr; d.sin_t = sin ? sin->data_ptr() : nullptr;
    d.k_cache = static_cast<char*>(kc.data_ptr()) + b0 * kc.stride(1) * kc.element_size();
    d.v_cache = static_cast<char*>(vc.data_ptr()) + b0 * vc.stride(1) * vc.element_size();
    d.k_ss = kc.stride(0); d.k_sb = kc.stride(1); d.v_ss = vc.stride(0); d.v_sb = vc.stride(1);
    d.x = x.data_ptr(); d.out = out.data_ptr();
    d.ws_bytes = K.decoder_step_scratch(&d);
    const Tensor ws = empty({d.ws_bytes > 0 ? d.ws_bytes : 1}, at::kByte, x);
    d.ws = ws.data_ptr();
    check(K.decoder_step(&d, stream()), "hg_decoder_step");
    for (const Tensor* c : {&kc, &vc})                     // as an in-place operation on the caches would
      if (!c->is_inference()) c->unsafeGetTensorImpl()->bump_version();
    count(d.launches);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// boundary(x, callback)
PyObject* py_boundary(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !tensors({a[0]}) || !PyCallable_Check(a[1])) Py_RETURN_NONE;
  const Tensor& x = arg(a[0]);
  if (!x.defined() || !at::GradMode::is_enabled() || at::isTensorSubclassLike(x) || x._fw_grad(0).defined()) Py_RETURN_NONE;
  const auto cb = c10::make_intrusive<Callback>(a[1]);
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = Boundary::apply(x, cb);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

void bind(const py::dict& fn, bool half, int pair_mode, py::object kernel_error) {
  auto at = [&](const char* name, auto& slot) {
    slot = reinterpret_cast<std::decay_t<decltype(slot)>>(py::cast<uintptr_t>(fn[name]));
  };
  at("hg_gemm_bf16", K.gemm); at("hg_gemm2_bf16", K.gemm2); at("hg_gemm2_scratch", K.gemm2_scratch); at("hg_gemm_skinny_bf16", K.gemm_skinny);
  at("hg_colsum_parts", K.colsum_parts); at("hg_colsum", K.colsum);
  at("hg_norm_fwd", K.norm_fwd); at("hg_norm_bwd", K.norm_bwd);
  at("hg_glu_fwd", K.glu_fwd); at("hg_glu_bwd", K.glu_bwd); at("hg_add_bf16", K.add); at("hg_rope", K.rope);
  at("hg_flash_fwd", K.flash_fwd); at("hg_flash_bwd_wants", K.flash_bwd_wants); at("hg_flash_bwd_has_room", K.flash_bwd_has_room); at("hg_flash_bwd_no_room", K.flash_bwd_no_room); at("hg_flash_bwd_ws", K.flash_bwd);
  at("hg_decoder_step_scratch", K.decoder_step_scratch); at("hg_decoder_step", K.decoder_step);
  g_lp = half ? at::kHalf : at::kBFloat16;
  g_pair_mode = pair_mode;
  g_kernel_error = kernel_error.release().ptr();
}

#define HG_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fn)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {HG_METHOD("linear", py_linear),
                          HG_METHOD("norm", py_norm),
                          HG_METHOD("activation", py_activation),
                          HG_METHOD("add", py_add),
                          HG_METHOD("rope_packed", py_rope),
                          HG_METHOD("flash_packed", py_flash_packed),
                          HG_METHOD("decoder_weights", py_decoder_weights),
                          HG_METHOD("decoder_step", py_decoder_step),
                          HG_METHOD("boundary", py_boundary),
                          {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(hg_torch_ops, m) {
  m.attr("interface") = kHgNativeInterface;
  m.def("bind", &bind);
  m.def("launches", [] { return g_launches.load(); });
  m.def("reset_launches", [] { g_launches = 0; });
  m.def("gemm_route", &route);
  PyModule_AddFunctions(m.ptr(), kMethods);
}
