// Torch binding of the layer calls: the autograd nodes of HQ_Linear and HQ_Conv2d, the plugin call and the stand-alone row
// quantiser, made without a Python frame between the caller and the C ABI.
//
// A small layer is bound by the host (1 x 197 tokens, 768 -> 768: 31 us of kernels in 123), so the node makes one C call per
// direction.  It reads the configuration module at forward and again at backward, as the reference does, and allocates
// through torch's caching allocator.  grad_out's g_x codes are one per byte at every contraction length, as the plugin's are.
//
// linear() and conv2d() answer None for whatever it does not cover (other transform schemes, the logarithmic quantiser, token
// bases above 64, other dtypes or devices, autocast, tracing, functorch transforms, forward-mode gradients, tensor
// subclasses and dispatch modes, arguments that are in error); the caller then takes the Python Function,
// which covers or refuses it.  A configuration that leaves the covered set between forward and backward
// goes to that Function's backward too.
#include <torch/extension.h>

#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/autocast_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/Exceptions.h>

#include "hot_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

PyObject* g_qm = nullptr;     // hot_b200.quant_matmul (owns the Philox call counter and finds the configuration module)
PyObject* g_error = nullptr;  // hot_b200._cabi.HotError

// The pending Python error as a C++ exception that may cross threads (the autograd engine runs the backward on its own).
[[noreturn]] void throw_python() {
  python_error err;
  err.persist();
  throw err;
}
[[noreturn]] void fail(int status, const char* where) {
  pybind11::gil_scoped_acquire gil;
  PyObject* e = PyObject_CallFunction(g_error, "iss", status, where, hot_last_error());
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  throw_python();
}
void check(int status, const char* where) {
  if (status != HOT_OK) fail(status, where);
}

// ---- the configuration module, read under the GIL ------------------------------------------------
struct Names {
  PyObject *args_fn, *philox, *fallback, *scheme, *t_gogi, *t_wgt, *t_gogw, *t_input, *b_gogi, *b_wgt, *b_gogw, *b_act, *q_gogi, *q_wgt,
      *q_gogw, *q_act, *autoq, *dict, *seed, *preset;
} N;

void intern_names() {
  auto s = [](const char* t) { return PyUnicode_InternFromString(t); };
  N = {s("_args"),          s("_philox_calls"), s("_native_fallback"), s("transform_scheme"), s("TransformGogi"),  s("TransformWgt"),
       s("TransformGogw"),  s("TransformInput"), s("GogiQuantBit"),    s("weightQuantBit"),   s("GogwQuantBit"),   s("actQuantBit"),
       s("quantBWDGogi"),   s("quantBWDWgt"),    s("quantBWDGogw"),    s("quantBWDAct"),      s("quantAuto"),      s("layer_quant_dict"),
       s("SEED"),           s("lowRankPreset")};
}

struct Ref {  // an owned Python reference
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  explicit operator bool() const { return p != nullptr; }
};

bool text_is(PyObject* o, const char* t) { return o && PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, t) == 0; }

// Attribute of the configuration module as a small integer; -1 where it is missing or no integer.
long attr_int(PyObject* mod, PyObject* name) {
  Ref v(PyObject_GetAttr(mod, name));
  if (!v) {
    PyErr_Clear();
    return -1;
  }
  const long n = PyLong_Check(v.p) ? PyLong_AsLong(v.p) : -1;
  if (PyErr_Occurred()) PyErr_Clear();
  return n;
}
bool attr_true(PyObject* mod, PyObject* name) {
  Ref v(PyObject_GetAttr(mod, name));
  if (!v) {
    PyErr_Clear();
    return false;
  }
  return PyObject_IsTrue(v.p) == 1;
}

// One quantiser by its configured name; false: not covered here.
bool quantiser(PyObject* name, long bits, bool row_ok, bool sawb_ok, hot_quant_t& q) {
  if (bits < 2 || bits > 8) return false;
  q.bits = (int32_t)bits;
  q.storage = HOT_STORE_INT8;
  q.noise = nullptr;
  if (text_is(name, "stoch") || text_is(name, "stoch_quantizer")) {
    q.rounding = HOT_ROUND_STOCH_PHILOX;
    q.scale_mode = HOT_SCALE_TENSOR;
  } else if (text_is(name, "int") || text_is(name, "int_quantizer")) {
    q.rounding = HOT_ROUND_NEAREST;
    q.scale_mode = HOT_SCALE_TENSOR;
  } else if (row_ok && (text_is(name, "nq") || text_is(name, "norm_quantizer"))) {
    q.rounding = HOT_ROUND_STOCH_PHILOX;
    q.scale_mode = HOT_SCALE_ROW;
  } else if (sawb_ok && text_is(name, "sawb")) {
    q.rounding = HOT_ROUND_NEAREST;
    q.scale_mode = HOT_SCALE_SAWB;
  } else {
    return false;
  }
  return true;
}
bool quantiser_attr(PyObject* mod, PyObject* attr, long bits, bool row_ok, bool sawb_ok, hot_quant_t& q) {
  Ref v(PyObject_GetAttr(mod, attr));
  if (!v) {
    PyErr_Clear();
    return false;
  }
  return quantiser(v.p, bits, row_ok, sawb_ok, q);
}

bool scheme_covered(PyObject* mod) {
  Ref v(PyObject_GetAttr(mod, N.scheme));
  if (!v) {
    PyErr_Clear();
    return false;
  }
  if (!text_is(v.p, "gih_gwlr") && !text_is(v.p, "hadamard")) return false;
  return attr_true(mod, N.t_gogi) && attr_true(mod, N.t_wgt) && attr_true(mod, N.t_gogw) && attr_true(mod, N.t_input);
}

// int(SEED or 0), whatever number SEED is; a Python error may be pending.
uint64_t seed_of(PyObject* mod) {
  Ref v(PyObject_GetAttr(mod, N.seed));
  if (!v) {
    PyErr_Clear();
    return 0;
  }
  if (PyObject_IsTrue(v.p) != 1) return 0;
  Ref n(PyNumber_Long(v.p));
  return n ? PyLong_AsUnsignedLongLongMask(n.p) : 0;
}

// Takes `count` offsets from the module's Philox call counter; the first of them.
uint64_t take_offsets(uint64_t count) {
  PyObject* d = PyModule_GetDict(g_qm);
  PyObject* cur = PyDict_GetItemWithError(d, N.philox);
  const uint64_t before = cur ? PyLong_AsUnsignedLongLong(cur) : 0;
  Ref next(PyLong_FromUnsignedLongLong(before + count));
  if (PyErr_Occurred() || !next || PyDict_SetItem(d, N.philox, next.p) != 0) throw_python();
  return before + 1;
}

// The three quantisers of a backward (grad_output on both sides and the weight), as configured now.
bool backward_quantisers(PyObject* layer_name, hot_linear_cfg_t& c) {
  Ref mod(PyObject_CallMethodNoArgs(g_qm, N.args_fn));
  if (!mod) throw_python();
  if (!scheme_covered(mod.p)) return false;
  bool ok = false;
  if (attr_true(mod.p, N.autoq)) {
    Ref dict(PyObject_GetAttr(mod.p, N.dict));
    if (!dict) {
      PyErr_Clear();
      return false;
    }
    const Py_ssize_t entries = PyObject_Length(dict.p);
    if (entries < 0) PyErr_Clear();
    if (entries > 0) {  // both sides take GogiQuantBit here, as the reference does (utils/quant_matmul.py:244-245, 307-308)
      Ref kx(PyUnicode_FromFormat("%S_gx", layer_name)), kw(PyUnicode_FromFormat("%S_gw", layer_name));
      Ref vx(kx ? PyObject_GetItem(dict.p, kx.p) : nullptr), vw(kw ? PyObject_GetItem(dict.p, kw.p) : nullptr);
      if (PyErr_Occurred()) PyErr_Clear();
      const long bits = attr_int(mod.p, N.b_gogi);
      if (!vx || !vw || text_is(vx.p, "stoch") || text_is(vx.p, "int") || text_is(vx.p, "nq") || text_is(vw.p, "stoch") ||
          text_is(vw.p, "int") || text_is(vw.p, "nq"))
        return false;  // the selection names whole quantisers
      if (!quantiser(vx.p, bits, true, false, c.q_gx) || !quantiser(vw.p, bits, true, false, c.q_gw)) return false;
      ok = true;
    }
  }
  if (!ok && (!quantiser_attr(mod.p, N.q_gogi, attr_int(mod.p, N.b_gogi), true, false, c.q_gx) ||
              !quantiser_attr(mod.p, N.q_gogw, attr_int(mod.p, N.b_gogw), true, false, c.q_gw)))
    return false;
  if (!quantiser_attr(mod.p, N.q_wgt, attr_int(mod.p, N.b_wgt), false, true, c.q_w)) return false;
  const uint64_t seed = seed_of(mod.p);
  if (PyErr_Occurred()) throw_python();
  const uint64_t first = take_offsets(3);
  c.q_gx.seed = c.q_gw.seed = c.q_w.seed = seed;
  c.q_gx.offset = first;
  c.q_gw.offset = first + 1;
  c.q_w.offset = first + 2;
  return true;
}

int dtype_code(at::ScalarType t) { return t == at::kFloat ? HOT_F32 : (t == at::kBFloat16 ? HOT_BF16 : -1); }

hot_stream_t current_stream() { return (hot_stream_t)c10::cuda::getCurrentCUDAStream().stream(); }
Tensor bytes(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }

// ---- the autograd nodes --------------------------------------------------------------------------
// What a layer keeps from forward to backward, and its two gradients from the gradient of its output rows.  The tensors are
// saved variables, in the order of FLinearQ: saved-tensor hooks (offloading, checkpoints) see each of them.
struct Saved {
  SavedVariable x_q_t, w, scale_x;  // w: [O, I], or a convolution's [O, C, kh, kw]
  hot_layer_t layer = {};
  PyObject* name = nullptr;

  ~Saved() {
    if (name && Py_IsInitialized()) {
      pybind11::gil_scoped_acquire gil;
      Py_DECREF(name);
    }
  }
  void release() {
    x_q_t.reset_data();
    w.reset_data();
    scale_x.reset_data();
  }
  // (batch, order_o, order_l, selection, q_x bits, q_x packed): what the Python backward needs to know of the forward
  Ref describe() const {
    const hot_linear_cfg_t& c = layer.cfg;
    PyObject* sel = PyList_New(c.rank_l);
    for (int i = 0; i < c.rank_l; ++i) PyList_SetItem(sel, i, PyLong_FromLong(c.sel_l[i]));
    return Ref(Py_BuildValue("(LiiNii)", (long long)layer.batch, c.order_o, c.order_l, sel, c.q_x.bits, c.q_x.storage == HOT_STORE_INT4));
  }
  // go: contiguous, w2: the weight as [O, I], both of one dtype; gx comes in the shape of go with I in place of O, or, for a
  // convolution whose product folds it, as the image's gradient (folded is then set)
  void backward(const std::shared_ptr<Node>& node, const Tensor& go, const Tensor& w2, bool need_x, bool need_w, bool need_b, Tensor& gx,
                Tensor& gw, Tensor& gb, const hot_conv_t* conv = nullptr, bool* folded = nullptr) const {
    const Tensor codes = x_q_t.unpack(node), scale = scale_x.unpack(node);
    hot_layer_t l = layer;
    {
      pybind11::gil_scoped_acquire gil;
      if (!backward_quantisers(name, l.cfg)) {
        Ref r(PyObject_CallMethodObjArgs(g_qm, N.fallback, Ref(THPVariable_Wrap(go)).p, Ref(THPVariable_Wrap(w2)).p,
                                         Ref(THPVariable_Wrap(codes)).p, Ref(THPVariable_Wrap(scale)).p, describe().p, name,
                                         need_x ? Py_True : Py_False, need_w ? Py_True : Py_False, nullptr));
        if (!r) throw_python();
        PyObject *px = PyTuple_GetItem(r.p, 0), *pw = PyTuple_GetItem(r.p, 1);
        if (px != Py_None) gx = THPVariable_Unpack(px);
        if (pw != Py_None) gw = THPVariable_Unpack(pw);
        if (need_b) gb = go.reshape({-1, l.O}).sum(0);
        return;
      }
    }
    const size_t ws_bytes = hot_layer_backward_workspace_bytes(&l);
    if (ws_bytes == 0) fail(HOT_ERR_UNSUPPORTED, "hot_layer_backward");
    const Tensor ws = bytes((int64_t)ws_bytes, go);
    const bool fold = need_x && conv && hot_conv_folds(&l, conv) != 0;
    if (folded) *folded = fold;
    if (fold) {
      gx = at::empty({conv->B, conv->C, conv->H, conv->W}, go.options());
    } else if (need_x) {
      std::vector<int64_t> shape = go.sizes().vec();
      shape.back() = l.I;
      gx = at::empty(shape, go.options());
    }
    // the product summed over samples is stored through a tensor map, whose rows begin at multiples of 16 bytes
    int64_t ldgw = l.I;
    const int64_t per16 = 16 / (int64_t)go.element_size();
    if (l.batch) ldgw = (ldgw + per16 - 1) / per16 * per16;
    if (need_w) gw = at::empty({l.O, ldgw}, go.options());
    // the bias gradient comes from the quantisers' own pass over grad_out where they can make it (they take channels in pairs)
    const bool sums = need_b && hot_layer_sums_rows(&l, go.data_ptr()) != 0;
    if (need_b) gb = sums ? at::empty({l.O}, go.options()) : go.reshape({-1, l.O}).sum(0);
    if (fold) {
      check(hot_layer_backward_conv(&l, conv, go.data_ptr(), w2.data_ptr(), w2.stride(0), codes.data_ptr(), (const float*)scale.data_ptr(),
                                    gx.data_ptr(), need_w ? gw.data_ptr() : nullptr, ldgw, sums ? gb.data_ptr() : nullptr, ws.data_ptr(), ws_bytes,
                                    nullptr, current_stream()),
            "hot_layer_backward_conv");
    } else {
      check(hot_layer_backward(&l, go.data_ptr(), w2.data_ptr(), w2.stride(0), codes.data_ptr(), (const float*)scale.data_ptr(),
                               need_x ? gx.data_ptr() : nullptr, l.I, need_w ? gw.data_ptr() : nullptr, ldgw, sums ? gb.data_ptr() : nullptr,
                               ws.data_ptr(), ws_bytes, nullptr, current_stream()),
            "hot_layer_backward");
    }
    if (need_w && ldgw != l.I) gw = gw.narrow(1, 0, l.I);
  }
};

struct HotLinearBackward : public Node {
  Saved s;
  bool has_bias = false;
  std::string name() const override { return "HotLinearBackward"; }
  void release_variables() override { s.release(); }

  variable_list apply(variable_list&& grads) override {
    variable_list out(has_bias ? 3 : 2);
    if (!grads[0].defined()) return out;
    at::NoGradGuard no_grad;
    Tensor go = grads[0];
    const bool need_x = task_should_compute_output(0), need_w = task_should_compute_output(1);
    bool need_b = has_bias && task_should_compute_output(2);
    if (!need_x && !need_w) {  // (needs nothing of what forward saved, and forward saved nothing where only the bias learns)
      if (need_b) out[2] = go.reshape({-1, go.size(-1)}).sum(0);
      return out;
    }
    const Tensor w = s.w.unpack(shared_from_this()).detach();
    c10::cuda::CUDAGuard guard(w.device());
    if (need_b && go.scalar_type() != w.scalar_type()) {  // (the sum is taken in the type the gradient came in)
      out[2] = go.reshape({-1, go.size(-1)}).sum(0);
      need_b = false;
    }
    go = go.contiguous();
    if (go.scalar_type() != w.scalar_type()) go = go.to(w.scalar_type());
    Tensor gb;
    s.backward(shared_from_this(), go, w, need_x, need_w, need_b, out[0], out[1], gb);
    if (need_b) out[2] = gb;
    return out;
  }
};

struct HotConvBackward : public Node {
  Saved s;
  hot_conv_t conv = {};
  int64_t positions = 0;  // output positions per image
  bool has_bias = false;
  std::string name() const override { return "HotConvBackward"; }
  void release_variables() override { s.release(); }

  variable_list apply(variable_list&& grads) override {
    variable_list out(has_bias ? 3 : 2);
    if (!grads[0].defined()) return out;
    at::NoGradGuard no_grad;
    Tensor go = grads[0];
    const bool need_x = task_should_compute_output(0), need_w = task_should_compute_output(1);
    bool need_b = has_bias && task_should_compute_output(2);
    if (!need_x && !need_w) {
      if (need_b) out[2] = go.sum({0, 2, 3});
      return out;
    }
    const Tensor w = s.w.unpack(shared_from_this()).detach();
    c10::cuda::CUDAGuard guard(w.device());
    if (need_b && go.scalar_type() != w.scalar_type()) {
      out[2] = go.sum({0, 2, 3});
      need_b = false;
    }
    go = go.contiguous();
    if (go.scalar_type() != w.scalar_type()) go = go.to(w.scalar_type());
    const Tensor rows = at::empty({conv.B, positions, s.layer.O}, go.options());
    check(hot_transpose(conv.dtype, conv.B, s.layer.O, positions, go.data_ptr(), nullptr, rows.data_ptr(), current_stream()), "hot_transpose");
    Tensor gcols;
    Tensor gb;
    bool folded = false;
    s.backward(shared_from_this(), rows, w.view({s.layer.O, s.layer.I}), need_x, need_w, need_b, gcols, out[1], gb, &conv, &folded);
    if (need_b) out[2] = gb;
    if (need_w) out[1] = out[1].reshape(w.sizes());  // (a copy where its rows are padded)
    if (need_x && folded) {
      out[0] = gcols;
    } else if (need_x) {
      gcols = gcols.contiguous();
      out[0] = at::empty({conv.B, conv.C, conv.H, conv.W}, go.options());
      check(hot_col2im(&conv, gcols.data_ptr(), out[0].data_ptr(), current_stream()), "hot_col2im");
    }
    return out;
  }
};

// Whether torch has to see the operations of a call one by one: kernels launched on raw pointers would be missing from a
// trace or a dispatch mode's record, lose a tangent, or meet a wrapper that has no memory.
bool seen_by_torch(const Tensor& t) { return at::isTensorSubclassLike(t) || t._fw_grad(0).defined(); }
bool torch_watches() {
  return torch::jit::tracer::isTracing() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// The part of a layer's configuration that forward fixes; false: not covered (a Python error may be pending).
// a: x, w, bias or None, order_o, order_l, selection, name
bool forward_config(PyObject* const* a, hot_linear_cfg_t& c, bool& preset) {
  if (at::autocast::is_autocast_enabled(at::kCUDA)) return false;  // the product would come in autocast's type, not the tensors'
  if (torch_watches()) return false;
  if (!THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !PyList_Check(a[5])) return false;
  const Tensor &x = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]);
  const int dt = dtype_code(x.scalar_type());
  const Py_ssize_t rank = PyList_GET_SIZE(a[5]);
  const long order_o = PyLong_AsLong(a[3]), order_l = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return false;
  if (seen_by_torch(x) || seen_by_torch(w)) return false;
  if (!x.is_cuda() || !w.is_cuda() || dt < 0 || x.scalar_type() != w.scalar_type() || x.device() != w.device() || x.numel() == 0 ||
      order_l < 1 || order_l > 64 || order_o < 1 || order_o > 16 || rank < 1 || rank > 64)
    return false;
  if (a[2] != Py_None) {
    const Tensor& bias = THPVariable_Unpack(a[2]);
    if (seen_by_torch(bias) || bias.device() != x.device() || bias.scalar_type() != x.scalar_type()) return false;
  }
  Ref mod(PyObject_CallMethodNoArgs(g_qm, N.args_fn));
  if (!mod || !scheme_covered(mod.p)) return false;
  c.dtype = dt;
  c.order_o = (int32_t)order_o;
  c.order_l = (int32_t)order_l;
  c.rank_l = (int32_t)rank;
  for (Py_ssize_t i = 0; i < rank; ++i) c.sel_l[i] = (int32_t)PyLong_AsLong(PyList_GET_ITEM(a[5], i));
  if (PyErr_Occurred() || !quantiser_attr(mod.p, N.q_act, attr_int(mod.p, N.b_act), false, true, c.q_x)) return false;
  Ref v(PyObject_GetAttr(mod.p, N.preset));
  if (!v) PyErr_Clear();
  preset = v && v.p != Py_None;
  c.q_x.seed = seed_of(mod.p);
  return !PyErr_Occurred();
}

// The activation buffer, made from the rows of x (contiguous).
struct Buffer {
  Tensor codes, scale;
};
Buffer compress(const hot_layer_t& l, const Tensor& x) {
  Buffer b;
  b.codes = at::empty({l.I, hot_layer_buffer_pitch(&l)}, x.options().dtype(at::kByte));
  b.scale = at::empty({std::max<int64_t>(l.batch, 1)}, x.options().dtype(at::kFloat));
  const size_t ws_bytes = hot_layer_compress_workspace_bytes(&l);
  if (ws_bytes == 0) fail(HOT_ERR_UNSUPPORTED, "hot_layer_compress");
  const Tensor ws = bytes((int64_t)ws_bytes, x);
  check(hot_layer_compress(&l, x.data_ptr(), l.I, b.codes.data_ptr(), (float*)b.scale.data_ptr(), ws.data_ptr(), ws_bytes, current_stream()),
        "hot_layer_compress");
  return b;
}

bool wants_grad(const Tensor& t) { return t.defined() && at::GradMode::is_enabled() && t.requires_grad(); }

template <typename NodeT>
void attach(const std::shared_ptr<NodeT>& node, Tensor& y, const Tensor& x, const Tensor& w, const Tensor& bias, const hot_layer_t& layer,
            const Buffer& buffer, PyObject* name) {
  node->set_next_edges(bias.defined() ? torch::autograd::collect_next_edges(x, w, bias) : torch::autograd::collect_next_edges(x, w));
  if (buffer.codes.defined()) {  // (else only the bias learns: nothing is needed of forward)
    node->s.x_q_t = SavedVariable(buffer.codes, false);
    node->s.w = SavedVariable(w, false);
    node->s.scale_x = SavedVariable(buffer.scale, false);
  }
  node->s.layer = layer;
  node->s.name = Py_NewRef(name);
  node->has_bias = bias.defined();
  torch::autograd::set_history(y, node);
}

// linear(x, w, bias or None, order_o, order_l, selection, name) -> output, or None (see the head of this file)
PyObject* linear_impl(PyObject* const* a) {
  hot_layer_t l = {};
  bool preset = false;
  if (!forward_config(a, l.cfg, preset)) return PyErr_Occurred() ? nullptr : Py_NewRef(Py_None);
  const Tensor x = THPVariable_Unpack(a[0]), w = THPVariable_Unpack(a[1]);
  const Tensor bias = a[2] == Py_None ? Tensor() : THPVariable_Unpack(a[2]);
  if (x.dim() < 2 || w.dim() != 2 || x.size(-1) != w.size(1) || w.stride(1) != 1) return Py_NewRef(Py_None);
  const bool per_sample = x.dim() == 3 && !preset;
  l.batch = per_sample ? x.size(0) : 0;
  l.I = x.size(-1);
  l.O = w.size(0);
  l.L = per_sample ? x.size(1) : x.numel() / l.I;
  if (l.L % l.cfg.order_l != 0 || l.batch > 65535) return Py_NewRef(Py_None);
  if (!per_sample && l.cfg.q_x.bits <= 4) l.cfg.q_x.storage = HOT_STORE_INT4;  // the saved buffer of the plain layout stays packed
  l.cfg.q_x.offset = take_offsets(1);
  Tensor y;
  Buffer buffer;
  std::shared_ptr<HotLinearBackward> node;
  const bool data_grads = wants_grad(x) || wants_grad(w);
  if (data_grads || wants_grad(bias)) node.reset(new HotLinearBackward(), torch::autograd::deleteNode);
  {
    pybind11::gil_scoped_release no_gil;
    at::AutoDispatchBelowADInplaceOrView below;
    c10::cuda::CUDAGuard guard(x.device());
    if (data_grads) buffer = compress(l, x.contiguous());
    // 16-bit tensors: the bias goes into the forward GEMM (one rounding of the output); float32 keeps the reference's
    // separate addition, whose result the parity tests pin bit for bit
    const bool fused = bias.defined() && l.cfg.dtype == HOT_BF16;
    y = fused ? at::linear(x, w, bias) : at::linear(x, w);
    if (bias.defined() && !fused) {
      if (y.scalar_type() == at::kFloat && y.is_contiguous() && bias.is_contiguous() && bias.numel() == l.O)
        check(hot_add_bias((float*)y.data_ptr(), (const float*)bias.data_ptr(), y.numel() / l.O, l.O, current_stream()), "hot_add_bias");
      else y.add_(bias);
    }
  }
  if (node) attach(node, y, x, w, bias, l, buffer, a[6]);
  return THPVariable_Wrap(y);
}

// conv2d(x, w, bias or None, order_o, order_l, selection, name, stride, padding, dilation (pairs)) -> output, or None
PyObject* conv2d_impl(PyObject* const* a) {
  hot_layer_t l = {};
  bool preset = false;
  if (!forward_config(a, l.cfg, preset)) return PyErr_Occurred() ? nullptr : Py_NewRef(Py_None);
  const Tensor x = THPVariable_Unpack(a[0]), w = THPVariable_Unpack(a[1]);
  const Tensor bias = a[2] == Py_None ? Tensor() : THPVariable_Unpack(a[2]);
  if (x.dim() != 4 || w.dim() != 4 || x.size(1) != w.size(1) || !w.is_contiguous()) return Py_NewRef(Py_None);
  if (bias.defined() && (bias.dim() != 1 || bias.size(0) != w.size(0) || !bias.is_contiguous())) return Py_NewRef(Py_None);  // (read as it lies)
  hot_conv_t v = {};
  v.dtype = l.cfg.dtype;
  v.B = x.size(0); v.C = x.size(1); v.H = x.size(2); v.W = x.size(3);
  v.kh = (int32_t)w.size(2); v.kw = (int32_t)w.size(3);
  if (!PyArg_ParseTuple(a[7], "ii", &v.sh, &v.sw) || !PyArg_ParseTuple(a[8], "ii", &v.ph, &v.pw) || !PyArg_ParseTuple(a[9], "ii", &v.dh, &v.dw)) {
    PyErr_Clear();
    return Py_NewRef(Py_None);
  }
  const int64_t oh = (v.H + 2 * v.ph - v.dh * (v.kh - 1) - 1) / v.sh + 1, ow = (v.W + 2 * v.pw - v.dw * (v.kw - 1) - 1) / v.sw + 1;
  if (v.H + 2 * v.ph < v.dh * (v.kh - 1) + 1 || v.W + 2 * v.pw < v.dw * (v.kw - 1) + 1 || v.B > 65535) return Py_NewRef(Py_None);
  const int64_t positions = oh * ow;
  if (positions > (1 << 30) || v.C * v.kh * v.kw > (1 << 30)) return Py_NewRef(Py_None);
  l.batch = preset ? 0 : v.B;
  l.L = preset ? v.B * positions : positions;
  l.I = v.C * v.kh * v.kw;
  l.O = w.size(0);
  if (l.L % l.cfg.order_l != 0) return Py_NewRef(Py_None);
  if (preset && l.cfg.q_x.bits <= 4) l.cfg.q_x.storage = HOT_STORE_INT4;
  l.cfg.q_x.offset = take_offsets(1);
  Tensor y;
  Buffer buffer;
  std::shared_ptr<HotConvBackward> node;
  const bool data_grads = wants_grad(x) || wants_grad(w);
  if (data_grads || wants_grad(bias)) {
    node.reset(new HotConvBackward(), torch::autograd::deleteNode);
    node->conv = v;
    node->positions = positions;
  }
  {
    pybind11::gil_scoped_release no_gil;
    at::AutoDispatchBelowADInplaceOrView below;
    c10::cuda::CUDAGuard guard(x.device());
    const Tensor xc = x.contiguous(), cols = at::empty({v.B, positions, l.I}, x.options());
    check(hot_im2col(&v, xc.data_ptr(), cols.data_ptr(), current_stream()), "hot_im2col");
    if (data_grads) buffer = compress(l, cols);
    const Tensor rows = at::linear(cols, w.view({l.O, l.I}));
    TORCH_CHECK(rows.scalar_type() == x.scalar_type() && rows.is_contiguous(), "HQ_Conv2d: the product came back in another type or layout");
    y = at::empty({v.B, l.O, oh, ow}, x.options());
    check(hot_transpose(v.dtype, v.B, positions, l.O, rows.data_ptr(), bias.defined() ? bias.data_ptr() : nullptr, y.data_ptr(), current_stream()),
          "hot_transpose");
  }
  if (node) attach(node, y, x, w, bias, l, buffer, a[6]);
  return THPVariable_Wrap(y);
}

// plugin_ready(go, w, x) -> whether the plugin call takes these three (a caller that gets False finds out why itself)
PyObject* plugin_ready_impl(PyObject* const* a) {
  for (int i = 0; i < 3; ++i)
    if (!THPVariable_Check(a[i])) Py_RETURN_FALSE;
  const Tensor &go = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]), &x = THPVariable_Unpack(a[2]);
  for (const Tensor* t : {&go, &w, &x})
    if (!t->is_cuda() || !t->is_contiguous() || t->dim() != 2 || t->scalar_type() != go.scalar_type()) Py_RETURN_FALSE;
  return PyBool_FromLong(w.size(0) == go.size(1) && x.size(0) == go.size(0) && x.size(1) == w.size(1));
}

// plugin(go, w, x, order_o, order_l, selection, per_token, philox, seed, base) -> (grad_x, grad_w, quantise seconds, product seconds)
PyObject* plugin_impl(PyObject* const* a) {
  const Tensor go = THPVariable_Unpack(a[0]), w = THPVariable_Unpack(a[1]), x = THPVariable_Unpack(a[2]);
  const int dt = dtype_code(go.scalar_type());
  TORCH_CHECK_TYPE(dt >= 0, "hot_b200 supports float32 and bfloat16 tensors, got ", go.scalar_type());
  const int64_t L = go.size(0), O = go.size(1), I = w.size(1);
  hot_linear_cfg_t c = {};
  c.dtype = dt;
  c.order_o = (int32_t)PyLong_AsLong(a[3]);
  c.order_l = (int32_t)PyLong_AsLong(a[4]);
  c.rank_l = (int32_t)std::min<Py_ssize_t>(PyList_Size(a[5]), 64);
  for (int i = 0; i < c.rank_l; ++i) c.sel_l[i] = (int32_t)PyLong_AsLong(PyList_GetItem(a[5], i));
  const bool per_token = PyObject_IsTrue(a[6]) == 1, philox = PyObject_IsTrue(a[7]) == 1;
  const uint64_t seed = PyLong_AsUnsignedLongLongMask(a[8]), base = PyLong_AsUnsignedLongLongMask(a[9]);
  if (PyErr_Occurred()) return nullptr;
  auto q = [&](int bits, int row, uint64_t k) {
    hot_quant_t r = {};
    r.bits = bits;
    r.storage = HOT_STORE_INT8;
    r.rounding = philox ? HOT_ROUND_STOCH_PHILOX : HOT_ROUND_NEAREST;
    r.scale_mode = row ? HOT_SCALE_ROW : HOT_SCALE_TENSOR;
    r.seed = seed;
    r.offset = base + k;
    return r;
  };
  c.q_gx = q(4, per_token, 1);
  c.q_w = q(4, 0, 2);
  c.q_gw = q(8, 0, 3);
  c.q_x = q(8, 0, 4);
  Tensor gx, gw;
  float ms[2] = {0.0f, 0.0f};
  {
    pybind11::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    c10::cuda::CUDAGuard guard(go.device());
    const size_t ws_bytes = hot_hlq_workspace_bytes(L, O, I, &c);
    if (ws_bytes == 0) fail(HOT_ERR_UNSUPPORTED, "HLQ_backward");
    const Tensor ws = bytes((int64_t)ws_bytes, go);
    gx = at::empty({L, I}, go.options());
    gw = at::empty({O, I}, go.options());
    const int rc = hot_hlq_backward(go.data_ptr(), w.data_ptr(), x.data_ptr(), L, O, I, &c, gx.data_ptr(), gw.data_ptr(), ws.data_ptr(),
                                    ws_bytes, ms, current_stream());
    check(rc, "HLQ_backward");
  }
  return Py_BuildValue("(NNdd)", THPVariable_Wrap(gx), THPVariable_Wrap(gw), 1e-3 * ms[0], 1e-3 * ms[1]);
}

// row_ht_quant(x, order, bits, packed, rounding, per_row, seed, offset, noise pointer) -> (codes, scales)
PyObject* row_ht_quant_impl(PyObject* const* a) {
  const Tensor x = THPVariable_Unpack(a[0]);
  const int dt = dtype_code(x.scalar_type());
  TORCH_CHECK_TYPE(dt >= 0, "hot_b200 supports float32 and bfloat16 tensors, got ", x.scalar_type());
  const long order = PyLong_AsLong(a[1]);
  hot_quant_t q = {};
  q.bits = (int32_t)PyLong_AsLong(a[2]);
  q.storage = PyObject_IsTrue(a[3]) == 1 ? HOT_STORE_INT4 : HOT_STORE_INT8;
  q.rounding = (int32_t)PyLong_AsLong(a[4]);
  q.scale_mode = PyObject_IsTrue(a[5]) == 1 ? HOT_SCALE_ROW : HOT_SCALE_TENSOR;
  q.seed = PyLong_AsUnsignedLongLongMask(a[6]);
  q.offset = PyLong_AsUnsignedLongLongMask(a[7]);
  q.noise = (const float*)(uintptr_t)PyLong_AsUnsignedLongLong(a[8]);
  if (PyErr_Occurred()) return nullptr;
  const int64_t rows = x.size(0), cols = x.size(1);
  const int64_t row_bytes = q.storage == HOT_STORE_INT4 ? cols / 2 : cols, pitch = (row_bytes + 15) / 16 * 16;
  Tensor codes, scales;
  {
    pybind11::gil_scoped_release no_gil;
    at::NoGradGuard no_grad;
    c10::cuda::CUDAGuard guard(x.device());
    codes = at::empty({rows, pitch}, x.options().dtype(at::kByte));
    scales = at::empty({q.scale_mode == HOT_SCALE_ROW ? rows : 1}, x.options().dtype(at::kFloat));
    const Tensor ws = q.scale_mode == HOT_SCALE_ROW ? Tensor() : at::empty({16}, x.options().dtype(at::kInt));
    check(hot_row_ht_quant(x.data_ptr(), dt, rows, cols, x.stride(0), (int)order, &q, codes.data_ptr(), pitch, (float*)scales.data_ptr(),
                           ws.defined() ? (uint32_t*)ws.data_ptr() : nullptr, current_stream()),
          "hot_row_ht_quant");
    if (pitch != row_bytes) codes = codes.narrow(1, 0, row_bytes);
  }
  return Py_BuildValue("(NN)", THPVariable_Wrap(codes), THPVariable_Wrap(scales));
}

template <PyObject* (*Impl)(PyObject* const*), int kArgs>
PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != kArgs) {
    PyErr_Format(PyExc_TypeError, "%d arguments expected, got %zd", kArgs, n);
    return nullptr;
  }
  return Impl(args);
  END_HANDLE_TH_ERRORS
}

PyObject* bind_impl(PyObject* const* a) {
  Py_XSETREF(g_qm, Py_NewRef(a[0]));
  Py_XSETREF(g_error, Py_NewRef(a[1]));
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)(void))call<bind_impl, 2>, METH_FASTCALL, "bind(quant_matmul, HotError)"},
    {"linear", (PyCFunction)(void (*)(void))call<linear_impl, 7>, METH_FASTCALL, "one HOT linear layer with its autograd node, or None"},
    {"conv2d", (PyCFunction)(void (*)(void))call<conv2d_impl, 10>, METH_FASTCALL, "one HOT convolution with its autograd node, or None"},
    {"plugin_ready", (PyCFunction)(void (*)(void))call<plugin_ready_impl, 3>, METH_FASTCALL, "whether plugin takes these tensors"},
    {"plugin", (PyCFunction)(void (*)(void))call<plugin_impl, 10>, METH_FASTCALL, "both gradients of one linear layer, complete on return"},
    {"row_ht_quant", (PyCFunction)(void (*)(void))call<row_ht_quant_impl, 9>, METH_FASTCALL, "codes and scales of the fused row quantiser"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "hot_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hot_torch(void) {
  intern_names();
  return PyModule_Create(&module);
}
