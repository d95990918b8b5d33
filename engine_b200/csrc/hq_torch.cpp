// Host path of the Python layer in native code: argument checks, output and scratch allocation and the calls into
// libhanzoquant_b200.so (the C ABI of include/hanzoquant_b200.h) for one QuantMethod / MoE call.  Written against the
// CPython API and ATen directly: a decode call is a few microseconds of GPU time, and the same steps through ctypes and
// torch's Python functions took 10 - 60 us per call (one linear 15 us, a one-token MoE layer 55 us).
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <unordered_map>

#include "../../include/hanzoquant_b200.h"

// three projections of one activation with a status word each (hq_api.cu; not part of the public header)
extern "C" int32_t hq_linear_qkv_run(const hq_weight* const w[3], const void* x, int32_t x_dtype, int64_t x_stride,
                                     void* const y[3], int32_t y_dtype, int64_t m, int32_t* const status_dev[3], void* stream);

namespace {

PyObject* g_error = nullptr;      // engine_b200._lib.HqError

struct Fail {};                   // a Python error has been set

[[noreturn]] void fail(const char* msg) {
  PyErr_SetString(g_error != nullptr ? g_error : PyExc_RuntimeError, msg);
  throw Fail{};
}
void check(int32_t rc, const char* what) {
  if (rc == HQ_OK) return;
  PyErr_Format(g_error != nullptr ? g_error : PyExc_RuntimeError, "%s: %s (%d)", what, hq_error_string(rc), (int)rc);
  throw Fail{};
}

int dt_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return HQ_DT_F32;
    case at::kHalf: return HQ_DT_F16;
    case at::kBFloat16: return HQ_DT_BF16;
    default: break;
  }
  PyErr_Format(g_error, "unsupported dtype %s: expected f32, f16 or bf16", c10::toString(t));
  throw Fail{};
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor", what);
    throw Fail{};
  }
  return THPVariable_Unpack(o);
}
const at::Tensor& cuda_tensor(PyObject* o, const char* what) {
  const at::Tensor& t = tensor(o, what);
  if (!t.is_cuda()) {
    PyErr_Format(g_error, "%s must be a CUDA tensor: this library has no CPU path", what);
    throw Fail{};
  }
  return t;
}
at::ScalarType dtype_or(PyObject* o, at::ScalarType other) {
  if (o == nullptr || o == Py_None) return other;
  if (!THPDtype_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "out_dtype must be a torch.dtype");
    throw Fail{};
  }
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}
cudaStream_t stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Tensor& like) {
  return at::empty(shape, like.options().dtype(dtype));
}
at::Tensor f32(const at::Tensor& t) { return t.scalar_type() == at::kFloat ? t.contiguous() : t.to(at::kFloat).contiguous(); }

// ---- a layer: its descriptor, its status words, its scratch per stream -------------------------------------------
struct Layer {
  PyObject_HEAD
  hq_weight w;
  at::Tensor* status;
  std::unordered_map<int64_t, int64_t>* need;                  // rows -> scratch bytes
  std::unordered_map<void*, at::Tensor>* scratch;              // stream -> zero-filled scratch
  int32_t* status_ptr() const { return status->data_ptr<int32_t>(); }
  int64_t scratch_bytes(int64_t m) {
    auto it = need->find(m);
    return it != need->end() ? it->second : (*need)[m] = hq_linear_workspace_bytes(&w, m);
  }
};
PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0) "engine_b200._hqtorch.Layer", sizeof(Layer)};

void layer_dealloc(PyObject* o) {
  Layer* l = reinterpret_cast<Layer*>(o);
  delete l->status;
  delete l->need;
  delete l->scratch;
  Py_TYPE(o)->tp_free(o);
}
Layer* layer(PyObject* o) {
  if (Py_TYPE(o) != &LayerType) {
    PyErr_SetString(PyExc_TypeError, "expected a layer handle");
    throw Fail{};
  }
  return reinterpret_cast<Layer*>(o);
}

// layer(address of an hq_weight, status tensor int32[4])
PyObject* py_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) return PyErr_Format(PyExc_TypeError, "layer(address, status)");
  const void* src = PyLong_AsVoidPtr(a[0]);
  if (src == nullptr || !THPVariable_Check(a[1])) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "layer(address, status)");
    return nullptr;
  }
  Layer* l = PyObject_New(Layer, &LayerType);
  if (l == nullptr) return nullptr;
  l->w = *static_cast<const hq_weight*>(src);
  l->status = new at::Tensor(THPVariable_Unpack(a[1]));
  l->need = new std::unordered_map<int64_t, int64_t>();
  l->scratch = new std::unordered_map<void*, at::Tensor>();
  return reinterpret_cast<PyObject*>(l);
}

// rows of a [.., k] activation as the library reads them
struct Rows {
  at::Tensor hold;
  const void* ptr;
  int dtype;
  int64_t m, stride;
};
Rows rows_of(const at::Tensor& a, int64_t k) {
  Rows r;
  const int64_t d = a.dim();
  if (d == 2 && a.stride(1) == 1) {
    r.hold = a;
    r.stride = a.stride(0);
  } else {
    r.hold = a.is_contiguous() ? a : a.reshape({-1, k}).contiguous();
    r.stride = k;
  }
  r.m = a.numel() / k;
  if (r.m <= 1) r.stride = k;
  r.ptr = r.hold.data_ptr();
  r.dtype = dt_code(a.scalar_type());
  return r;
}
void to_f16(Rows& r, int64_t k, const at::Tensor& like, int32_t* status, cudaStream_t s) {
  if (r.dtype == HQ_DT_F16) return;
  if (r.m > 1 && r.stride != k) {
    r.hold = r.hold.contiguous();
    r.ptr = r.hold.data_ptr();
    r.stride = k;
  }
  at::Tensor h = empty({r.m, k}, at::kHalf, like);
  check(hq_convert_status(r.ptr, r.dtype, h.data_ptr(), HQ_DT_F16, r.m * k, status, s), "hq_convert_status");
  r.hold = h;
  r.ptr = h.data_ptr();
  r.dtype = HQ_DT_F16;
}
at::Tensor out_like(const at::Tensor& a, int64_t n, at::ScalarType dtype) {
  if (a.dim() == 2) return empty({a.size(0), n}, dtype, a);
  std::vector<int64_t> shape(a.sizes().begin(), a.sizes().end());
  shape.back() = n;
  return empty(shape, dtype, a);
}

at::Tensor run_linear(Layer* l, const at::Tensor& a, at::ScalarType out_dtype, Rows& x, cudaStream_t s) {
  at::Tensor y = out_like(a, l->w.n, out_dtype);
  void* ws = nullptr;
  int64_t ws_bytes = 0;
  const int64_t need = l->scratch_bytes(x.m);
  if (need > 0) {
    at::Tensor& t = (*l->scratch)[s];
    if (!t.defined() || t.numel() < need) t = at::zeros({need}, a.options().dtype(at::kByte));
    ws = t.data_ptr();
    ws_bytes = t.numel();
  }
  check(hq_linear_forward_ws(&l->w, x.ptr, x.dtype, x.stride, y.data_ptr(), dt_code(out_dtype), l->w.n, x.m, ws, ws_bytes,
                             l->status_ptr(), s),
        "hq_linear_forward_ws");
  return y;
}


#define HQ_TRY try {
#define HQ_CATCH                                                          \
  }                                                                       \
  catch (const Fail&) {                                                   \
    return nullptr;                                                       \
  }                                                                       \
  catch (const std::exception& e) {                                       \
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what()); \
    return nullptr;                                                       \
  }

// linear(layer, a, out_dtype or None): y = a . W^T (+ b), leading dims flattened to rows
PyObject* py_linear(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 3) return PyErr_Format(PyExc_TypeError, "linear(layer, a, out_dtype)");
  Layer* l = layer(p[0]);
  const at::Tensor& a = cuda_tensor(p[1], "a");
  if (l->w.n_experts != 1) fail("forward on an expert bank: use gather_forward");
  if (a.dim() < 1 || a.size(-1) != l->w.k) {
    PyErr_Format(g_error, "shape mismatch: input has %lld features, weight expects %lld",
                 a.dim() < 1 ? 0ll : (long long)a.size(-1), (long long)l->w.k);
    return nullptr;
  }
  const c10::cuda::CUDAGuard guard(a.device());
  const cudaStream_t s = stream_of(a);
  const at::ScalarType od = dtype_or(p[2], a.scalar_type());
  Rows x = rows_of(a, l->w.k);
  if (hq_tensor_path(&l->w, x.m, 1)) to_f16(x, l->w.k, a, l->status_ptr(), s);
  return THPVariable_Wrap(run_linear(l, a, od, x, s));
  HQ_CATCH
}

// qkv(q, k, v, xs, out_dtype or None): three projections of one activation
PyObject* py_qkv(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 5) return PyErr_Format(PyExc_TypeError, "qkv(q, k, v, xs, out_dtype)");
  Layer* l[3] = {layer(p[0]), layer(p[1]), layer(p[2])};
  const at::Tensor& a = cuda_tensor(p[3], "xs");
  const c10::cuda::CUDAGuard guard(a.device());
  const cudaStream_t s = stream_of(a);
  const at::ScalarType od = dtype_or(p[4], a.scalar_type());
  Rows x = rows_of(a, l[0]->w.k);
  if (hq_tensor_path(&l[0]->w, x.m, 1)) to_f16(x, l[0]->w.k, a, l[0]->status_ptr(), s);
  bool scratch = false;
  for (int i = 0; i < 3; ++i) scratch = scratch || l[i]->scratch_bytes(x.m) > 0 || l[i]->w.k != l[0]->w.k;
  if (!scratch) {
    at::Tensor y[3];
    const hq_weight* w[3];
    void* yp[3];
    int32_t* status[3];
    for (int i = 0; i < 3; ++i) {
      y[i] = out_like(a, l[i]->w.n, od);
      w[i] = &l[i]->w;
      yp[i] = y[i].data_ptr();
      status[i] = l[i]->status_ptr();
    }
    check(hq_linear_qkv_run(w, x.ptr, x.dtype, x.stride, yp, dt_code(od), x.m, status, s), "hq_linear_qkv_forward");
    return Py_BuildValue("(NNN)", THPVariable_Wrap(y[0]), THPVariable_Wrap(y[1]), THPVariable_Wrap(y[2]));
  }
  PyObject* out = PyTuple_New(3);
  if (out == nullptr) return nullptr;
  for (int i = 0; i < 3; ++i) {
    try {
      PyTuple_SET_ITEM(out, i, THPVariable_Wrap(run_linear(l[i], a, od, x, s)));
    } catch (...) {
      Py_DECREF(out);
      throw;
    }
  }
  return out;
  HQ_CATCH
}

// glu(gate, up, xs, address of an hq_act_args, out_dtype or None): act(xs . Wg^T) * (xs . Wu^T) in one launch
PyObject* py_glu(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 5) return PyErr_Format(PyExc_TypeError, "glu(gate, up, xs, act, out_dtype)");
  Layer *g = layer(p[0]), *u = layer(p[1]);
  const at::Tensor& a = cuda_tensor(p[2], "xs");
  const hq_act_args* act = static_cast<const hq_act_args*>(PyLong_AsVoidPtr(p[3]));
  if (act == nullptr) return nullptr;
  const c10::cuda::CUDAGuard guard(a.device());
  const cudaStream_t s = stream_of(a);
  const at::ScalarType od = dtype_or(p[4], a.scalar_type());
  Rows x = rows_of(a, g->w.k);
  if (hq_tensor_path(&g->w, x.m, 1)) to_f16(x, g->w.k, a, g->status_ptr(), s);
  at::Tensor y = out_like(a, g->w.n, od);
  check(hq_linear_glu_forward(&g->w, &u->w, act, x.ptr, x.dtype, x.stride, y.data_ptr(), dt_code(od), g->w.n, x.m,
                              g->status_ptr(), s),
        "hq_linear_glu_forward");
  return THPVariable_Wrap(y);
  HQ_CATCH
}

// ---- router ------------------------------------------------------------------------------------------------------
struct RouterNames {
  PyObject *top_k, *score, *selected, *renorm, *norm_min, *scale, *clip;
};
RouterNames g_names;

double number(PyObject* o, PyObject* name) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (v == nullptr) throw Fail{};
  const double d = PyFloat_AsDouble(v);
  Py_DECREF(v);
  if (d == -1.0 && PyErr_Occurred()) throw Fail{};
  return d;
}
hq_router_args router_args(int64_t n_experts, PyObject* config, const at::Tensor& bias, const at::Tensor& scale) {
  hq_router_args r{};
  r.n_experts = (int32_t)n_experts;
  r.top_k = (int32_t)number(config, g_names.top_k);
  r.score_mode = (int32_t)number(config, g_names.score);
  r.weight_mode = (int32_t)number(config, g_names.selected);
  r.renormalize = number(config, g_names.renorm) != 0.0;
  r.norm_min = (float)number(config, g_names.norm_min);
  r.output_scale = (float)number(config, g_names.scale);
  PyObject* clip = PyObject_GetAttr(config, g_names.clip);
  if (clip == nullptr) throw Fail{};
  if (clip != Py_None) {
    r.clamp_logits = 1;
    PyObject *lo = PySequence_GetItem(clip, 0), *hi = PySequence_GetItem(clip, 1);
    r.clamp_min = lo != nullptr ? (float)PyFloat_AsDouble(lo) : 0.f;
    r.clamp_max = hi != nullptr ? (float)PyFloat_AsDouble(hi) : 0.f;
    Py_XDECREF(lo);
    Py_XDECREF(hi);
  }
  Py_DECREF(clip);
  if (PyErr_Occurred()) throw Fail{};
  r.selection_bias = bias.defined() ? bias.data_ptr<float>() : nullptr;
  r.expert_scale = scale.defined() ? scale.data_ptr<float>() : nullptr;
  return r;
}
at::Tensor optional_f32(PyObject* o, const char* what) { return o == Py_None ? at::Tensor() : f32(tensor(o, what)); }

// router(logits, config, selection_bias, expert_scale, n_group, topk_group, group mode) -> (weights f32, ids int32)
PyObject* py_router(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 7) return PyErr_Format(PyExc_TypeError, "router(logits, config, bias, scale, n_group, topk_group, mode)");
  const at::Tensor& in = cuda_tensor(p[0], "logits");
  if (in.dim() != 2) fail("logits must be [tokens, experts]");
  const c10::cuda::CUDAGuard guard(in.device());
  const at::Tensor logits = in.contiguous(), bias = optional_f32(p[2], "selection_bias"), scale = optional_f32(p[3], "expert_scale");
  const int64_t t = logits.size(0), e = logits.size(1);
  const hq_router_args r = router_args(e, p[1], bias, scale);
  const long n_group = PyLong_AsLong(p[4]), topk_group = PyLong_AsLong(p[5]), mode = PyLong_AsLong(p[6]);
  if (PyErr_Occurred()) return nullptr;
  if (r.top_k < 0) fail("top_k must not be negative");
  at::Tensor ids = empty({t, r.top_k}, at::kInt, logits), w = empty({t, r.top_k}, at::kFloat, logits);
  const cudaStream_t s = stream_of(logits);
  uint32_t* idp = reinterpret_cast<uint32_t*>(ids.data_ptr<int32_t>());
  if (n_group > 1)
    check(hq_router_topk_grouped(logits.data_ptr(), dt_code(logits.scalar_type()), t, &r, (int32_t)n_group,
                                 (int32_t)topk_group, (int32_t)mode, idp, w.data_ptr<float>(), s),
          "hq_router_topk_grouped");
  else
    check(hq_router_topk(logits.data_ptr(), dt_code(logits.scalar_type()), t, &r, idp, w.data_ptr<float>(), s), "hq_router_topk");
  return Py_BuildValue("(NN)", THPVariable_Wrap(w), THPVariable_Wrap(ids));
  HQ_CATCH
}

// ---- MoE layers --------------------------------------------------------------------------------------------------
// One allocation for a call's scratch, cut into 256-byte aligned pieces
struct Scratch {
  int64_t total = 0;
  at::Tensor hold;
  uint8_t* base = nullptr;
  int64_t add(int64_t bytes) {
    const int64_t at = total;
    total += (bytes + 255) / 256 * 256;
    return at;
  }
  void alloc(const at::Tensor& like) {
    hold = empty({total > 0 ? total : 256}, at::kByte, like);
    base = hold.data_ptr<uint8_t>();
  }
};
// the dispatch tables of one call
struct Tables {
  int64_t bounds, sa, st, inv, ws, ws_bytes;
  Tables(Scratch& s, int64_t t, int32_t k, int32_t e) {
    bounds = s.add((e + 1) * 4);
    sa = s.add(t * k * 4);
    st = s.add(t * k * 4);
    inv = s.add(t * k * 4);
    ws_bytes = hq_moe_dispatch_workspace_bytes(t, k, e);
    ws = s.add(ws_bytes);
  }
  void build(const Scratch& s, const uint32_t* ids, int64_t t, int32_t k, int32_t e, cudaStream_t stream) const {
    check(hq_moe_dispatch_build(ids, t, k, e, (int32_t*)(s.base + bounds), (int32_t*)(s.base + sa), (int32_t*)(s.base + st),
                                (int32_t*)(s.base + inv), s.base + ws, ws_bytes, stream),
          "hq_moe_dispatch_build");
  }
};

// moe_layer(gate or gate_up, up or None, down, act address, xs, logits, config, bias, scale, shared_out, out_dtype)
PyObject* py_moe_layer(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 11) return PyErr_Format(PyExc_TypeError, "moe_layer: 11 arguments");
  Layer *g = layer(p[0]), *u = p[1] == Py_None ? nullptr : layer(p[1]), *d = layer(p[2]);
  const hq_act_args* act = static_cast<const hq_act_args*>(PyLong_AsVoidPtr(p[3]));
  if (act == nullptr) return nullptr;
  const at::Tensor& xs = cuda_tensor(p[4], "xs");
  const c10::cuda::CUDAGuard guard(xs.device());
  const cudaStream_t s = stream_of(xs);
  const at::Tensor x = xs.contiguous();
  const int64_t hidden = xs.size(-1), t = hidden > 0 ? xs.numel() / hidden : 0;
  const at::Tensor logits = tensor(p[5], "logits").contiguous();
  const at::Tensor bias = optional_f32(p[7], "selection_bias"), scale = optional_f32(p[8], "expert_scale");
  if (hidden != g->w.k || logits.numel() != t * d->w.n_experts)
    fail("forward_layer: input / logits / weight shapes disagree");
  const at::ScalarType od = dtype_or(p[10], xs.scalar_type());
  hq_moe_layer layer_args{};
  layer_args.gate = &g->w;
  layer_args.up = u != nullptr ? &u->w : nullptr;
  layer_args.down = &d->w;
  layer_args.act = *act;
  layer_args.router = router_args(d->w.n_experts, p[6], bias, scale);
  const int xdt = dt_code(x.scalar_type());
  const int64_t need = hq_moe_layer_workspace_bytes(&layer_args, t, xdt);
  if (need == 0 && t > 0) fail("hq_moe_layer_workspace_bytes: the layer description is inconsistent");
  Scratch sc;
  sc.add(need);
  sc.alloc(x);
  at::Tensor out = out_like(xs, d->w.n, od), add;
  if (p[9] != Py_None) {
    add = tensor(p[9], "shared_out");
    add = add.scalar_type() == od ? add.contiguous() : add.to(od).contiguous();
    if (add.numel() != t * d->w.n) fail("forward_layer: shared_out does not match the output");
  }
  check(hq_moe_layer_forward(&layer_args, logits.data_ptr(), dt_code(logits.scalar_type()), x.data_ptr(), xdt, t,
                             add.defined() ? add.data_ptr() : nullptr, out.data_ptr(), dt_code(od), sc.base, sc.total,
                             g->status_ptr(), s),
        "hq_moe_layer_forward");
  return THPVariable_Wrap(out);
  HQ_CATCH
}

// ids as int32 [T, k], weights as f32 [T, k]
struct Routing {
  at::Tensor ids, w;
  int64_t t;
  int32_t k;
  Routing(PyObject* weights, PyObject* indices) {
    ids = cuda_tensor(indices, "topk_ids");
    if (ids.dim() != 2) fail("topk_ids must be [tokens, top_k]");
    if (ids.scalar_type() != at::kInt && ids.scalar_type() != at::kUInt32) ids = ids.to(at::kInt);
    ids = ids.contiguous();
    w = f32(cuda_tensor(weights, "topk_weights"));
    t = ids.size(0);
    k = (int32_t)ids.size(1);
    if (w.numel() != t * k) fail("topk_weights and topk_ids disagree");
  }
  const uint32_t* id_ptr() const { return static_cast<const uint32_t*>(ids.data_ptr()); }
};
at::ScalarType row_dtype(at::ScalarType out) { return out == at::kHalf || out == at::kBFloat16 ? out : at::kFloat; }

// the addend of the weighted reduce in the output's dtype
at::Tensor addend(PyObject* shared, at::ScalarType od, int64_t elems) {
  if (shared == Py_None) return at::Tensor();
  at::Tensor a = tensor(shared, "shared_out");
  a = a.scalar_type() == od ? a.contiguous() : a.to(od).contiguous();
  if (a.numel() != elems) fail("shared_out does not match the output");
  return a;
}

// moe_fp8(gate, up, down, act address, xs, topk_weights, topk_ids, shared_out, out_dtype)
PyObject* py_moe_fp8(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 9) return PyErr_Format(PyExc_TypeError, "moe_fp8: 9 arguments");
  Layer *g = layer(p[0]), *u = layer(p[1]), *d = layer(p[2]);
  const hq_act_args* act = static_cast<const hq_act_args*>(PyLong_AsVoidPtr(p[3]));
  if (act == nullptr) return nullptr;
  const at::Tensor& xs = cuda_tensor(p[4], "xs");
  const c10::cuda::CUDAGuard guard(xs.device());
  const cudaStream_t s = stream_of(xs);
  const at::Tensor x = xs.contiguous();
  const Routing r(p[5], p[6]);
  const int64_t hidden = xs.size(-1), inter = g->w.n, rows = r.t * r.k;
  if (hidden != g->w.k || x.numel() != r.t * hidden) fail("forward_fp8_act: input / indices / weight shapes disagree");
  const int32_t e = d->w.n_experts;
  const at::ScalarType od = dtype_or(p[8], xs.scalar_type()), yd = row_dtype(od);
  Scratch sc;
  const Tables tb(sc, r.t, r.k, e);
  const int64_t xq = sc.add(rows * hidden), xsc = sc.add(rows * (hidden / 128) * 4), hq = sc.add(rows * inter),
                hs = sc.add(rows * (inter / 128) * 4), y = sc.add(rows * d->w.n * (yd == at::kFloat ? 4 : 2));
  // A token's row stands in the sorted order once per slot.  Quantizing it each time is bound by the divisions (4,096 tokens x
  // 8 slots x 7,168: 270 us); from about a thousand rows the tokens are quantized once and their codes copied (launch and copy
  // cost less than the divisions saved).
  const bool once = r.k > 1 && rows >= 1024;
  const int64_t tq = once ? sc.add(r.t * hidden) : 0, ts = once ? sc.add(r.t * (hidden / 128) * 4) : 0;
  sc.alloc(x);
  const int32_t* bounds = (const int32_t*)(sc.base + tb.bounds);
  at::Tensor out = out_like(xs, d->w.n, od);
  const at::Tensor add = addend(p[7], od, out.numel());
  tb.build(sc, r.id_ptr(), r.t, r.k, e, s);
  if (once) {
    check(hq_fp8_quant_rows(x.data_ptr(), dt_code(x.scalar_type()), hidden, nullptr, r.t, hidden, sc.base + tq,
                            (float*)(sc.base + ts), s),
          "hq_fp8_quant_rows");
    check(hq_fp8_gather_rows(sc.base + tq, hidden, (const float*)(sc.base + ts), hidden / 128 * 4, (const int32_t*)(sc.base + tb.st),
                             bounds + e, rows, hidden, sc.base + xq, (float*)(sc.base + xsc), s),
          "hq_fp8_gather_rows");
  } else {
    check(hq_fp8_quant_rows_n(x.data_ptr(), dt_code(x.scalar_type()), hidden, (const int32_t*)(sc.base + tb.st), bounds + e,
                              rows, hidden, sc.base + xq, (float*)(sc.base + xsc), s),
          "hq_fp8_quant_rows_n");
  }
  check(hq_moe_fp8_gate_up_forward(&g->w, &u->w, act, sc.base + xq, (const float*)(sc.base + xsc), r.t, r.k, bounds,
                                   sc.base + hq, (float*)(sc.base + hs), g->status_ptr(), s),
        "hq_moe_fp8_gate_up_forward");
  check(hq_moe_fp8_gather_forward(&d->w, sc.base + hq, (const float*)(sc.base + hs), r.t, r.k, bounds,
                                  (const int32_t*)(sc.base + tb.sa), nullptr, sc.base + y, dt_code(yd), d->w.n, HQ_ROWS_SORTED,
                                  g->status_ptr(), s),
        "hq_moe_fp8_gather_forward(down)");
  check(hq_moe_weighted_reduce(sc.base + y, dt_code(yd), r.w.data_ptr<float>(), (const int32_t*)(sc.base + tb.inv),
                               add.defined() ? add.data_ptr() : nullptr, out.data_ptr(), dt_code(od), r.t, r.k, d->w.n, s),
        "hq_moe_weighted_reduce");
  return THPVariable_Wrap(out);
  HQ_CATCH
}

// moe_mx(gate_up, down, act address, xs, topk_weights, topk_ids, shared_out, out_dtype): interleaved gate/up rows
PyObject* py_moe_mx(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 8) return PyErr_Format(PyExc_TypeError, "moe_mx: 8 arguments");
  Layer *g = layer(p[0]), *d = layer(p[1]);
  const hq_act_args* act = static_cast<const hq_act_args*>(PyLong_AsVoidPtr(p[2]));
  if (act == nullptr) return nullptr;
  const at::Tensor& xs = cuda_tensor(p[3], "xs");
  const c10::cuda::CUDAGuard guard(xs.device());
  const cudaStream_t s = stream_of(xs);
  const at::Tensor x = xs.contiguous();
  const Routing r(p[4], p[5]);
  const int64_t hidden = xs.size(-1), inter = g->w.n / 2, rows = r.t * r.k;
  if (hidden != g->w.k || x.numel() != r.t * hidden) fail("forward_mx_act: input / indices / weight shapes disagree");
  const int32_t e = d->w.n_experts;
  const at::ScalarType od = dtype_or(p[7], xs.scalar_type()), yd = row_dtype(od);
  Scratch sc;
  const Tables tb(sc, r.t, r.k, e);
  const int64_t xq = sc.add(rows * hidden), xsc = sc.add(rows * (hidden / 32)), hq = sc.add(rows * inter),
                hs = sc.add(rows * (inter / 32)), y = sc.add(rows * d->w.n * (yd == at::kFloat ? 4 : 2));
  sc.alloc(x);
  const int32_t* bounds = (const int32_t*)(sc.base + tb.bounds);
  at::Tensor out = out_like(xs, d->w.n, od);
  const at::Tensor add = addend(p[6], od, out.numel());
  tb.build(sc, r.id_ptr(), r.t, r.k, e, s);
  check(hq_mxfp8_quant_rows(x.data_ptr(), dt_code(x.scalar_type()), hidden, (const int32_t*)(sc.base + tb.st), bounds + e, rows,
                            hidden, sc.base + xq, sc.base + xsc, s),
        "hq_mxfp8_quant_rows");
  check(hq_moe_mx_gather_forward(&g->w, act, sc.base + xq, sc.base + xsc, r.t, r.k, bounds, nullptr, nullptr, 0, 0,
                                 HQ_ROWS_SORTED, sc.base + hq, sc.base + hs, g->status_ptr(), s),
        "hq_moe_mx_gather_forward(gate_up)");
  check(hq_moe_mx_gather_forward(&d->w, nullptr, sc.base + hq, sc.base + hs, r.t, r.k, bounds, nullptr, sc.base + y, dt_code(yd),
                                 d->w.n, HQ_ROWS_SORTED, nullptr, nullptr, g->status_ptr(), s),
        "hq_moe_mx_gather_forward(down)");
  check(hq_moe_weighted_reduce(sc.base + y, dt_code(yd), r.w.data_ptr<float>(), (const int32_t*)(sc.base + tb.inv),
                               add.defined() ? add.data_ptr() : nullptr, out.data_ptr(), dt_code(od), r.t, r.k, d->w.n, s),
        "hq_moe_weighted_reduce");
  return THPVariable_Wrap(out);
  HQ_CATCH
}

// fp8_dense(gate, up, down, act address, xs, bounds int32 {0, rows}, out_dtype): a one-expert block over every row
PyObject* py_fp8_dense(PyObject*, PyObject* const* p, Py_ssize_t n) {
  HQ_TRY
  if (n != 7) return PyErr_Format(PyExc_TypeError, "fp8_dense: 7 arguments");
  Layer *g = layer(p[0]), *u = layer(p[1]), *d = layer(p[2]);
  const hq_act_args* act = static_cast<const hq_act_args*>(PyLong_AsVoidPtr(p[3]));
  if (act == nullptr) return nullptr;
  const at::Tensor& xs = cuda_tensor(p[4], "xs");
  const c10::cuda::CUDAGuard guard(xs.device());
  const cudaStream_t s = stream_of(xs);
  const at::Tensor x = xs.contiguous();
  const at::Tensor& bounds = cuda_tensor(p[5], "bounds");
  const int64_t hidden = xs.size(-1), inter = g->w.n, t = hidden > 0 ? x.numel() / hidden : 0;
  if (hidden != g->w.k) fail("forward_fp8_dense: input and weight shapes disagree");
  const at::ScalarType od = dtype_or(p[6], xs.scalar_type());
  Scratch sc;
  const int64_t xq = sc.add(t * hidden), xsc = sc.add(t * (hidden / 128) * 4), hq = sc.add(t * inter),
                hs = sc.add(t * (inter / 128) * 4);
  sc.alloc(x);
  at::Tensor y = out_like(xs, d->w.n, od);
  check(hq_fp8_quant_rows(x.data_ptr(), dt_code(x.scalar_type()), hidden, nullptr, t, hidden, sc.base + xq,
                          (float*)(sc.base + xsc), s),
        "hq_fp8_quant_rows");
  check(hq_moe_fp8_gate_up_forward(&g->w, &u->w, act, sc.base + xq, (const float*)(sc.base + xsc), t, 1,
                                   bounds.data_ptr<int32_t>(), sc.base + hq, (float*)(sc.base + hs), g->status_ptr(), s),
        "hq_moe_fp8_gate_up_forward(shared)");
  check(hq_fp8_linear_forward(&d->w, sc.base + hq, (const float*)(sc.base + hs), t, y.data_ptr(), dt_code(od), d->w.n,
                              g->status_ptr(), s),
        "hq_fp8_linear_forward(shared)");
  return THPVariable_Wrap(y);
  HQ_CATCH
}

// scratch(layer) -> the scratch tensors in use (one per stream)
PyObject* py_scratch(PyObject*, PyObject* h) {
  HQ_TRY
  const Layer* l = layer(h);
  PyObject* out = PyList_New(0);
  if (out == nullptr) return nullptr;
  for (const auto& kv : *l->scratch) {
    PyObject* t = THPVariable_Wrap(kv.second);
    if (t == nullptr || PyList_Append(out, t) != 0) {
      Py_XDECREF(t);
      Py_DECREF(out);
      return nullptr;
    }
    Py_DECREF(t);
  }
  return out;
  HQ_CATCH
}

PyObject* py_set_error(PyObject*, PyObject* cls) {
  Py_XDECREF(g_error);
  Py_INCREF(cls);
  g_error = cls;
  Py_RETURN_NONE;
}

#define HQ_FAST(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {HQ_FAST("layer", py_layer),         HQ_FAST("linear", py_linear),   HQ_FAST("qkv", py_qkv),
                           HQ_FAST("glu", py_glu),             HQ_FAST("router", py_router),   HQ_FAST("moe_layer", py_moe_layer),
                           HQ_FAST("moe_fp8", py_moe_fp8),     HQ_FAST("moe_mx", py_moe_mx),   HQ_FAST("fp8_dense", py_fp8_dense),
                           {"scratch", py_scratch, METH_O, nullptr},
                           {"set_error", py_set_error, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_hqtorch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hqtorch() {
  LayerType.tp_dealloc = layer_dealloc;
  LayerType.tp_flags = Py_TPFLAGS_DEFAULT;
  if (PyType_Ready(&LayerType) < 0) return nullptr;
  g_names = {PyUnicode_InternFromString("top_k"),       PyUnicode_InternFromString("score_function"),
             PyUnicode_InternFromString("selected_weight"), PyUnicode_InternFromString("renormalize"),
             PyUnicode_InternFromString("norm_min"),    PyUnicode_InternFromString("output_scale"),
             PyUnicode_InternFromString("logit_clip")};
  return PyModule_Create(&g_module);
}
