// Native host path of the Python package: torch tensors -> FhobProblem -> libfhob.so, and the
// autograd functions of fhob.attention.
//
// A call of a small problem is bound by what the host does before the launches.  Measured for
// flash_bwdbwd (fp32, 2 heads, N = 256): 79 us a call with the checks, the strides and the struct
// in Python and ctypes; the fields of a tensor alone cost about 100 ns each there.
//
// Everything here serves well-formed calls on CUDA tensors.  A function returns None for any other
// call (a check that fails, host tensors, a view that cannot be read in place, a stream that is
// being captured, an error from the library), and the caller then takes the Python path, which
// makes copies where they help and otherwise raises the error.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include "../../include/fhob.h"

namespace {

using at::Tensor;

PyObject* g_workspaces = nullptr;   // the package's dict (device, stream) -> workspace tensor

struct Mask {
  bool causal;
  int64_t window;   // 0 = none
};

// Index order of FhobLayout.
enum { kQ = 0, kK, kV, kO, kDO, kDDQ, kDDK, kDDV, kTensors };

struct Call {
  FhobProblem p;
  FhobLayout lay;
  int device = -1;
  cudaStream_t stream = nullptr;
};

bool is_tc_capable(at::ScalarType t, int64_t d, int64_t dv) {
  if (t == at::kFloat) return d <= 64 && dv <= 64 && d % 4 == 0 && dv % 4 == 0;
  return d <= 128 && dv <= 128 && d % 8 == 0 && dv % 8 == 0;
}

// Fills the problem from up to eight matrices (NULL = not part of this call).  False: not a call for this path.
bool fill(Call& c, const Tensor* const (&t)[kTensors], double scale, const Mask& m, int impl) {
  const Tensor& q = *t[kQ];
  if (!q.is_cuda() || impl < 0) return false;
  const auto dtype = q.scalar_type();
  const int ft = dtype == at::kBFloat16 ? FHOB_BF16 : dtype == at::kHalf ? FHOB_F16 : dtype == at::kFloat ? FHOB_F32 : -1;
  if (ft < 0) return false;
  const int dim = static_cast<int>(q.dim());
  if (dim != 3 && dim != 4) return false;
  const auto device = q.device();
  const int64_t batches = dim == 4 ? q.size(0) : 1, heads = dim == 4 ? q.size(1) : q.size(0), bh = batches * heads;
  const int64_t n_q = q.size(dim - 2), d = q.size(dim - 1);
  const Tensor& k = *t[kK];
  if (k.dim() < 3 || k.dim() > 4) return false;
  const int64_t n_k = k.size(k.dim() - 2), dv = t[kV] ? t[kV]->size(-1) : d;
  if (bh <= 0 || n_q <= 0 || n_k <= 0 || d <= 0 || dv <= 0) return false;
  if (bh > INT32_MAX || n_q > INT32_MAX || n_k > INT32_MAX || d > 128 || dv > 128) return false;
  const int64_t align = 16 / static_cast<int64_t>(q.element_size());
  if (d % align || dv % align) return false;
  bool contiguous = true;
  const void* ptr[kTensors];
  for (int i = 0; i < kTensors; ++i) {
    ptr[i] = nullptr;
    if (!t[i]) continue;
    const Tensor& x = *t[i];
    const int xd = static_cast<int>(x.dim());
    if ((xd != 3 && xd != 4) || x.scalar_type() != dtype || x.device() != device) return false;
    const int64_t xb = xd == 4 ? x.size(0) * x.size(1) : x.size(0);
    const bool q_side = i == kQ || i == kO || i == kDO || i == kDDQ, v_side = i == kV || i == kO || i == kDO || i == kDDV;
    if (xb != bh || x.size(xd - 2) != (q_side ? n_q : n_k) || x.size(xd - 1) != (v_side ? dv : d)) return false;
    contiguous = contiguous && x.is_contiguous();
    ptr[i] = x.const_data_ptr();
    if (reinterpret_cast<uintptr_t>(ptr[i]) & 15u) return false;
  }
  FhobProblem& p = c.p;
  memset(&p, 0, sizeof(p));
  p.bh = static_cast<int32_t>(bh); p.n_q = static_cast<int32_t>(n_q); p.n_k = static_cast<int32_t>(n_k);
  p.d = static_cast<int32_t>(d); p.d_v = dv == d ? 0 : static_cast<int32_t>(dv);
  p.dtype = ft; p.causal = m.causal ? 1 : 0; p.window = static_cast<int32_t>(m.window);
  p.impl = impl; p.scale = static_cast<float>(scale);
  p.q = ptr[kQ]; p.k = ptr[kK]; p.v = ptr[kV]; p.o = ptr[kO]; p.d_o = ptr[kDO];
  p.ddq = ptr[kDDQ]; p.ddk = ptr[kDDK]; p.ddv = ptr[kDDV];
  if (!contiguous) {
    // views are read in place through the tensor maps of the tensor-core kernels, if every stride
    // stays on the 16-byte grid
    if (impl == FHOB_IMPL_SIMT || !is_tc_capable(dtype, d, dv)) return false;
    memset(&c.lay, 0, sizeof(c.lay));
    c.lay.heads = static_cast<int32_t>(heads);
    for (int i = 0; i < kTensors; ++i) {
      if (!t[i]) continue;
      const Tensor& x = *t[i];
      const int xd = static_cast<int>(x.dim());
      if (x.size(xd - 1) > 1 && x.stride(xd - 1) != 1) return false;
      if (xd == 4 && (x.size(0) != batches || x.size(1) != heads)) return false;
      const int64_t head = x.stride(xd - 3), batch = xd == 4 ? x.stride(0) : head * heads;
      const int64_t row = x.size(xd - 2) == 1 ? x.size(xd - 1) : x.stride(xd - 2);   // a single row: any stride describes it
      if (row <= 0 || head < 0 || batch < 0 || row % align || head % align || batch % align) return false;
      c.lay.row[i] = row; c.lay.head[i] = head; c.lay.batch[i] = batch;
    }
    c.lay.lse_head = n_q;
    c.lay.lse_batch = heads * n_q;
    p.layout = &c.lay;
  }
  c.device = device.index();
  return true;
}

bool fill_lse(Call& c, const Tensor& lse) {
  if (!lse.is_cuda() || lse.get_device() != c.device || lse.scalar_type() != at::kFloat || !lse.is_contiguous()) return false;
  if (lse.dim() < 1 || lse.size(-1) != c.p.n_q || lse.numel() != static_cast<int64_t>(c.p.bh) * c.p.n_q) return false;
  c.p.lse = static_cast<const float*>(lse.const_data_ptr());
  return (reinterpret_cast<uintptr_t>(c.p.lse) & 15u) == 0;
}

// The stream and its workspace, from the dict the Python path uses too (needs the GIL).  Threads on one stream
// share it: the library queues the kernels of a call without another's between them.  Memory
// allocated while a stream is captured belongs to the graph: that is left to the Python path.
bool take_workspace(Call& c, Tensor& keep) {
  if (at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None) return false;
  c.stream = at::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(c.device)).stream();
  const size_t need = fhob_workspace_bytes_problem(&c.p);
  py::tuple key = py::make_tuple(c.device, reinterpret_cast<uintptr_t>(c.stream));
  PyObject* have = PyDict_GetItemWithError(g_workspaces, key.ptr());   // borrowed
  if (have && THPVariable_Check(have)) keep = THPVariable_Unpack(have);
  if (!keep.defined() || static_cast<size_t>(keep.numel()) < need) {
    PyErr_Clear();
    const int64_t bytes = static_cast<int64_t>(need > (1u << 20) ? need : (1u << 20));
    keep = at::empty({bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, c.device));
    py::object value = py::reinterpret_steal<py::object>(THPVariable_Wrap(keep));
    if (PyDict_SetItem(g_workspaces, key.ptr(), value.ptr()) != 0) throw py::error_already_set();
  }
  c.p.workspace = keep.data_ptr();
  c.p.workspace_bytes = static_cast<size_t>(keep.numel());
  return true;
}

Tensor empty_like_shape(const Tensor& t) {   // contiguous, same shape, type and device
  return at::detail::empty_cuda(t.sizes(), t.scalar_type(), t.device(), std::nullopt);
}

// Runs `launch` with the call's device current and without the GIL; false on an error (the Python
// path then repeats the call and raises).
template <class F>
bool launched(const Call& c, F&& launch) {
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != c.device) guard.set_index(static_cast<c10::DeviceIndex>(c.device));
  py::gil_scoped_release nogil;
  return launch() == FHOB_OK;
}

// ---- the three operators (with the GIL held); false = not for this path

bool run_bwdbwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor* o, const Tensor& d_o, const Tensor& ddq,
                const Tensor& ddk, const Tensor& ddv, const Tensor& lse, double scale, const Mask& m, int impl,
                Tensor (&out)[4]) {
  Call c;
  Tensor ws;
  if (!fill(c, {&q, &k, &v, o, &d_o, &ddq, &ddk, &ddv}, scale, m, impl) || !fill_lse(c, lse)) return false;
  if (!take_workspace(c, ws)) return false;
  const Tensor* like[4] = {&q, &k, &v, &d_o};
  for (int i = 0; i < 4; ++i) out[i] = empty_like_shape(*like[i]);
  c.p.dq2 = out[0].data_ptr(); c.p.dk2 = out[1].data_ptr(); c.p.dv2 = out[2].data_ptr(); c.p.ddo = out[3].data_ptr();
  return launched(c, [&] { return fhob_bwdbwd(&c.p, c.stream); });
}

bool run_forward(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const Mask& m, int impl, bool need_o,
                 Tensor& o, Tensor& lse) {
  Call c;
  Tensor ws;
  if (!fill(c, {&q, &k, &v, nullptr, nullptr, nullptr, nullptr, nullptr}, scale, m, impl)) return false;
  if (!take_workspace(c, ws)) return false;
  at::DimVector shape(q.sizes().begin(), q.sizes().end());
  if (need_o) {
    shape.back() = v.size(-1);
    o = at::detail::empty_cuda(shape, q.scalar_type(), q.device(), std::nullopt);
  }
  shape.pop_back();
  lse = at::detail::empty_cuda(shape, at::kFloat, q.device(), std::nullopt);
  return launched(c, [&] { return fhob_forward(&c.p, need_o ? o.data_ptr() : nullptr, static_cast<float*>(lse.data_ptr()), c.stream); });
}

bool run_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& d_o, const Tensor& lse,
                  double scale, const Mask& m, int impl, Tensor (&out)[3]) {
  Call c;
  Tensor ws;
  if (!fill(c, {&q, &k, &v, &o, &d_o, nullptr, nullptr, nullptr}, scale, m, impl) || !fill_lse(c, lse)) return false;
  if (!take_workspace(c, ws)) return false;
  const Tensor* like[3] = {&q, &k, &v};
  for (int i = 0; i < 3; ++i) out[i] = empty_like_shape(*like[i]);
  return launched(c, [&] { return fhob_backward(&c.p, out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(), c.stream); });
}

// ---- fhob.attention: twice differentiable.  The derivative of the first backward is taken with O
// and L regarded as functions of q, k, v (jax.vjp(attn_bwd), jax_refs/flash_impl.py:408-417), so O
// enters it detached and no gradient flows into it.

py::object python_fn(const char* module, const char* name) { return py::module_::import(module).attr(name); }
py::dict mask_kwargs(const Mask& m) {
  py::dict kw;
  kw["is_causal"] = m.causal;
  kw["sliding_window"] = m.window ? py::cast(m.window) : py::object(py::none());
  return kw;
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct AttentionBackward : torch::autograd::Function<AttentionBackward> {
  static variable_list forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse, Tensor d_o,
                               double scale, bool causal, int64_t window) {
    ctx->save_for_backward({q, k, v, o, lse, d_o});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["window"] = window;
    const Mask m{causal, window};
    py::gil_scoped_acquire gil;
    Tensor g[3];
    if (run_backward(q, k, v, o, d_o, lse, scale, m, FHOB_IMPL_AUTO, g)) return {g[0], g[1], g[2]};
    return py::cast<std::vector<Tensor>>(python_fn("fhob.autograd", "attention_backward")(q, k, v, o, d_o, lse, scale, **mask_kwargs(m)));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const double scale = ctx->saved_data["scale"].toDouble();
    const Mask m{ctx->saved_data["causal"].toBool(), ctx->saved_data["window"].toInt()};
    py::gil_scoped_acquire gil;
    Tensor r[4];
    if (!run_bwdbwd(s[0], s[1], s[2], &s[3], s[5], g[0], g[1], g[2], s[4], scale, m, FHOB_IMPL_AUTO, r)) {
      const auto got = py::cast<std::vector<Tensor>>(python_fn("fhob.ops", "flash_bwdbwd")(
          s[0], s[1], s[2], s[3], s[5], g[0].contiguous(), g[1].contiguous(), g[2].contiguous(), s[4], scale, **mask_kwargs(m)));
      for (int i = 0; i < 4; ++i) r[i] = got[i];
    }
    return {r[0], r[1], r[2], Tensor(), Tensor(), r[3], Tensor(), Tensor(), Tensor()};
  }
};

struct Attention : torch::autograd::Function<Attention> {
  static Tensor forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, double scale, bool causal, int64_t window) {
    const Mask m{causal, window};
    Tensor o, lse;
    {
      py::gil_scoped_acquire gil;
      if (!run_forward(q, k, v, scale, m, FHOB_IMPL_AUTO, true, o, lse)) {
        const auto got = py::cast<std::vector<Tensor>>(python_fn("fhob.ops", "attention_forward")(q, k, v, scale, **mask_kwargs(m)));
        o = got[0];
        lse = got[1];
      }
    }
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["window"] = window;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const auto r = AttentionBackward::apply(s[0], s[1], s[2], s[3].detach(), s[4], g[0], ctx->saved_data["scale"].toDouble(),
                                            ctx->saved_data["causal"].toBool(), ctx->saved_data["window"].toInt());
    return {r[0], r[1], r[2], Tensor(), Tensor(), Tensor()};
  }
};

// ---- module functions (vector call, positional arguments)

const Tensor* tensor_arg(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// sliding_window: None, or a positive int together with a causal mask
bool mask_args(PyObject* causal, PyObject* window, Mask& m) {
  const int c = PyObject_IsTrue(causal);
  if (c < 0) { PyErr_Clear(); return false; }
  m.causal = c == 1;
  m.window = 0;
  if (window == Py_None) return true;
  if (!PyLong_CheckExact(window)) return false;
  int overflow = 0;
  const long long w = PyLong_AsLongLongAndOverflow(window, &overflow);
  if (overflow || w < 1 || w > INT32_MAX || !m.causal) return false;
  m.window = w;
  return true;
}

bool scale_arg(PyObject* o, double& scale) {
  scale = PyFloat_CheckExact(o) ? PyFloat_AS_DOUBLE(o) : PyFloat_AsDouble(o);
  if (scale == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}

int impl_arg(PyObject* o) {   // "auto", "simt", "tcgen05"; -1 = something else
  if (!PyUnicode_Check(o)) return -1;
  if (PyUnicode_CompareWithASCIIString(o, "auto") == 0) return FHOB_IMPL_AUTO;
  if (PyUnicode_CompareWithASCIIString(o, "simt") == 0) return FHOB_IMPL_SIMT;
  if (PyUnicode_CompareWithASCIIString(o, "tcgen05") == 0) return FHOB_IMPL_TCGEN05;
  return -1;
}

PyObject* wrapped(const Tensor* t, int n) {
  PyObject* r = PyTuple_New(n);
  for (int i = 0; r && i < n; ++i) PyTuple_SET_ITEM(r, i, THPVariable_Wrap(t[i]));
  return r;
}

// bwdbwd(Q, K, V, O, dO, ddQ, ddK, ddV, L, scale, is_causal, sliding_window, impl)
PyObject* py_bwdbwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Mask m;
  double scale;
  if (n != 13 || !mask_args(a[10], a[11], m) || !scale_arg(a[9], scale)) Py_RETURN_NONE;
  const Tensor* t[9];
  for (int i = 0; i < 9; ++i) {
    t[i] = tensor_arg(a[i]);
    if (!t[i] && !(i == kO && a[i] == Py_None)) Py_RETURN_NONE;
  }
  Tensor out[4];
  if (!run_bwdbwd(*t[0], *t[1], *t[2], t[3], *t[4], *t[5], *t[6], *t[7], *t[8], scale, m, impl_arg(a[12]), out)) Py_RETURN_NONE;
  return wrapped(out, 4);
  END_HANDLE_TH_ERRORS
}

// forward(Q, K, V, scale, is_causal, sliding_window, impl, need_o) -> (O, L) | (None, L)
PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Mask m;
  if (n != 8 || !mask_args(a[4], a[5], m)) Py_RETURN_NONE;
  const Tensor *q = tensor_arg(a[0]), *k = tensor_arg(a[1]), *v = tensor_arg(a[2]);
  if (!q || !k || !v || q->dim() < 1) Py_RETURN_NONE;
  double scale = 1.0 / std::sqrt(static_cast<double>(q->size(-1)));
  if (a[3] != Py_None && !scale_arg(a[3], scale)) Py_RETURN_NONE;
  const int need_o = PyObject_IsTrue(a[7]);
  Tensor r[2];
  if (!run_forward(*q, *k, *v, scale, m, impl_arg(a[6]), need_o == 1, r[0], r[1])) Py_RETURN_NONE;
  if (need_o == 1) return wrapped(r, 2);
  PyObject* out = PyTuple_New(2);
  Py_INCREF(Py_None);
  PyTuple_SET_ITEM(out, 0, Py_None);
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(r[1]));
  return out;
  END_HANDLE_TH_ERRORS
}

// backward(Q, K, V, O, dO, L, scale, is_causal, sliding_window, impl) -> (dQ, dK, dV)
PyObject* py_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Mask m;
  double scale;
  if (n != 10 || !mask_args(a[7], a[8], m) || !scale_arg(a[6], scale)) Py_RETURN_NONE;
  const Tensor* t[6];
  for (int i = 0; i < 6; ++i)
    if (!(t[i] = tensor_arg(a[i]))) Py_RETURN_NONE;
  Tensor out[3];
  if (!run_backward(*t[0], *t[1], *t[2], *t[3], *t[4], *t[5], scale, m, impl_arg(a[9]), out)) Py_RETURN_NONE;
  return wrapped(out, 3);
  END_HANDLE_TH_ERRORS
}

// attention(q, k, v, scale, is_causal, window): window 0 = none (validated by the caller)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n == 6, "attention takes 6 arguments");
  const Tensor* t[3];
  for (int i = 0; i < 3; ++i) {
    t[i] = tensor_arg(a[i]);
    TORCH_CHECK_TYPE(t[i], "q, k and v must be tensors");
  }
  const double scale = PyFloat_AsDouble(a[3]);
  const int causal = PyObject_IsTrue(a[4]);
  const long long window = PyLong_AsLongLong(a[5]);
  if (PyErr_Occurred()) return nullptr;
  Tensor o;
  try {
    pybind11::gil_scoped_release nogil;
    o = Attention::apply(*t[0], *t[1], *t[2], scale, causal == 1, static_cast<int64_t>(window));
  } catch (py::error_already_set& e) {   // from the Python path: keep its type
    e.restore();
    return nullptr;
  }
  return THPVariable_Wrap(o);
  END_HANDLE_TH_ERRORS
}

// use_workspaces(dict): where workspaces are kept between calls
PyObject* py_use_workspaces(PyObject*, PyObject* d) {
  if (!PyDict_Check(d)) {
    PyErr_SetString(PyExc_TypeError, "a dict is expected");
    return nullptr;
  }
  Py_INCREF(d);
  Py_XSETREF(g_workspaces, d);
  Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"bwdbwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bwdbwd)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_forward)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_backward)), METH_FASTCALL, nullptr},
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL, nullptr},
    {"use_workspaces", py_use_workspaces, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Native host path of fhob", -1, g_methods};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&g_module); }
