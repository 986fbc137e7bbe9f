// Native call path of the Python entry points on CUDA tensors: lib/_ft_torch.so.
//
// A small reduction is bound by the host: walking the tensors through Python attributes, building a ctypes
// array, the device guard and the stream lookup took 15 us around a kernel of 2 us.  Here the same checks read
// the tensors' C++ objects and the library is called directly: 18.4 -> 6.9 us per call for four fp32 vectors of
// 4099 elements, launches back to back (two launches then; with one, 3.0 us, of which everything here is 0.3 and
// the launch the rest; a new result tensor adds 0.8).
//
// Every function answers one of
//   a tensor (or None where the caller has the result already)   done;
//   an int                                                       the library's status, the call failed;
//   NotImplemented                                               anything out of the ordinary (CPU tensors, tensor
//       subclasses, mixed types or sizes, ...): the caller's Python path checks it and reports it in words.
// A C++ exception (a tensor without memory inside vmap, a dispatch mode that raises, ...) becomes the Python exception
// it would be in torch: guarded() stands between every function and the interpreter.
//
// libflextree.so is not linked: its entry points arrive as addresses through bind(), so that the checked
// build (FT_LIB=bounds) and the normal one share this module.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cstring>
#include <exception>
#include <optional>

#include "../api/ft_types.h"

namespace {

int (*p_reduce_nway)(int, int, const void* const*, void*, int, size_t, int, void*) = nullptr;
int (*p_reduce_nway_scaled)(int, int, const void* const*, void*, int, size_t, float, void*) = nullptr;

int (*p_local_world_run)(void* const*, int, const void* const*, void* const*, size_t, int, int, const int*, int, int, int, int, int, float, void*) = nullptr;

int (*p_host_pipe_reduce)(void*, int, int, const void* const*, int, const int*, void* const*, int, size_t, void*) = nullptr;

PyObject* other() { Py_RETURN_NOTIMPLEMENTED; }

int dtype_of(at::ScalarType t) {
  switch (t) {
    case at::kByte: return FT_U8;
    case at::kChar: return FT_I8;
    case at::kShort: return FT_I16;
    case at::kInt: return FT_I32;
    case at::kLong: return FT_I64;
    case at::kFloat: return FT_F32;
    case at::kDouble: return FT_F64;
    case at::kBool: return FT_BOOL;
    case at::kBFloat16: return FT_BF16;
    case at::kHalf: return FT_F16;
    default: return -1;
  }
}

int op_of(PyObject* o) {
  const char* s = PyUnicode_Check(o) ? PyUnicode_AsUTF8(o) : nullptr;
  if (!s) { PyErr_Clear(); return -1; }
  return !std::strcmp(s, "sum") ? FT_SUM : !std::strcmp(s, "band") ? FT_BAND : -1;
}

// A plain, contiguous tensor; null for anything else.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.layout() == at::kStrided && t.is_contiguous() ? &t : nullptr;
}
// ... on a CUDA device.
const at::Tensor* plain_cuda(PyObject* o) {
  const at::Tensor* t = plain(o);
  return t && t->is_cuda() ? t : nullptr;
}

// References to the tensors of a call.  The calls give up the GIL, and the caller's lists are only borrowed: a thread that
// changes one in the meantime would otherwise free the tensors whose memory the call is about to use.  Destroyed with
// the GIL held.
struct Kept {
  PyObject* o[2 * FT_MAX_FANIN];
  int n = 0;
  Kept() = default;
  Kept(const Kept&) = delete;
  Kept& operator=(const Kept&) = delete;
  ~Kept() { while (n) Py_DECREF(o[--n]); }
  void add(PyObject* p) { Py_INCREF(p); o[n++] = p; }
};

// n tensors that share type, size and device.  Returns n, or 0.
int gather_inputs(PyObject* seq, const void** src, const at::Tensor** first, Kept* kept) {
  const bool list = PyList_CheckExact(seq);
  if (!list && !PyTuple_CheckExact(seq)) return 0;
  const Py_ssize_t n = list ? PyList_GET_SIZE(seq) : PyTuple_GET_SIZE(seq);
  if (n < 1 || n > FT_MAX_FANIN) return 0;
  for (Py_ssize_t k = 0; k < n; ++k) {
    PyObject* o = list ? PyList_GET_ITEM(seq, k) : PyTuple_GET_ITEM(seq, k);
    const at::Tensor* t = plain_cuda(o);
    if (!t) return 0;
    kept->add(o);
    if (k == 0) *first = t;
    else if (t->scalar_type() != (*first)->scalar_type() || t->numel() != (*first)->numel() || t->device() != (*first)->device()) return 0;
    src[k] = t->const_data_ptr();
  }
  return (int)n;
}

PyObject* answer(int code, PyObject* out, std::optional<at::Tensor>& made) {
  if (code) return PyLong_FromLong(code);
  if (made) return THPVariable_Wrap(std::move(*made));
  Py_INCREF(out);
  return out;
}

// reduce_nway(tensors, op, out | None, variant)
PyObject* reduce_nway(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4 || !p_reduce_nway) return other();
  const void* src[FT_MAX_FANIN];
  const at::Tensor* t0 = nullptr;
  Kept kept;   // (args[] themselves are held by the caller's frame)
  const int n = gather_inputs(args[0], src, &t0, &kept);
  const int op = op_of(args[1]);
  if (!n || op < 0 || !PyLong_CheckExact(args[3])) return other();
  const int dt = dtype_of(t0->scalar_type());
  const long variant = PyLong_AsLong(args[3]);
  if (dt < 0 || (variant == -1 && PyErr_Occurred())) { PyErr_Clear(); return other(); }
  const at::Tensor* dst = nullptr;
  if (args[2] != Py_None) {
    dst = plain_cuda(args[2]);
    if (!dst || dst->scalar_type() != t0->scalar_type() || dst->numel() != t0->numel() || dst->device() != t0->device()) return other();
  }
  std::optional<at::Tensor> made;
  int code = 0;
  Py_BEGIN_ALLOW_THREADS
  try {
    c10::cuda::CUDAGuard guard(t0->device());
    if (!dst) made.emplace(at::detail::empty_cuda(t0->sizes(), t0->scalar_type(), t0->device(), std::nullopt));
    void* out = dst ? dst->mutable_data_ptr() : made->mutable_data_ptr();
    code = p_reduce_nway(op, dt, src, out, n, (size_t)t0->numel(), (int)variant, c10::cuda::getCurrentCUDAStream(t0->device().index()).stream());
  } catch (...) {
    code = -1;   // e.g. out of memory: the Python path asks again and raises what torch raises
  }
  Py_END_ALLOW_THREADS
  if (code < 0) return other();
  return answer(code, args[2], made);
}

// reduce_nway_scaled(tensors, scale, out_dtype | None, out | None)
PyObject* reduce_nway_scaled(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4 || !p_reduce_nway_scaled) return other();
  const void* src[FT_MAX_FANIN];
  const at::Tensor* t0 = nullptr;
  Kept kept;   // (args[] themselves are held by the caller's frame)
  const int n = gather_inputs(args[0], src, &t0, &kept);
  if (!n || !PyFloat_CheckExact(args[1])) return other();
  const float scale = (float)PyFloat_AS_DOUBLE(args[1]);
  const at::Tensor* dst = nullptr;
  at::ScalarType to = t0->scalar_type();
  if (args[3] != Py_None) {
    dst = plain_cuda(args[3]);
    if (!dst || dst->numel() != t0->numel() || dst->device() != t0->device()) return other();
    to = dst->scalar_type();
  } else if (args[2] != Py_None) {
    if (!THPDtype_Check(args[2])) return other();
    to = reinterpret_cast<THPDtype*>(args[2])->scalar_type;
  }
  const int in_dt = dtype_of(t0->scalar_type()), out_dt = dtype_of(to);
  if ((in_dt != FT_F32 && in_dt != FT_BF16) || (out_dt != FT_F32 && out_dt != FT_BF16)) return other();
  std::optional<at::Tensor> made;
  int code = 0;
  Py_BEGIN_ALLOW_THREADS
  try {
    c10::cuda::CUDAGuard guard(t0->device());
    if (!dst) made.emplace(at::detail::empty_cuda(t0->sizes(), to, t0->device(), std::nullopt));
    void* out = dst ? dst->mutable_data_ptr() : made->mutable_data_ptr();
    code = p_reduce_nway_scaled(in_dt, out_dt, src, out, n, (size_t)t0->numel(), scale, c10::cuda::getCurrentCUDAStream(t0->device().index()).stream());
  } catch (...) {
    code = -1;
  }
  Py_END_ALLOW_THREADS
  if (code < 0) return other();
  return answer(code, args[3], made);
}

// local_world_run(handles, tensors, outs, op, widths, lonely, ring, algo, phase, scale): `handles` is a list
// and `widths` a tuple of ints.  None when done; outs is tensors for a call in place.
PyObject* local_world_run(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 10 || !p_local_world_run || !PyList_CheckExact(args[0]) || !PyTuple_CheckExact(args[4])) return other();
  const Py_ssize_t n = PyList_GET_SIZE(args[0]), nw = PyTuple_GET_SIZE(args[4]);
  void* handles[FT_MAX_FANIN];
  int widths[FT_MAX_FANIN];
  const void *in[FT_MAX_FANIN], *res[FT_MAX_FANIN];
  const at::Tensor *t0 = nullptr, *o0 = nullptr;
  Kept kept;
  if (n < 1 || n > FT_MAX_FANIN || nw > FT_MAX_FANIN) return other();   // no handles: a closed world
  if (gather_inputs(args[1], in, &t0, &kept) != n) return other();
  if (args[2] == args[1]) {
    std::memcpy(res, in, sizeof(void*) * n);
    o0 = t0;
  } else if (gather_inputs(args[2], res, &o0, &kept) != n) {
    return other();
  }
  if (o0->scalar_type() != t0->scalar_type() || o0->numel() != t0->numel() || o0->device() != t0->device()) return other();
  for (Py_ssize_t k = 0; k < n; ++k) handles[k] = PyLong_AsVoidPtr(PyList_GET_ITEM(args[0], k));
  for (Py_ssize_t k = 0; k < nw; ++k) widths[k] = (int)PyLong_AsLong(PyTuple_GET_ITEM(args[4], k));
  const int op = op_of(args[3]), dt = dtype_of(t0->scalar_type());
  const int lonely = (int)PyLong_AsLong(args[5]), ring = (int)PyLong_AsLong(args[6]), algo = (int)PyLong_AsLong(args[7]);
  const int phase = (int)PyLong_AsLong(args[8]);
  const double scale = PyFloat_AsDouble(args[9]);
  if (op < 0 || dt < 0 || PyErr_Occurred()) { PyErr_Clear(); return other(); }
  int code = 0;
  Py_BEGIN_ALLOW_THREADS
  try {
    c10::cuda::CUDAGuard guard(t0->device());
    code = p_local_world_run(handles, (int)n, in, const_cast<void* const*>(res), (size_t)t0->numel(), dt, op, widths, (int)nw, lonely, ring, algo,
                             phase, (float)scale, c10::cuda::getCurrentCUDAStream(t0->device().index()).stream());
  } catch (...) {
    code = FT_ERR_NOT_AVAILABLE;
  }
  Py_END_ALLOW_THREADS
  if (code == FT_ERR_NOT_AVAILABLE) return other();
  if (code) return PyLong_FromLong(code);
  Py_RETURN_NONE;
}

// Plain, contiguous CPU tensors that share type and size with *first (set by the first one).  Returns their number, or 0.
int gather_host(PyObject* seq, const void** ptr, const at::Tensor** first, Kept* kept) {
  const bool list = PyList_CheckExact(seq);
  if (!list && !PyTuple_CheckExact(seq)) return 0;
  const Py_ssize_t n = list ? PyList_GET_SIZE(seq) : PyTuple_GET_SIZE(seq);
  if (n < 1 || n > FT_MAX_FANIN) return 0;
  for (Py_ssize_t k = 0; k < n; ++k) {
    PyObject* o = list ? PyList_GET_ITEM(seq, k) : PyTuple_GET_ITEM(seq, k);
    const at::Tensor* t = plain(o);
    if (!t || !t->is_cpu()) return 0;
    kept->add(o);
    if (!*first) *first = t;
    else if (t->scalar_type() != (*first)->scalar_type() || t->numel() != (*first)->numel()) return 0;
    ptr[k] = t->const_data_ptr();
  }
  return (int)n;
}

// host_pipe_run(pipeline, device, inputs, fanins, outs, op): on the current stream of `device`.  None when done.
PyObject* host_pipe_run(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 6 || !p_host_pipe_reduce || !PyList_CheckExact(args[3])) return other();
  const void *src[FT_MAX_FANIN], *dst[FT_MAX_FANIN];
  int fanin[FT_MAX_FANIN];
  const at::Tensor* t0 = nullptr;
  Kept kept;
  const int n_in = gather_host(args[2], src, &t0, &kept), n_out = n_in ? gather_host(args[4], dst, &t0, &kept) : 0;
  if (!n_out || PyList_GET_SIZE(args[3]) != n_out) return other();
  for (int j = 0; j < n_out; ++j) fanin[j] = (int)PyLong_AsLong(PyList_GET_ITEM(args[3], j));
  void* pipe = PyLong_AsVoidPtr(args[0]);
  const long device = PyLong_AsLong(args[1]);
  const int op = op_of(args[5]), dt = dtype_of(t0->scalar_type());
  if (!pipe || op < 0 || dt < 0 || PyErr_Occurred()) { PyErr_Clear(); return other(); }
  int code = 0;
  Py_BEGIN_ALLOW_THREADS
  try {
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
    code = p_host_pipe_reduce(pipe, op, dt, src, n_in, fanin, const_cast<void* const*>(dst), n_out, (size_t)t0->numel(),
                              c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream());
  } catch (...) {
    code = -1;
  }
  Py_END_ALLOW_THREADS
  if (code < 0) return other();
  if (code) return PyLong_FromLong(code);
  Py_RETURN_NONE;
}

// narrow_all(tensors, ranges): for each tensor the list of its flat [lo, hi) views; ranges[k] is a tuple of (lo, hi).
PyObject* narrow_all(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2 || !PyList_CheckExact(args[0]) || !PyTuple_CheckExact(args[1])) return other();
  const Py_ssize_t n = PyList_GET_SIZE(args[0]);
  if (n < 1 || PyTuple_GET_SIZE(args[1]) != n) return other();
  THPObjectPtr all(PyList_New(n));
  if (!all) return nullptr;
  int64_t numel = -1;   // one size for all, as the ranges are
  for (Py_ssize_t k = 0; k < n; ++k) {
    // looked up for each tensor: a dispatch mode runs Python code below, which may change the list
    const at::Tensor* p = k < PyList_GET_SIZE(args[0]) ? plain(PyList_GET_ITEM(args[0], k)) : nullptr;
    PyObject* ranges = PyTuple_GET_ITEM(args[1], k);
    if (!p || !PyTuple_CheckExact(ranges)) return other();
    const at::Tensor t = *p;
    if (k == 0) numel = t.numel();
    else if (t.numel() != numel) return other();
    // nothing to record for a tensor without a gradient: past the autograd layer, but not past the one that makes it a view
    std::optional<at::AutoDispatchBelowAutograd> below;
    if (!t.requires_grad() && !t._fw_grad(0).defined()) below.emplace();
    PyObject* mine = PyList_New(PyTuple_GET_SIZE(ranges));
    if (!mine) return nullptr;
    PyList_SET_ITEM(all.get(), k, mine);
    for (Py_ssize_t j = 0; j < PyTuple_GET_SIZE(ranges); ++j) {
      PyObject* range = PyTuple_GET_ITEM(ranges, j);
      if (!PyTuple_CheckExact(range) || PyTuple_GET_SIZE(range) != 2) return other();
      const int64_t lo = PyLong_AsLongLong(PyTuple_GET_ITEM(range, 0)), hi = PyLong_AsLongLong(PyTuple_GET_ITEM(range, 1));
      if (PyErr_Occurred()) return nullptr;
      if (lo < 0 || hi < lo || hi > numel) return other();
      PyObject* view = THPVariable_Wrap(t.as_strided({hi - lo}, {1}, t.storage_offset() + lo));
      if (!view) return nullptr;
      PyList_SET_ITEM(mine, j, view);
    }
  }
  return all.release();
}

// bind({name: address}): entry points of the libflextree build this process uses.
PyObject* bind(PyObject*, PyObject* d) {
  if (!PyDict_Check(d)) { PyErr_SetString(PyExc_TypeError, "bind() takes a dict"); return nullptr; }
  auto get = [&](const char* name, auto& fn) {
    PyObject* v = PyDict_GetItemString(d, name);
    if (!v) { PyErr_Format(PyExc_KeyError, "%s", name); return false; }
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(PyLong_AsVoidPtr(v));
    return !PyErr_Occurred();
  };
  if (!get("ft_reduce_nway", p_reduce_nway) || !get("ft_reduce_nway_scaled", p_reduce_nway_scaled) ||
      !get("ft_local_world_run", p_local_world_run) || !get("ft_host_pipe_reduce", p_host_pipe_reduce))
    return nullptr;
  Py_RETURN_NONE;
}

// No C++ exception may leave through the interpreter's C frames.  (Torch's own wrapper for this also collects warnings,
// which costs a call 15 to 20 ns; nothing here warns.)
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
  try {
    return F(self, args, nargs);
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
constexpr PyMethodDef method(const char* name, const char* doc) {
  return {name, (PyCFunction)(void (*)(void))guarded<F>, METH_FASTCALL, doc};
}

PyMethodDef methods[] = {
    {"bind", bind, METH_O, "bind({name: address})"},
    method<reduce_nway>("reduce_nway", "reduce_nway(tensors, op, out, variant)"),
    method<reduce_nway_scaled>("reduce_nway_scaled", "reduce_nway_scaled(tensors, scale, out_dtype, out)"),
    method<local_world_run>("local_world_run", "local_world_run(handles, tensors, outs, op, widths, lonely, ring, algo, phase, scale)"),
    method<host_pipe_run>("host_pipe_run", "host_pipe_run(pipeline, device, inputs, fanins, outs, op)"),
    method<narrow_all>("narrow_all", "narrow_all(tensors, ranges)"),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ft_torch", "native call path of the Python entry points", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__ft_torch(void) { return PyModule_Create(&module); }
