// Python module `_host`: the host path of one call (output and scratch allocation, strides, current
// stream, device guard, the C ABI calls) in native code.
//
// Through ctypes and torch's Python front end that path took 45 us of a forward call and 130 us of a
// backward call, more than the kernels of a short sequence.  The functions here do the same steps in the
// same order on the same tensors and keep nothing between calls.  Plain CPython entry points with
// torch's own exception translation (an out-of-memory error arrives as torch.OutOfMemoryError); the
// interpreter lock is released around allocations and launches, as ctypes does around a call.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include "../../include/fa2_b200.h"

namespace {

// A [B, H, N, D] tensor the kernels can read through its own strides: unit last stride, 16-byte
// aligned base, batch / head / row strides that are positive multiples of 8 elements (those of
// size-1 dimensions do not matter), rows that do not overlap.
bool readable_in_place(const at::Tensor& t) {
  if (t.stride(3) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
  for (int i = 0; i < 3; ++i)
    if (t.size(i) > 1 && (t.stride(i) <= 0 || t.stride(i) % 8)) return false;
  return t.size(2) == 1 || t.stride(2) >= t.size(3);
}
at::Tensor kernel_input(const at::Tensor& t) { return readable_in_place(t) ? t : t.contiguous(); }

template <size_t N>
struct StrideArray {
  long long v[3 * N];
  explicit StrideArray(const std::array<const at::Tensor*, N>& ts) {
    for (size_t i = 0; i < N; ++i)
      for (int d = 0; d < 3; ++d) v[3 * i + d] = ts[i]->stride(d);
  }
};

int dtype_code(const at::Tensor& t) { return t.scalar_type() == at::kHalf ? FA2_DTYPE_FP16 : FA2_DTYPE_BF16; }

bool tensors(PyObject* const* args, int n) {
  for (int i = 0; i < n; ++i)
    if (!THPVariable_Check(args[i]) || THPVariable_Unpack(args[i]).dim() < 3) {
      PyErr_Format(PyExc_TypeError, "argument %d must be a [B, H, N, ..] tensor", i);
      return false;
    }
  return true;
}

// forward(q, k, v, scale, f32) -> (code, output, lse, fp32 output or None).  Shapes, devices and
// dtypes are the caller's business; a non-zero code is that of fa2_fwd_strided / fa2_fwd_strided_f32.
PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) return PyErr_Format(PyExc_TypeError, "forward takes 5 arguments");
  if (!tensors(args, 3)) return nullptr;
  const double scale = PyFloat_AsDouble(args[3]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  const bool f32 = args[4] == Py_True;
  at::Tensor q = THPVariable_Unpack(args[0]), k = THPVariable_Unpack(args[1]), v = THPVariable_Unpack(args[2]);
  at::Tensor output, lse, output32;
  int code;
  {
    pybind11::gil_scoped_release no_gil;
    q = kernel_input(q), k = kernel_input(k), v = kernel_input(v);
    output = at::empty(q.sizes(), q.options().memory_format(at::MemoryFormat::Contiguous));
    lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
    const c10::cuda::CUDAGuard guard(q.device());
    if (f32) output32 = at::empty(q.sizes(), output.options().dtype(at::kFloat));
    const StrideArray<5> strides({&q, &k, &v, &output, f32 ? &output32 : &output});
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    const int b = q.size(0), h = q.size(1), n = q.size(2), nk = k.size(2), d = q.size(3);
    code = f32 ? fa2_fwd_strided_f32(q.data_ptr(), k.data_ptr(), v.data_ptr(), output.data_ptr(),
                                     output32.data_ptr<float>(), lse.data_ptr<float>(), b, h, n, nk, d,
                                     dtype_code(q), static_cast<float>(scale), strides.v, stream)
               : fa2_fwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), output.data_ptr(),
                                 lse.data_ptr<float>(), b, h, n, nk, d, dtype_code(q),
                                 static_cast<float>(scale), strides.v, stream);
  }
  return Py_BuildValue("iNNN", code, THPVariable_Wrap(output), THPVariable_Wrap(lse), THPVariable_Wrap(output32));
  END_HANDLE_TH_ERRORS
}

// preprocess(output, d_output, lse) -> (code, rowstats, d_output as the kernels read it)
PyObject* preprocess(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3) return PyErr_Format(PyExc_TypeError, "preprocess takes 3 arguments");
  if (!tensors(args, 3)) return nullptr;
  const at::Tensor output = THPVariable_Unpack(args[0]), lse = THPVariable_Unpack(args[2]);
  at::Tensor d_output = THPVariable_Unpack(args[1]), rowstats;
  int code;
  {
    pybind11::gil_scoped_release no_gil;
    d_output = kernel_input(d_output);
    const int b = output.size(0), h = output.size(1), n = output.size(2);
    rowstats = at::empty({static_cast<int64_t>(fa2_rowstats_bytes(b, h, n) / 4)}, lse.options());
    const c10::cuda::CUDAGuard guard(output.device());
    const StrideArray<2> strides({&output, &d_output});
    code = fa2_bwd_preprocess_strided(output.data_ptr(), d_output.data_ptr(), lse.data_ptr<float>(),
                                      rowstats.data_ptr<float>(), b, h, n, output.size(3), dtype_code(output),
                                      strides.v,
                                      c10::cuda::getCurrentCUDAStream(output.device().index()).stream());
  }
  return Py_BuildValue("iNN", code, THPVariable_Wrap(rowstats), THPVariable_Wrap(d_output));
  END_HANDLE_TH_ERRORS
}

// gradients(q, k, v, f32) -> dense uninitialised (dq, dk, dv), fp32 or in the dtype of q, k, v
PyObject* gradients(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4) return PyErr_Format(PyExc_TypeError, "gradients takes 4 arguments");
  if (!tensors(args, 3)) return nullptr;
  at::Tensor d[3];
  for (int i = 0; i < 3; ++i) {
    const at::Tensor& t = THPVariable_Unpack(args[i]);
    const auto options = t.options().memory_format(at::MemoryFormat::Contiguous);
    d[i] = at::empty(t.sizes(), args[3] == Py_True ? options.dtype(at::kFloat) : options);
  }
  return Py_BuildValue("NNN", THPVariable_Wrap(d[0]), THPVariable_Wrap(d[1]), THPVariable_Wrap(d[2]));
  END_HANDLE_TH_ERRORS
}

// backward(q, k, v, d_output, dq, dk, dv, rowstats, workspace or None, scale, mode) -> code; dq, dk
// and dv all in the dtype of q, or all fp32
PyObject* backward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 11) return PyErr_Format(PyExc_TypeError, "backward takes 11 arguments");
  if (!tensors(args, 7)) return nullptr;
  if (!THPVariable_Check(args[7]) || !(args[8] == Py_None || THPVariable_Check(args[8])))
    return PyErr_Format(PyExc_TypeError, "rowstats and workspace must be tensors");
  const double scale = PyFloat_AsDouble(args[9]);
  const long mode = PyLong_AsLong(args[10]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor t[7];
  for (int i = 0; i < 7; ++i) t[i] = THPVariable_Unpack(args[i]);
  const at::Tensor rowstats = THPVariable_Unpack(args[7]);
  const at::Tensor workspace = args[8] == Py_None ? at::Tensor() : THPVariable_Unpack(args[8]);
  const bool f32 = t[4].scalar_type() == at::kFloat;
  for (int i = 4; i < 7; ++i)
    if (t[i].scalar_type() != (f32 ? at::kFloat : t[0].scalar_type()))
      return PyErr_Format(PyExc_TypeError, "dq, dk and dv must be all fp32 or all of the dtype of q");
  int code;
  {
    pybind11::gil_scoped_release no_gil;
    for (int i = 0; i < 4; ++i) t[i] = kernel_input(t[i]);
    const at::Tensor& q = t[0];
    const c10::cuda::CUDAGuard guard(q.device());
    const StrideArray<7> strides({&t[0], &t[1], &t[2], &t[3], &t[4], &t[5], &t[6]});
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    void* ws = workspace.defined() ? workspace.data_ptr() : nullptr;
    const size_t ws_bytes = workspace.defined() ? workspace.nbytes() : 0;
    const int b = q.size(0), h = q.size(1), n = q.size(2), nk = t[1].size(2), d = q.size(3);
    code = f32 ? fa2_bwd_strided_f32(q.data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                                     rowstats.data_ptr<float>(), t[4].data_ptr<float>(), t[5].data_ptr<float>(),
                                     t[6].data_ptr<float>(), ws, ws_bytes, b, h, n, nk, d, dtype_code(q),
                                     static_cast<float>(scale), static_cast<int>(mode), strides.v, stream)
               : fa2_bwd_strided(q.data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                                 rowstats.data_ptr<float>(), t[4].data_ptr(), t[5].data_ptr(), t[6].data_ptr(),
                                 ws, ws_bytes, b, h, n, nk, d, dtype_code(q), static_cast<float>(scale),
                                 static_cast<int>(mode), strides.v, stream);
  }
  return PyLong_FromLong(code);
  END_HANDLE_TH_ERRORS
}

PyObject* is_readable_in_place(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  if (!THPVariable_Check(arg) || THPVariable_Unpack(arg).dim() != 4)
    return PyErr_Format(PyExc_TypeError, "expected a [B, H, N, D] tensor");
  return PyBool_FromLong(readable_in_place(THPVariable_Unpack(arg)));
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(forward)), METH_FASTCALL, nullptr},
    {"preprocess", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(preprocess)), METH_FASTCALL, nullptr},
    {"gradients", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(gradients)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(backward)), METH_FASTCALL, nullptr},
    {"readable_in_place", is_readable_in_place, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
