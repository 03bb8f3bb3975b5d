// Python module `_host`: the host path of one call (output and scratch allocation, strides, current
// stream, device guard, the C ABI calls) in native code.
//
// Through ctypes and torch's Python front end that path took 45 us of a forward call and 130 us of a
// backward call, more than the kernels of a short sequence.  The functions here do the same steps in the
// same order on the same tensors and keep nothing between calls.  `attention` is the whole call as a C++
// autograd function.  Plain CPython entry points with
// torch's own exception translation (an out-of-memory error arrives as torch.OutOfMemoryError); the
// interpreter lock is released around allocations and launches, as ctypes does around a call.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <exception>

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

struct Forward {
  int code;
  at::Tensor output, lse, output32;
};
// q, k and v are replaced by what the kernels read.
Forward run_forward(at::Tensor& q, at::Tensor& k, at::Tensor& v, double scale, bool f32) {
  Forward r;
  q = kernel_input(q), k = kernel_input(k), v = kernel_input(v);
  r.output = at::empty(q.sizes(), q.options().memory_format(at::MemoryFormat::Contiguous));
  r.lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
  const c10::cuda::CUDAGuard guard(q.device());
  if (f32) r.output32 = at::empty(q.sizes(), r.output.options().dtype(at::kFloat));
  const StrideArray<5> strides({&q, &k, &v, &r.output, f32 ? &r.output32 : &r.output});
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  const int b = q.size(0), h = q.size(1), n = q.size(2), nk = k.size(2), d = q.size(3);
  r.code = f32 ? fa2_fwd_strided_f32(q.data_ptr(), k.data_ptr(), v.data_ptr(), r.output.data_ptr(),
                                     r.output32.data_ptr<float>(), r.lse.data_ptr<float>(), b, h, n, nk, d,
                                     dtype_code(q), static_cast<float>(scale), strides.v, stream)
               : fa2_fwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), r.output.data_ptr(),
                                 r.lse.data_ptr<float>(), b, h, n, nk, d, dtype_code(q),
                                 static_cast<float>(scale), strides.v, stream);
  return r;
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
  Forward r;
  {
    pybind11::gil_scoped_release no_gil;
    r = run_forward(q, k, v, scale, f32);
  }
  return Py_BuildValue("iNNN", r.code, THPVariable_Wrap(r.output), THPVariable_Wrap(r.lse),
                       THPVariable_Wrap(r.output32));
  END_HANDLE_TH_ERRORS
}

// Launches the preprocess; d_output is replaced by what the kernels read.
int run_preprocess(const at::Tensor& output, at::Tensor& d_output, const at::Tensor& lse, at::Tensor& rowstats) {
  d_output = kernel_input(d_output);
  const int b = output.size(0), h = output.size(1), n = output.size(2);
  rowstats = at::empty({static_cast<int64_t>(fa2_rowstats_bytes(b, h, n) / 4)}, lse.options());
  const c10::cuda::CUDAGuard guard(output.device());
  const StrideArray<2> strides({&output, &d_output});
  return fa2_bwd_preprocess_strided(output.data_ptr(), d_output.data_ptr(), lse.data_ptr<float>(),
                                    rowstats.data_ptr<float>(), b, h, n, output.size(3), dtype_code(output),
                                    strides.v, c10::cuda::getCurrentCUDAStream(output.device().index()).stream());
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
    code = run_preprocess(output, d_output, lse, rowstats);
  }
  return Py_BuildValue("iNN", code, THPVariable_Wrap(rowstats), THPVariable_Wrap(d_output));
  END_HANDLE_TH_ERRORS
}

at::Tensor empty_gradient(const at::Tensor& t, bool f32) {
  const auto options = t.options().memory_format(at::MemoryFormat::Contiguous);
  return at::empty(t.sizes(), f32 ? options.dtype(at::kFloat) : options);
}

// gradients(q, k, v, f32) -> dense uninitialised (dq, dk, dv), fp32 or in the dtype of q, k, v
PyObject* gradients(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4) return PyErr_Format(PyExc_TypeError, "gradients takes 4 arguments");
  if (!tensors(args, 3)) return nullptr;
  at::Tensor d[3];
  for (int i = 0; i < 3; ++i) d[i] = empty_gradient(THPVariable_Unpack(args[i]), args[3] == Py_True);
  return Py_BuildValue("NNN", THPVariable_Wrap(d[0]), THPVariable_Wrap(d[1]), THPVariable_Wrap(d[2]));
  END_HANDLE_TH_ERRORS
}

// t = q, k, v, d_output, dq, dk, dv
int run_backward(at::Tensor (&t)[7], const at::Tensor& rowstats, const at::Tensor& workspace, double scale, int mode) {
  const bool f32 = t[4].scalar_type() == at::kFloat;
  for (int i = 0; i < 4; ++i) t[i] = kernel_input(t[i]);
  const at::Tensor& q = t[0];
  const c10::cuda::CUDAGuard guard(q.device());
  const StrideArray<7> strides({&t[0], &t[1], &t[2], &t[3], &t[4], &t[5], &t[6]});
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  void* ws = workspace.defined() ? workspace.data_ptr() : nullptr;
  const size_t ws_bytes = workspace.defined() ? workspace.nbytes() : 0;
  const int b = q.size(0), h = q.size(1), n = q.size(2), nk = t[1].size(2), d = q.size(3);
  return f32 ? fa2_bwd_strided_f32(q.data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                                   rowstats.data_ptr<float>(), t[4].data_ptr<float>(), t[5].data_ptr<float>(),
                                   t[6].data_ptr<float>(), ws, ws_bytes, b, h, n, nk, d, dtype_code(q),
                                   static_cast<float>(scale), mode, strides.v, stream)
             : fa2_bwd_strided(q.data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                               rowstats.data_ptr<float>(), t[4].data_ptr(), t[5].data_ptr(), t[6].data_ptr(),
                               ws, ws_bytes, b, h, n, nk, d, dtype_code(q), static_cast<float>(scale), mode,
                               strides.v, stream);
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
    code = run_backward(t, rowstats, workspace, scale, static_cast<int>(mode));
  }
  return PyLong_FromLong(code);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------------------
// The whole call as a C++ autograd function: FlashAttentionV2Function of api.py without the interpreter in
// forward and backward, for plain CUDA tensors of one of the kernels' dtypes or fp32 (`eligible`); whatever else
// the entry point takes goes through the Python function.  [2,4,256,64] fp16, microseconds a pass on the host:
// forward and backward 112 -> 76 (52 of them torch's engine and an empty function), forward alone 17.6 -> 7.3.
// ---------------------------------------------------------------------------------------------------------
constexpr const char* kApiModule = "flash_attention_triton_b200.api";
constexpr const char* kLibModule = "flash_attention_triton_b200._lib";

// Environment switches that api.py serves.  Called with the interpreter lock, under which os.environ changes them.
bool python_path_asked() {
  const char* check = std::getenv("FA2_B200_CHECK_STATUS");
  const char* mode = std::getenv("FA2_B200_BWD_MODE");
  return (check && std::strcmp(check, "1") == 0) || (mode && *mode);
}

// Raises _lib.Fa2Error for a non-zero code.  Called without the interpreter lock.
void check_code(const char* fn, int code) {
  if (code == 0) return;
  pybind11::gil_scoped_acquire gil;
  try {
    pybind11::module_::import(kLibModule).attr("check")(fn, code);
  } catch (pybind11::error_already_set& e) {
    e.restore();
    python_error error;
    error.persist();
    throw error;
  }
}

constexpr int kModeAtomic = 0, kModeRecompute = 1, kModeSpill = 2;
constexpr long long kScratchMaxBytesPerHead = 2ll << 30;

long long scratch_bytes_per_head(long long n) {
  const long long tiles = (n + 127) / 128;
  return tiles * (tiles + 1) / 2 * 32768;
}

// Which dQ strategy serves a call (the rule, with its reasons: _backward_mode of api.py).
int backward_mode(bool deterministic, int d, long long n) {
  if (d > 128) return kModeSpill;
  if (d <= 64) return deterministic ? kModeRecompute : kModeAtomic;
  return scratch_bytes_per_head(n) <= kScratchMaxBytesPerHead ? kModeSpill : kModeRecompute;
}

// The workspace of a backward mode, and the mode that will run: less scratch, or the mode that needs none, when memory is
// short (_allocate_workspace of api.py).  `allocate` gives back an undefined tensor when it has no memory.  False: no
// memory for the least the mode needs, `bytes`.
template <typename Allocate>
bool allocate_workspace(int b, int h, int n, int d, int& mode, long long& bytes, at::Tensor& workspace, Allocate&& allocate) {
  const long long want = static_cast<long long>(fa2_bwd_workspace_bytes(b, h, n, d, mode));
  workspace = at::Tensor();
  bytes = want;
  if (want == 0) return true;
  const long long one_head = scratch_bytes_per_head(n);
  long long sizes[3] = {want, 0, 0};
  int count = 1;
  if (mode == kModeSpill)
    for (const long long less : {want / 8 / one_head * one_head, one_head})
      if (less >= one_head && less < sizes[count - 1]) sizes[count++] = less;
  for (int i = 0; i < count; ++i) {
    workspace = allocate(bytes = sizes[i]);
    if (workspace.defined()) return true;
  }
  if (mode != kModeSpill || d > 128) return false;
  mode = kModeRecompute, bytes = 0;
  return true;
}

// backward_mode(deterministic, head dim, rows) -> mode
PyObject* py_backward_mode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3) return PyErr_Format(PyExc_TypeError, "backward_mode takes 3 arguments");
  const int deterministic = PyObject_IsTrue(args[0]);
  const long d = PyLong_AsLong(args[1]);
  const long long n = PyLong_AsLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromLong(backward_mode(deterministic != 0, static_cast<int>(d), n));
  END_HANDLE_TH_ERRORS
}

// allocate_workspace(allocate, batch, heads, rows, head dim, mode) -> (workspace or None, bytes, mode), mode -1: no memory.
// allocate(bytes) gives a tensor, or None when it has no memory.
PyObject* py_allocate_workspace(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 6) return PyErr_Format(PyExc_TypeError, "allocate_workspace takes 6 arguments");
  long v[5];
  for (int i = 0; i < 5; ++i) v[i] = PyLong_AsLong(args[i + 1]);
  if (PyErr_Occurred()) return nullptr;
  int mode = static_cast<int>(v[4]);
  long long bytes = 0;
  at::Tensor workspace;
  const bool ok = allocate_workspace(v[0], v[1], v[2], v[3], mode, bytes, workspace, [&](long long size) {
    const auto given = pybind11::reinterpret_steal<pybind11::object>(PyObject_CallFunction(args[0], "L", size));
    if (!given) throw python_error();
    TORCH_CHECK_TYPE(given.is_none() || THPVariable_Check(given.ptr()), "allocate must give a tensor or None");
    return given.is_none() ? at::Tensor() : THPVariable_Unpack(given.ptr());
  });
  return Py_BuildValue("NLi", THPVariable_Wrap(workspace), bytes, ok ? mode : -1);
  END_HANDLE_TH_ERRORS
}

// Saved-tensor hooks must give back what was saved.  False for what _flash_attention_backward of api.py asserts.
bool as_saved(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& output, const at::Tensor& lse,
              const at::Tensor& d_output) {
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4, "the saved q, k and v must be [B, H, N, D] tensors");
  if (lse.sizes() != q.sizes().slice(0, 3) || !output.is_contiguous() ||
      (q.scalar_type() != at::kHalf && q.scalar_type() != at::kBFloat16))
    return false;
  TORCH_CHECK(k.size(0) == q.size(0) && k.size(1) == q.size(1) && k.size(3) == q.size(3) && k.size(2) <= q.size(2) &&
                  v.sizes() == k.sizes() && output.sizes() == q.sizes() && d_output.sizes() == q.sizes(),
              "the saved tensors have changed their shapes");
  for (const at::Tensor* t : {&k, &v, &output, &lse, &d_output})
    TORCH_CHECK(t->device() == q.device() && t->scalar_type() == (t == &lse ? at::kFloat : q.scalar_type()),
                "the saved tensors have changed their type or device");
  TORCH_CHECK(q.is_cuda() && lse.is_contiguous(), "the saved tensors have changed their device or strides");
  return true;
}

struct Attention : torch::autograd::Function<Attention> {
  // `r` holds the outputs of the forward kernel, already launched on saved_q, saved_k and saved_v.
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor&, const at::Tensor&,
                            const at::Tensor&, const std::array<at::Tensor, 3>& saved, const Forward& r,
                            double scale, bool deterministic) {
    ctx->save_for_backward({saved[0], saved[1], saved[2], r.output, r.lse});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["deterministic"] = deterministic;
    ctx->saved_data["f32"] = r.output32.defined();
    // the tensor that is saved is not the one handed out
    return r.output32.defined() ? r.output32 : r.output.view(r.output.sizes());
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &q = saved[0], &k = saved[1], &v = saved[2], &output = saved[3], &lse = saved[4];
    const double scale = ctx->saved_data["scale"].toDouble();
    const bool deterministic = ctx->saved_data["deterministic"].toBool(), f32 = ctx->saved_data["f32"].toBool();
    at::Tensor d_output = grads[0];
    if (d_output.scalar_type() != q.scalar_type()) d_output = d_output.to(q.scalar_type());
    bool python = !as_saved(q, k, v, output, lse, d_output);
    if (!python) {
      pybind11::gil_scoped_acquire gil;
      python = python_path_asked();
    }
    at::Tensor dq = empty_gradient(q, f32), dk = empty_gradient(k, f32), dv = empty_gradient(v, f32);
    if (python) {
      pybind11::gil_scoped_acquire gil;
      try {
        pybind11::module_::import(kApiModule)
            .attr("_flash_attention_backward")(q, k, v, output, lse, dq, dk, dv, d_output, scale, deterministic);
      } catch (pybind11::error_already_set& e) {
        e.restore();
        python_error error;
        error.persist();
        throw error;
      }
    } else {
      at::Tensor rowstats;
      check_code("fa2_bwd_preprocess_strided", run_preprocess(output, d_output, lse, rowstats));
      int mode = backward_mode(deterministic, q.size(3), q.size(2));
      at::Tensor workspace;
      long long bytes = 0;
      std::exception_ptr no_memory;
      const auto allocate = [&](long long size) {
        try {
          return at::empty({size}, q.options().dtype(at::kByte).memory_format(at::MemoryFormat::Contiguous));
        } catch (const c10::OutOfMemoryError&) {
          no_memory = std::current_exception();
          return at::Tensor();
        }
      };
      if (!allocate_workspace(q.size(0), q.size(1), q.size(2), q.size(3), mode, bytes, workspace, allocate))
        std::rethrow_exception(no_memory);
      at::Tensor t[7] = {q, k, v, d_output, dq, dk, dv};
      check_code("fa2_bwd_strided", run_backward(t, rowstats, workspace, scale, mode));
    }
    return {dq, dk, dv, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

// Plain tensors outside every mode, transform and trace that an autograd function written in Python would see.
bool eligible(PyObject* const* args) {
  for (int i = 0; i < 3; ++i)
    if (!THPVariable_CheckExact(args[i])) return false;
  const at::Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
  for (const at::Tensor* t : {&q, &k, &v}) {
    if (!t->defined() || t->dim() != 4 || !t->is_cuda() || t->layout() != at::kStrided || !t->has_storage() ||
        t->numel() == 0 || t->is_neg() || t->unsafeGetTensorImpl()->is_python_dispatch())
      return false;
    if (t->scalar_type() != q.scalar_type() || t->device() != q.device()) return false;
    if (t->_fw_grad(0).defined()) return false;
  }
  const auto dtype = q.scalar_type();
  if (dtype != at::kHalf && dtype != at::kBFloat16 && dtype != at::kFloat) return false;
  if (k.size(0) != q.size(0) || k.size(1) != q.size(1) || k.size(3) != q.size(3) || k.sizes() != v.sizes()) return false;
  if (k.size(2) > q.size(2) || q.size(3) % 8 != 0 || q.size(3) > 256) return false;
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !torch::jit::tracer::isTracing() && !python_path_asked();
}

// attention(q, k, v, scale or None, deterministic) -> output, or None: the caller's general path takes this call
// (and reports what is wrong with it).
PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) return PyErr_Format(PyExc_TypeError, "attention takes 5 arguments");
  if (!eligible(args) || !(args[3] == Py_None || PyFloat_CheckExact(args[3]))) Py_RETURN_NONE;
  const int deterministic = PyObject_IsTrue(args[4]);
  if (deterministic < 0) return nullptr;
  double scale = args[3] == Py_None ? 0.0 : PyFloat_AS_DOUBLE(args[3]);
  const at::Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
  if (scale == 0.0) scale = 1.0 / std::sqrt(static_cast<double>(q.size(3)));
  at::Tensor result;
  {
    pybind11::gil_scoped_release no_gil;
    std::array<at::Tensor, 3> in{q, k, v};
    Forward r;
    {
      const at::AutoGradMode no_grad(false);
      const bool f32 = q.scalar_type() == at::kFloat;
      if (f32)
        for (at::Tensor& t : in) t = t.to(at::kHalf);
      r = run_forward(in[0], in[1], in[2], scale, f32);
    }
    if (r.code == 0) {
      const bool graph = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
      result = graph ? Attention::apply(q, k, v, in, r, scale, deterministic != 0)
                     : (r.output32.defined() ? r.output32 : r.output);
    }
  }
  if (!result.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(result);
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
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(attention)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(forward)), METH_FASTCALL, nullptr},
    {"preprocess", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(preprocess)), METH_FASTCALL, nullptr},
    {"gradients", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(gradients)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(backward)), METH_FASTCALL, nullptr},
    {"backward_mode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_backward_mode)), METH_FASTCALL, nullptr},
    {"allocate_workspace", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_allocate_workspace)), METH_FASTCALL, nullptr},
    {"readable_in_place", is_readable_in_place, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
