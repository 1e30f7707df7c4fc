// The hot calls of the Python binding as an extension module: tensor checks, output allocation, stream lookup and the call
// into the C ABI in one native step (through ctypes the same calls spent 3 to 4 us in the interpreter, more than a launch).
//
// Every function takes the plain form of its call only and returns NotImplemented for anything else (other tensor types,
// layouts, dtypes or devices, a closed handle, a scratch of another size): engine.py then takes its general path, which
// checks and reports as it always did.  Errors of the C ABI raise engine.Q35bError.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/Context.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>

#include "../../../include/q35b_nvfp4.h"

namespace {

PyObject * g_error_type = nullptr;  // engine.Q35bError
PyObject * g_workspaces = nullptr;  // engine._workspaces: (device index, stream) -> uint8 tensor

PyObject * not_plain() { Py_RETURN_NOTIMPLEMENTED; }

PyObject * raise_status(int status) {
  PyObject * e = PyObject_CallFunction(g_error_type, "is", status, q35b_last_error());
  if (e != nullptr) {
    PyErr_SetObject(g_error_type, e);
    Py_DECREF(e);
  }
  return nullptr;
}

// An int (kernel numbers) or a float or int (scales), as the general path takes them: anything else is left to it.
bool int_arg(PyObject * o, int * out) {
  if (!PyLong_Check(o)) return false;
  const long v = PyLong_AsLong(o);
  if (v < INT32_MIN || v > INT32_MAX || PyErr_Occurred() != nullptr) {
    PyErr_Clear();
    return false;
  }
  *out = static_cast<int>(v);
  return true;
}
bool float_arg(PyObject * o, float * out) {
  if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
  *out = static_cast<float>(PyFloat_AsDouble(o));
  if (PyErr_Occurred() == nullptr) return true;
  PyErr_Clear();
  return false;
}

// A tensor of exactly torch.Tensor on the current CUDA device, strided and with memory behind it.
bool plain_cuda(PyObject * o, at::ScalarType type, c10::DeviceIndex device, const at::Tensor ** out) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor & t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.scalar_type() != type || t.device().index() != device || t.layout() != at::kStrided) return false;
  if (t.key_set().has(c10::DispatchKey::FuncTorchBatched) || t.key_set().has(c10::DispatchKey::FuncTorchGradWrapper)) return false;
  *out = &t;
  return true;
}

const q35b_weight * weight_arg(PyObject * o) { return static_cast<const q35b_weight *>(PyLong_AsVoidPtr(o)); }

void * stream_of(c10::DeviceIndex device) { return c10::cuda::getCurrentCUDAStream(device).stream(); }

template <typename F>
int without_gil(F && f) {
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = f();
  Py_END_ALLOW_THREADS
  return status;
}

// A new tensor.  Without the dispatcher, unless a dispatch mode or a profiler listens to it, or new memory is to be filled: 0.9 us
// instead of 1.4, of 4.2 for the smallest projection; asking takes some 0.03.
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, c10::DeviceIndex device) {
  const c10::Device where(at::kCUDA, device);
  const at::Context & context = at::globalContext();
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::getStepCallbacksUnlessEmpty(at::RecordScope::FUNCTION).has_value() ||
      (context.deterministicAlgorithms() && context.deterministicFillUninitializedMemory())) return at::empty(size, at::TensorOptions().dtype(type).device(where));
  return at::detail::empty_cuda(size, type, where, std::nullopt);
}

// The caller's output [m, cols] BF16 with unit column stride, or a new one in `made`; NULL: not the plain form.
const at::Tensor * output(PyObject * o, int64_t m, int64_t cols, c10::DeviceIndex device, at::Tensor & made) {
  if (o == Py_None) {
    made = empty({m, cols}, at::kBFloat16, device);
    return &made;
  }
  const at::Tensor * t = nullptr;
  if (!plain_cuda(o, at::kBFloat16, device, &t) || t->dim() != 2 || t->size(0) != m || t->size(1) != cols || t->stride(1) != 1) return nullptr;
  return t;
}

PyObject * returned(PyObject * given, at::Tensor & made) {
  if (given == Py_None) return THPVariable_Wrap(std::move(made));
  Py_INCREF(given);
  return given;
}

// gemv(weight, x [m, K] or [K], out or None, kernel) -> out
PyObject * gemv(PyObject *, PyObject * const * args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const q35b_weight * w = n == 4 ? weight_arg(args[0]) : nullptr;
  if (w == nullptr) return not_plain();
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::Tensor * x = nullptr;
  if (!plain_cuda(args[1], at::kBFloat16, device, &x) || !x->is_contiguous() || x->dim() < 1 || x->dim() > 2) return not_plain();
  const int64_t m = x->dim() == 2 ? x->size(0) : 1;
  if (x->size(-1) != q35b_weight_cols(w) || m < 1 || m > 8) return not_plain();
  int kernel = 0;
  if (!int_arg(args[3], &kernel)) return not_plain();
  at::Tensor made;
  const at::Tensor * y = output(args[2], m, q35b_weight_rows(w), device, made);
  if (y == nullptr || !y->is_contiguous()) return not_plain();
  const void * xp = x->const_data_ptr();
  void * yp = y->mutable_data_ptr(), * stream = stream_of(device);
  if (const int st = without_gil([&] { return q35b_gemv_w4a16_bf16(w, xp, static_cast<int>(m), yp, kernel, stream); })) return raise_status(st);
  return returned(args[2], made);
  END_HANDLE_TH_ERRORS
}

// gemv_f32(weight, x [K], input_scale, kernel) -> y [rows]
PyObject * gemv_f32(PyObject *, PyObject * const * args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const q35b_weight * w = n == 4 ? weight_arg(args[0]) : nullptr;
  if (w == nullptr) return not_plain();
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::Tensor * x = nullptr;
  if (!plain_cuda(args[1], at::kFloat, device, &x) || !x->is_contiguous() || x->numel() != q35b_weight_cols(w)) return not_plain();
  float scale = 0.0f;
  int kernel = 0;
  if (!float_arg(args[2], &scale) || !int_arg(args[3], &kernel)) return not_plain();
  at::Tensor y = empty({q35b_weight_rows(w)}, at::kFloat, device);
  const float * xp = x->const_data_ptr<float>();
  float * yp = y.mutable_data_ptr<float>();
  void * stream = stream_of(device);
  if (const int st = without_gil([&] { return q35b_gemv_w4a16_f32(w, xp, scale, yp, kernel, stream); })) return raise_status(st);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// batch_run(batch)
PyObject * batch_run(PyObject *, PyObject * batch) {
  HANDLE_TH_ERRORS
  const auto * b = static_cast<const q35b_gemv_batch *>(PyLong_AsVoidPtr(batch));
  if (b == nullptr) return not_plain();
  void * stream = stream_of(c10::cuda::current_device());
  if (const int st = without_gil([&] { return q35b_gemv_batch_run(b, stream); })) return raise_status(st);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// Contiguous [m, k] BF16 or fp32 activations and their scratch (codes, tiled scales, scale word).
struct Activations {
  const at::Tensor * x = nullptr, * codes = nullptr, * scales = nullptr, * g = nullptr;
  int m = 0, k = 0;
  bool bf16 = false;
  float scale = 0.0f;
  void * workspace = nullptr;
  bool take(PyObject * px, PyObject * const * scratch, PyObject * global_scale, c10::DeviceIndex device, void * stream) {
    bf16 = plain_cuda(px, at::kBFloat16, device, &x);
    if ((!bf16 && !plain_cuda(px, at::kFloat, device, &x)) || x->dim() != 2 || !x->is_contiguous()) return false;
    if (x->size(0) < 1 || x->size(0) > INT32_MAX || x->size(1) < 1 || x->size(1) > INT32_MAX) return false;
    m = static_cast<int>(x->size(0));
    k = static_cast<int>(x->size(1));
    if (!plain_cuda(scratch[0], at::kByte, device, &codes) || !plain_cuda(scratch[1], at::kByte, device, &scales) ||
        !plain_cuda(scratch[2], at::kFloat, device, &g)) {
      return false;
    }
    if (!codes->is_contiguous() || codes->numel() != static_cast<int64_t>(m) * (k / 2)) return false;
    if (!float_arg(global_scale, &scale)) return false;
    PyObject * key = Py_BuildValue("(iK)", static_cast<int>(device), static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
    if (key == nullptr) {
      PyErr_Clear();
      return false;
    }
    PyObject * ws = PyDict_GetItem(g_workspaces, key);  // borrowed; engine.py makes it on the first call of a stream
    Py_DECREF(key);
    const at::Tensor * w = nullptr;
    if (ws == nullptr || !plain_cuda(ws, at::kByte, device, &w)) return false;
    workspace = w->mutable_data_ptr();
    return true;
  }
  int quantize(void * stream) const {
    auto * c = static_cast<uint8_t *>(codes->mutable_data_ptr());
    auto * s = static_cast<uint8_t *>(scales->mutable_data_ptr());
    auto * word = static_cast<float *>(g->mutable_data_ptr());
    const void * xp = x->const_data_ptr();
    return bf16 ? q35b_quantize_nvfp4_bf16(xp, m, k, scale, c, s, word, workspace, stream)
                : q35b_quantize_nvfp4_f32(static_cast<const float *>(xp), m, k, scale, c, s, word, workspace, stream);
  }
};

int gemm_call(const q35b_weight * w, const at::Tensor & codes, const at::Tensor & scales, const at::Tensor & g, int m,
              const at::Tensor * residual, const at::Tensor & out, void * stream) {
  const auto * c = static_cast<const uint8_t *>(codes.const_data_ptr());
  const auto * s = static_cast<const uint8_t *>(scales.const_data_ptr());
  const auto * word = static_cast<const float *>(g.const_data_ptr());
  const int ldc = static_cast<int>(out.stride(0));
  if (residual == nullptr) return q35b_gemm_w4a4_bf16(w, c, s, word, m, out.mutable_data_ptr(), ldc, nullptr, stream);
  return q35b_gemm_w4a4_bf16_residual(w, c, s, word, m, residual->const_data_ptr(), static_cast<int>(residual->stride(0)),
                                      out.mutable_data_ptr(), ldc, nullptr, stream);
}

bool residual_arg(PyObject * o, int m, int rows, c10::DeviceIndex device, const at::Tensor ** out) {
  if (o == Py_None) return true;
  return plain_cuda(o, at::kBFloat16, device, out) && (*out)->dim() == 2 && (*out)->size(0) == m && (*out)->size(1) == rows &&
         (*out)->stride(1) == 1 && (*out)->stride(0) <= INT32_MAX;
}

// project_prefill(weight, x, out or None, codes, scales, g, global_scale, residual or None) -> out
PyObject * project_prefill(PyObject *, PyObject * const * args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const q35b_weight * w = n == 8 ? weight_arg(args[0]) : nullptr;
  if (w == nullptr) return not_plain();
  const c10::DeviceIndex device = c10::cuda::current_device();
  void * stream = stream_of(device);
  Activations a;
  if (!a.take(args[1], args + 3, args[6], device, stream) || a.k != q35b_weight_cols(w)) return not_plain();
  const int rows = q35b_weight_rows(w);
  const at::Tensor * residual = nullptr;
  if (!residual_arg(args[7], a.m, rows, device, &residual)) return not_plain();
  at::Tensor made;
  const at::Tensor * out = output(args[2], a.m, q35b_weight_is_gate_up(w) != 0 ? rows / 2 : rows, device, made);
  if (out == nullptr || out->stride(0) > INT32_MAX) return not_plain();
  auto * codes = static_cast<uint8_t *>(a.codes->mutable_data_ptr()), * scales = static_cast<uint8_t *>(a.scales->mutable_data_ptr());
  auto * word = static_cast<float *>(a.g->mutable_data_ptr());
  const void * xp = a.x->const_data_ptr(), * rp = residual != nullptr ? residual->const_data_ptr() : nullptr;
  const int ldr = residual != nullptr ? static_cast<int>(residual->stride(0)) : 0, ldc = static_cast<int>(out->stride(0));
  void * cp = out->mutable_data_ptr();
  const int st = without_gil([&] {
    return q35b_project_prefill(w, xp, a.bf16 ? 0 : 1, a.m, a.scale, codes, scales, word, a.workspace, rp, ldr, cp, ldc, nullptr, stream);
  });
  if (st != 0) return raise_status(st);
  return returned(args[2], made);
  END_HANDLE_TH_ERRORS
}

// quantize(x, codes, scales, g, global_scale): writes the scratch
PyObject * quantize(PyObject *, PyObject * const * args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5) return not_plain();
  const c10::DeviceIndex device = c10::cuda::current_device();
  void * stream = stream_of(device);
  Activations a;
  if (!a.take(args[0], args + 1, args[4], device, stream)) return not_plain();
  if (const int st = without_gil([&] { return a.quantize(stream); })) return raise_status(st);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// gemm(weight, codes, scales, g, m, out or None, residual or None) -> out
PyObject * gemm(PyObject *, PyObject * const * args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const q35b_weight * w = n == 7 ? weight_arg(args[0]) : nullptr;
  if (w == nullptr) return not_plain();
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::Tensor * codes = nullptr, * scales = nullptr, * g = nullptr, * residual = nullptr;
  if (!plain_cuda(args[1], at::kByte, device, &codes) || !plain_cuda(args[2], at::kByte, device, &scales) || !plain_cuda(args[3], at::kFloat, device, &g)) return not_plain();
  int m = 0;
  const int rows = q35b_weight_rows(w);
  if (!int_arg(args[4], &m) || m < 1 || !residual_arg(args[6], m, rows, device, &residual)) return not_plain();
  at::Tensor made;
  const at::Tensor * out = output(args[5], m, q35b_weight_is_gate_up(w) != 0 ? rows / 2 : rows, device, made);
  if (out == nullptr || out->stride(0) > INT32_MAX) return not_plain();
  void * stream = stream_of(device);
  if (const int st = without_gil([&] { return gemm_call(w, *codes, *scales, *g, m, residual, *out, stream); })) return raise_status(st);
  return returned(args[5], made);
  END_HANDLE_TH_ERRORS
}

// setup(Q35bError, workspaces)
PyObject * setup(PyObject *, PyObject * const * args, Py_ssize_t n) {
  if (n != 2 || !PyDict_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "setup(error type, dict)");
    return nullptr;
  }
  Py_XDECREF(g_error_type);
  Py_XDECREF(g_workspaces);
  Py_INCREF(args[0]);
  Py_INCREF(args[1]);
  g_error_type = args[0];
  g_workspaces = args[1];
  Py_RETURN_NONE;
}

template <PyObject * (*F)(PyObject *, PyObject * const *, Py_ssize_t)>
PyMethodDef fast(const char * name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL, nullptr};
}

PyMethodDef g_methods[] = {fast<setup>("setup"),       fast<gemv>("gemv"),     fast<gemv_f32>("gemv_f32"), {"batch_run", batch_run, METH_O, nullptr},
                           fast<quantize>("quantize"), fast<gemm>("gemm"),     fast<project_prefill>("project_prefill"), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "q35b_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_q35b_torch() { return PyModule_Create(&g_module); }
