// The host side of one eager weight-only product: what torchao_fork_b200/ops.py does between the decision that nobody but the kernels has a say in
// the call (no mode, tracer, transform, gradient or wrapper: runs_eagerly) and the launch -- checks, output, workspace, stream, device -- as native code.
// Through Python and ctypes these take about 5 us more, of about 22 that a call of one row takes, while its kernel takes 5.  Everything that is not
// plainly in order (shapes, types, strides, alignment, no rows) is left to the Python code, which mends or refuses it: the answer is then None.
// An error code of the library comes back as an int.  The functions' types are those of the header that this module is built with, and a library of another
// version is refused (bind).
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/ao_b200.h"

namespace {

decltype(&ao_b200_int4_mm_workspace_bytes) int4_bytes;
decltype(&ao_b200_int8_mm_workspace_bytes) int8_bytes;
decltype(&ao_b200_int4_mm) int4_mm_fn;
decltype(&ao_b200_int8_mm) int8_mm_fn;

// rows as the kernels read them: bf16 [m][k], whole 16-byte pieces
bool rows_ok(const at::Tensor& x) {
  return x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.size(0) > 0 && x.size(1) > 0 && x.size(1) % 8 == 0 && x.stride(1) == 1 &&
         x.stride(0) % 8 == 0 && x.stride(0) >= x.size(1) && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0;
}

struct Owned {   // a reference that goes with the scope
  PyObject* p;
  ~Owned() { Py_XDECREF(p); }
};

// workspace(device index, stream, bytes) -> a uint8 tensor that the caller's table keeps, or None
bool workspace_of(PyObject* workspace, int device, cudaStream_t stream, int64_t bytes, Owned& tensor, void** at) {
  *at = nullptr;
  if (bytes == 0) return true;
  Owned index{PyLong_FromLong(device)}, where{PyLong_FromVoidPtr(stream)}, size{PyLong_FromLongLong(bytes)};
  if (!index.p || !where.p || !size.p) return false;
  PyObject* args[3] = {index.p, where.p, size.p};
  tensor.p = PyObject_Vectorcall(workspace, args, 3, nullptr);
  if (tensor.p == nullptr) return false;
  if (!THPVariable_Check(tensor.p)) {
    PyErr_SetString(PyExc_TypeError, "workspace: a tensor is wanted");
    return false;
  }
  *at = THPVariable_Unpack(tensor.p).data_ptr();
  return true;
}

PyObject* int4_mm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !THPVariable_Check(a[3]) || !PyLong_Check(a[2]) || !PyLong_Check(a[4])) Py_RETURN_NONE;
  const at::Tensor &x = THPVariable_Unpack(a[0]), &packed = THPVariable_Unpack(a[1]), &sz = THPVariable_Unpack(a[3]);
  int over = 0;
  const int64_t group = PyLong_AsLongLongAndOverflow(a[2], &over), out = over ? 0 : PyLong_AsLongLongAndOverflow(a[4], &over);
  if (over || !(group == 32 || group == 64 || group == 128 || group == 256) || !rows_ok(x)) Py_RETURN_NONE;
  if (!(packed.is_cuda() && packed.dim() == 4 && packed.scalar_type() == at::kInt && packed.size(2) == 32 && packed.size(3) == 4 && packed.is_contiguous()))
    Py_RETURN_NONE;
  const int64_t np = packed.size(0) * 16, kp = packed.size(1) * 64;
  if (!(sz.is_cuda() && sz.dim() == 4 && sz.scalar_type() == at::kBFloat16 && sz.size(0) == packed.size(0) && sz.size(1) == kp / group && sz.size(2) == 16 &&
        sz.size(3) == 2 && sz.is_contiguous() && x.size(1) <= kp && out > 0 && out <= np))
    Py_RETURN_NONE;
  const c10::DeviceIndex device = x.device().index();
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  const int64_t m = x.size(0), bytes = int4_bytes(m, np, kp);
  Owned held{nullptr};
  void* ws = nullptr;
  if (!workspace_of(a[5], device, stream, bytes, held, &ws)) return nullptr;
  at::Tensor y = at::empty({m, out}, at::TensorOptions().dtype(at::kBFloat16).device(x.device()));
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = int4_mm_fn(x.data_ptr(), m, x.size(1), x.stride(0), packed.data_ptr(), sz.data_ptr(), np, kp, (int)group, y.data_ptr(), out, out, ws, bytes, stream);
  Py_END_ALLOW_THREADS
  return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyObject* int8_mm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) Py_RETURN_NONE;
  const at::Tensor &x = THPVariable_Unpack(a[0]), &packed = THPVariable_Unpack(a[1]), &scale = THPVariable_Unpack(a[2]);
  if (!rows_ok(x) || !(packed.is_cuda() && packed.dim() == 3 && packed.scalar_type() == at::kByte && packed.size(2) == 1024 && packed.is_contiguous()))
    Py_RETURN_NONE;
  const int64_t np = packed.size(0) * 16, kp = packed.size(1) * 64, out = scale.numel();
  if (!(scale.is_cuda() && scale.scalar_type() == at::kBFloat16 && scale.is_contiguous() && x.size(1) <= kp && out > 0 && out <= np)) Py_RETURN_NONE;
  const c10::DeviceIndex device = x.device().index();
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  const int64_t m = x.size(0), bytes = int8_bytes(m, np, kp);
  Owned held{nullptr};
  void* ws = nullptr;
  if (!workspace_of(a[3], device, stream, bytes, held, &ws)) return nullptr;
  at::Tensor y = at::empty({m, out}, at::TensorOptions().dtype(at::kBFloat16).device(x.device()));
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = int8_mm_fn(x.data_ptr(), m, x.size(1), x.stride(0), packed.data_ptr(), scale.data_ptr(), np, kp, y.data_ptr(), out, out, ws, bytes, stream);
  Py_END_ALLOW_THREADS
  return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// the library's version, and its functions by their addresses: int4_mm, its workspace_bytes, int8_mm, its workspace_bytes
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long f[4];
  int version;
  if (!PyArg_ParseTuple(args, "iKKKK", &version, f, f + 1, f + 2, f + 3)) return nullptr;
  if (version != AO_B200_ABI_VERSION) return PyErr_Format(PyExc_ImportError, "built for version %d of the library, which is %d", AO_B200_ABI_VERSION, version);
  int4_mm_fn = reinterpret_cast<decltype(int4_mm_fn)>(f[0]);
  int4_bytes = reinterpret_cast<decltype(int4_bytes)>(f[1]);
  int8_mm_fn = reinterpret_cast<decltype(int8_mm_fn)>(f[2]);
  int8_bytes = reinterpret_cast<decltype(int8_bytes)>(f[3]);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"int4_mm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(int4_mm)), METH_FASTCALL, nullptr},
    {"int8_mm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(int8_mm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ao_b200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ao_b200_host() { return PyModule_Create(&module); }
