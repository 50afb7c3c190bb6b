// The host side of one call of a compiled graph, as a CPython extension: check the tensors, allocate
// the results, hand the pointers to kb200_plan_run.  Takes the place of GPUExecutable.__call__ of the
// reference (kiln/gpu/runtime.py:206-217), which copies the inputs into fixed buffers, replays a graph
// and clones the results out.
//
// A small kernel takes 2 to 5 us, so what such a call costs is the host's work and the launches around
// the kernel.  The same steps from Python (current stream, torch.empty, ctypes, a copy in and a clone
// out around a graph replay) took 17.5 us a call whatever the kernel was; these take about 1 us and one
// launch per kernel.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/copy.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <mutex>
#include <string>
#include <vector>

#include "kb200.h"

namespace {

constexpr int kMaxBuffers = 16;       // what kb200_plan_run takes

struct Caller {
  kb200_plan* plan;
  c10::Device device{c10::kCUDA, 0};
  std::vector<std::vector<int64_t>> in_shapes, out_shapes;
  std::vector<at::Tensor> fixed_inputs;      // where an input goes that the kernels cannot read as it is
  std::mutex copies;                         // held from such a copy to the launches that read it
};

// The interpreter is left to other threads; taken again on the way out, by an exception too.
struct WithoutInterpreter {
  PyThreadState* const state = PyEval_SaveThread();
  ~WithoutInterpreter() { PyEval_RestoreThread(state); }
};

constexpr const char* kCapsule = "kb200.caller";

void destroy(PyObject* capsule) { delete static_cast<Caller*>(PyCapsule_GetPointer(capsule, kCapsule)); }

bool read_shapes(PyObject* list, std::vector<std::vector<int64_t>>* out) {
  const Py_ssize_t n = PySequence_Size(list);
  if (n < 0) return false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* shape = PySequence_GetItem(list, i);
    const Py_ssize_t rank = shape ? PySequence_Size(shape) : -1;
    std::vector<int64_t> dims;
    for (Py_ssize_t d = 0; d < rank; ++d) {
      PyObject* v = PySequence_GetItem(shape, d);
      dims.push_back(v ? PyLong_AsLongLong(v) : -1);
      Py_XDECREF(v);
    }
    Py_XDECREF(shape);
    if (rank < 0 || PyErr_Occurred()) return false;
    out->push_back(std::move(dims));
  }
  return true;
}

// caller(plan address, device index, input shapes, output shapes, fixed input tensors)
PyObject* make_caller(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  unsigned long long plan;
  int device;
  PyObject *in_shapes, *out_shapes, *fixed;
  if (!PyArg_ParseTuple(args, "KiOOO", &plan, &device, &in_shapes, &out_shapes, &fixed)) return nullptr;
  auto c = std::make_unique<Caller>();
  c->plan = reinterpret_cast<kb200_plan*>(plan);
  c->device = c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device));
  if (!read_shapes(in_shapes, &c->in_shapes) || !read_shapes(out_shapes, &c->out_shapes)) return nullptr;
  const Py_ssize_t n = PySequence_Size(fixed);
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* t = PySequence_GetItem(fixed, i);
    if (!t || !THPVariable_Check(t)) {
      Py_XDECREF(t);
      PyErr_SetString(PyExc_TypeError, "fixed inputs must be tensors");
      return nullptr;
    }
    c->fixed_inputs.push_back(THPVariable_Unpack(t));
    Py_DECREF(t);
  }
  if (c->in_shapes.size() > kMaxBuffers || c->out_shapes.size() > kMaxBuffers || c->fixed_inputs.size() != c->in_shapes.size()) {
    PyErr_SetString(PyExc_ValueError, "caller: bad number of inputs or outputs");
    return nullptr;
  }
  return PyCapsule_New(c.release(), kCapsule, destroy);
  END_HANDLE_TH_ERRORS
}

std::string text(c10::IntArrayRef shape) {
  std::string s = "(";
  for (size_t i = 0; i < shape.size(); ++i) s += (i ? ", " : "") + std::to_string(shape[i]);
  return s + (shape.size() == 1 ? ",)" : ")");
}

PyObject* raise(int status) {
  PyObject* type = status == KB200_ERR_ARGUMENT || status == KB200_ERR_BOUNDS ? PyExc_ValueError
                   : status == KB200_ERR_UNSUPPORTED                          ? PyExc_NotImplementedError
                                                                              : PyExc_RuntimeError;
  PyErr_Format(type, "kb200: %s (status %d)", kb200_last_error(), status);
  return nullptr;
}

// run(caller, *inputs) -> [outputs]
PyObject* run(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  Caller* c = n_args > 0 ? static_cast<Caller*>(PyCapsule_GetPointer(args[0], kCapsule)) : nullptr;
  if (!c) return PyErr_Occurred() ? nullptr : (PyErr_SetString(PyExc_TypeError, "run(caller, *inputs)"), nullptr);
  const size_t n_in = c->in_shapes.size(), n_out = c->out_shapes.size();
  if ((size_t)(n_args - 1) != n_in)
    return PyErr_Format(PyExc_TypeError, "expected %zu inputs, got %zd", n_in, n_args - 1);
  for (size_t i = 0; i < n_in; ++i) {
    if (!THPVariable_Check(args[1 + i])) return PyErr_Format(PyExc_TypeError, "input %zu is not a tensor", i);
    const at::Tensor& t = THPVariable_Unpack(args[1 + i]);
    if (t.sizes() != c10::IntArrayRef(c->in_shapes[i]))
      return PyErr_Format(PyExc_ValueError, "Kiln was compiled for input shape %s, got %s", text(c->in_shapes[i]).c_str(),
                          text(t.sizes()).c_str());
  }
  const c10::cuda::CUDAGuard guard(c->device);
  void* in[kMaxBuffers];
  bool copied = false;
  for (size_t i = 0; i < n_in; ++i) {
    const at::Tensor& t = THPVariable_Unpack(args[1 + i]);
    // read where it is: float32, dense, on this device, 16-byte aligned (128-bit loads, tensor maps); a tensor without memory
    // (zeros that autograd made, a wrapper) has its values copied
    const bool direct = t.layout() == c10::kStrided && t.scalar_type() == c10::kFloat && t.device() == c->device && t.is_contiguous() && !t.is_neg() &&
                        !t._is_zerotensor();
    const void* at = direct ? t.const_data_ptr() : nullptr;
    in[i] = (reinterpret_cast<uintptr_t>(at) & 15) == 0 ? const_cast<void*>(at) : nullptr;
    copied = copied || in[i] == nullptr;
  }
  void* out[kMaxBuffers];
  std::vector<at::Tensor> results;
  results.reserve(n_out);
  for (size_t i = 0; i < n_out; ++i) {
    results.push_back(at::detail::empty_cuda(c->out_shapes[i], c10::kFloat, c->device, std::nullopt));
    out[i] = results[i].data_ptr();
  }
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(c->device.index()).stream();
  int status;
  {
    const WithoutInterpreter others_run;
    std::unique_lock<std::mutex> one_copy(c->copies, std::defer_lock);
    if (copied) {
      one_copy.lock();
      const c10::NoGradGuard no_grad;
      for (size_t i = 0; i < n_in; ++i)
        if (in[i] == nullptr) c->fixed_inputs[i].copy_(THPVariable_Unpack(args[1 + i]).detach(), /*non_blocking=*/true);
    }
    status = kb200_plan_run(c->plan, in, (int)n_in, out, (int)n_out, stream);
  }
  if (status != KB200_OK) return raise(status);
  PyObject* list = PyList_New((Py_ssize_t)n_out);
  for (size_t i = 0; list && i < n_out; ++i) PyList_SET_ITEM(list, (Py_ssize_t)i, THPVariable_Wrap(std::move(results[i])));
  return list;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"caller", make_caller, METH_VARARGS, "caller(plan, device, input_shapes, output_shapes, fixed_inputs)"},
    {"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(run)), METH_FASTCALL, "run(caller, *inputs) -> list of output tensors"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_kb200_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__kb200_call() { return PyModule_Create(&module); }
