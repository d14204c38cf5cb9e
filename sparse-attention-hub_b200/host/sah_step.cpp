// Host side of a decode call whose mask is bands (sink, local window) and, at most, an exact top-k
// of q.k on top of them: tensors in, output out, in one call from Python.
//
// Such a call is one to four short kernels (10 us of a float32 call over 4096 keys), and the Python
// that checked the tensors, built Mask objects, allocated seven buffers and converted a hundred
// arguments took longer than they did: 48 us; with this entry the call takes 10 us, as long as its kernel.  Here the
// tensors are looked at in C++, one scratch tensor is allocated, with a top-k two (with the output all that a call
// allocates, whatever the key count of the call before), and the kernels are launched by sah_fixed_step_run.
//
// fixed_step(...) returns None for tensors that this path does not serve; the caller then takes the
// general path, which serves them or says what is wrong with them.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/version.h>

#include "sah_b200.h"

namespace {

int (*plan_fn)(const sah_fixed_step*, sah_fixed_step_layout*) = nullptr;
int (*run_fn)(const sah_fixed_step*, const sah_fixed_step_layout*, void*) = nullptr;
int64_t (*capture_fn)(void*) = nullptr;

// bind(addresses of sah_fixed_step_plan, sah_fixed_step_run and sah_stream_capture)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "bind: three addresses expected");
    return nullptr;
  }
  void* address[3];
  for (int i = 0; i < 3; ++i) {
    address[i] = PyLong_AsVoidPtr(args[i]);
    if (address[i] == nullptr && PyErr_Occurred()) return nullptr;
  }
  plan_fn = reinterpret_cast<decltype(plan_fn)>(address[0]);
  run_fn = reinterpret_cast<decltype(run_fn)>(address[1]);
  capture_fn = reinterpret_cast<decltype(capture_fn)>(address[2]);
  Py_RETURN_NONE;
}

bool rows_of(const at::Tensor& t, int64_t* strides) {
  if (t.dim() != 4 || t.layout() != at::kStrided || t.stride(3) != 1) return false;
  for (int i = 0; i < 3; ++i) strides[i] = t.stride(i);
  return true;
}

// fixed_step(queries, keys, values, attention_mask or None, sinks or None, scaling, bands, heavy, tickets,
//            sm_count, stream, whether a capture may keep the tickets)
// -> None, a non-zero status, (identity of the capture that the stream is in,) for tickets that it may not keep, or (out, scratch, offsets of ucols (-1: there is no list), umemb and ucount in it, groups,
//     rows per group)
PyObject* fixed_step(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 12 || plan_fn == nullptr) {
    PyErr_SetString(PyExc_TypeError, "fixed_step: twelve arguments expected, after bind()");
    return nullptr;
  }
  for (int i = 0; i < 3; ++i)
    if (!THPVariable_CheckExact(args[i])) Py_RETURN_NONE;
  if ((args[3] != Py_None && !THPVariable_CheckExact(args[3])) || (args[4] != Py_None && !THPVariable_CheckExact(args[4])) ||
      !THPVariable_CheckExact(args[8]) || !PyTuple_CheckExact(args[6]))
    Py_RETURN_NONE;
  const at::Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
  const at::Tensor& tickets = THPVariable_Unpack(args[8]);
  sah_fixed_step s = {};
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device() || tickets.device() != q.device())
    Py_RETURN_NONE;
  const at::ScalarType dtype = q.scalar_type();
  if (dtype != at::kFloat && dtype != at::kBFloat16) Py_RETURN_NONE;
  if (k.scalar_type() != dtype || v.scalar_type() != dtype) Py_RETURN_NONE;
  if (!rows_of(q, s.q_stride) || !rows_of(k, s.k_stride) || !rows_of(v, s.v_stride)) Py_RETURN_NONE;
  if (k.sizes() != v.sizes() || k.size(0) != q.size(0) || k.size(3) != q.size(3)) Py_RETURN_NONE;
  if (q.numel() == 0 || k.numel() == 0 || q.size(1) % k.size(1) != 0) Py_RETURN_NONE;
  for (int i = 0; i < 3; ++i)
    if (q.size(i) > INT32_MAX) Py_RETURN_NONE;
  s.dtype = dtype == at::kBFloat16 ? SAH_BF16 : SAH_F32;
  s.B = (int32_t)q.size(0);
  s.Hq = (int32_t)q.size(1);
  s.Hkv = (int32_t)k.size(1);
  s.Sq = (int32_t)q.size(2);
  s.D = (int32_t)q.size(3);
  s.S = k.size(2);
  if (args[3] != Py_None) {
    const at::Tensor& bias = THPVariable_Unpack(args[3]);
    int64_t stride[3];
    if (bias.device() != q.device() || bias.scalar_type() != dtype || !rows_of(bias, stride) || bias.size(3) < s.S)
      Py_RETURN_NONE;
    for (int i = 0; i < 3; ++i) s.bias_stride[i] = bias.size(i) > 1 ? stride[i] : 0;
    s.bias = bias.data_ptr();
  }
  if (args[4] != Py_None) {
    const at::Tensor& sinks = THPVariable_Unpack(args[4]);
    if (sinks.device() != q.device() || sinks.scalar_type() != at::kFloat || sinks.dim() != 1 || sinks.size(0) != s.Hq ||
        !sinks.is_contiguous())
      Py_RETURN_NONE;
    s.sinks = sinks.data_ptr<float>();
  }
  s.scaling = (float)PyFloat_AsDouble(args[5]);
  const Py_ssize_t words = PyTuple_GET_SIZE(args[6]);
  if (words % 5 != 0 || words > 5 * SAH_STEP_MAX_BANDS) Py_RETURN_NONE;
  s.n_bands = (int32_t)(words / 5);
  for (Py_ssize_t i = 0; i < words; ++i) s.bands[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[6], i));
  s.heavy = PyLong_AsLongLong(args[7]);
  s.sm_count = (int32_t)PyLong_AsLong(args[9]);
  void* stream = PyLong_AsVoidPtr(args[10]);
  if (PyErr_Occurred()) return nullptr;
  s.q = q.data_ptr();
  s.k = k.data_ptr();
  s.v = v.data_ptr();
  s.tickets = tickets.data_ptr<int32_t>();
  s.n_tickets = tickets.numel();
  sah_fixed_step_layout layout;
  if (plan_fn(&s, &layout) != SAH_OK) Py_RETURN_NONE;
  if (args[11] != Py_True) {
    const int64_t capture = capture_fn(stream);
    if (capture != 0) return Py_BuildValue("(L)", (long long)capture);
  }
  at::Tensor out, scratch, scores;
  int status;
  {
    pybind11::gil_scoped_release no_gil;
    out = at::empty({s.B, s.Sq, s.Hq, s.D}, q.options().requires_grad(false));
    scratch = at::empty({layout.total}, q.options().dtype(at::kByte).requires_grad(false));
    if (layout.scores_total > 0) {  // apart from the list, which outlives the call for those who ask about it
      scores = at::empty({layout.scores_total}, q.options().dtype(at::kByte).requires_grad(false));
      s.scores = scores.data_ptr();
    }
    s.out = out.data_ptr();
    s.scratch = scratch.data_ptr();
    status = run_fn(&s, &layout, stream);
  }
  if (status != SAH_OK) return PyLong_FromLong(status);
  PyObject* result = PyTuple_New(7);
  if (result == nullptr) return nullptr;
  PyTuple_SET_ITEM(result, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(result, 1, THPVariable_Wrap(std::move(scratch)));
  PyTuple_SET_ITEM(result, 2, PyLong_FromLongLong(layout.planned ? layout.ucols : -1));
  PyTuple_SET_ITEM(result, 3, PyLong_FromLongLong(layout.umemb));
  PyTuple_SET_ITEM(result, 4, PyLong_FromLongLong(layout.ucount));
  PyTuple_SET_ITEM(result, 5, PyLong_FromLong(layout.sizes.groups));
  PyTuple_SET_ITEM(result, 6, PyLong_FromLong(layout.sizes.rows_per_group));
  return result;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"fixed_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fixed_step)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_sah_step", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__sah_step() {
  PyObject* m = PyModule_Create(&module);
  // the torch that the tensors' layout was compiled for
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
