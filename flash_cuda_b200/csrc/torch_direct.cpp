// torch_direct.cpp — `call_fwd` without the dispatcher: a Python function that hands plain CUDA tensors straight to the
// implementation of the torch op `fwd` (torch_op.cpp).
//
// A call through `torch.ops` spent 8 of its 15 us on taking 37 arguments through the schema, the boxed stack and the
// dispatcher; a decode step of one sequence is 9.4 us on the GPU.  This function reads its 23 arguments from the vector
// call and does nothing else the dispatcher would not: it declines (returns None, and the caller goes through the op)
// unless the dispatcher would have nothing to do but call the CUDA kernel - see `plain` and `nothing_active`.
// Measured per call, one sequence of 1000 keys: 14.6 -> 11.3 us, now bound by the GPU.
//
// A library of its own, because it needs the Python runtime: the op's library does not.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/grad_mode.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "torch_op.h"

namespace {

// No tracing, functorch transform, dispatch or function mode, or profiler callback: none of the keys that these put into
// the thread's included set, and no mode on the stacks.  (Inference mode only takes keys out.)
bool nothing_active() {
  const c10::impl::LocalDispatchKeySet tls = c10::impl::tls_local_dispatch_key_set();
  const c10::DispatchKeySet usual({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView});
  return usual.isSupersetOf(tls.included_) && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         !at::impl::torch_function_mode_enabled() && !at::hasCallbacks();
}

// A torch.Tensor (no subclass) on CUDA whose dispatch keys are the CUDA kernel's and those that fall through to it, without
// a gradient or a tangent that somebody would expect the result to carry.
bool plain(PyObject* o, std::optional<at::Tensor>* out) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::DispatchKeySet usual({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                                   c10::DispatchKey::AutocastCUDA});
  if (!t.defined() || !usual.isSupersetOf(t.key_set())) return false;
  if (t.unsafeGetTensorImpl()->autograd_meta() != nullptr &&
      ((t.requires_grad() && at::GradMode::is_enabled()) || t._fw_grad(/*level=*/0).defined()))
    return false;
  *out = t;
  return true;
}
bool plain_or_none(PyObject* o, std::optional<at::Tensor>* out) { return o == Py_None || plain(o, out); }

bool integer(PyObject* o, int64_t* out) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *out = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
bool number(PyObject* o, double* out) {
  if (!PyFloat_CheckExact(o)) return false;
  *out = PyFloat_AS_DOUBLE(o);
  return true;
}

// fwd(q, k, v, out, cu_seqlens_q, cu_seqlens_k, seqused_k, max_seqlen_q, max_seqlen_k, page_table, leftpad_k, q_descale,
//     k_descale, v_descale, softmax_scale, causal, window_left, window_right, softcap, scheduler_metadata, num_splits,
//     sm_margin, s_aux) -> (out, lse), or None: not a call for this path
PyObject* direct_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 23 || !nothing_active()) Py_RETURN_NONE;
  std::optional<at::Tensor> q, k, v, out, cu_q, cu_k, used_k, table, leftpad, qd, kd, vd, metadata, s_aux;
  int64_t max_q, max_k, wl, wr, splits, margin;
  double scale, cap;
  if (!plain(a[0], &q) || !plain(a[1], &k) || !plain(a[2], &v) || !plain_or_none(a[3], &out) || !plain_or_none(a[4], &cu_q) ||
      !plain_or_none(a[5], &cu_k) || !plain_or_none(a[6], &used_k) || !integer(a[7], &max_q) || !integer(a[8], &max_k) ||
      !plain_or_none(a[9], &table) || !plain_or_none(a[10], &leftpad) || !plain_or_none(a[11], &qd) ||
      !plain_or_none(a[12], &kd) || !plain_or_none(a[13], &vd) || !number(a[14], &scale) || !PyBool_Check(a[15]) ||
      !integer(a[16], &wl) || !integer(a[17], &wr) || !number(a[18], &cap) || !plain_or_none(a[19], &metadata) ||
      !integer(a[20], &splits) || !integer(a[21], &margin) || !plain_or_none(a[22], &s_aux))
    Py_RETURN_NONE;
  const bool causal = a[15] == Py_True;
  std::pair<at::Tensor, at::Tensor> r;
  {
    pybind11::gil_scoped_release no_gil;      // (as the op's call does)
    r = fa_b200::attention(*q, *k, *v, {}, {}, {}, out, cu_q, cu_k, {}, {}, used_k, max_q, max_k, table, {}, leftpad, {}, {},
                           {}, qd, kd, vd, scale, causal, wl, wr, cap, true, metadata, splits, {}, margin, s_aux, 1, 0, {});
  }
  PyObject* o0 = THPVariable_Wrap(std::move(r.first));
  PyObject* o1 = THPVariable_Wrap(std::move(r.second));
  PyObject* t = o0 && o1 ? PyTuple_Pack(2, o0, o1) : nullptr;
  Py_XDECREF(o0);
  Py_XDECREF(o1);
  return t;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"fwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(direct_fwd)), METH_FASTCALL,
                          "(out, lse) of the torch op `fwd`, or None where the call has to go through the op"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "fa_b200_direct", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_fa_b200_direct(void) { return PyModule_Create(&module); }
