// Arguments and results of the Python bindings.
#pragma once

#include "host.h"

#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace t5b_host {

inline Tensor tensor_arg(PyObject* o) {
  if (o == Py_None) return Tensor();
  TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor, got ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
inline int64_t int_arg(PyObject* o) {
  PyObject* n = PyLong_Check(o) ? (Py_INCREF(o), o) : PyNumber_Long(o);
  if (!n) throw python_error();
  const int64_t v = (int64_t)PyLong_AsLongLong(n);
  Py_DECREF(n);
  if (v == -1 && PyErr_Occurred()) throw python_error();       // does not fit in 64 bits
  return v;
}
inline double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
inline bool bool_arg(PyObject* o) {
  if (o == Py_True) return true;
  if (o == Py_False || o == Py_None) return false;
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
inline std::optional<int64_t> opt_int(PyObject* o) { return o == Py_None ? std::nullopt : std::optional<int64_t>(int_arg(o)); }
inline PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
inline PyObject* wrap2(const Tensor& a, const Tensor& b) {
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, wrap(a));
  PyTuple_SET_ITEM(r, 1, wrap(b));
  return r;
}
inline void expect(Py_ssize_t got, Py_ssize_t want) { TORCH_CHECK_TYPE(got == want, "expected ", want, " arguments, got ", got); }

#define T5B_METHOD(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
extern PyMethodDef stack_methods[];

}  // namespace t5b_host
