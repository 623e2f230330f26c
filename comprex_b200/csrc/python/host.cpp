// Host work of an optimizer step that is proportional to the number of parameters, for the Python
// side: walking 161 parameters for the addresses of their gradients takes 60 us of attribute look-ups
// in Python and 3 us here, and a ResNet-50 step is 110 us of GPU work.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

// the same memory order: strides of dimensions of size 1 say nothing
bool same_layout(const at::Tensor& a, const at::Tensor& b) {
  const auto n = b.sizes();
  if (a.sizes() != n) return false;
  const auto x = a.strides(), y = b.strides();
  for (size_t d = 0; d < n.size(); ++d)
    if (n[d] != 1 && x[d] != y[d]) return false;
  return true;
}

// collect(params, scalar_type, zeros, out) -> 0: the table at address `out` (one int64 per parameter)
// already held these addresses, 1: it has changed, 2: some gradient has another element type or
// memory order than its parameter (the table is incomplete).  `zeros` stands in for a missing one.
PyObject* collect(PyObject*, PyObject* args) {
  PyObject* params;
  int scalar_type;
  unsigned long long zeros, out;
  if (!PyArg_ParseTuple(args, "O!iKK", &PyList_Type, &params, &scalar_type, &zeros, &out)) return nullptr;
  int64_t* table = reinterpret_cast<int64_t*>(out);
  long changed = 0;
  const Py_ssize_t n = PyList_GET_SIZE(params);
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* o = PyList_GET_ITEM(params, i);
    if (!THPVariable_Check(o)) {
      PyErr_SetString(PyExc_TypeError, "collect: not a tensor");
      return nullptr;
    }
    const at::Tensor& p = THPVariable_Unpack(o);
    const at::Tensor& g = p.grad();
    int64_t a = static_cast<int64_t>(zeros);
    if (g.defined()) {
      if (static_cast<int>(g.scalar_type()) != scalar_type || g.layout() != at::kStrided || !same_layout(g, p))
        return PyLong_FromLong(2);
      a = reinterpret_cast<int64_t>(g.data_ptr());
    }
    changed |= table[i] != a;
    table[i] = a;
  }
  return PyLong_FromLong(changed);
}

// the value `collect` wants for a dtype, from a tensor of that dtype
PyObject* scalar_type(PyObject*, PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "scalar_type: not a tensor");
    return nullptr;
  }
  return PyLong_FromLong(static_cast<long>(THPVariable_Unpack(o).scalar_type()));
}

PyMethodDef methods[] = {{"collect", collect, METH_VARARGS, nullptr},
                         {"scalar_type", scalar_type, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_cxhost", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__cxhost(void) { return PyModule_Create(&module); }
