// Host work on torch tensors for the Python side, where attribute look-ups in Python would cost as
// much as the GPU's work:
//  * collect: the addresses of an optimizer's gradients (161 parameters: 60 us in Python, 3 us here,
//    next to 110 us of GPU work for the step),
//  * run_vector: the launches of one message of a prepared connection.  Checks of the vector,
//    descriptors and native calls took 20 us per exchange in Python, the kernels of a 64 k-element
//    exchange take 15 us.
// Tensors of unusual kinds (nested, sparse, wrapped by a transform) throw at the questions asked here.  No
// exception may leave these functions: such a tensor is not the plain case, and the caller's general path
// says what is wrong with it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../cx_common.h"

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
    int64_t a = static_cast<int64_t>(zeros);
    try {
      const at::Tensor& p = THPVariable_Unpack(o);
      const at::Tensor& g = p.grad();
      if (g.defined()) {
        if (static_cast<int>(g.scalar_type()) != scalar_type || g.layout() != at::kStrided || !same_layout(g, p))
          return PyLong_FromLong(2);
        a = reinterpret_cast<int64_t>(g.data_ptr());
      }
    } catch (const std::exception&) {
      return PyLong_FromLong(2);
    }
    changed |= table[i] != a;
    table[i] = a;
  }
  return PyLong_FromLong(changed);
}

int element_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return CX_F32;
    case at::kBFloat16: return CX_BF16;
    case at::kHalf: return CX_F16;
    default: return -1;
  }
}

typedef int (*RunOps)(CxOp*, int, uint64_t, void*);
enum Role { kSend = 0, kApply = 1, kDenseSend = 2, kDenseRead = 3, kDenseAdd = 4, kRleRead = 5 };

// run_vector(role, run_ops, ops, count, seq, stream, vector, device, n) -> what cx_run_ops returns, or
// None when the vector is not the plain case (a contiguous CUDA tensor of the right size and type on
// `device`): nothing has happened then, the caller takes its general path.
//   kSend: input of a threshold + compress (or run-length send) list, n elements.  kApply: destination of an
//   apply op, n elements.  kDense*: a dense message of the vector's length, at most n, of the op's element type.
//   kRleRead: destination of a run-length receive, n fp32 elements.
PyObject* run_vector(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 9) {
    PyErr_SetString(PyExc_TypeError, "run_vector: nine arguments");
    return nullptr;
  }
  const long role = PyLong_AsLong(a[0]);
  RunOps run = reinterpret_cast<RunOps>(PyLong_AsUnsignedLongLong(a[1]));
  CxOp* ops = reinterpret_cast<CxOp*>(PyLong_AsUnsignedLongLong(a[2]));
  const long count = PyLong_AsLong(a[3]);
  const uint64_t seq = PyLong_AsUnsignedLongLong(a[4]);
  void* stream = reinterpret_cast<void*>(PyLong_AsUnsignedLongLong(a[5]));
  const long device = PyLong_AsLong(a[7]);
  const int64_t n = PyLong_AsLongLong(a[8]);
  if (PyErr_Occurred()) return nullptr;
  if (!THPVariable_CheckExact(a[6])) Py_RETURN_NONE;
  int code;
  int64_t len;
  void* ptr;
  try {
    const at::Tensor& t = THPVariable_Unpack(a[6]);
    if (!t.is_cuda() || t.device().index() != device || t.layout() != at::kStrided || !t.is_contiguous()) Py_RETURN_NONE;
    code = element_code(t);
    if (code < 0) Py_RETURN_NONE;
    len = t.numel();
    ptr = t.data_ptr();
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
  if (role == kSend) {
    if (len != n) Py_RETURN_NONE;
    for (long i = 0; i < count; ++i) {
      ops[i].g = ptr;
      ops[i].dtype = code;
    }
  } else if (role == kApply) {
    if (len < n) Py_RETURN_NONE;
    ops[0].apply.out = ptr;
    ops[0].apply.out_dtype = code;
  } else if (role == kRleRead) {
    if (len != n || code != CX_F32) Py_RETURN_NONE;
    ops[0].out = ptr;
  } else {
    if (len > n || code != ops[0].dtype) Py_RETURN_NONE;
    ops[0].n = len;
    if (role == kDenseSend) ops[0].g = ptr;
    else ops[0].out = ptr;
    if (role == kDenseAdd) ops[0].own = ptr;
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = run(ops, static_cast<int>(count), seq, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// install(pairs): `v.grad = g` for every (g, v); the checks of the attribute are left to it whenever
// the pair is not plainly two tensors of the same kind.
PyObject* install(PyObject*, PyObject* pairs) {
  PyObject* it = PyObject_GetIter(pairs);
  if (!it) return nullptr;
  while (PyObject* pair = PyIter_Next(it)) {
    PyObject* two = PySequence_Fast(pair, "install: (gradient, variable) pairs");
    Py_DECREF(pair);
    bool ok = two && PySequence_Fast_GET_SIZE(two) == 2;
    if (two && !ok) PyErr_SetString(PyExc_ValueError, "install: (gradient, variable) pairs");
    if (ok) {
      PyObject* g = PySequence_Fast_GET_ITEM(two, 0);
      PyObject* v = PySequence_Fast_GET_ITEM(two, 1);
      bool done = false;
      if (THPVariable_Check(g) && THPVariable_Check(v) && g != v) {
        try {
          const at::Tensor& gt = THPVariable_Unpack(g);
          const at::Tensor& vt = THPVariable_Unpack(v);
          if (gt.defined() && vt.defined() && vt.is_leaf() && gt.layout() == at::kStrided && vt.layout() == at::kStrided &&
              gt.scalar_type() == vt.scalar_type() && vt.grad_dtype() == vt.scalar_type() && gt.device() == vt.device() && gt.sizes() == vt.sizes()) {
            vt.mutable_grad() = gt;
            done = true;
          }
        } catch (const std::exception&) {
          done = false;
        }
      }
      ok = done || PyObject_SetAttrString(v, "grad", g) == 0;
    }
    Py_XDECREF(two);
    if (!ok) break;
  }
  Py_DECREF(it);
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// the value `collect` wants for a dtype, from a tensor of that dtype
PyObject* scalar_type(PyObject*, PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "scalar_type: not a tensor");
    return nullptr;
  }
  return PyLong_FromLong(static_cast<long>(THPVariable_Unpack(o).scalar_type()));      // (does not throw)
}

PyMethodDef methods[] = {{"collect", collect, METH_VARARGS, nullptr},
                         {"run_vector", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(run_vector)),
                          METH_FASTCALL, nullptr},
                         {"install", install, METH_O, nullptr},
                         {"scalar_type", scalar_type, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_cxhost", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__cxhost(void) { return PyModule_Create(&module); }
