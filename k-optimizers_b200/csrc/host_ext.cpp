// Per-step host work over a parameter list, in native code: the CPython module kaon_b200._kaon_host.
//
// A step has to look at every tensor of every parameter group: does it have a gradient, where is it, is it of a
// kind the kernels read, have the weights moved, is it still the tensor and the state the plan was built for.  In Python that
// costs about 0.6 us a tensor (a 720-tensor adapter list: 440 us of host time beside 60 us of device work); here
// about 24 ns.  Anything unusual is only reported: the Python path then runs and raises or rebuilds.
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>
#include <new>
#include <unordered_map>
#include <vector>

#ifndef KAON_HOST_ABI
#error "KAON_HOST_ABI: the torch and Python this is compiled for (kaon_b200/_build.py)"
#endif

namespace {

const char g_abi[] = "kaon host module for " KAON_HOST_ABI;   // _build.py looks for it in the file

enum : long { ANY_GRAD = 1, GRADS_CHANGED = 2, UNUSUAL = 4 };

PyTypeObject* g_parameter = nullptr;   // torch.nn.Parameter (a subclass of torch.Tensor without a `grad` of its own)
PyTypeObject* g_tensor = nullptr;

// The tensor behind `o`, or null where attribute lookups may not mean what they mean on a plain tensor.
const at::Tensor* plain(PyObject* o) {
  PyTypeObject* t = Py_TYPE(o);
  if (t != g_parameter && t != g_tensor) return nullptr;
  return &THPVariable_Unpack(o);
}

// scan(params, states, param_ptrs, grad_ptrs): `params` and `states` are lists of equal length, the other two
// addresses of int64 arrays as long: where the weights were when the plan was built (read), where the gradients
// were at the last step (0: none; updated unless UNUSUAL is returned).  Returns a mask of the values above.
PyObject* scan(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4 || !PyList_CheckExact(args[0]) || !PyList_CheckExact(args[1])) {
    PyErr_SetString(PyExc_TypeError, "scan(params: list, states: list, param_ptrs: int, grad_ptrs: int)");
    return nullptr;
  }
  const int64_t* was = reinterpret_cast<const int64_t*>(PyLong_AsUnsignedLongLong(args[2]));
  int64_t* grads = reinterpret_cast<int64_t*>(PyLong_AsUnsignedLongLong(args[3]));
  if (PyErr_Occurred()) return nullptr;
  const Py_ssize_t n = PyList_GET_SIZE(args[0]);
  if (PyList_GET_SIZE(args[1]) != n) return PyLong_FromLong(UNUSUAL);
  static thread_local std::vector<int64_t> now;
  now.assign(static_cast<size_t>(n), 0);
  long mask = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const at::Tensor* p = plain(PyList_GET_ITEM(args[0], i));
    PyObject* st = PyList_GET_ITEM(args[1], i);
    if (!p || !PyDict_CheckExact(st) || PyDict_GET_SIZE(st) == 0 || reinterpret_cast<int64_t>(p->const_data_ptr()) != was[i])
      return PyLong_FromLong(UNUSUAL);
    const at::Tensor& g = p->unsafeGetTensorImpl()->grad();   // (Tensor::grad() asks whether it is a leaf, to warn)
    if (g.defined()) {
      if (g.layout() != at::kStrided || g.scalar_type() != p->scalar_type() || !g.is_contiguous())
        return PyLong_FromLong(UNUSUAL);
      now[i] = reinterpret_cast<int64_t>(g.const_data_ptr());
      if (now[i] != 0) mask |= ANY_GRAD;
    }
  }
  if (n > 0 && std::memcmp(grads, now.data(), sizeof(int64_t) * n) != 0) {
    std::memcpy(grads, now.data(), sizeof(int64_t) * n);
    mask |= GRADS_CHANGED;
  }
  return PyLong_FromLong(mask);
}

// entries(state, params, pos): pos[i] (int64 array at an address) = where PyDict_Next finds params[i] in the dict `state`,
// -1 where it is no key.
PyObject* entries(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3 || !PyDict_Check(args[0]) || !PyList_CheckExact(args[1])) {
    PyErr_SetString(PyExc_TypeError, "entries(state: dict, params: list, pos: int)");
    return nullptr;
  }
  int64_t* pos = reinterpret_cast<int64_t*>(PyLong_AsUnsignedLongLong(args[2]));
  if (PyErr_Occurred()) return nullptr;
  try {
    std::unordered_map<PyObject*, int64_t> at;
    PyObject *k, *v;
    for (Py_ssize_t next = 0, here = 0; PyDict_Next(args[0], &next, &k, &v); here = next) at[k] = here;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[1]); ++i) {
      const auto it = at.find(PyList_GET_ITEM(args[1], i));
      pos[i] = it == at.end() ? -1 : it->second;
    }
  } catch (const std::bad_alloc&) {
    return PyErr_NoMemory();
  }
  Py_RETURN_NONE;
}

// settled(params, seen, state, states, pos): whether a group is what its plans were built for: the live list `params`
// holds the tensors of `seen` in their order, and the live dict `state` maps each that has a dict in `states` (not
// None) to that very dict; the others have no gradient.  pos: as `entries` left it.  A key occurs once in a dict, so finding
// (tensor, dict) at the position noted proves the mapping, without hashing the tensor (a call back into Python); a
// dict that was rearranged since only looks changed.
PyObject* settled(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 5 || !PyList_CheckExact(args[1]) || !PyList_CheckExact(args[3]) ||
      PyList_GET_SIZE(args[1]) != PyList_GET_SIZE(args[3])) {
    PyErr_SetString(PyExc_TypeError, "settled(params, seen: list, state, states: list, pos: int)");
    return nullptr;
  }
  const int64_t* pos = reinterpret_cast<const int64_t*>(PyLong_AsUnsignedLongLong(args[4]));
  if (PyErr_Occurred()) return nullptr;
  const Py_ssize_t n = PyList_GET_SIZE(args[1]);
  if (!PyList_CheckExact(args[0]) || PyList_GET_SIZE(args[0]) != n || !PyDict_Check(args[2])) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject *p = PyList_GET_ITEM(args[1], i), *st = PyList_GET_ITEM(args[3], i);
    if (PyList_GET_ITEM(args[0], i) != p) Py_RETURN_FALSE;
    if (st == Py_None) {
      const at::Tensor* t = plain(p);
      if (!t || t->grad().defined()) Py_RETURN_FALSE;
      continue;
    }
    Py_ssize_t at = static_cast<Py_ssize_t>(pos[i]);
    PyObject *k, *v;
    if (at < 0 || !PyDict_Next(args[2], &at, &k, &v) || k != p || v != st) Py_RETURN_FALSE;
    if (!PyDict_CheckExact(st) || PyDict_GET_SIZE(st) == 0) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}

// grads_present(params): 0 no tensor of the list has a gradient, 1 some have, 2 all have (an empty list: 0); -1: unusual.
PyObject* grads_present(PyObject*, PyObject* list) {
  if (!PyList_CheckExact(list)) return PyLong_FromLong(-1);
  const Py_ssize_t n = PyList_GET_SIZE(list);
  Py_ssize_t have = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const at::Tensor* p = plain(PyList_GET_ITEM(list, i));
    if (!p) return PyLong_FromLong(-1);
    have += p->grad().defined() ? 1 : 0;
  }
  return PyLong_FromLong(have == 0 ? 0 : have == n ? 2 : 1);
}

// bump(states, key, grad_ptrs): states[i][key] += 1 for every tensor with a gradient (grad_ptrs as scan left it).
PyObject* bump(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3 || !PyList_CheckExact(args[0])) {
    PyErr_SetString(PyExc_TypeError, "bump(states: list, key: str, grad_ptrs: int)");
    return nullptr;
  }
  const int64_t* grads = reinterpret_cast<const int64_t*>(PyLong_AsUnsignedLongLong(args[2]));
  if (PyErr_Occurred()) return nullptr;
  const Py_ssize_t n = PyList_GET_SIZE(args[0]);
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (grads[i] == 0) continue;
    PyObject* st = PyList_GET_ITEM(args[0], i);
    PyObject* v = PyDict_CheckExact(st) ? PyDict_GetItemWithError(st, args[1]) : nullptr;
    if (!v || !PyLong_CheckExact(v)) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, "bump: a state has no integer counter");
      return nullptr;
    }
    PyObject* next = PyLong_FromLongLong(PyLong_AsLongLong(v) + 1);
    const int rc = next ? PyDict_SetItem(st, args[1], next) : -1;
    Py_XDECREF(next);
    if (rc < 0) return nullptr;
  }
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"scan", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(scan)), METH_FASTCALL, nullptr},
    {"entries", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entries)), METH_FASTCALL, nullptr},
    {"settled", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(settled)), METH_FASTCALL, nullptr},
    {"grads_present", grads_present, METH_O, nullptr},
    {"bump", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bump)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_kaon_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

PyTypeObject* type_of(const char* mod, const char* name) {
  PyObject* m = PyImport_ImportModule(mod);
  PyObject* t = m ? PyObject_GetAttrString(m, name) : nullptr;
  Py_XDECREF(m);
  return reinterpret_cast<PyTypeObject*>(t);   // kept for the life of the process
}

}  // namespace

PyMODINIT_FUNC PyInit__kaon_host() {
  g_tensor = type_of("torch", "Tensor");
  g_parameter = type_of("torch.nn", "Parameter");
  if (!g_tensor || !g_parameter) return nullptr;
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "abi", g_abi + sizeof("kaon host module for ") - 1) < 0) Py_CLEAR(m);
  return m;
}
