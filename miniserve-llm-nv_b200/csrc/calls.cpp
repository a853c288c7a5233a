// Calls of the library's entry points from Python.  ctypes builds an object for every argument, 0.12 us each, and the entry points take ten to fifty: a
// call of thirty arguments took 3.7 us and takes 0.4 here, of a pass that is bound by the host where the step has few tokens.
//
// An Entry has the function's address and a trampoline for its types (`trampolines`, a table made from the prototypes in the sources, says which
// name has which).  Numbers are taken as ctypes takes them (integers modulo their size, None as a null pointer), and the interpreter's lock is released
// while the function runs, as there.  Whatever else comes (objects of ctypes, other counts, other types) goes to the ctypes function, which accepts or refuses it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstring>
#include <tuple>
#include <utility>

namespace {

bool take(PyObject* from, void*& to) {
  if (from == Py_None) {
    to = nullptr;
    return true;
  }
  if (!PyLong_Check(from)) return false;
  to = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(from));
  return true;
}
bool take(PyObject* from, int& to) {
  if (!PyLong_Check(from)) return false;
  to = (int)PyLong_AsUnsignedLongLongMask(from);
  return true;
}
bool take(PyObject* from, long long& to) {
  if (!PyLong_Check(from)) return false;
  to = (long long)PyLong_AsUnsignedLongLongMask(from);
  return true;
}
bool take(PyObject* from, float& to) {
  if (!PyFloat_Check(from)) return false;
  to = (float)PyFloat_AS_DOUBLE(from);
  return true;
}
PyObject* give(int v) { return PyLong_FromLong(v); }
PyObject* give(long long v) { return PyLong_FromLongLong(v); }

// The result, or null without an exception set: not these arguments.
using Trampoline = PyObject* (*)(void* function, PyObject* const* arguments, Py_ssize_t count);

template <typename R, typename... A, size_t... I>
PyObject* call_with(void* function, PyObject* const* arguments, std::index_sequence<I...>) {
  std::tuple<A...> values;
  if (!(take(arguments[I], std::get<I>(values)) && ...)) return nullptr;
  R result;
  Py_BEGIN_ALLOW_THREADS
  result = reinterpret_cast<R (*)(A...)>(function)(std::get<I>(values)...);
  Py_END_ALLOW_THREADS
  return give(result);
}
template <typename R, typename... A>
PyObject* call(void* function, PyObject* const* arguments, Py_ssize_t count) {
  if (count != (Py_ssize_t)sizeof...(A)) return nullptr;
  return call_with<R, A...>(function, arguments, std::index_sequence_for<A...>{});
}

using pointer = void*;
using longlong = long long;
struct Named { const char* name; Trampoline trampoline; };
const Named trampolines[] = {
#include TRAMPOLINES
};

struct Entry {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  PyObject *general, *attributes;            // the ctypes function; what a caller sets
  void* function;
  Trampoline trampoline;
};

PyObject* entry_call(PyObject* self, PyObject* const* arguments, size_t flags, PyObject* names) {
  Entry* entry = reinterpret_cast<Entry*>(self);
  if (names == nullptr) {
    PyObject* result = entry->trampoline(entry->function, arguments, PyVectorcall_NARGS(flags));
    if (result != nullptr || PyErr_Occurred()) return result;
  }
  return PyObject_Vectorcall(entry->general, arguments, flags & ~PY_VECTORCALL_ARGUMENTS_OFFSET, names);
}
int entry_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<Entry*>(self)->general);
  Py_VISIT(reinterpret_cast<Entry*>(self)->attributes);
  return 0;
}
int entry_clear(PyObject* self) {
  Py_CLEAR(reinterpret_cast<Entry*>(self)->attributes);
  return 0;
}
void entry_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  Py_CLEAR(reinterpret_cast<Entry*>(self)->general);
  Py_CLEAR(reinterpret_cast<Entry*>(self)->attributes);
  PyObject_GC_Del(self);
}

PyTypeObject entry_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// entry(name, address, ctypes function): the Entry, or None where the name has no trampoline.
PyObject* make_entry(PyObject*, PyObject* arguments) {
  const char* name;
  unsigned long long address;
  PyObject* general;
  if (!PyArg_ParseTuple(arguments, "sKO", &name, &address, &general)) return nullptr;
  for (const Named& named : trampolines) {
    if (std::strcmp(named.name, name) != 0) continue;
    Entry* entry = PyObject_GC_New(Entry, &entry_type);
    if (entry == nullptr) return nullptr;
    entry->vectorcall = entry_call;
    Py_INCREF(general);
    entry->general = general;
    entry->attributes = nullptr;
    entry->function = reinterpret_cast<void*>(address);
    entry->trampoline = named.trampoline;
    PyObject_GC_Track(reinterpret_cast<PyObject*>(entry));
    return reinterpret_cast<PyObject*>(entry);
  }
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"entry", make_entry, METH_VARARGS, "entry(name, address, general) -> callable or None"}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "miniserve_b200_calls", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_miniserve_b200_calls() {
  entry_type.tp_name = "miniserve_b200_calls.Entry";
  entry_type.tp_basicsize = sizeof(Entry);
  entry_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL;
  entry_type.tp_vectorcall_offset = offsetof(Entry, vectorcall);
  entry_type.tp_dictoffset = offsetof(Entry, attributes);
  entry_type.tp_call = PyVectorcall_Call;
  entry_type.tp_getattro = PyObject_GenericGetAttr;
  entry_type.tp_setattro = PyObject_GenericSetAttr;
  entry_type.tp_traverse = entry_traverse;
  entry_type.tp_clear = entry_clear;
  entry_type.tp_dealloc = entry_dealloc;
  if (PyType_Ready(&entry_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
