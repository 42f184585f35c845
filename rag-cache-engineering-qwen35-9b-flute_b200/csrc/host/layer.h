// Native description of one palettized projection, kept in its module's __dict__ as "_native".
//
// The module stays the owner of its state: a description remembers which objects it was built from and
// what its tensors looked like (storage, type, shape), and is only used while the module still holds
// exactly those, so .to(), drop_blob(), a replaced palette or a changed option all lead back to the
// Python route, which builds a new one.
#pragma once

#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <string>
#include <vector>

#include "../../../include/b200_lut.h"

namespace b200host {

// What a tensor looks like from outside: its address, type, sizes and strides. A tensor can change all of
// them and stay the same object (set_, t_, an assignment to .data).
struct Look {
  const void* data = nullptr;
  at::ScalarType type = at::kFloat;
  c10::SmallVector<int64_t, 4> sizes, strides;
};

// One entry of the module (or of the module it is tied to) that the description depends on.
struct Watch {
  PyObject* key;        // interned name
  PyObject* value;      // the object found under it when the description was built, or null
  PyObject* dict;       // the other module's __dict__, or null: the module's own
  bool in_params;       // looked up in _parameters instead of _buffers / __dict__
  bool tensor;
  Look look;
};

struct Layer {
  PyObject_HEAD
  bool ready;
  int N, K, bits, bits2, group, n_groups, device, dtype;     // dtype: B200LUT_BF16 / B200LUT_F16
  at::ScalarType scalar;
  bool two, res, res_ok, rotated, kgrouped;
  int pow2_segments;
  PyObject* rotation;                       // key of the fold (equal keys: the same rotation), or null
  at::Tensor *packed, *lut, *packed2, *lut2, *bias, *resA, *resB, *signs, *awq;
  std::vector<Watch>* watches;
};

inline PyObject* name_buffers() { static PyObject* s = PyUnicode_InternFromString("_buffers"); return s; }
inline PyObject* name_params() { static PyObject* s = PyUnicode_InternFromString("_parameters"); return s; }
inline PyObject* name_modules() { static PyObject* s = PyUnicode_InternFromString("_modules"); return s; }
inline PyObject* name_native() { static PyObject* s = PyUnicode_InternFromString("_native"); return s; }

// Where a module keeps `key`: a buffer shadows a plain attribute (both exist for optional tensors).
inline PyObject* lookup(PyObject* dict, PyObject* key, bool in_params) {
  PyObject* group = PyDict_GetItemWithError(dict, in_params ? name_params() : name_buffers());
  if (group && PyDict_Check(group)) {
    PyObject* v = PyDict_GetItemWithError(group, key);
    if (v) return v;
  }
  return PyDict_GetItemWithError(dict, key);
}

inline Look look_of(const at::Tensor& t) {
  Look l;
  l.data = t.const_data_ptr();
  l.type = t.scalar_type();
  l.sizes.assign(t.sizes().begin(), t.sizes().end());
  l.strides.assign(t.strides().begin(), t.strides().end());
  return l;
}

inline bool looks_the_same(const at::Tensor& t, const Look& l) {
  return t.const_data_ptr() == l.data && t.scalar_type() == l.type && t.sizes() == at::IntArrayRef(l.sizes) &&
         t.strides() == at::IntArrayRef(l.strides);
}

inline bool current(const Layer& l, PyObject* dict) {
  for (const Watch& w : *l.watches) {
    PyObject* v = lookup(w.dict ? w.dict : dict, w.key, w.in_params);
    if (v != w.value) return false;
    if (w.tensor && !looks_the_same(THPVariable_Unpack(v), w.look)) return false;
  }
  return true;
}

extern PyTypeObject LayerType;

// The module's description if it may be used, else null (never sets an exception).
inline Layer* layer_of(PyObject* dict) {
  PyObject* o = PyDict_GetItemWithError(dict, name_native());
  if (!o || Py_TYPE(o) != &LayerType) return nullptr;
  Layer* l = reinterpret_cast<Layer*>(o);
  if (!l->ready) return nullptr;
  if (!current(*l, dict)) {
    PyDict_SetItem(dict, name_native(), Py_None);     // the Python route builds a new one
    return nullptr;
  }
  return l;
}

// Lets other Python threads run while this one allocates and launches (a launch blocks when the stream's
// queue is full, and what drains the queue may be a host function that needs the interpreter). Whatever
// the launches use is held by the caller: layers by Held, tensors by reference.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};
struct Held {
  PyObject* o;
  explicit Held(void* p) : o(static_cast<PyObject*>(p)) { Py_XINCREF(o); }
  ~Held() { Py_XDECREF(o); }
  Held(const Held&) = delete;
};

// Child module `name` of a module's __dict__: its own __dict__ (borrowed), or null.
inline PyObject* child_dict(PyObject* dict, PyObject* name, PyObject** child = nullptr) {
  PyObject* mods = PyDict_GetItemWithError(dict, name_modules());
  PyObject* m = mods && PyDict_Check(mods) ? PyDict_GetItemWithError(mods, name) : nullptr;
  if (child) *child = m;
  if (!m) return nullptr;
  PyObject* d = PyObject_GenericGetDict(m, nullptr);
  if (!d) { PyErr_Clear(); return nullptr; }
  Py_DECREF(d);                                       // the object keeps it
  return d;
}

// The Python route's rule: "1", "true" or "True", whitespace around it aside.
inline bool env_on(const char* name) {
  const char* e = std::getenv(name);
  if (!e) return false;
  std::string v(e);
  v.erase(0, std::min(v.find_first_not_of(" \t\r\n\v\f"), v.size()));
  v.erase(v.find_last_not_of(" \t\r\n\v\f") + 1);
  return v == "1" || v == "true" || v == "True";
}

}  // namespace b200host
