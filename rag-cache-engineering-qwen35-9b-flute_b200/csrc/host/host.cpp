// Native forward of the palettized modules (extension module _b200lut_host).
//
// An eager forward of a small projection is bound by the host: the Python route (argument checks,
// segment tables through ctypes, device guards) took 29-31 us around a 5-9 us kernel. The functions
// here do the same work for the shapes and dtypes that need no conversion: look the module's native
// description up, allocate the outputs, call the C entries. They return None, having launched
// nothing, when a call is not one of those; the Python route then runs.
#include <cstring>

#include "merged.h"

using namespace b200host;

namespace b200host {

// ---- Layer objects ----------------------------------------------------------------------
static void layer_clear(Layer* l) {
  for (at::Tensor* t : {l->packed, l->lut, l->packed2, l->lut2, l->bias, l->resA, l->resB, l->signs, l->awq}) delete t;
  if (l->watches) {
    for (Watch& w : *l->watches) {
      Py_XDECREF(w.key);
      Py_XDECREF(w.value);
      Py_XDECREF(w.dict);
    }
    delete l->watches;
  }
  Py_XDECREF(l->rotation);
}
static void layer_dealloc(PyObject* o) {
  layer_clear(reinterpret_cast<Layer*>(o));
  PyObject_Free(o);
}
// A copied or pickled module builds its own description: this object travels as None.
static PyObject* reduce_none(PyObject*, PyObject*) {
  return Py_BuildValue("(O())", reinterpret_cast<PyObject*>(Py_TYPE(Py_None)));
}
static PyMethodDef reduce_methods[] = {{"__reduce__", reduce_none, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};

PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

static int ready_type(PyTypeObject* t, const char* name, size_t size, destructor d) {
  t->tp_name = name;
  t->tp_basicsize = Py_ssize_t(size);
  t->tp_dealloc = d;
  t->tp_flags = Py_TPFLAGS_DEFAULT;
  t->tp_methods = reduce_methods;
  return PyType_Ready(t);
}

static at::Tensor* tensor_or_null(PyObject* o) {
  return o && THPVariable_Check(o) ? new at::Tensor(THPVariable_Unpack(o)) : nullptr;
}
static long int_of(PyObject* d, const char* key) {
  PyObject* v = PyDict_GetItemString(d, key);
  return v ? PyLong_AsLong(v) : 0;
}

static PyObject* g_library_error = nullptr;   // LibraryError(code, message) of the ctypes layer

template <typename F>
static PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const LaunchError& e) {
    if (!PyErr_Occurred()) {
      PyObject* args = Py_BuildValue("(is)", e.code, e.what());
      if (args) PyErr_SetObject(g_library_error ? g_library_error : PyExc_RuntimeError, args);
      Py_XDECREF(args);
    }
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// Fills `l` (zeroed) from the spec of bind(); null with an exception set, or a C++ exception, where it cannot.
static PyObject* describe(Layer* l, PyObject* dict, PyObject* spec) {
  auto t = [&](const char* k) { return tensor_or_null(PyDict_GetItemString(spec, k)); };
  l->packed = t("packed"); l->lut = t("lut"); l->packed2 = t("packed2"); l->lut2 = t("lut2");
  l->bias = t("bias"); l->resA = t("resA"); l->resB = t("resB"); l->signs = t("signs"); l->awq = t("awq");
  l->watches = new std::vector<Watch>();
  l->rotation = PyDict_GetItemString(spec, "rotation");
  Py_XINCREF(l->rotation);
  l->N = int(int_of(spec, "N")); l->K = int(int_of(spec, "K"));
  l->bits = int(int_of(spec, "bits")); l->bits2 = int(int_of(spec, "bits2"));
  l->group = int(int_of(spec, "group_size")); l->n_groups = int(int_of(spec, "n_groups"));
  l->two = l->packed2 && l->lut2;
  l->res = l->resA && l->resB;
  l->kgrouped = int_of(spec, "kgrouped") != 0;
  l->rotated = l->signs != nullptr;
  l->pow2_segments = __builtin_popcount(unsigned(l->K));
  l->ready = l->packed && l->lut && l->lut->is_cuda() &&
             (l->lut->scalar_type() == at::kBFloat16 || l->lut->scalar_type() == at::kHalf);
  l->device = l->ready ? l->lut->get_device() : -1;
  l->scalar = l->ready ? l->lut->scalar_type() : at::kFloat;
  l->dtype = l->scalar == at::kHalf ? B200LUT_F16 : B200LUT_BF16;
  l->res_ok = false;
  if (l->res) {
    const at::Tensor &A = *l->resA, &B = *l->resB;
    auto fine = [&](const at::Tensor& x) {
      return x.is_cuda() && x.scalar_type() == l->scalar && x.is_contiguous() &&
             (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15) == 0;
    };
    l->res_ok = A.dim() == 2 && B.dim() == 2 && A.size(1) <= 1024 && A.size(1) % 8 == 0 && fine(A) && fine(B);
  }
  PyObject* tied = PyDict_GetItemString(spec, "tied");
  PyObject* names[3] = {PyDict_GetItemString(spec, "watch"), PyDict_GetItemString(spec, "watch_params"),
                        tied ? PyDict_GetItemString(spec, "watch_tied") : nullptr};
  for (int g = 0; g < 3; ++g) {
    if (!names[g]) continue;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(names[g]); ++i) {
      PyObject* key = PyTuple_GET_ITEM(names[g], i);
      Py_INCREF(key);
      PyUnicode_InternInPlace(&key);
      PyObject* v = lookup(g == 2 ? tied : dict, key, g == 1);
      Py_XINCREF(v);
      if (g == 2) Py_INCREF(tied);
      l->watches->push_back(Watch{key, v, g == 2 ? tied : nullptr, g == 1, v && THPVariable_Check(v), Look()});
      if (l->watches->back().tensor) l->watches->back().look = look_of(THPVariable_Unpack(v));
    }
  }
  return PyErr_Occurred() ? nullptr : reinterpret_cast<PyObject*>(l);
}

// bind(module_dict, spec): spec is a dict with the layer's tensors and integers, "watch" (names in
// the module whose objects it was built from) and "watch_params"; "tied" and "watch_tied" name what
// belongs to another module, by its __dict__.
static PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyDict_Check(a[0]) || !PyDict_Check(a[1])) {
    PyErr_SetString(PyExc_TypeError, "bind(module_dict, spec)");
    return nullptr;
  }
  PyObject *dict = a[0], *spec = a[1];
  Layer* l = PyObject_New(Layer, &LayerType);
  if (!l) return nullptr;
  std::memset(reinterpret_cast<char*>(l) + sizeof(PyObject), 0, sizeof(Layer) - sizeof(PyObject));
  PyObject* done = guarded([&]() -> PyObject* { return describe(l, dict, spec); });
  if (!done) Py_DECREF(l);
  return done;
}

// ---- forwards ---------------------------------------------------------------------------------------
// The launch context of tensors on `device`; false when that is not the current device.
static bool context(int device, bool pdl, Ctx* c) {
  if (int(c10::cuda::current_device()) != device) return false;
  c->device = device;
  c->stream = c10::cuda::getCurrentCUDAStream(c10::DeviceIndex(device)).stream();
  c->flags = pdl ? B200LUT_FLAG_PDL : 0;
  return true;
}

// [..., cols] shaped like x up to its last dimension
static at::Tensor output_like(const at::Tensor& x, int64_t cols, const Layer& l) {
  c10::SmallVector<int64_t, 6> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = cols;
  return empty(sizes, l.scalar, l.device);
}

static bool arguments(const char* what, PyObject* const* a, Py_ssize_t n) {
  if (n == 3 && PyDict_Check(a[0])) return true;
  PyErr_Format(PyExc_TypeError, "%s(module_dict, x, pdl)", what);
  return false;
}

static PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arguments("linear", a, n)) return nullptr;
  if (!THPVariable_Check(a[1])) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    Layer* l = layer_of(a[0]);
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    Rows r;
    Ctx c;
    if (!l || !rows_of(x, *l, &r) || linear_kind(*l, r.M) == Kind::kNotServed || !context(l->device, a[2] == Py_True, &c))
      Py_RETURN_NONE;
    const bool fused = rotation_fuses(*l, r.M);
    const Held held(l);
    at::Tensor out;
    {
      const WithoutGil free;
      out = output_like(x, l->N, *l);
      linear_into(*l, r, out.mutable_data_ptr(), l->N, fused, c);
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// Q/K/V: outputs side by side in one [..., sum N] tensor.
static PyObject* qkv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arguments("qkv", a, n)) return nullptr;
  if (!THPVariable_Check(a[1])) Py_RETURN_NONE;
  static PyObject* names[3] = {PyUnicode_InternFromString("q_proj"), PyUnicode_InternFromString("k_proj"),
                               PyUnicode_InternFromString("v_proj")};
  return guarded([&]() -> PyObject* {
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    Layer* ls[3];
    int64_t total = 0;
    for (int i = 0; i < 3; ++i) {
      PyObject* d = child_dict(a[0], names[i]);
      ls[i] = d ? layer_of(d) : nullptr;
      if (!ls[i]) Py_RETURN_NONE;
      total += ls[i]->N;
    }
    Rows r;
    Ctx c;
    if (!rows_of(x, *ls[0], &r) || !mergeable(a[0], ls, 3, r.M) || !context(ls[0]->device, a[2] == Py_True, &c)) Py_RETURN_NONE;
    const bool fused = merged_rotation_fuses(ls, 3, r.M);
    const at::Tensor stack = stack_or_none(a[0], ls, 3, r.M);
    const Held h0(ls[0]), h1(ls[1]), h2(ls[2]);
    at::Tensor out;
    {
      const WithoutGil free;
      out = output_like(x, total, *ls[0]);
      char* p = static_cast<char*>(out.mutable_data_ptr());
      void* outs[3];
      for (int i = 0; i < 3; p += 2 * int64_t(ls[i]->N), ++i) outs[i] = p;
      merged_into(stack, ls, 3, r, outs, total, B200LUT_EPI_NONE, fused, c);
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// down(silu(gate(x)) * up(x)); the caller has checked that the activation is SiLU.
static PyObject* mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arguments("mlp", a, n)) return nullptr;
  if (!THPVariable_Check(a[1])) Py_RETURN_NONE;
  static PyObject* names[3] = {PyUnicode_InternFromString("gate_proj"), PyUnicode_InternFromString("up_proj"),
                               PyUnicode_InternFromString("down_proj")};
  return guarded([&]() -> PyObject* {
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    Layer* ls[3];
    for (int i = 0; i < 3; ++i) {
      PyObject* d = child_dict(a[0], names[i]);
      ls[i] = d ? layer_of(d) : nullptr;
      if (!ls[i]) Py_RETURN_NONE;
    }
    const Layer& down = *ls[2];
    const int I = ls[0]->N;
    Rows r;
    Ctx c;
    if (!rows_of(x, *ls[0], &r) || ls[1]->N != I || down.K != I || down.dtype != ls[0]->dtype ||
        down.device != ls[0]->device || !mergeable(a[0], ls, 2, r.M) || linear_kind(down, r.M) == Kind::kNotServed ||
        !context(down.device, a[2] == Py_True, &c))
      Py_RETURN_NONE;
    const bool fused = merged_rotation_fuses(ls, 2, r.M), down_fused = rotation_fuses(down, r.M);
    const at::Tensor stack = stack_or_none(a[0], ls, 2, r.M);
    const Held h0(ls[0]), h1(ls[1]), h2(ls[2]);
    at::Tensor out;
    {
      const WithoutGil free;
      at::Tensor g = empty({r.M, I}, down.scalar, down.device), u;
      void* outs[2] = {g.mutable_data_ptr(), nullptr};
      if (r.M > kGemvMaxM) {
        u = empty({r.M, I}, down.scalar, down.device);
        outs[1] = u.mutable_data_ptr();
      }
      merged_into(stack, ls, 2, r, outs, I, r.M > kGemvMaxM ? B200LUT_EPI_NONE : B200LUT_EPI_SILU_MUL, fused, c);
      if (r.M > kGemvMaxM) check(b200lut_silu_mul(outs[0], outs[1], r.M, I, I, I, down.dtype, c.stream));
      out = output_like(x, down.N, down);
      linear_into(down, Rows{outs[0], I, r.M}, out.mutable_data_ptr(), down.N, down_fused, c);
    }
    return THPVariable_Wrap(std::move(out));
  });
}

static PyObject* kgrouped(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arguments("kgrouped", a, n)) return nullptr;
  if (!THPVariable_Check(a[1])) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    Layer* l = layer_of(a[0]);
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    Rows r;
    Ctx c;
    if (!l || !l->kgrouped || !rows_of(x, *l, &r) || !context(l->device, a[2] == Py_True, &c)) Py_RETURN_NONE;
    const Held held(l);
    at::Tensor out;
    {
      const WithoutGil free;
      out = output_like(x, l->N, *l);
      const void* bias = l->bias ? l->bias->const_data_ptr() : nullptr;
      if (r.M <= kGemvMaxM) {
        // without a scratch the entry refuses the shapes that need one: the Python route brings it
        const int rc = b200lut_gemv_kgrouped(r.ptr, r.ld, r.M, l->K, l->dtype, l->packed->const_data_ptr(),
                                             l->lut->const_data_ptr(), bias, l->N, l->bits, out.mutable_data_ptr(), l->N, 0,
                                             nullptr, 0, c.stream);
        if (rc == B200LUT_ERR_WORKSPACE) out.reset();
        else check(rc);
      } else {
        const size_t need = b200lut_gemm_workspace_bytes(r.M, l->N, l->K);
        at::Tensor ws;
        if (need) ws = scratch_pool().get(Scratch::kSplit, c.device, c.stream, need);
        check(b200lut_gemm_kgrouped(r.ptr, r.ld, r.M, l->K, l->dtype, l->packed->const_data_ptr(), l->lut->const_data_ptr(),
                                    bias, l->N, l->bits, out.mutable_data_ptr(), l->N, c.flags,
                                    need ? ws.mutable_data_ptr() : nullptr, need ? size_t(ws.numel()) : 0, c.stream));
      }
    }
    if (!out.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
  });
}

// embed(module_dict, ids, bad): rows of the table; `bad` (int32 [1]) is set when an id is out of range.
static PyObject* embed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arguments("embed", a, n)) return nullptr;
  if (!THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    Layer* l = layer_of(a[0]);
    const at::Tensor &ids = THPVariable_Unpack(a[1]), &bad = THPVariable_Unpack(a[2]);
    Ctx c;
    if (!l || l->rotated || (l->res && !l->res_ok) || !ids.is_cuda() || ids.get_device() != l->device ||
        ids.scalar_type() != at::kLong || !ids.is_contiguous() || ids.numel() == 0 || !context(l->device, false, &c))
      Py_RETURN_NONE;
    c10::SmallVector<int64_t, 6> sizes(ids.sizes().begin(), ids.sizes().end());
    sizes.push_back(l->K);
    const Held held(l);
    at::Tensor out;
    {
      const WithoutGil free;
      out = empty(sizes, l->scalar, l->device);
      b200lut_segment s = segment(*l, out.mutable_data_ptr(), l->K);
      if (l->res) {
        s.resA = l->resA->const_data_ptr();
        s.res_rank = int(l->resA->size(1));
      }
      check(b200lut_embed_gather_checked(ids.const_data_ptr<int64_t>(), ids.numel(), l->K, l->dtype, &s,
                                         l->res ? l->resB->const_data_ptr() : nullptr, 0,
                                         static_cast<int32_t*>(bad.mutable_data_ptr()), c.stream));
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// fht(x, signs or None, scale or None, mode, block): the transform of x's last dimension.
static PyObject* fht(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "fht(x, signs, scale, mode, block)");
    return nullptr;
  }
  if (!THPVariable_Check(a[0])) Py_RETURN_NONE;
  const long mode = PyLong_AsLong(a[3]), block = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor& x = THPVariable_Unpack(a[0]);
    Ctx c;
    if (!x.is_cuda() || x.dim() < 1 || !x.is_contiguous() || x.numel() == 0 || !context(x.get_device(), false, &c))
      Py_RETURN_NONE;
    const int64_t K = x.size(-1), M = x.numel() / K;
    if (M > 0x7fffffff || K > 0x7fffffff) Py_RETURN_NONE;
    int dtype;
    if (x.scalar_type() == at::kBFloat16) dtype = B200LUT_BF16;
    else if (x.scalar_type() == at::kHalf) dtype = B200LUT_F16;
    else if (x.scalar_type() == at::kFloat) dtype = 2;
    else Py_RETURN_NONE;
    const float* v[2] = {nullptr, nullptr};
    for (int i = 0; i < 2; ++i) {
      if (a[1 + i] == Py_None) continue;
      if (!THPVariable_Check(a[1 + i])) Py_RETURN_NONE;
      const at::Tensor& t = THPVariable_Unpack(a[1 + i]);
      if (!t.is_cuda() || t.get_device() != c.device || t.scalar_type() != at::kFloat || !t.is_contiguous() || t.numel() != K)
        Py_RETURN_NONE;
      v[i] = static_cast<const float*>(t.const_data_ptr());
    }
    at::Tensor y;
    {
      const WithoutGil free;
      y = empty(x.sizes(), x.scalar_type(), c.device);
      check(b200lut_fht(x.const_data_ptr(), y.mutable_data_ptr(), v[0], v[1], int(M), int(K), K, K, dtype, int(mode),
                        int(block), c.stream));
    }
    return THPVariable_Wrap(std::move(y));
  });
}

// workspace(device, bytes): the split schedule's scratch of the current stream (zero-filled when new).
static PyObject* workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "workspace(device, bytes)");
    return nullptr;
  }
  const long device = PyLong_AsLong(a[0]);
  const size_t bytes = PyLong_AsSize_t(a[1]);
  if (PyErr_Occurred()) return nullptr;
  return guarded([&]() -> PyObject* {
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(c10::DeviceIndex(device)).stream();
    at::Tensor t;
    {
      const WithoutGil free;      // the pool's lock is only ever taken without the interpreter's
      t = scratch_pool().get(Scratch::kSplit, int(device), st, bytes);
    }
    return THPVariable_Wrap(std::move(t));
  });
}

static PyObject* set_library_error(PyObject*, PyObject* type) {
  Py_INCREF(type);
  Py_XDECREF(g_library_error);
  g_library_error = type;
  Py_RETURN_NONE;
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL, nullptr
static PyMethodDef methods[] = {{"bind", FAST(bind)},
                                {"linear", FAST(linear)},
                                {"qkv", FAST(qkv)},
                                {"mlp", FAST(mlp)},
                                {"kgrouped", FAST(kgrouped)},
                                {"embed", FAST(embed)},
                                {"fht", FAST(fht)},
                                {"workspace", FAST(workspace)},
                                {"set_library_error", set_library_error, METH_O, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200lut_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace b200host

PyMODINIT_FUNC PyInit__b200lut_host(void) {
  if (ready_type(&LayerType, "_b200lut_host.Layer", sizeof(Layer), layer_dealloc) < 0) return nullptr;
  return PyModule_Create(&module);
}
