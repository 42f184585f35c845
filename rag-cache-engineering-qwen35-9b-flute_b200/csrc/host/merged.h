// Projections that share x as one launch: Q/K/V side by side, or gate and up under SiLU*mul.
#pragma once

#include "route.h"

namespace b200host {

constexpr int kMaxMerged = 4;

// The residual's first factors of the merged projections, stacked along r so that one projection launch
// serves them all: the record that the Python route keeps in the owning module's __dict__ as "_resB_stack",
// (stack, factors, (address, version) of each factor). Null when there is none for the factors as they are
// now; the Python route then builds it, outside of any stream capture.
inline PyObject* name_stack() { static PyObject* s = PyUnicode_InternFromString("_resB_stack"); return s; }

inline const at::Tensor* residual_stack(PyObject* owner_dict, Layer* const* ls, int n) {
  PyObject* o = PyDict_GetItemWithError(owner_dict, name_stack());
  if (!o || !PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 3) return nullptr;
  PyObject *stack = PyTuple_GET_ITEM(o, 0), *factors = PyTuple_GET_ITEM(o, 1), *marks = PyTuple_GET_ITEM(o, 2);
  if (!THPVariable_Check(stack) || !PyTuple_Check(factors) || !PyTuple_Check(marks) ||
      PyTuple_GET_SIZE(marks) != 2 * PyTuple_GET_SIZE(factors))
    return nullptr;
  Py_ssize_t at_factor = 0;
  for (int i = 0; i < n; ++i) {
    if (!ls[i]->res) continue;
    const at::Tensor& b = *ls[i]->resB;
    if (at_factor >= PyTuple_GET_SIZE(factors)) return nullptr;
    PyObject* f = PyTuple_GET_ITEM(factors, at_factor);
    if (!THPVariable_Check(f) || !THPVariable_Unpack(f).is_same(b)) return nullptr;
    const unsigned long long address = PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(marks, 2 * at_factor));
    const long long version = PyLong_AsLongLong(PyTuple_GET_ITEM(marks, 2 * at_factor + 1));
    if (PyErr_Occurred()) { PyErr_Clear(); return nullptr; }
    if (address != reinterpret_cast<uintptr_t>(b.const_data_ptr()) || version != (b.is_inference() ? -1 : b._version()))
      return nullptr;
    ++at_factor;
  }
  return at_factor == PyTuple_GET_SIZE(factors) ? &THPVariable_Unpack(stack) : nullptr;
}

// The stack that a launch of M rows reads, undefined where there is none to read.
inline at::Tensor stack_or_none(PyObject* owner_dict, Layer* const* ls, int n, int M) {
  bool any_res = false;
  for (int i = 0; i < n; ++i) any_res = any_res || ls[i]->res;
  return any_res && M <= kGemvMaxM ? *residual_stack(owner_dict, ls, n) : at::Tensor();
}

inline bool same_fold(const Layer& a, const Layer& b) {
  if (!a.rotated || !b.rotated) return !a.rotated && !b.rotated;
  return a.rotation && b.rotation && PyObject_RichCompareBool(a.rotation, b.rotation, Py_EQ) == 1;
}

// One dtype, K and fold; every residual of a kind the launch carries (at decode with its stack at hand).
inline bool mergeable(PyObject* owner_dict, Layer* const* ls, int n, int M) {
  if (env_on("FLUTE_NO_MERGE")) return false;
  const Layer& a = *ls[0];
  bool any_res = false;
  for (int i = 0; i < n; ++i) {
    const Layer& l = *ls[i];
    any_res = any_res || l.res;
    if (l.kgrouped || l.K != a.K || l.dtype != a.dtype || l.device != a.device || !same_fold(a, l)) return false;
    if (l.res && !residual_served(l, M)) return false;
    if (M > kGemvMaxM && (l.K < 128 || l.two || l.bits != a.bits || l.group != a.group || l.group < 64)) return false;
  }
  return !any_res || M > kGemvMaxM || residual_stack(owner_dict, ls, n) != nullptr;
}

inline bool merged_rotation_fuses(Layer* const* ls, int n, int M) {
  bool fused = ls[0]->rotated;
  for (int i = 0; i < n; ++i) fused = fused && rotation_fuses(*ls[i], M);
  return fused;
}

// The merged launch into outs[i] (row stride ld): M <= 16 the decode kernels, with EPI_SILU_MUL only
// outs[0] is written; M > 16 the tensor-core GEMM (no epilogue there).
// `fused` is merged_rotation_fuses(), `stack` the residual_stack() of M <= 16. Runs without the interpreter lock.
inline void merged_into(const at::Tensor& stack, Layer* const* ls, int n, Rows r, void* const* outs, int64_t ld, int epilogue,
                        bool fused, const Ctx& c) {
  const Layer& a = *ls[0];
  bool any_res = false;
  for (int i = 0; i < n; ++i) any_res = any_res || ls[i]->res;
  at::Tensor rotated, t;
  if (a.rotated && !fused) {
    rotated = rotate(a, r, c);
    r = Rows{rotated.const_data_ptr(), a.K, r.M};
  }
  b200lut_segment segs[kMaxMerged];
  int64_t rows = 0;
  for (int i = 0; i < n; ++i) {
    segs[i] = segment(*ls[i], outs[i], ld);
    rows += ls[i]->N;
  }
  if (r.M <= kGemvMaxM) {
    if (any_res) {
      const int cols = int(stack.size(0));
      t = empty({r.M, cols}, at::kFloat, c.device);
      float* tp = static_cast<float*>(t.mutable_data_ptr());
      check(b200lut_residual_project(r.ptr, r.ld, r.M, a.K, a.dtype, stack.const_data_ptr(), cols, tp, cols, c.flags,
                                     c.stream));
      for (int i = 0; i < n; ++i) {
        if (!ls[i]->res) continue;
        add_residual(&segs[i], *ls[i], tp, cols);
        tp += ls[i]->resB->size(0);
      }
    }
    if (fused) {
      b200lut_input in = {};
      in.rot_signs = signs_of(a);
      in.awq_scale = awq_of(a);
      check(b200lut_gemv_input(r.ptr, r.ld, r.M, a.K, a.dtype, segs, n, epilogue, 0, nullptr, 0, c.flags, nullptr, &in,
                               c.stream));
    } else {
      check(b200lut_gemv_multi(r.ptr, r.ld, r.M, a.K, a.dtype, segs, n, epilogue, 0, nullptr, 0, c.flags, c.stream));
    }
    return;
  }
  if (any_res) {                       // the projections' t blocks lie side by side in one matrix
    int64_t cols = 0;
    for (int i = 0; i < n; ++i) cols += ls[i]->res ? padded_cols(int(ls[i]->resB->size(0))) : 0;
    t = empty({r.M, cols}, a.scalar, c.device);
    char* tp = static_cast<char*>(t.mutable_data_ptr());
    for (int i = 0; i < n; ++i) {
      if (!ls[i]->res) continue;
      const int R = int(ls[i]->resB->size(0));
      const int64_t w = padded_cols(R);
      check(b200lut_residual_project_rows(r.ptr, r.ld, r.M, a.K, a.dtype, ls[i]->resB->const_data_ptr(), R, tp, cols, int(w),
                                          c.flags, c.stream));
      add_residual(&segs[i], *ls[i], tp, cols);
      tp += 2 * w;
    }
  }
  gemm_launch(r, a.K, a.dtype, segs, n, rows, c);
}

}  // namespace b200host
