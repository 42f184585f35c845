// Projections that share x as one launch: Q/K/V side by side, or gate and up under SiLU*mul.
#pragma once

#include "route.h"

namespace b200host {

constexpr int kMaxMerged = 4;

// The residual's first factors of the merged projections, stacked along r so that one projection
// launch serves them all; kept in the owning module's __dict__ and rebuilt when a factor changes.
struct Stack {
  PyObject_HEAD
  int n, cols;                     // layers, columns of t
  Layer* layers[kMaxMerged];       // borrowed for identity; `keep` owns them
  PyObject* keep;
  int offset[kMaxMerged];          // first row of each layer's factor
  at::Tensor* resB;
};
extern PyTypeObject StackType;

inline PyObject* name_stack() { static PyObject* s = PyUnicode_InternFromString("_native_stack"); return s; }

inline Stack* stack_of(PyObject* owner_dict, Layer* const* ls, int n) {
  PyObject* o = PyDict_GetItemWithError(owner_dict, name_stack());
  if (o && Py_TYPE(o) == &StackType) {
    Stack* st = reinterpret_cast<Stack*>(o);
    bool same = st->n == n && st->resB;
    for (int i = 0; same && i < n; ++i) same = st->layers[i] == ls[i];
    if (same) return st;
  }
  Stack* st = PyObject_New(Stack, &StackType);
  if (!st) throw LaunchError(0, "out of memory");
  st->n = n;
  st->resB = nullptr;
  st->keep = PyList_New(0);
  std::vector<at::Tensor> parts;
  int off = 0;
  for (int i = 0; i < n; ++i) {
    st->layers[i] = ls[i];
    PyList_Append(st->keep, reinterpret_cast<PyObject*>(ls[i]));
    st->offset[i] = off;
    if (ls[i]->res) {
      parts.push_back(*ls[i]->resB);
      off += int(ls[i]->resB->size(0));
    }
  }
  st->cols = off;
  st->resB = new at::Tensor(at::cat(parts, 0).contiguous());
  PyDict_SetItem(owner_dict, name_stack(), reinterpret_cast<PyObject*>(st));
  Py_DECREF(st);                   // the dict holds it
  return st;
}

inline bool same_fold(const Layer& a, const Layer& b) {
  if (!a.rotated || !b.rotated) return !a.rotated && !b.rotated;
  return a.rotation && b.rotation && PyObject_RichCompareBool(a.rotation, b.rotation, Py_EQ) == 1;
}

// One dtype, K and fold; every residual of a kind the launch carries.
inline bool mergeable(Layer* const* ls, int n, int M) {
  if (env_on("FLUTE_NO_MERGE")) return false;
  const Layer& a = *ls[0];
  for (int i = 0; i < n; ++i) {
    const Layer& l = *ls[i];
    if (l.kgrouped || l.K != a.K || l.dtype != a.dtype || l.device != a.device || !same_fold(a, l)) return false;
    if (l.res && !residual_served(l, M)) return false;
    if (M > kGemvMaxM && (l.K < 128 || l.two || l.bits != a.bits || l.group != a.group || l.group < 64)) return false;
  }
  return true;
}

// The merged launch into outs[i] (row stride ld): M <= 16 the decode kernels, with EPI_SILU_MUL only
// outs[0] is written; M > 16 the tensor-core GEMM (no epilogue there).
inline void merged_into(PyObject* owner_dict, Layer* const* ls, int n, Rows r, void* const* outs, int64_t ld, int epilogue,
                        const Ctx& c) {
  const Layer& a = *ls[0];
  bool fused = a.rotated, any_res = false;
  for (int i = 0; i < n; ++i) {
    fused = fused && rotation_fuses(*ls[i], r.M);
    any_res = any_res || ls[i]->res;
  }
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
      Stack* st = stack_of(owner_dict, ls, n);
      t = empty({r.M, st->cols}, at::kFloat, c.device);
      float* tp = static_cast<float*>(t.mutable_data_ptr());
      check(b200lut_residual_project(r.ptr, r.ld, r.M, a.K, a.dtype, st->resB->const_data_ptr(), st->cols, tp, st->cols,
                                     c.flags, c.stream));
      for (int i = 0; i < n; ++i)
        if (ls[i]->res) add_residual(&segs[i], *ls[i], tp + st->offset[i], st->cols);
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
