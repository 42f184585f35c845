// Launches of the projection forward: which C entry serves a row count, and its arguments. The rules
// are those of the Python route (palettized_modules.py); what they do not cover returns kNotServed
// before anything has been launched, and the Python route runs.
#pragma once

#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <stdexcept>
#include <string>

#include "layer.h"
#include "scratch.h"

namespace b200host {

constexpr int kGemvMaxM = 16;

// A 2-D view [M, K] of the activation rows.
struct Rows {
  const void* ptr;
  int64_t ld;
  int M;
};

struct Ctx {
  int device;
  cudaStream_t stream;
  int flags;
};

struct LaunchError : std::runtime_error {
  int code;
  LaunchError(int c, const char* m) : std::runtime_error(m), code(c) {}
};

inline void check(int rc) {
  if (rc != B200LUT_OK) throw LaunchError(rc, b200lut_last_error());
}

inline at::Tensor empty(at::IntArrayRef sizes, at::ScalarType st, int device) {
  return at::Tensor(at::detail::empty_cuda(sizes, st, at::Device(at::kCUDA, device), std::nullopt));
}

// x as rows of l.K values in the layer's dtype on the current device; false: not served natively.
inline bool rows_of(const at::Tensor& x, const Layer& l, Rows* r) {
  if (!x.is_cuda() || x.scalar_type() != l.scalar || x.get_device() != l.device || x.dim() < 1) return false;
  if (x.requires_grad() && c10::GradMode::is_enabled()) return false;
  if (l.K <= 0 || x.size(-1) != l.K) return false;
  const int64_t n = x.numel() / l.K;
  if (n < 1 || n > 0x7fffffff) return false;
  int64_t ld = l.K;
  if (!x.is_contiguous()) {
    if (x.dim() != 2 || x.stride(1) != 1 || x.stride(0) % 8 || x.stride(0) < l.K) return false;
    ld = x.stride(0);
  }
  r->ptr = x.const_data_ptr();
  if (reinterpret_cast<uintptr_t>(r->ptr) & 15) return false;
  r->ld = ld;
  r->M = int(n);
  return true;
}

inline b200lut_segment segment(const Layer& l, void* out, int64_t ldo) {
  b200lut_segment s = {};
  s.packed = l.packed->const_data_ptr();
  s.lut = l.lut->const_data_ptr();
  if (l.two) {
    s.packed2 = l.packed2->const_data_ptr();
    s.lut2 = l.lut2->const_data_ptr();
    s.bits2 = l.bits2;
  }
  if (l.bias) s.bias = l.bias->const_data_ptr();
  s.out = out;
  s.ldo = ldo;
  s.N = l.N;
  s.group_size = l.group;
  s.n_groups = l.n_groups;
  s.bits = l.bits;
  return s;
}

inline void add_residual(b200lut_segment* s, const Layer& l, const void* t, int64_t ldt) {
  s->resA = l.resA->const_data_ptr();
  s->res_rank = int(l.resA->size(1));
  s->res_t = t;
  s->res_ldt = ldt;
}

inline const float* signs_of(const Layer& l) { return static_cast<const float*>(l.signs->const_data_ptr()); }
inline const float* awq_of(const Layer& l) { return l.awq ? static_cast<const float*>(l.awq->const_data_ptr()) : nullptr; }

// The residual rides the projection launch.
inline bool residual_served(const Layer& l, int M) {
  if (!l.res_ok) return false;
  if (M <= kGemvMaxM) return true;
  if (l.group < 64 || l.K < 128) return false;
  return !(l.two && l.bits == 4 && l.bits2 == 4);      // the 4 + 4 pair is one one-tile launch
}

inline bool rows_kernel_shape(const Layer& l, int M) { return M <= 8 && l.bits == 4 && !l.two && l.group >= 32; }

// The rotation runs inside the decode launch.
inline bool rotation_fuses(const Layer& l, int M) {
  return l.rotated && rows_kernel_shape(l, M) && !l.res && l.pow2_segments <= 8 && !env_on("FLUTE_NO_FHT_FUSE");
}

enum class Kind { kNotServed, kGemv, kGemm, kTwoStream };

inline Kind linear_kind(const Layer& l, int M) {
  if (l.kgrouped || (l.res && !residual_served(l, M))) return Kind::kNotServed;
  if (M <= kGemvMaxM) return Kind::kGemv;
  if ((l.bits == 4 && (!l.two || l.bits2 == 4)) || (!l.two && l.group >= 64 && l.K >= 128)) return Kind::kGemm;
  if (l.two && l.group >= 64 && l.K >= 128) return Kind::kTwoStream;
  return Kind::kNotServed;
}

// The layer's input fold as its own launch: rows in the layer's dtype, a fresh [M, K] tensor.
inline at::Tensor rotate(const Layer& l, const Rows& r, const Ctx& c) {
  at::Tensor y = empty({r.M, l.K}, l.scalar, c.device);
  check(b200lut_fht(r.ptr, y.mutable_data_ptr(), signs_of(l), awq_of(l), r.M, l.K, r.ld, l.K, l.dtype,
                    l.awq ? B200LUT_FHT_AWQ : B200LUT_FHT_FORWARD, 0, c.stream));
  return y;
}

inline int64_t padded_cols(int rank) { return 64 * ((int64_t(rank) + 63) / 64); }

// `n` projections that share x as one prefill launch, with the split schedule's scratch.
inline void gemm_launch(const Rows& r, int K, int dtype, const b200lut_segment* segs, int n, int64_t rows, const Ctx& c) {
  const size_t need = segs[0].packed2 ? 0 : b200lut_gemm_launch_workspace_bytes(r.M, int(rows), K, segs[0].bits, segs[0].group_size);
  at::Tensor ws;
  if (need) ws = scratch_pool().get(Scratch::kSplit, c.device, c.stream, need);
  void* wp = need ? ws.mutable_data_ptr() : nullptr;
  const size_t wb = need ? size_t(ws.numel()) : 0;
  if (n == 1) check(b200lut_gemm_ws(r.ptr, r.ld, r.M, K, dtype, segs, B200LUT_EPI_NONE, c.flags, wp, wb, c.stream));
  else check(b200lut_gemm_multi(r.ptr, r.ld, r.M, K, dtype, segs, n, c.flags, wp, wb, c.stream));
}

// out[M, N] (row stride ldo) = the layer on rows r; linear_kind() has said it is served, `fused` is
// rotation_fuses(). Runs without the interpreter lock.
inline void linear_into(const Layer& l, Rows r, void* out, int64_t ldo, bool fused, const Ctx& c) {
  const Kind kind = linear_kind(l, r.M);
  at::Tensor rotated, t;
  if (l.rotated && !fused) {
    rotated = rotate(l, r, c);
    r = Rows{rotated.const_data_ptr(), l.K, r.M};
  }
  b200lut_segment s = segment(l, out, ldo);
  if (l.res) {
    const int R = int(l.resB->size(0));
    if (kind == Kind::kGemv) {
      t = empty({r.M, R}, at::kFloat, c.device);
      check(b200lut_residual_project(r.ptr, r.ld, r.M, l.K, l.dtype, l.resB->const_data_ptr(), R,
                                     static_cast<float*>(t.mutable_data_ptr()), R, c.flags, c.stream));
      add_residual(&s, l, t.const_data_ptr(), R);
    } else {
      const int64_t cols = padded_cols(R);
      t = empty({r.M, cols}, l.scalar, c.device);
      check(b200lut_residual_project_rows(r.ptr, r.ld, r.M, l.K, l.dtype, l.resB->const_data_ptr(), R,
                                          t.mutable_data_ptr(), cols, int(cols), c.flags, c.stream));
      add_residual(&s, l, t.const_data_ptr(), cols);
    }
  }
  if (fused) {
    b200lut_input in = {};
    in.rot_signs = signs_of(l);
    in.awq_scale = awq_of(l);
    check(b200lut_gemv_input(r.ptr, r.ld, r.M, l.K, l.dtype, &s, 1, B200LUT_EPI_NONE, 0, nullptr, 0, c.flags, nullptr,
                             &in, c.stream));
  } else if (kind == Kind::kGemv) {
    check(b200lut_gemv_multi(r.ptr, r.ld, r.M, l.K, l.dtype, &s, 1, B200LUT_EPI_NONE, 0, nullptr, 0, c.flags, c.stream));
  } else if (kind == Kind::kGemm) {
    gemm_launch(r, l.K, l.dtype, &s, 1, l.N, c);
  } else {
    const size_t need = b200lut_gemm_two_stream_bytes(r.M, l.N);
    at::Tensor ws = scratch_pool().get(Scratch::kTwoStream, c.device, c.stream, need);
    // two launches that share the scratch: another thread's on this stream must not come between them
    const std::lock_guard<std::mutex> both(scratch_pool().two_stream_launches());
    check(b200lut_gemm_two_stream(r.ptr, r.ld, r.M, l.K, l.dtype, &s, c.flags, ws.mutable_data_ptr(),
                                  size_t(ws.numel()), c.stream));
  }
}

}  // namespace b200host
