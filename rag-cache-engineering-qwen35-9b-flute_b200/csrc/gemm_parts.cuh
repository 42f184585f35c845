// What the tensor-core GEMM kernels share: the description of a merged launch's projections, the
// bulk-load wrapper, the code-field arithmetic of the slab layout, the activation tensor map.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "pairtable.cuh"
#include "tc05.cuh"

namespace b200lut {
namespace {

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

constexpr int kPMaxSeg = 4;             // projections that share x in one launch (Q/K/V/z, gate/up)

// One projection of a launch: its row tiles are the global row tiles [row0, next row0).
struct PersistSeg {
  const uint8_t* packed;
  const uint16_t* lut;
  const uint16_t* bias;
  uint16_t* out;
  long long ldo;
  int row0, n_groups, out_aligned;
  int res_rank;            // rank of the low-rank residual, 0 if the projection has none
  const uint16_t* resA;    // [N, res_rank], row-major
  int t_col0, pad;         // first column of this projection's block of the t matrix
};

// The projection that owns global row tile `row` (static indexing of the parameter block: a
// chain of selects, no local copy).
template <typename P>
__device__ __forceinline__ PersistSeg segment_of_row(const P& p, int row) {
  PersistSeg sd = p.seg[0];
#pragma unroll
  for (int i = 1; i < kPMaxSeg; ++i)
    if (i < p.nsegs && row >= p.seg[i].row0) sd = p.seg[i];
  return sd;
}

// Pair-table address of field i (0..15) of local slab sl (0, 1): the field's 2 * BITS bits
// moved to address bits 8.., joined with the lane base.
template <int BITS>
__device__ __forceinline__ uint32_t slab_field_addr(const uint32_t (&w)[2 * BITS], int sl, int i,
                                                    uint32_t base) {
  if constexpr (BITS == 4) {
    return __byte_perm(w[4 * sl + (i >> 2)], base, 0x7604u | (uint32_t(i & 3) << 4));
  } else {
    constexpr uint32_t kMask = ((1u << (2 * BITS)) - 1u) << 8;
    const int pos = 32 * BITS * sl + 2 * BITS * i, m = pos >> 5, sh = pos & 31;
    uint32_t v;
    if (sh + 2 * BITS > 32) v = __funnelshift_r(w[m], w[(m + 1) % (2 * BITS)], sh - 8);
    else if (sh >= 8) v = w[m] >> (sh - 8);
    else v = w[m] << (8 - sh);
    return (v & kMask) | base;
  }
}

// The 2 * BITS bits of field i (0..15) of local slab sl (0, 1): two codes, the lower one first.
template <int BITS>
__device__ __forceinline__ uint32_t slab_field(const uint32_t (&w)[2 * BITS], int sl, int i) {
  constexpr uint32_t kMask = (1u << (2 * BITS)) - 1u;
  const int pos = 32 * BITS * sl + 2 * BITS * i, m = pos >> 5, sh = pos & 31;
  if (sh + 2 * BITS > 32) return __funnelshift_r(w[m], w[(m + 1) % (2 * BITS)], sh) & kMask;
  return (w[m] >> sh) & kMask;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

inline int encode_x_map(CUtensorMap* map, const void* x, int64_t ldx, int M, int K, int dtype, int NT) {
  EncodeTiledFn enc = encode_fn();
  B200LUT_REQUIRE(enc != nullptr, B200LUT_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {cuuint64_t(K), cuuint64_t(M)};
  const cuuint64_t strides[1] = {cuuint64_t(ldx) * 2};
  const cuuint32_t box[2] = {cuuint32_t(kChunkK), cuuint32_t(NT)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, dtype == B200LUT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                     : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                         2, const_cast<void*>(x), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200LUT_REQUIRE(r == CUDA_SUCCESS, B200LUT_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", int(r));
  return B200LUT_OK;
}

}  // namespace
}  // namespace b200lut
