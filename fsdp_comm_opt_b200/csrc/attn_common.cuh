// Helpers shared by the attention kernels that were written after the first two generations:
// 4-D tensor maps over packed [B, S, H, D] projections, the TMA load they feed, and a
// bounded mbarrier wait for single-thread roles that also watches a CTA-wide abort flag.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdio>

#include "attn_sm100.cuh"
#include "umma.cuh"

namespace zc {
namespace attn {
using namespace umma;

constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Bounded wait for the TMA and MMA threads: parked in hardware (no issue slots taken from the
// softmax warps on the same scheduler), woken when the phase completes, given up after two
// seconds or as soon as another role has raised `*abort_flag`.
__device__ __forceinline__ bool role_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_wait_parked(bar, parity, abort_flag);
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(ptr);
  }
  return fn;
}

// bf16 [B, S, H, D] with element strides (s_b, s_s, s_h), heads of D contiguous elements, viewed as
// (D, H, S, B); box = one 64-wide slab of `rows` sequence positions of one head, SWIZZLE_128B,
// zero fill outside the tensor
inline bool make_map_bshd(CUtensorMap* m, const void* base, int D, int H, int S, int B, int64_t s_b, int64_t s_s,
                          int64_t s_h, int rows) {
  EncodeFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)s_h * 2, (cuuint64_t)s_s * 2, (cuuint64_t)s_b * 2};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)rows, 1};
  cuuint32_t el[4] = {1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, el,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    fprintf(stderr, "[zc_attn] cuTensorMapEncodeTiled failed (%d): base=%p D=%d H=%d S=%d B=%d rows=%d\n", (int)r,
            base, D, H, S, B, rows);
  return r == CUDA_SUCCESS;
}

}  // namespace attn
}  // namespace zc
