// What the two-SM kernel and the one of small products share: eight columns of C at a time, and the operands' tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdint>
#include <cstdio>

namespace zc {

// f[j] += bias[col + j], j = 0..7 (col is a multiple of 8; the last group of a ragged N is read element-wise)
__device__ __forceinline__ void add_bias8(const __nv_bfloat16* bias, int64_t col, int64_t N, float (&f)[8]) {
  if (col + 8 <= N) {
    const uint4 b = *reinterpret_cast<const uint4*>(bias + col);
    const __nv_bfloat162* bb = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(bb[j]);
      f[2 * j] += t.x;
      f[2 * j + 1] += t.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (col + j < N) f[j] += __bfloat162float(bias[col + j]);
  }
}

// f += the eight old bf16 values of C
__device__ __forceinline__ void add_old8(const uint4& old, float (&f)[8]) {
  const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 o2 = __bfloat1622float2(ob[j]);
    f[2 * j] += o2.x;
    f[2 * j + 1] += o2.y;
  }
}
__device__ __forceinline__ uint4 round8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162 a0 = __floats2bfloat162_rn(f[0], f[1]), a1 = __floats2bfloat162_rn(f[2], f[3]);
  __nv_bfloat162 a2 = __floats2bfloat162_rn(f[4], f[5]), a3 = __floats2bfloat162_rn(f[6], f[7]);
  v.x = *reinterpret_cast<uint32_t*>(&a0);
  v.y = *reinterpret_cast<uint32_t*>(&a1);
  v.z = *reinterpret_cast<uint32_t*>(&a2);
  v.w = *reinterpret_cast<uint32_t*>(&a3);
  return v;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}
// 2-D bf16 row-major tensor [rows][cols] with rows `ld` elements apart; box = (box_cols inner, box_rows),
// 128B swizzle.  Elements past `cols` in a row (padding up to ld) are outside the map and read as zeros.
inline bool make_map(CUtensorMap* m, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t el[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, el,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    fprintf(stderr, "[zc_gemm] cuTensorMapEncodeTiled failed (%d): ptr=%p rows=%lld cols=%lld box=(%d,%d)\n",
            (int)r, ptr, (long long)rows, (long long)cols, box_cols, box_rows);
  return r == CUDA_SUCCESS;
}

// The launcher of csrc/gemm_small.cu, and in how many parts it would cut K (cut_k: it may): 0 when the product is not one of
// its own, or expected to take longer there than `other_us`.
int gemm_small_parts(int64_t M, int64_t N, int64_t K, bool cut_k, double other_us);
int gemm_small_launch(const void* A, const void* B, void* C, const void* bias, int64_t M, int64_t N, int64_t K, int64_t lda,
                      int64_t ldb, int64_t ldc, int a_major, int b_major, int accumulate, int parts, int* status,
                      cudaStream_t st);

}  // namespace zc
