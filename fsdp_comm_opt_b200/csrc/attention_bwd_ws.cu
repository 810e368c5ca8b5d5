// Causal GQA attention backward for sm_100a.  Two kernels: the warp-specialised kernel below
// (ZC_ATTN_BWD=ws) and, further down, the key-row kernel that is the default.
//
// One CTA (320 threads) per (128-key block, kv head, batch); it loops over the query heads of the
// group and over the query blocks at or below the diagonal, with dK and dV accumulating in TMEM.
//   warp 0      TMA producer: K, V once; then Q_i and dO_i per iteration (4-D tensor maps,
//               SWIZZLE_128B, zero fill past S).  The next iteration's loads start as soon as the
//               MMAs that read the buffers have completed, and overlap the dQ reduction below.
//   warp 1      MMA issuer: S = Q K^T and dP = dO V^T, then dV += P^T dO, dK += dS^T Q and
//               dQ_i = dS K (P / dS are read through MN-major descriptors: no transposes)
//   warps 2-9   256 compute threads: two threads share a query row and take 64 columns each;
//               P = exp2(S*c - lse), dS = P (dP - delta) scale, written to smem as bf16; then the
//               dQ_i tile is read from TMEM and reduced into the fp32 accumulator with red.add
// TMEM (512 columns): dK | dV | R0 (S, later dQ_i) | R1 (dP).  Shared memory: K V Q dO P dS, 32 KB
// each.  Every wait is bounded; a timed-out role raises a CTA-wide abort flag.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "attn_sm100.cuh"
#include "launch_util.h"
#include "umma.cuh"

namespace zc {
namespace bws {
using namespace umma;

constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// global[tile at (c0..c3)] += smem tile  (element-wise fp32 add done by the TMA unit; rows past the
// tensor's extent are clipped)
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2,
                                                  int c3) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(map), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void bulk_commit_and_wait_read() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ uint64_t desc_k(uint32_t base, int k) {
  return smem_desc(base + (k >> 2) * 16384 + (k & 3) * 32, 16, 1024);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t base, int k) { return smem_desc(base + k * 2048, 16384, 1024); }

__device__ __forceinline__ void store_chunk32(uint8_t* tile, int row, int col0, const float (&v)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int col = col0 + q * 8;
    __nv_bfloat162 a = __floats2bfloat162_rn(v[q * 8 + 0], v[q * 8 + 1]);
    __nv_bfloat162 b = __floats2bfloat162_rn(v[q * 8 + 2], v[q * 8 + 3]);
    __nv_bfloat162 c = __floats2bfloat162_rn(v[q * 8 + 4], v[q * 8 + 5]);
    __nv_bfloat162 d = __floats2bfloat162_rn(v[q * 8 + 6], v[q * 8 + 7]);
    uint4 u;
    u.x = *reinterpret_cast<uint32_t*>(&a);
    u.y = *reinterpret_cast<uint32_t*>(&b);
    u.z = *reinterpret_cast<uint32_t*>(&c);
    u.w = *reinterpret_cast<uint32_t*>(&d);
    *reinterpret_cast<uint4*>(tile + (col >> 6) * 16384 + sw128_off(row, (col >> 3) & 7)) = u;
  }
}

struct BwdParams {
  const float *lse, *delta;
  float* dq_acc;
  __nv_bfloat16 *dk, *dv;
  int B, S, Hq, Hkv;
  int64_t dks0, dks1, dks2, dvs0, dvs1, dvs2;
  float scale;
  int* status;
  int parts;  // CTAs that share a key block's query heads (the key-row kernel)
};

template <int D>
__global__ void __launch_bounds__(320, 1) attn_bwd_ws_kernel(const __grid_constant__ CUtensorMap mapQ,
                                                             const __grid_constant__ CUtensorMap mapK,
                                                             const __grid_constant__ CUtensorMap mapV,
                                                             const __grid_constant__ CUtensorMap mapdO,
                                                             const __grid_constant__ CUtensorMap mapdQ,
                                                             const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int TILE = 128 * D * 2;
  constexpr int SLABS = D / 64;
  uint8_t* sK = smem;
  uint8_t* sV = smem + 1 * 32768;
  uint8_t* sQ = smem + 2 * 32768;
  uint8_t* sdO = smem + 3 * 32768;
  uint8_t* sP = smem + 4 * 32768;
  uint8_t* sdS = smem + 5 * 32768;
  __shared__ uint64_t kv_full, qdo_full, qdo_empty, sdp_full, pds_full, dq_full, dq_empty;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nkb = gridDim.x;
  const int jb = blockIdx.x;
  const int hk = blockIdx.y, b = blockIdx.z;
  const int group = p.Hq / p.Hkv;
  const int k0 = jb * 128;
  const int iters = group * (nkb - jb);
  if (tid == 0) {
    mbar_init(&kv_full, 1);
    mbar_init(&qdo_full, 1);
    mbar_init(&qdo_empty, 1);
    mbar_init(&sdp_full, 1);
    mbar_init(&pds_full, 1);
    mbar_init(&dq_full, 1);
    mbar_init(&dq_empty, 1);
    mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm_dk = tmem_base, tm_dv = tmem_base + 128, tm_r0 = tmem_base + 256, tm_r1 = tmem_base + 384;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(&kv_full, 2 * TILE);
#pragma unroll
      for (int sl = 0; sl < SLABS; ++sl) {
        tma_load_4d(sK + sl * 16384, &mapK, &kv_full, sl * 64, hk, k0, b);
        tma_load_4d(sV + sl * 16384, &mapV, &kv_full, sl * 64, hk, k0, b);
      }
      for (int it = 0; it < iters; ++it) {
        const int h = hk * group + it / (nkb - jb);
        const int q0 = (jb + it % (nkb - jb)) * 128;
        if (!mbar_wait_relaxed(&qdo_empty, (it & 1) ^ 1)) { s_abort = 1; break; }
        mbar_expect_tx(&qdo_full, 2 * TILE);
#pragma unroll
        for (int sl = 0; sl < SLABS; ++sl) {
          tma_load_4d(sQ + sl * 16384, &mapQ, &qdo_full, sl * 64, h, q0, b);
          tma_load_4d(sdO + sl * 16384, &mapdO, &qdo_full, sl * 64, h, q0, b);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t id_s = idesc_bf16(128, 128, MAJOR_K, MAJOR_K);
      const uint32_t id_kv = idesc_bf16(128, D, MAJOR_MN, MAJOR_MN);
      const uint32_t id_dq = idesc_bf16(128, D, MAJOR_K, MAJOR_MN);
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aQ = smem_u32(sQ), adO = smem_u32(sdO), aP = smem_u32(sP),
                     adS = smem_u32(sdS);
      bool ok = mbar_wait_relaxed(&kv_full, 0);
      for (int it = 0; it < iters && ok; ++it) {
        if (!(ok = mbar_wait_relaxed(&qdo_full, it & 1))) break;
        if (!(ok = mbar_wait_relaxed(&dq_empty, (it & 1) ^ 1))) break;
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) mma_bf16(tm_r0, desc_k(aQ, k), desc_k(aK, k), id_s, k != 0);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) mma_bf16(tm_r1, desc_k(adO, k), desc_k(aV, k), id_s, k != 0);
        mma_commit(&sdp_full);
        if (!(ok = mbar_wait_relaxed(&pds_full, it & 1))) break;
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 8; ++k) mma_bf16(tm_dv, desc_mn(aP, k), desc_mn(adO, k), id_kv, (it | k) != 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) mma_bf16(tm_dk, desc_mn(adS, k), desc_mn(aQ, k), id_kv, (it | k) != 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) mma_bf16(tm_r0, desc_k(adS, k), desc_mn(aK, k), id_dq, k != 0);
        mma_commit(&dq_full);
        mma_commit(&qdo_empty);
      }
      if (!ok) s_abort = 1;
    }
  } else {
    const int cw = warp - 2;
    const int quarter = warp & 3;
    const int half = cw >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32);
    const float sl2 = p.scale * LOG2E;
    for (int it = 0; it < iters; ++it) {
      const int h = hk * group + it / (nkb - jb);
      const int ib = jb + it % (nkb - jb);
      const int q0 = ib * 128;
      const int row = q0 + r;
      float lse2 = 0.f, dl = 0.f;
      if (row < p.S) {
        lse2 = __ldg(p.lse + ((int64_t)b * p.Hq + h) * p.S + row) * LOG2E;
        dl = __ldg(p.delta + ((int64_t)b * p.Hq + h) * p.S + row);
      }
      if (!mbar_wait(&sdp_full, it & 1)) s_abort = 1;
      tc_fence_after_sync();
      const bool diag = (ib == jb) || (q0 + 128 > p.S) || (k0 + 128 > p.S);
#pragma unroll 1
      for (int c = half * 64; c < half * 64 + 64; c += 32) {
        uint32_t rs[32], rp[32];
        tmem_ld32(tmem_addr(tm_r0, lane_base, c), rs);
        tmem_ld32(tmem_addr(tm_r1, lane_base, c), rp);
        tmem_ld_wait();
        float pv[32], ds[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float e = exp2f(__uint_as_float(rs[i]) * sl2 - lse2);
          if (diag && (k0 + c + i > row || k0 + c + i >= p.S || row >= p.S)) e = 0.f;
          pv[i] = e;
          ds[i] = e * (__uint_as_float(rp[i]) - dl) * p.scale;
        }
        store_chunk32(sP, r, c, pv);
        store_chunk32(sdS, r, c, ds);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(1, 256);
      if (s_abort) break;
      if (tid == 64) mbar_arrive(&pds_full);
      // ---- dQ_i partial: this thread reduces its row's columns [half*D/2, half*D/2 + D/2) ---------
      if (!mbar_wait(&dq_full, it & 1)) s_abort = 1;
      tc_fence_after_sync();
      // The dV/dK/dQ MMAs have finished reading P and dS, so their 64 KB of shared memory are
      // free: stage the fp32 dQ_i tile there (32-column slabs, 128B swizzle) and let one thread add
      // it into the global accumulator with bulk tensor reductions instead of 4096 red.add per CTA.
#pragma unroll 1
      for (int c = half * (D / 2); c < half * (D / 2) + D / 2; c += 32) {
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm_r0, lane_base, c), rr);
        tmem_ld_wait();
        uint8_t* slab = sP + (c >> 5) * 16384;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<uint4*>(slab + sw128_off(r, i)) =
              make_uint4(rr[4 * i], rr[4 * i + 1], rr[4 * i + 2], rr[4 * i + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      named_bar_sync(1, 256);
      if (s_abort) break;
      if (tid == 64) {
#pragma unroll
        for (int t = 0; t < D / 32; ++t) tma_reduce_add_4d(&mapdQ, sP + t * 16384, t * 32, h, q0, b);
        bulk_commit_and_wait_read();
        mbar_arrive(&dq_empty);
      }
    }
    if (!s_abort) {
      // all MMAs into dK / dV have completed (dq_full of the last iteration covers them)
      const int krow = k0 + r;
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t tmx = which ? tm_dv : tm_dk;
        __nv_bfloat16* dst = which ? p.dv + b * p.dvs0 + (int64_t)krow * p.dvs1 + hk * p.dvs2
                                   : p.dk + b * p.dks0 + (int64_t)krow * p.dks1 + hk * p.dks2;
#pragma unroll 1
        for (int c = half * (D / 2); c < half * (D / 2) + D / 2; c += 32) {
          uint32_t rr[32];
          tmem_ld32(tmem_addr(tmx, lane_base, c), rr);
          tmem_ld_wait();
          if (krow < p.S) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              __nv_bfloat162 a0 = __floats2bfloat162_rn(__uint_as_float(rr[i]), __uint_as_float(rr[i + 1]));
              __nv_bfloat162 a1 = __floats2bfloat162_rn(__uint_as_float(rr[i + 2]), __uint_as_float(rr[i + 3]));
              __nv_bfloat162 a2 = __floats2bfloat162_rn(__uint_as_float(rr[i + 4]), __uint_as_float(rr[i + 5]));
              __nv_bfloat162 a3 = __floats2bfloat162_rn(__uint_as_float(rr[i + 6]), __uint_as_float(rr[i + 7]));
              uint4 u;
              u.x = *reinterpret_cast<uint32_t*>(&a0);
              u.y = *reinterpret_cast<uint32_t*>(&a1);
              u.z = *reinterpret_cast<uint32_t*>(&a2);
              u.w = *reinterpret_cast<uint32_t*>(&a3);
              *reinterpret_cast<uint4*>(dst + c + i) = u;
            }
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(p.status, 5);
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeFn encode_fn() {
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
// bf16 [B, S, H, D] with element strides (s_b, s_s, s_h), viewed as (D, H, S, B); box = one 64-wide
// slab of `rows` sequence positions of one head
static bool make_map4(CUtensorMap* m, const void* base, int D, int H, int S, int B, int64_t s_b, int64_t s_s,
                      int64_t s_h, int rows = 128) {
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
    fprintf(stderr, "[zc_attn_bwd] cuTensorMapEncodeTiled failed (%d): base=%p D=%d H=%d S=%d B=%d\n", (int)r, base, D,
            H, S, B);
  return r == CUDA_SUCCESS;
}

// fp32 accumulator [B, S, Hq, D] viewed as (D, Hq, S, B); box = 32 columns x `rows` rows of one head
static bool make_map4_f32(CUtensorMap* m, const void* base, int D, int H, int S, int B, int rows = 128,
                          bool swizzle = true) {
  EncodeFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 4, (cuuint64_t)H * D * 4, (cuuint64_t)S * H * D * 4};
  cuuint32_t box[4] = {32, 1, (cuuint32_t)rows, 1};
  cuuint32_t el[4] = {1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(base), dims, strides, box, el,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fprintf(stderr, "[zc_attn_bwd] fp32 tensor map failed (%d)\n", (int)r);
  return r == CUDA_SUCCESS;
}

struct Scratch {
  int* status = nullptr;
};
static Scratch g_scratch[64];

__global__ void __launch_bounds__(256) delta_kernel(const __nv_bfloat16* __restrict__ o,
                                                    const __nv_bfloat16* __restrict__ dout, float* __restrict__ delta,
                                                    int B, int S, int Hq, int D) {
  const int64_t wid = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t total = (int64_t)B * S * Hq;
  if (wid >= total) return;
  const __nv_bfloat16* po = o + wid * D;
  const __nv_bfloat16* pd = dout + wid * D;
  float acc = 0.f;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(po + i));
    const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(pd + i));
    acc += a.x * g.x + a.y * g.y;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (lane == 0) {
    const int64_t bs = wid / Hq;
    const int hh = (int)(wid % Hq);
    delta[((bs / S) * Hq + hh) * S + bs % S] = acc;
  }
}

__global__ void __launch_bounds__(256) dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                                         int64_t rows, int Hq, int D, int64_t s_bs, int64_t s_h) {
  const int vpr = D / 4;
  const int64_t total = rows * Hq * vpr;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
    const int v = (int)(i % vpr);
    const int h = (int)((i / vpr) % Hq);
    const int64_t r = i / ((int64_t)vpr * Hq);
    const float4 f = *reinterpret_cast<const float4*>(acc + (r * Hq + h) * D + v * 4);
    __nv_bfloat162 a = __floats2bfloat162_rn(f.x, f.y), c = __floats2bfloat162_rn(f.z, f.w);
    uint2 u;
    u.x = *reinterpret_cast<uint32_t*>(&a);
    u.y = *reinterpret_cast<uint32_t*>(&c);
    *reinterpret_cast<uint2*>(dq + r * s_bs + h * s_h + v * 4) = u;
  }
}

// delta[b, h, s] = sum_d o * dout and the cleared fp32 accumulator of dQ in one pass: D / 8 threads a (row, head), 16
// bytes of each input and 32 of the accumulator a thread.  Bound by HBM; 4096 x 32 x 128: 20.5 us, with a warp a
// (row, head), four-byte loads and a memset 28.5 + 12.2.
template <int D>
__global__ void __launch_bounds__(256) delta_zero_kernel(const uint4* o, const uint4* dout,
                                                         float* __restrict__ delta, float4* __restrict__ dq_acc, int S,
                                                         int Hq, int64_t total) {
  chain();
  constexpr int T = D / 8;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  float acc = 0.f;
  if (i < total * T) {
    const uint4 a = o[i], g = dout[i];
    dq_acc[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f);
    dq_acc[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&av[k]));
      const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gv[k]));
      acc += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int k = T / 2; k > 0; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
  if (i < total * T && threadIdx.x % T == 0) {
    const int64_t row = i / T, bs = row / Hq, b = bs / S;
    delta[(b * Hq + row % Hq) * S + bs % S] = acc;
  }
}

// acc [rows, Hq, D] fp32 -> dq bf16 (16-byte aligned, element strides multiples of 8): eight elements a thread.
// Bound by HBM; 4096 x 32 x 128: 24 us with four elements and 64-bit divisions a thread, 13 so.
template <int D>
__global__ void __launch_bounds__(256) dq_convert8_kernel(const float4* acc, __nv_bfloat16* __restrict__ dq,
                                                          int64_t units, uint32_t Hq, int64_t s_bs, int64_t s_h) {
  chain();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= units) return;
  const float4 a = ld_once(acc + 2 * i), c = ld_once(acc + 2 * i + 1);
  const uint32_t rh = (uint32_t)(i / (D / 8)), r = rh / Hq, h = rh - r * Hq;
  uint4 v;
  __nv_bfloat162 p0 = __floats2bfloat162_rn(a.x, a.y), p1 = __floats2bfloat162_rn(a.z, a.w);
  __nv_bfloat162 p2 = __floats2bfloat162_rn(c.x, c.y), p3 = __floats2bfloat162_rn(c.z, c.w);
  v.x = *reinterpret_cast<uint32_t*>(&p0);
  v.y = *reinterpret_cast<uint32_t*>(&p1);
  v.z = *reinterpret_cast<uint32_t*>(&p2);
  v.w = *reinterpret_cast<uint32_t*>(&p3);
  *reinterpret_cast<uint4*>(dq + r * s_bs + h * s_h + (i % (D / 8)) * 8) = v;
}

}  // namespace bws

// =================================================================================================
// Key-row ("transposed") backward, head dimensions 64 and 128: the default.
//
// One CTA (512 threads) per (128-key block, kv head, batch); 128 queries an iteration, with the KEY index on the
// TMEM lanes:
//   S^T  = K Q^T,  dP^T = V dO^T                     (128 keys x 128 queries each)
//   P^T  = exp2(S^T c - lse[q])                      bf16 into TMEM, over the scores that it came from
//   dS^T = P^T (dP^T - delta[q]) scale               bf16 into shared memory
//   dV  += P^T dO (A from TMEM),  dK += dS^T Q       (accumulate in TMEM over all iterations)
//   dQ   = dS K                                      (dS^T read MN-major; at head dimension 128 over dP^T)
// Roles, by warpgroup (registers are moved with setmaxnreg, 48 + 2 x 152 + 160 = the launch's 4 x 128 a thread):
//   0     warp 0: TMA producer (K, V once, then Q two iterations ahead and dO one or two), warp 1: MMA issuer,
//         warp 2: lse and delta of the iteration's queries into shared memory
//   1, 2  P^T and dS^T; a thread owns a key row and 64 of the queries
//   3     drains dQ: TMEM -> registers -> 16 KB pieces of 32 dimensions in shared memory -> bulk tensor reduction
//         into the fp32 accumulator [B, S, Hq, D]
// Order of the MMAs: dV(i), S(i+1), dQ(i), dK(i), dP(i+1): the exponentials of i+1 run beside dQ(i) and dK(i), dS(i+1)
// beside dV(i+1) and S(i+2), the drain of dQ(i) beside dK(i).  (At head dimension 64, where dQ has columns of its own,
// dP(i+1) ahead of dQ(i) was slower: 1927 against 1754 us for 2 x 8192 keys and 25 heads.)
// What bounds it: the issue of the MMAs, which take 70 to 110 clocks each whatever their width (an operand's bytes
// move at about 70 B per clock from shared memory), 40 of them an iteration at head dimension 128 and 32 at 64.  With 64
// queries an iteration and P^T in shared memory it was 64 for the same work.  16384 keys, 32 / 8 heads of 128: 7200 ->
// 4884 us; 8 x 1024 keys, 25 heads of 64: 259 -> 180, and 175 -> 168 since dK and dV are stored in whole lines.
// CTAs are numbered heaviest first (key block 0 has the most query blocks below the diagonal).
namespace bkt {
using namespace bws;

template <int D>
struct Cfg {
  static constexpr int TILE = 128 * D * 2;               // K, V, Q or dO
  static constexpr int DO_STAGES = D == 128 ? 1 : 2;
  static constexpr bool ALIAS = D == 128;                // dQ takes the columns of dP^T
  static constexpr int TILES = 4 + DO_STAGES;            // K, V, 2 Q, dO
  static constexpr int DS = TILES * TILE, STAGE = DS + 32768, STAT = STAGE + 32768, BARS = STAT + 2048;
  static constexpr int SMEM = BARS + 256;
  static constexpr int TM_S = 0, TM_DP = 128, TM_DK = 256, TM_DV = 256 + D, TM_DQ = ALIAS ? TM_DP : 256 + 2 * D;
};
struct Bars {
  uint64_t kv_full, q_full[2], q_empty[2], do_full[2], do_empty[2], s_full, dp_full, p_full, ds_full, dv_done, dq_full,
      dq_empty, stat_full[2], stat_empty[2], all_done;
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(Bars) <= 256, "the barriers' space");

// MMAs whose shared-memory operands are given by the low words of their descriptors: 1024 bytes between groups of eight
// rows, SWIZZLE_128B and the sm_100 version field are the same for all of this kernel's
constexpr uint32_t DESC_HI = (1024 >> 4) | 1u << 14 | 2u << 29;
__device__ __forceinline__ void mma_ss(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "mov.b64 da, {%1, %5};\n"
      "mov.b64 db, {%2, %5};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
      "}\n" ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "n"(DESC_HI)
      : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t tmem_a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 db;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "mov.b64 db, {%2, %5};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n"
      "}\n" ::"r"(d), "r"(tmem_a), "r"(b), "r"(idesc), "r"(accumulate), "n"(DESC_HI)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// four floats at the shared-memory address `at` of CTA `rank` of the cluster
__device__ __forceinline__ float4 ld_cluster(uint32_t at, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(at), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// SHARED: a cluster of p.parts CTAs works on one key block.  (The kernel of its own without it: the few instructions more
// before a CTA's first load cost 3 % where CTAs are short.)
template <int D, bool SHARED>
__global__ void __launch_bounds__(512, 1) attn_bwd_kt_kernel(const __grid_constant__ CUtensorMap mapQ,
                                                             const __grid_constant__ CUtensorMap mapK,
                                                             const __grid_constant__ CUtensorMap mapV,
                                                             const __grid_constant__ CUtensorMap mapdO,
                                                             const __grid_constant__ CUtensorMap mapdQ,
                                                             const BwdParams p) {
  using C = Cfg<D>;
  // No static shared memory: the dynamic part starts at the (1024-byte aligned) beginning of the block's window
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) atomicExch(p.status, 9);
    return;
  }
  uint8_t* sK = smem;  // [128 keys x D] bf16, D / 64 column slabs of 16 KB
  uint8_t* sV = smem + C::TILE;
  uint8_t* sQ = smem + 2 * C::TILE;
  uint8_t* sdO = smem + 4 * C::TILE;
  uint8_t* sdS = smem + C::DS;        // [128 keys x 128 queries] bf16, two slabs of 64 queries
  uint8_t* sStage = smem + C::STAGE;  // 2 x [128 queries x 32 dims] fp32
  float* s_stat = reinterpret_cast<float*>(smem + C::STAT);  // per stage: -lse * log2(e) of 128 queries, their -delta * scale
  Bars& m = *reinterpret_cast<Bars*>(smem + C::BARS);
  volatile int* s_abort = &m.abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_jb = p.Hkv * p.B;
  const int parts = SHARED ? p.parts : 1;
  const int part = SHARED ? blockIdx.x % parts : 0, unit = SHARED ? blockIdx.x / parts : blockIdx.x;
  const int jb = unit / per_jb;
  const int hk = (unit % per_jb) % p.Hkv, b = (unit % per_jb) / p.Hkv;
  const int group = p.Hq / p.Hkv / parts;  // query heads of this CTA
  const int h0 = hk * (p.Hq / p.Hkv) + part * group;
  const int k0 = jb * 128;
  const int nqb = (p.S + 127) / 128;
  const int iters = group * (nqb - jb);  // query blocks at or below this key block's diagonal
  if (tid == 0) {
    mbar_init(&m.kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&m.q_full[i], 1);
      mbar_init(&m.q_empty[i], 1);
      mbar_init(&m.do_full[i], 1);
      mbar_init(&m.do_empty[i], 1);
      mbar_init(&m.stat_full[i], 1);
      mbar_init(&m.stat_empty[i], 8);
    }
    mbar_init(&m.s_full, 1);
    mbar_init(&m.dp_full, 1);
    mbar_init(&m.p_full, 8);
    mbar_init(&m.ds_full, 8);
    mbar_init(&m.dv_done, 1);
    mbar_init(&m.dq_full, 1);
    mbar_init(&m.dq_empty, 4);
    mbar_init(&m.all_done, 1);
    mbar_fence_init();
    m.abort = 0;
  }
  if (warp == 1) {
    tmem_alloc(&m.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = m.tmem_base;
  chain_wait();
  if (warp == 1) chain_next();  // which has its TMEM
  // bounded wait: parked in hardware, woken when the phase completes, given up after two seconds or when another role
  // raised the abort flag
  auto role_wait = [&](uint64_t* bar, uint32_t parity) -> bool { return mbar_wait_parked(bar, parity, s_abort); };

  if (warp < 4) {
    regs_dec<48>();
    if (warp == 0 && lane == 0) {
      mbar_expect_tx(&m.kv_full, 2 * C::TILE);
#pragma unroll
      for (int sl = 0; sl < D / 64; ++sl) {
        tma_load_4d(sK + sl * 16384, &mapK, &m.kv_full, sl * 64, hk, k0, b);
        tma_load_4d(sV + sl * 16384, &mapV, &m.kv_full, sl * 64, hk, k0, b);
      }
      int h = h0, ib = jb;
      for (int i = 0; i < iters; ++i) {
        const int sq = i & 1, sd = i % C::DO_STAGES;
        if (!role_wait(&m.q_empty[sq], ((i >> 1) & 1) ^ 1)) { *s_abort = 1; break; }
        mbar_expect_tx(&m.q_full[sq], C::TILE);
#pragma unroll
        for (int sl = 0; sl < D / 64; ++sl)
          tma_load_4d(sQ + sq * C::TILE + sl * 16384, &mapQ, &m.q_full[sq], sl * 64, h, ib * 128, b);
        if (!role_wait(&m.do_empty[sd], ((i / C::DO_STAGES) & 1) ^ 1)) { *s_abort = 1; break; }
        mbar_expect_tx(&m.do_full[sd], C::TILE);
#pragma unroll
        for (int sl = 0; sl < D / 64; ++sl)
          tma_load_4d(sdO + sd * C::TILE + sl * 16384, &mapdO, &m.do_full[sd], sl * 64, h, ib * 128, b);
        if (++ib == nqb) { ib = jb; ++h; }
      }
    } else if (warp == 1 && lane == 0) {
      const uint32_t id_s = idesc_bf16(128, 128, MAJOR_K, MAJOR_K);    // S^T, dP^T
      const uint32_t id_kv = idesc_bf16(128, D, MAJOR_K, MAJOR_MN);    // dV, dK
      const uint32_t id_dq = idesc_bf16(128, D, MAJOR_MN, MAJOR_MN);   // dQ
      // Operand descriptors at offset 0; an MMA adds (byte offset >> 4) to the start-address field (shared memory is
      // below 256 KB, the 14-bit field never carries).  K-major: 16 KB slabs of 64 elements; MN-major: the same slabs.
      uint32_t dK_k = (uint32_t)smem_desc(smem_u32(sK), 16, 1024), dV_k = (uint32_t)smem_desc(smem_u32(sV), 16, 1024);
      uint32_t dQ_k = (uint32_t)smem_desc(smem_u32(sQ), 16, 1024), ddO_k = (uint32_t)smem_desc(smem_u32(sdO), 16, 1024);
      uint32_t ddS_k = (uint32_t)smem_desc(smem_u32(sdS), 16, 1024);
      constexpr uint32_t MN = ((16384 - 16) >> 4) << 16;  // added, K-major -> MN-major: the slab stride
      auto off_k = [](int k) { return (uint32_t)(((k >> 2) * 16384 + (k & 3) * 32) >> 4); };
      auto off_mn = [](int k) { return (uint32_t)((k * 2048) >> 4); };
      auto issue_s = [&](int i) {  // S^T(i)
        const uint32_t dq = dQ_k + (uint32_t)((i & 1) * (C::TILE >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k) mma_ss(tm + C::TM_S, dK_k + off_k(k), dq + off_k(k), id_s, k != 0);
        mma_commit(&m.s_full);
      };
      auto issue_dp = [&](int i) {  // dP^T(i)
        const uint32_t dd = ddO_k + (uint32_t)((i % C::DO_STAGES) * (C::TILE >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k) mma_ss(tm + C::TM_DP, dV_k + off_k(k), dd + off_k(k), id_s, k != 0);
        mma_commit(&m.dp_full);
      };
      auto run = [&]() -> bool {
        if (!role_wait(&m.kv_full, 0) || !role_wait(&m.q_full[0], 0)) return false;
        tc_fence_after_sync();
        issue_s(0);
        if (!role_wait(&m.do_full[0], 0)) return false;
        tc_fence_after_sync();
        issue_dp(0);
        for (int i = 0; i < iters; ++i) {
          // the sums with constants are made where they are used, not kept over the loop in registers that are not there
          asm volatile("" : "+r"(dK_k), "+r"(dV_k), "+r"(dQ_k), "+r"(ddO_k), "+r"(ddS_k));
          const int sq = i & 1, sd = i % C::DO_STAGES;
          if (!role_wait(&m.p_full, i & 1)) return false;
          tc_fence_after_sync();
          // dV += P^T dO: the thread that owns queries [64 g, 64 g + 64) keeps its P at column 64 g
          const uint32_t dd = (ddO_k + MN) + (uint32_t)(sd * (C::TILE >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            mma_ts(tm + C::TM_DV, tm + C::TM_S + (uint32_t)((k >> 2) * 64 + (k & 3) * 8), dd + off_mn(k), id_kv, (i | k) != 0);
          mma_commit(&m.dv_done);
          mma_commit(&m.do_empty[sd]);
          if (i + 1 < iters) {  // S^T(i+1) overwrites P^T(i)
            if (!role_wait(&m.q_full[(i + 1) & 1], ((i + 1) >> 1) & 1) || !role_wait(&m.dv_done, i & 1)) return false;
            tc_fence_after_sync();
            issue_s(i + 1);
          }
          if (!role_wait(&m.ds_full, i & 1)) return false;
          if (!C::ALIAS && i > 0 && !role_wait(&m.dq_empty, (i - 1) & 1)) return false;
          tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            mma_ss(tm + C::TM_DQ, (ddS_k + MN) + off_mn(k), (dK_k + MN) + off_mn(k), id_dq, k != 0);
          mma_commit(&m.dq_full);
          const uint32_t dq = (dQ_k + MN) + (uint32_t)(sq * (C::TILE >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k) mma_ss(tm + C::TM_DK, ddS_k + off_k(k), dq + off_mn(k), id_kv, (i | k) != 0);
          mma_commit(&m.q_empty[sq]);
          if (i + 1 < iters) {  // at head dimension 128 dP^T(i+1) overwrites dQ(i)
            if (!role_wait(&m.do_full[(i + 1) % C::DO_STAGES], ((i + 1) / C::DO_STAGES) & 1)) return false;
            if (C::ALIAS && !role_wait(&m.dq_empty, i & 1)) return false;
            tc_fence_after_sync();
            issue_dp(i + 1);
          }
        }
        mma_commit(&m.all_done);
        return true;
      };
      if (!run()) *s_abort = 1;
    } else if (warp == 2) {
      int h = h0, ib = jb;
      for (int i = 0; i < iters; ++i) {
        const int st = i & 1;
        const int64_t row = ((int64_t)b * p.Hq + h) * p.S;
        float vl[4], vd[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          // queries past the end: P = exp2(0 - inf) = 0
          const int q = ib * 128 + lane * 4 + k;
          vl[k] = q < p.S ? -p.lse[row + q] * LOG2E : -CUDART_INF_F;
          vd[k] = q < p.S ? -p.delta[row + q] * p.scale : 0.f;
        }
        const bool ok = role_wait(&m.stat_empty[st], ((i >> 1) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, ok)) { *s_abort = 1; break; }
        float4* dst = reinterpret_cast<float4*>(s_stat + st * 256);
        dst[lane] = make_float4(vl[0], vl[1], vl[2], vl[3]);
        dst[32 + lane] = make_float4(vd[0], vd[1], vd[2], vd[3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&m.stat_full[st]);
        if (++ib == nqb) { ib = jb; ++h; }
      }
    }
  } else if (warp < 12) {
    regs_inc<152>();
    const int quarter = warp & 3;          // TMEM lane quarter this warp may access
    const int half = (warp - 4) >> 2;      // which 64 of the 128 query columns
    const int r = quarter * 32 + lane;     // key row of the tile == TMEM lane
    const uint32_t lane_base = (uint32_t)(quarter * 32);
    const int c0 = half * 64;
    const uint64_t sl22 = pack2(p.scale * LOG2E, p.scale * LOG2E), scale2 = pack2(p.scale, p.scale);
    int ib = jb;
    bool fail = false;
    for (int i = 0; i < iters; ++i) {
      const int st = i & 1;
      fail = !mbar_wait_parked(&m.stat_full[st], (i >> 1) & 1, s_abort) || !mbar_wait_parked(&m.s_full, i & 1, s_abort);
      if (__any_sync(0xffffffffu, fail || *s_abort)) { fail = true; break; }
      tc_fence_after_sync();
      uint32_t e[2][32];
      tmem_ld32(tmem_addr(tm + C::TM_S, lane_base, c0), e[0]);
      tmem_ld32(tmem_addr(tm + C::TM_S, lane_base, c0 + 32), e[1]);
      tmem_ld_wait();
      const ulonglong2* nl = reinterpret_cast<const ulonglong2*>(s_stat + st * 256 + c0);        // pairs of floats
      const ulonglong2* nd = reinterpret_cast<const ulonglong2*>(s_stat + st * 256 + 128 + c0);
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        const ulonglong2 l4 = nl[g];
        uint32_t* v = &e[g >> 3][(g & 7) * 4];
        float x[4];
        unpack2(fma2(pack2(__uint_as_float(v[0]), __uint_as_float(v[1])), sl22, l4.x), x[0], x[1]);
        unpack2(fma2(pack2(__uint_as_float(v[2]), __uint_as_float(v[3])), sl22, l4.y), x[2], x[3]);
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = __float_as_uint(exp2f(x[k]));
      }
      if (ib == jb) {  // the block on the diagonal; keys past the end of the sequence lie below it
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (r > c0 + c) e[c >> 5][c & 31] = 0u;
      }
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 32; ++c)
        pk[c] = pack_bf16(__uint_as_float(e[c >> 4][(c & 15) * 2]), __uint_as_float(e[c >> 4][(c & 15) * 2 + 1]));
      tmem_st32(tmem_addr(tm + C::TM_S, lane_base, c0), pk);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&m.p_full);
      __syncwarp();
      // dp_full(i) also tells that dQ(i-1) and dK(i-1), issued before it, have read dS^T(i-1)
      fail = !mbar_wait_parked(&m.dp_full, i & 1, s_abort);
      if (__any_sync(0xffffffffu, fail || *s_abort)) { fail = true; break; }
      tc_fence_after_sync();
      uint8_t* slab = sdS + half * 16384;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t dp[32];
        tmem_ld32(tmem_addr(tm + C::TM_DP, lane_base, c0 + c * 32), dp);
        tmem_ld_wait();
        uint32_t ds[16];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const ulonglong2 d4 = nd[c * 8 + g];
          float x[4];
          unpack2(mul2(pack2(__uint_as_float(e[c][4 * g]), __uint_as_float(e[c][4 * g + 1])),
                       fma2(pack2(__uint_as_float(dp[4 * g]), __uint_as_float(dp[4 * g + 1])), scale2, d4.x)), x[0], x[1]);
          unpack2(mul2(pack2(__uint_as_float(e[c][4 * g + 2]), __uint_as_float(e[c][4 * g + 3])),
                       fma2(pack2(__uint_as_float(dp[4 * g + 2]), __uint_as_float(dp[4 * g + 3])), scale2, d4.y)), x[2], x[3]);
          ds[2 * g] = pack_bf16(x[0], x[1]);
          ds[2 * g + 1] = pack_bf16(x[2], x[3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(slab + sw128_off(r, c * 4 + j)) =
              make_uint4(ds[4 * j], ds[4 * j + 1], ds[4 * j + 2], ds[4 * j + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&m.ds_full);
        mbar_arrive(&m.stat_empty[st]);
      }
      __syncwarp();
      if (++ib == nqb) ib = jb;
    }
    if (!fail) fail = !mbar_wait_parked(&m.all_done, 0, s_abort);
    if (__any_sync(0xffffffffu, fail)) {
      *s_abort = 1;
    } else if (SHARED) {
      // fp32 sums of this CTA's heads into its own shared memory (K, V, Q and dO are done with), four columns of 128 rows
      // after each other
      tc_fence_after_sync();
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        float4* dst = reinterpret_cast<float4*>(smem) + which * (D / 4) * 128 + r;
#pragma unroll 1
        for (int c = half * (D / 2); c < (half + 1) * (D / 2); c += 32) {
          uint32_t rr[32];
          tmem_ld32(tmem_addr(tm + (which ? C::TM_DV : C::TM_DK), lane_base, c), rr);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q)
            dst[(c / 4 + q) * 128] = make_float4(__uint_as_float(rr[4 * q]), __uint_as_float(rr[4 * q + 1]),
                                                 __uint_as_float(rr[4 * q + 2]), __uint_as_float(rr[4 * q + 3]));
        }
      }
    } else {
      // half of the warps dK, half dV; K, V, Q and dO are done with
      tc_fence_after_sync();
      const uint32_t tmx = tm + (half ? C::TM_DV : C::TM_DK);
      const int key = k0 + quarter * 32;
      const int64_t stride = half ? p.dvs1 : p.dks1;
      __nv_bfloat16* dst = half ? p.dv + b * p.dvs0 + hk * p.dvs2 : p.dk + b * p.dks0 + hk * p.dks2;
#pragma unroll 1
      for (int c = 0; c < D; c += 64) {
        uint32_t pk[32];
#pragma unroll
        for (int k = 0; k < 64; k += 32) {
          uint32_t rr[32];
          tmem_ld32(tmem_addr(tmx, lane_base, c + k), rr);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 16; ++q) pk[k / 2 + q] = pack_bf16(__uint_as_float(rr[2 * q]), __uint_as_float(rr[2 * q + 1]));
        }
        store_rows64(smem + (warp - 4) * 4096, pk, dst + key * stride + c, stride, p.S - key);
      }
    }
  } else {
    regs_inc<160>();
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;     // query row of the tile == TMEM lane
    const uint32_t lane_base = (uint32_t)(quarter * 32);
    int h = h0, ib = jb;
    bool fail = false;
    for (int i = 0; i < iters; ++i) {
      fail = !mbar_wait_parked(&m.dq_full, i & 1, s_abort) || *s_abort;
      // all four warps leave together: they share the named barriers below
      if (named_bar_or(1, 128, fail)) { fail = true; break; }
      tc_fence_after_sync();
      uint32_t rr[D / 32][32];
#pragma unroll
      for (int c = 0; c < D / 32; ++c) tmem_ld32(tmem_addr(tm + C::TM_DQ, lane_base, c * 32), rr[c]);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&m.dq_empty);
      __syncwarp();
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint8_t* buf = sStage + (c & 1) * 16384;
        if (tid == 384) bulk_wait_read<1>();  // the reduction before the last one has read this buffer
        named_bar_sync(2, 128);
#pragma unroll
        for (int t = 0; t < 8; ++t)
          *reinterpret_cast<uint4*>(buf + sw128_off(r, t)) =
              make_uint4(rr[c][4 * t], rr[c][4 * t + 1], rr[c][4 * t + 2], rr[c][4 * t + 3]);
        fence_proxy_async_smem();
        named_bar_sync(3, 128);
        if (tid == 384) {
          tma_reduce_add_4d(&mapdQ, buf, c * 32, h, ib * 128, b);
          bulk_commit();
        }
      }
      __syncwarp();
      if (++ib == nqb) { ib = jb; ++h; }
    }
    if (tid == 384) bulk_wait0();
    if (fail) *s_abort = 1;
  }
  tc_fence_before_sync();
  if constexpr (SHARED) {
    __syncwarp();
    cluster_sync();
    if (warp >= 4 && warp < 12) {
      // Each CTA of the cluster adds up its share of the columns, in the order of the parts, eight of a row a thread; a warp
      // has up to four such groups next to each other, of eight rows or more.
      const int groups = 2 * (D / 8) / parts, wide = min(groups, 4), high = 32 / wide;
      for (int w = warp - 4; w < groups / wide * (128 / high); w += 8) {
        const int row = (w % (128 / high)) * high + lane % high, key = k0 + row;
        const int g = part * groups + w / (128 / high) * wide + lane / high;  // dK's groups of eight columns, then dV's
        const uint32_t at = smem_u32(smem) + (uint32_t)(2 * g * 128 + row) * 16;
        float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
        for (int c = 0; c < parts; ++c) {
          const float4 x = ld_cluster(at, c), y = ld_cluster(at + 128 * 16, c);
          f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
          f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
        }
        if (key < p.S) {
          const int col = (g % (D / 8)) * 8;
          __nv_bfloat16* dst = g >= D / 8 ? p.dv + b * p.dvs0 + (int64_t)key * p.dvs1 + hk * p.dvs2
                                          : p.dk + b * p.dks0 + (int64_t)key * p.dks1 + hk * p.dks2;
          *reinterpret_cast<uint4*>(dst + col) =
              make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        }
      }
    }
    cluster_sync();  // the others have read this CTA's sums
  } else {
    __syncthreads();
  }
  if (tid == 0 && *s_abort) atomicExch(p.status, 6);
  if (warp == 1) tmem_dealloc(tm, 512);
}

// Key blocks whose `parts` CTAs each, a cluster, run at once.
template <int D>
static int blocks_at_once(int parts) {
  static int two[64], four[64], eight[64];
  const auto kernel = attn_bwd_kt_kernel<D, true>;
  switch (parts) {
    case 1: return sm_count();
    case 2: return clusters_at_once(kernel, 2, 512, Cfg<D>::SMEM, two);
    case 4: return clusters_at_once(kernel, 4, 512, Cfg<D>::SMEM, four);
    default: return clusters_at_once(kernel, 8, 512, Cfg<D>::SMEM, eight);
  }
}

// How many CTAs (a cluster) share the query heads of a key block.  A key block's iterations follow one another, so with few
// key blocks, batches and KV heads the chip waits for the longest of them: 1024 keys, 8 / 2 heads of 128 are 16 CTAs of up to
// 32 iterations, 83 us.  Counted in iterations (2.3 us at head dimension 128, 2 at 64): the longest CTA or the average of all
// SMs, and for every wave of clusters (74 of two, 33 of four, 15 of eight run at once) what one costs beside its iterations, 4 alone
// and a few more for adding up the shares.  (us, alone and shared) 1024 keys, 8 / 2 heads: 83, by four 31; 2048, 32 / 8: 166, by
// two 100; 4096, 8 / 2: 308, by four 108; 1024, 64 / 8: 167, by two 97; 4096, 64 / 8: 713, by two 683; 4096, 32 / 8: 337, by two 353,
// so alone.
// A query block's dQ gets its key blocks' tiles in the order of time.  By heads and not by query blocks the tiles come an
// iteration after each other, and where all CTAs run at once they come in the same order at every run; in a second wave they do not
// (1920 keys, 16 / 8 heads of 64: alone none of 2998 runs differed from the first, by two all of 39).  So where dQ repeats without
// sharing, key blocks are shared only as far as all clusters run at once.  What that costs: 1024 keys, 64 / 8 heads of 128, 97 us
// where four would take 75; 1280 keys, 212 where they would take 115.  Without sharing it repeats in one wave while
// CTAs do not drift apart by an iteration, with few key blocks or few CTAs (of 174 to 2340 runs in several places of memory that
// differed: head dimension 128, none at 1536 keys, 8 / 2 heads, nor at 2048, 323 at 1920, 16 / 8; 64, none up to 3584 keys with any heads or
// 7168 with 8 / 1, 116 of 174 at 4096, 32 / 4).
template <int D>
static int parts_of(int S, int Hq, int Hkv, int B) {
  const int sms = sm_count(), nqb = (S + 127) / 128, group = Hq / Hkv;
  const double alone = 4.0, shared = D == 128 ? 7.0 : 5.5;
  const double ctas = (double)nqb * Hkv * B, longest = (double)group * nqb, all = ctas * group * (nqb + 1) / 2;
  const bool repeats = ctas <= sms && (D == 128 ? nqb <= 12 || ctas <= 32 : nqb <= 28 || ctas <= 56);
  int best = 1;
  double least = 0;
  for (int c = 1; c <= 8 && group % c == 0; c *= 2) {
    const double waves = std::ceil(ctas / blocks_at_once<D>(c));
    if (c > 1 && repeats && waves > 1) break;
    const double t = std::max(longest / c, all / sms) + waves * (c > 1 ? shared : alone);
    if (c == 1 || t < least) { best = c; least = t; }
  }
  return best;
}

template <int D>
static int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                  const CUtensorMap& mdq, BwdParams p, cudaStream_t st) {
  using C = Cfg<D>;
  static_assert(2 * 128 * D * 4 <= C::DS, "the shares' sums take the place of K, V, Q and dO");
  p.parts = parts_of<D>(p.S, p.Hq, p.Hkv, p.B);
  const int units = (p.S + 127) / 128 * p.Hkv * p.B;
  if (p.parts == 1) {
    if (cudaFuncSetAttribute(attn_bwd_kt_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
      return launch_status();
    zc::launch_chained(attn_bwd_kt_kernel<D, false>, units, 512, C::SMEM, st, mq, mk, mv, mdo, mdq, p);
    return launch_status();
  }
  if (cudaFuncSetAttribute(attn_bwd_kt_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
    return launch_status();
  zc::launch_chained_cluster(p.parts, attn_bwd_kt_kernel<D, true>, units * p.parts, 512, C::SMEM, st, mq, mk, mv, mdo, mdq, p);
  return launch_status();
}

}  // namespace bkt
}  // namespace zc

extern "C" {

int zc_attn_bwd_ws_status_read_and_clear() {
  int dev = 0;
  cudaGetDevice(&dev);
  zc::bws::Scratch& sc = zc::bws::g_scratch[dev];
  if (!sc.status) return 0;
  int v = 0;
  cudaMemcpy(&v, sc.status, sizeof(int), cudaMemcpyDeviceToHost);
  if (v) cudaMemset(sc.status, 0, sizeof(int));
  return v;
}

// Same argument list as zc_attn_bwd: `dq_acc` is the fp32 accumulator of dQ, B * S * Hq * D floats that the launcher
// clears.
int zc_attn_bwd_ws(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                   float* delta, void* dq, void* dk, void* dv, int B, int S, int Hq, int Hkv, int D, int64_t qs0,
                   int64_t qs1, int64_t qs2, int64_t ks0, int64_t ks1, int64_t ks2, int64_t vs0, int64_t vs1,
                   int64_t vs2, int64_t dqs0, int64_t dqs1, int64_t dqs2, int64_t dks0, int64_t dks1, int64_t dks2,
                   int64_t dvs0, int64_t dvs1, int64_t dvs2, float scale, float* dq_acc, cudaStream_t st) {
  using namespace zc;
  using namespace zc::bws;
  if ((D != 64 && D != 128) || Hq % Hkv) return ERR_UNSUPPORTED;
  if ((qs1 | qs2 | ks1 | ks2 | vs1 | vs2 | qs0 | ks0 | vs0 | dqs1 | dqs2 | dks1 | dks2 | dvs1 | dvs2 | dqs0 | dks0 | dvs0) % 8)
    return ERR_UNSUPPORTED;
  if (dqs0 != (int64_t)S * dqs1) return ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(dout)) & 15)
    return ERR_UNSUPPORTED;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaSetDevice(dev);
  Scratch& sc = g_scratch[dev];
  if (!sc.status) {
    if (cudaMalloc(&sc.status, sizeof(int)) != cudaSuccess) return ERR_BAD_ARG;
    cudaMemset(sc.status, 0, sizeof(int));
  }
  const size_t need = (size_t)B * S * Hq * D * sizeof(float);
  cudaMemsetAsync(dq_acc, 0, need, st);
  CUtensorMap mq, mk, mv, mdo, mdq;
  if (!make_map4(&mq, q, D, Hq, S, B, qs0, qs1, qs2) || !make_map4(&mk, k, D, Hkv, S, B, ks0, ks1, ks2) ||
      !make_map4(&mv, v, D, Hkv, S, B, vs0, vs1, vs2) ||
      !make_map4(&mdo, dout, D, Hq, S, B, (int64_t)S * Hq * D, (int64_t)Hq * D, D) ||
      !make_map4_f32(&mdq, dq_acc, D, Hq, S, B))
    return ERR_BAD_ARG;
  BwdParams p;
  p.lse = lse; p.delta = delta; p.dq_acc = dq_acc; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.dks0 = dks0; p.dks1 = dks1; p.dks2 = dks2; p.dvs0 = dvs0; p.dvs1 = dvs1; p.dvs2 = dvs2;
  p.scale = scale; p.status = sc.status;
  const int64_t rows = (int64_t)B * S * Hq;
  delta_kernel<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)dout,
                                                                   delta, B, S, Hq, D);
  const int smem = 6 * 32768 + 1024;
  static bool attr[2] = {false, false};
  const dim3 grid((S + 127) / 128, Hkv, B);
  if (D == 128) {
    if (!attr[0]) { cudaFuncSetAttribute(attn_bwd_ws_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); attr[0] = true; }
    attn_bwd_ws_kernel<128><<<grid, 320, smem, st>>>(mq, mk, mv, mdo, mdq, p);
  } else {
    if (!attr[1]) { cudaFuncSetAttribute(attn_bwd_ws_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); attr[1] = true; }
    attn_bwd_ws_kernel<64><<<grid, 320, smem, st>>>(mq, mk, mv, mdo, mdq, p);
  }
  const int cgrid = (int)std::min<int64_t>((rows * (D / 4) + 255) / 256, (int64_t)sm_count() * 16);
  dq_convert_kernel<<<cgrid, 256, 0, st>>>(dq_acc, (__nv_bfloat16*)dq, (int64_t)B * S, Hq, D, dqs1, dqs2);
  return launch_status();
}

// Same argument list as zc_attn_bwd: the key-row kernel.
int zc_attn_bwd_kt(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                   float* delta, void* dq, void* dk, void* dv, int B, int S, int Hq, int Hkv, int D, int64_t qs0,
                   int64_t qs1, int64_t qs2, int64_t ks0, int64_t ks1, int64_t ks2, int64_t vs0, int64_t vs1,
                   int64_t vs2, int64_t dqs0, int64_t dqs1, int64_t dqs2, int64_t dks0, int64_t dks1, int64_t dks2,
                   int64_t dvs0, int64_t dvs1, int64_t dvs2, float scale, float* dq_acc, cudaStream_t st) {
  using namespace zc;
  using namespace zc::bws;
  if ((D != 64 && D != 128) || Hq % Hkv) return ERR_UNSUPPORTED;
  if ((qs1 | qs2 | ks1 | ks2 | vs1 | vs2 | qs0 | ks0 | vs0 | dqs1 | dqs2 | dks1 | dks2 | dvs1 | dvs2 | dqs0 | dks0 | dvs0) % 8)
    return ERR_UNSUPPORTED;
  if (dqs0 != (int64_t)S * dqs1) return ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(dout)) & 15)
    return ERR_UNSUPPORTED;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaSetDevice(dev);
  Scratch& sc = g_scratch[dev];
  if (!sc.status) {
    if (cudaMalloc(&sc.status, sizeof(int)) != cudaSuccess) return ERR_BAD_ARG;
    cudaMemset(sc.status, 0, sizeof(int));
  }
  CUtensorMap mq, mk, mv, mdo, mdq;
  if (!make_map4(&mq, q, D, Hq, S, B, qs0, qs1, qs2) || !make_map4(&mk, k, D, Hkv, S, B, ks0, ks1, ks2) ||
      !make_map4(&mv, v, D, Hkv, S, B, vs0, vs1, vs2) ||
      !make_map4(&mdo, dout, D, Hq, S, B, (int64_t)S * Hq * D, (int64_t)Hq * D, D) ||
      !make_map4_f32(&mdq, dq_acc, D, Hq, S, B))
    return ERR_BAD_ARG;
  BwdParams p;
  p.lse = lse; p.delta = delta; p.dq_acc = dq_acc; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.dks0 = dks0; p.dks1 = dks1; p.dks2 = dks2; p.dvs0 = dvs0; p.dvs1 = dvs1; p.dvs2 = dvs2;
  p.scale = scale; p.status = sc.status;
  const int64_t rows = (int64_t)B * S * Hq, units = rows * (D / 8);
  const unsigned ugrid = (unsigned)((units + 255) / 256);
  if (reinterpret_cast<uintptr_t>(o) & 15) {  // a saved output that came back from a hook at an odd address
    cudaMemsetAsync(dq_acc, 0, (size_t)rows * D * sizeof(float), st);
    delta_kernel<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)dout,
                                                                     delta, B, S, Hq, D);
  } else if (D == 128) {
    zc::launch_chained(delta_zero_kernel<128>, ugrid, 256, 0, st, (const uint4*)o, (const uint4*)dout, delta, (float4*)dq_acc, S, Hq, rows);
  } else {
    zc::launch_chained(delta_zero_kernel<64>, ugrid, 256, 0, st, (const uint4*)o, (const uint4*)dout, delta, (float4*)dq_acc, S, Hq, rows);
  }
  const int rc = D == 128 ? bkt::launch<128>(mq, mk, mv, mdo, mdq, p, st) : bkt::launch<64>(mq, mk, mv, mdo, mdq, p, st);
  if (rc) return rc;
  if ((reinterpret_cast<uintptr_t>(dq) & 15) || rows >= (1ll << 32))
    dq_convert_kernel<<<(unsigned)(sm_count() * 16), 256, 0, st>>>(dq_acc, (__nv_bfloat16*)dq, (int64_t)B * S, Hq, D, dqs1, dqs2);
  else if (D == 128)
    zc::launch_chained(dq_convert8_kernel<128>, ugrid, 256, 0, st, (const float4*)dq_acc, (__nv_bfloat16*)dq, units, Hq, dqs1, dqs2);
  else
    zc::launch_chained(dq_convert8_kernel<64>, ugrid, 256, 0, st, (const float4*)dq_acc, (__nv_bfloat16*)dq, units, Hq, dqs1, dqs2);
  return launch_status();
}

// For a look at the rule: how many CTAs share a key block's query heads, and how many key blocks so shared run at once.
int zc_attn_bwd_parts(int S, int Hq, int Hkv, int B, int D) {
  return D == 128 ? zc::bkt::parts_of<128>(S, Hq, Hkv, B) : zc::bkt::parts_of<64>(S, Hq, Hkv, B);
}
int zc_attn_bwd_blocks_at_once(int parts, int D) { return D == 128 ? zc::bkt::blocks_at_once<128>(parts) : zc::bkt::blocks_at_once<64>(parts); }

}  // extern "C"
