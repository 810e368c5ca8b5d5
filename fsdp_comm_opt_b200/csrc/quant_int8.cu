// int8 absmax quantisation of one buffer and dequantisation of all ranks' buffers (the arithmetic of
// QuantizedAllGather).  Packed buffer: word 0 = fp32 scale, word 1 = bits of the absolute maximum,
// words 2-3 zero, bytes [16, 16 + n) = int8 payload.
//
// All three passes are bound by memory, so they move 16-byte vectors of the wide type and keep several
// of them in flight per thread.  One element per thread and trip (2-byte loads, a 64-bit division per
// element in the dequantiser) ran at 0.2 of the copy bandwidth: 508 us for eight ranks' 27 264 000
// elements, against 101 us that the bytes need.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch_util.h"

namespace zc {
namespace q8 {

constexpr int THREADS = 256;
constexpr int MAX_GRID_Y = 65535;

__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float widen(float v) { return v; }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T narrow(float v);
template <> __device__ __forceinline__ __nv_bfloat16 narrow<__nv_bfloat16>(float v) { return __float2bfloat16(v); }
template <> __device__ __forceinline__ float narrow<float>(float v) { return v; }
template <> __device__ __forceinline__ __half narrow<__half>(float v) { return __float2half(v); }

// sixteen bytes of T
template <typename T> struct alignas(16) Vec {
  static constexpr int N = 16 / sizeof(T);
  T v[N];
};
template <typename T> __device__ __forceinline__ Vec<T> load_vec(const T* p) {
  return *reinterpret_cast<const Vec<T>*>(p);
}

__device__ __forceinline__ float scale_of(float absmax) { return fmaxf(absmax / 127.f, 1e-8f); }
__device__ __forceinline__ int8_t quant1(float x, float scale) {
  return (int8_t)fminf(fmaxf(rintf(x / scale), -127.f), 127.f);
}

__device__ __forceinline__ float block_absmax(float m, float* red) {  // result in thread 0
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = fmaxf(m, red[i]);
  return m;
}

// |maximum| of the elements that thread `t` of `nt` owns: whole 16-byte vectors (four in flight), then
// the tail; `vec` false (an unaligned input): one element at a time
template <typename T>
__device__ __forceinline__ float thread_absmax(const T* __restrict__ x, int64_t n, bool vec, int64_t t, int64_t nt) {
  constexpr int N = Vec<T>::N;
  const int64_t nv = vec ? n / N : 0;
  float m = 0.f;
  // the last trip too has its loads in flight together, one at a time they are a memory's latency each (27 264 000 elements:
  // 17.1 -> 14.4 us)
  for (int64_t i = t; i < nv; i += 4 * nt) {
    Vec<T> a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * nt < nv) a[k] = load_vec(x + (i + k * nt) * N);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * nt < nv) {
#pragma unroll
        for (int j = 0; j < N; ++j) m = fmaxf(m, fabsf(widen(a[k].v[j])));
      }
  }
  for (int64_t i = nv * N + t; i < n; i += nt) m = fmaxf(m, fabsf(widen(x[i])));
  return m;
}

// quantise the elements of thread `t` of `nt`, sixteen at a time (one 16-byte store)
template <typename T>
__device__ __forceinline__ void thread_quant(const T* __restrict__ x, int64_t n, bool vec, float scale,
                                             int8_t* __restrict__ q, int64_t t, int64_t nt) {
  constexpr int N = Vec<T>::N, L = 16 / N;
  const int64_t nv = vec ? n / 16 : 0;
  for (int64_t i = t; i < nv; i += nt) {
    Vec<T> a[L];
#pragma unroll
    for (int k = 0; k < L; ++k) a[k] = load_vec(x + i * 16 + k * N);
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w[k] = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = 4 * k + j;
        w[k] |= (uint32_t)(uint8_t)quant1(widen(a[e / N].v[e % N]), scale) << (8 * j);
      }
    }
    *reinterpret_cast<uint4*>(q + i * 16) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  for (int64_t i = nv * 16 + t; i < n; i += nt) q[i] = quant1(widen(x[i]), scale);
}

template <typename T>
__global__ void __launch_bounds__(THREADS) absmax_kernel(const T* __restrict__ x, int64_t n, bool vec,
                                                         uint32_t* __restrict__ hdr) {
  __shared__ float red[32];
  float m = thread_absmax<T>(x, n, vec, (int64_t)blockIdx.x * THREADS + threadIdx.x, (int64_t)gridDim.x * THREADS);
  m = block_absmax(m, red);
  if (threadIdx.x == 0) atomicMax(hdr + 1, __float_as_uint(m));  // non-negative floats order like their bit patterns
}

// The second read of x comes from L2 for buffers below its 126 MB.
template <typename T>
__global__ void __launch_bounds__(THREADS) quant_kernel(const T* __restrict__ x, int64_t n, bool vec,
                                                        uint8_t* __restrict__ out) {
  const float scale = scale_of(__uint_as_float(reinterpret_cast<const uint32_t*>(out)[1]));
  if (blockIdx.x == 0 && threadIdx.x == 0) reinterpret_cast<float*>(out)[0] = scale;
  thread_quant<T>(x, n, vec, scale, reinterpret_cast<int8_t*>(out + 16), (int64_t)blockIdx.x * THREADS + threadIdx.x,
                  (int64_t)gridDim.x * THREADS);
}

// Small buffers: one cluster of eight CTAs finds the maximum, exchanges it through distributed shared
// memory and quantises, in one launch instead of three (the header's clearing, maximum, quantise).
constexpr int SMALL_CTAS = 8, SMALL_THREADS = 1024;
template <typename T>
__global__ void __cluster_dims__(SMALL_CTAS, 1, 1) __launch_bounds__(SMALL_THREADS)
    quant_small_kernel(const T* __restrict__ x, int64_t n, bool vec, uint8_t* __restrict__ out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float red[32];
  __shared__ float part;
  const int64_t t = (int64_t)blockIdx.x * SMALL_THREADS + threadIdx.x, nt = SMALL_CTAS * SMALL_THREADS;
  float m = block_absmax(thread_absmax<T>(x, n, vec, t, nt), red);
  if (threadIdx.x == 0) part = m;
  cluster.sync();
  m = 0.f;
#pragma unroll
  for (int i = 0; i < SMALL_CTAS; ++i) m = fmaxf(m, *cluster.map_shared_rank(&part, i));
  cluster.sync();  // nobody leaves while its maximum may still be read
  const float scale = scale_of(m);
  if (t == 0) *reinterpret_cast<uint4*>(out) = make_uint4(__float_as_uint(scale), __float_as_uint(m), 0u, 0u);
  thread_quant<T>(x, n, vec, scale, reinterpret_cast<int8_t*>(out + 16), t, nt);
}

// One grid row per rank.  Units of eight elements start where the output row reaches a 16-byte boundary
// (`head` elements in: row r starts at r * n elements, any alignment), so every store is whole; the
// payload bytes of a unit then start `head` bytes past an 8-byte boundary and are cut out of two
// aligned words.  Eight units per thread and trip keep enough loads in flight.
template <typename T>
__global__ void __launch_bounds__(THREADS) dequant_kernel(const uint8_t* __restrict__ gathered, int64_t stride,
                                                          int64_t n, T* __restrict__ out) {
  constexpr int U = 8;
  const uint8_t* slot = gathered + blockIdx.y * stride;
  const float scale = __ldg(reinterpret_cast<const float*>(slot));
  const uint8_t* q = slot + 16;
  T* dst = out + blockIdx.y * n;
  const int mis = (int)(reinterpret_cast<uintptr_t>(dst) & 15);
  const int64_t head = mis ? (16 - mis) / (int)sizeof(T) : 0;  // below eight elements
  const int64_t nu = n > head ? (n - head) / 8 : 0;
  const uint32_t sh = (uint32_t)head * 8;
  // 8388608 + u in fp32 has the byte u as its low mantissa byte: two cheap instructions per element
  // instead of an integer conversion
  auto value = [&](uint32_t w, int j) -> float {
    const uint32_t u = __byte_perm(w ^ 0x80808080u, 0x4B000000u, 0x7540 | j);
    return (__uint_as_float(u) - 8388736.f) * scale;
  };
  auto emit = [&](int64_t u, uint2 a, uint2 b) {
    const uint64_t lo = ((uint64_t)a.y << 32) | a.x, hi = ((uint64_t)b.y << 32) | b.x;
    const uint64_t w = sh ? (lo >> sh) | (hi << (64 - sh)) : lo;
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[j] = value((uint32_t)w, j);
      f[4 + j] = value((uint32_t)(w >> 32), j);
    }
    T* d = dst + head + u * 8;
#pragma unroll
    for (int k = 0; k < 8 / Vec<T>::N; ++k) {
      Vec<T> o;
#pragma unroll
      for (int j = 0; j < Vec<T>::N; ++j) o.v[j] = narrow<T>(f[k * Vec<T>::N + j]);
      *reinterpret_cast<Vec<T>*>(d + k * Vec<T>::N) = o;
    }
  };
  // the word after a unit's own is read only when the unit reaches into it, so never past the payload
  auto word = [&](int64_t u) { return __ldg(reinterpret_cast<const uint2*>(q) + u); };
  const int64_t step = (int64_t)gridDim.x * THREADS;
  int64_t u = (int64_t)blockIdx.x * THREADS + threadIdx.x;
  const uint2 none = make_uint2(0u, 0u);
  for (; u + (U - 1) * step < nu; u += U * step) {
    uint2 a[U], b[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      a[k] = word(u + k * step);
      b[k] = sh ? word(u + k * step + 1) : none;
    }
#pragma unroll
    for (int k = 0; k < U; ++k) emit(u + k * step, a[k], b[k]);
  }
  for (; u < nu; u += step) emit(u, word(u), sh ? word(u + 1) : none);
  if (blockIdx.x == 0) {  // the elements before the first unit and after the last one
    const int64_t tail = head + nu * 8;
    for (int64_t k = threadIdx.x; k < n; k += THREADS) {
      if (k >= head && k < tail) k += (tail - k + THREADS - 1) / THREADS * THREADS;
      if (k < n) dst[k] = narrow<T>((float)(int8_t)q[k] * scale);
    }
  }
}

// payloads or outputs that no vector access can reach (a buffer or a row stride off its boundary)
template <typename T>
__global__ void __launch_bounds__(THREADS) dequant_unaligned_kernel(const uint8_t* __restrict__ gathered, int64_t stride,
                                                                    int64_t n, T* __restrict__ out) {
  const uint8_t* slot = gathered + blockIdx.y * stride;
  const float scale = *reinterpret_cast<const float*>(slot);
  for (int64_t k = (int64_t)blockIdx.x * THREADS + threadIdx.x; k < n; k += (int64_t)gridDim.x * THREADS)
    out[blockIdx.y * n + k] = narrow<T>((float)(int8_t)slot[16 + k] * scale);
}

template <typename T>
int quantise(const void* x, int64_t n, uint8_t* out, cudaStream_t st) {
  // a payload that is not on a 16-byte boundary takes the element-wise loops of the same kernels
  const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  // Up to 512 K elements eight SMs read the buffer twice in less time than two more launches take (a
  // launch costs 2-3 us, 1 MB through eight SMs about 1.5 us a pass).
  if (vec && n <= (1 << 19)) {
    quant_small_kernel<T><<<SMALL_CTAS, SMALL_THREADS, 0, st>>>((const T*)x, n, vec, out);
    return launch_status();
  }
  cudaMemsetAsync(out, 0, 16, st);
  const int64_t units = (n + 15) / 16;
  const int grid = (int)std::min<int64_t>((units + THREADS - 1) / THREADS, (int64_t)sm_count() * 8);
  absmax_kernel<T><<<grid, THREADS, 0, st>>>((const T*)x, n, vec, (uint32_t*)out);
  quant_kernel<T><<<grid, THREADS, 0, st>>>((const T*)x, n, vec, out);
  return launch_status();
}

template <typename T>
int dequantise(const uint8_t* gathered, int64_t stride, int world, int64_t n, T* out, cudaStream_t st) {
  const bool ok = ((reinterpret_cast<uintptr_t>(gathered) | (uintptr_t)stride) & 15) == 0 &&
                  reinterpret_cast<uintptr_t>(out) % sizeof(T) == 0;
  const int64_t units = (n + 7) / 8;
  // 32 CTAs per SM (four waves): 108 us for the eight ranks above, 121 with one wave, which reads too many pages
  // at a time
  const int64_t most = std::max<int64_t>(1, (int64_t)sm_count() * 32 / world);
  for (; world > 0; world -= MAX_GRID_Y, gathered += MAX_GRID_Y * stride, out += MAX_GRID_Y * n) {
    const int rows = std::min(world, MAX_GRID_Y);
    if (ok) {
      const dim3 grid((unsigned)std::min<int64_t>((units + THREADS - 1) / THREADS, most), rows);
      dequant_kernel<T><<<grid, THREADS, 0, st>>>(gathered, stride, n, out);
    } else {
      const dim3 grid((unsigned)std::min<int64_t>((n + THREADS - 1) / THREADS, 2 * most), rows);
      dequant_unaligned_kernel<T><<<grid, THREADS, 0, st>>>(gathered, stride, n, out);
    }
  }
  return launch_status();
}

}  // namespace q8
}  // namespace zc

extern "C" {

int zc_quant_int8(const void* x, int64_t n, int dtype, void* out, cudaStream_t st) {
  using namespace zc;
  if (n == 0) {
    cudaMemsetAsync(out, 0, 16, st);
    return launch_status();
  }
  switch (dtype) {
    case 0: return q8::quantise<__nv_bfloat16>(x, n, (uint8_t*)out, st);
    case 1: return q8::quantise<float>(x, n, (uint8_t*)out, st);
    case 2: return q8::quantise<__half>(x, n, (uint8_t*)out, st);
    default: return ERR_UNSUPPORTED;
  }
}

int zc_dequant_int8(const void* gathered, int64_t stride, int world, int64_t n, int dtype, void* out,
                    cudaStream_t st) {
  using namespace zc;
  if (world <= 0 || n <= 0) return 0;
  switch (dtype) {
    case 0: return q8::dequantise<__nv_bfloat16>((const uint8_t*)gathered, stride, world, n, (__nv_bfloat16*)out, st);
    case 1: return q8::dequantise<float>((const uint8_t*)gathered, stride, world, n, (float*)out, st);
    case 2: return q8::dequantise<__half>((const uint8_t*)gathered, stride, world, n, (__half*)out, st);
    default: return ERR_UNSUPPORTED;
  }
}

}  // extern "C"
