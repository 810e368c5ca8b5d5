// Gradient of an embedding table, added up into the bf16 buffer that holds it.
//
// grad[v] (+)= sum over the positions t with ids[t] = v of dout[t], fp32 sums in a fixed order, rounded once.
// One block per position: it compares its id with all of them (n * 8 bytes from L2, so n is limited) and finds how many
// positions share it and how many of these come before its own.  The block of a rare id's first position sums it; a
// frequent id's blocks divide the row's columns among themselves, each reading 128 bytes or more of every row with
// 2048 / columns groups of threads that take every so many words of 32 positions.  No sort, no atomics in
// memory, no dense gradient beside the buffer.
// A table of 128256 x 4096 and 4096 positions took a cleared dense gradient (175 us), a sort and scatter
// (about 290) and a copy into the buffer (340).  Now the buffer is cleared (the rows that no position names are zeros, which
// is most of the bytes) and this kernel runs: 212 us for uniform ids, of which the kernel takes 62, and 193 for 4096 equal
// ones (2869 when an id's first block summed all of them).  What bounds it: the gradient's rows, and the comparisons of n
// blocks with n ids (8192 positions 64 wide: 85 us, the sort 140), eight of which are in flight per thread.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "launch_util.h"

namespace zc {
namespace emb {

constexpr int THREADS = 256;
constexpr int MAX_N = 8192;    // positions: their matches are a bit each of MAX_N / 32 words
constexpr int WARPS = THREADS / 32;
constexpr int IDS_AHEAD = 8;   // ids in flight per thread
constexpr int AHEAD = 8;       // rows in flight per thread
constexpr int MIN_COLS = 64, MAX_COLS = THREADS * 8;   // columns of a block at least and at most

__global__ void __launch_bounds__(THREADS, 3) embedding_grad_kernel(const int64_t* ids,
                                                                 const __nv_bfloat16* dout,
                                                                 __nv_bfloat16* __restrict__ grad, int n, int dim,
                                                                 int64_t rows, int accumulate) {
  chain();
  __shared__ uint32_t match[MAX_N / 32];
  __shared__ uint32_t any[MAX_N / 1024];   // which words of `match` are not zero
  __shared__ uint32_t count;               // positions with this id: all, and in the upper half those before this block's
  __shared__ __align__(16) float part[THREADS * 8];
  const int i = blockIdx.x, lane = threadIdx.x & 31;
  const int64_t id = ids[i];
  if (id < 0 || id >= rows) return;        // the lookup has refused these
  if (threadIdx.x < MAX_N / 1024) any[threadIdx.x] = 0;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  const int words = (n + 31) / 32;
  for (int w0 = threadIdx.x >> 5; w0 < words; w0 += WARPS * IDS_AHEAD) {
    int64_t other[IDS_AHEAD];
#pragma unroll
    for (int k = 0; k < IDS_AHEAD; ++k) {
      const int j = (w0 + k * WARPS) * 32 + lane;
      other[k] = j < n ? ids[j] : -1;
    }
#pragma unroll
    for (int k = 0; k < IDS_AHEAD; ++k) {
      const int w = w0 + k * WARPS;
      const uint32_t b = __ballot_sync(0xffffffffu, other[k] == id);
      if (lane == 0 && w < words) {
        match[w] = b;
        if (b) {
          atomicOr(&any[w >> 5], 1u << (w & 31));
          const uint32_t earlier = w < (i >> 5) ? b : w == (i >> 5) ? b & ((1u << (i & 31)) - 1) : 0u;
          atomicAdd(&count, (uint32_t)__popc(b) | (uint32_t)__popc(earlier) << 16);
        }
      }
    }
  }
  __syncthreads();
  // An id of up to AHEAD positions, one round trip, is its first block's alone.  The columns of a frequent one are halved
  // for every doubling of the blocks that can help, down to a full line of 128 bytes.
  const int total = (int)(count & 0xffffu), mine = (int)(count >> 16);
  const bool frequent = total > AHEAD;
  if (!frequent && mine > 0) return;
  const int blocks = frequent ? total : 1;
  int cols = MAX_COLS;
  while (frequent && cols > MIN_COLS && (int64_t)cols * blocks >= 2 * (int64_t)dim) cols >>= 1;
  const int groups = MAX_COLS / cols, group = threadIdx.x / (cols / 8);
  uint32_t my_words = 0;                   // of 32 words, those of this thread's group
  for (int k = group; k < 32; k += groups) my_words |= 1u << k;
  for (int64_t c0 = (int64_t)mine * cols; c0 < dim; c0 += (int64_t)blocks * cols) {
    const int c = (int)c0 + (threadIdx.x % (cols / 8)) * 8;
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    if (c < dim) {
      int pos[AHEAD], m = 0;
      auto flush = [&]() {
        uint4 v[AHEAD];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
          if (a < m) v[a] = *reinterpret_cast<const uint4*>(dout + (int64_t)pos[a] * dim + c);
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
          if (a < m) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[a]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 f = __bfloat1622float2(h[k]);
              acc[2 * k] += f.x;
              acc[2 * k + 1] += f.y;
            }
          }
        m = 0;
      };
      for (int s = 0; s * 1024 < n; ++s)
        for (uint32_t aw = any[s] & my_words; aw; aw &= aw - 1) {
          const int w = s * 32 + __ffs(aw) - 1;
          for (uint32_t b = match[w]; b; b &= b - 1) {
            const int t = w * 32 + __ffs(b) - 1;
#pragma unroll
            for (int a = 0; a < AHEAD; ++a)
              if (a == m) pos[a] = t;
            if (++m == AHEAD) flush();
          }
        }
      flush();
    }
    if (groups > 1) {                      // the groups' sums, in the groups' order
      __syncthreads();
      float4* p = reinterpret_cast<float4*>(part + threadIdx.x * 8);
      p[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      p[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      __syncthreads();
      if (group == 0)
        for (int g = 1; g < groups; ++g)
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] += part[g * cols + threadIdx.x * 8 + k];
    }
    if (group > 0 || c >= dim) continue;
    __nv_bfloat16* dst = grad + id * dim + c;
    const uint4 old = accumulate ? *reinterpret_cast<const uint4*>(dst) : make_uint4(0, 0, 0, 0);
    const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old);
    uint32_t out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(o2[k]);
      const __nv_bfloat162 r = __floats2bfloat162_rn(acc[2 * k] + f.x, acc[2 * k + 1] + f.y);
      out[k] = *reinterpret_cast<const uint32_t*>(&r);
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(out[0], out[1], out[2], out[3]);
  }
}

}  // namespace emb
}  // namespace zc

extern "C" {

// `grad` [rows, dim] bf16 is overwritten (`accumulate` 0: rows that no id names become zeros) or added to.  dim a multiple of
// 8, both tensors 16-byte aligned, 1 <= n <= 8192; else ERR_UNSUPPORTED and nothing is written.
int zc_embedding_grad(const void* ids, const void* dout, void* grad, int64_t n, int64_t dim, int64_t rows, int accumulate,
                      cudaStream_t st) {
  using namespace zc;
  if (n < 1 || n > emb::MAX_N || dim < 8 || dim % 8 || dim > (1 << 24) || rows < 1) return ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(grad)) & 15) return ERR_UNSUPPORTED;
  if (!accumulate) cudaMemsetAsync(grad, 0, (size_t)rows * dim * 2, st);
  zc::launch_chained(emb::embedding_grad_kernel, (unsigned)n, emb::THREADS, 0, st, (const int64_t*)ids, (const __nv_bfloat16*)dout,
                                                                   (__nv_bfloat16*)grad, (int)n, (int)dim, rows, accumulate);
  return launch_status();
}

}  // extern "C"
