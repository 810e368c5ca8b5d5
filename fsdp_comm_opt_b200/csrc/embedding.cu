// Gradient of an embedding table, added up into the bf16 buffer that holds it.
//
// grad[v] (+)= sum over the positions t with ids[t] = v of dout[t], fp32 sums in the order of the positions, rounded once.
// One block per position: it compares its id with all of them (n * 8 bytes from L2, so n is limited), leaves when an
// earlier position has the same id, and otherwise adds up that id's rows.  No sort, no atomics, no dense gradient beside
// the buffer: a table of 128256 x 4096 and 4096 positions took a cleared dense gradient (175 us), a sort and scatter
// (about 290) and a copy into the buffer (340); now the buffer is cleared (the rows that no position names are zeros, which
// is most of the bytes) and this kernel runs (219 + 93 us).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "launch_util.h"

namespace zc {
namespace emb {

constexpr int THREADS = 256;
constexpr int MAX_N = 8192;    // positions: their matches are a bit each of MAX_N / 32 words
constexpr int AHEAD = 8;       // rows in flight per thread

__global__ void __launch_bounds__(THREADS) embedding_grad_kernel(const int64_t* __restrict__ ids,
                                                                 const __nv_bfloat16* __restrict__ dout,
                                                                 __nv_bfloat16* __restrict__ grad, int n, int dim,
                                                                 int64_t rows, int accumulate) {
  __shared__ uint32_t match[MAX_N / 32];
  __shared__ uint32_t any[MAX_N / 1024];   // which words of `match` are not zero
  const int i = blockIdx.x, lane = threadIdx.x & 31;
  const int64_t id = ids[i];
  if (id < 0 || id >= rows) return;        // the lookup has refused these
  if (threadIdx.x < MAX_N / 1024) any[threadIdx.x] = 0;
  __syncthreads();
  const int words = (n + 31) / 32;
  for (int w = threadIdx.x >> 5; w < words; w += THREADS / 32) {
    const int j = w * 32 + lane;
    const uint32_t b = __ballot_sync(0xffffffffu, j < n && ids[j] == id);
    if (lane == 0) {
      match[w] = b;
      if (b) atomicOr(&any[w >> 5], 1u << (w & 31));
    }
  }
  __syncthreads();
  // an earlier position with this id?  Its block does the sum.
  const uint32_t below = (1u << (i & 31)) - 1;
  if (match[i >> 5] & below) return;
  for (int s = 0; s <= i >> 10; ++s)
    if (any[s] & (s == i >> 10 ? (1u << ((i >> 5) & 31)) - 1 : 0xffffffffu)) return;
  for (int c = threadIdx.x * 8; c < dim; c += THREADS * 8) {
    float acc[8];
    __nv_bfloat16* dst = grad + id * dim + c;
    const uint4 old = accumulate ? *reinterpret_cast<const uint4*>(dst) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    int pos[AHEAD], m = 0;
    auto flush = [&]() {
      uint4 v[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a)
        if (a < m) v[a] = __ldg(reinterpret_cast<const uint4*>(dout + (int64_t)pos[a] * dim + c));
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
    for (int s = i >> 10; s * 1024 < n; ++s)
      for (uint32_t aw = any[s]; aw; aw &= aw - 1) {
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
  emb::embedding_grad_kernel<<<(unsigned)n, emb::THREADS, 0, st>>>((const int64_t*)ids, (const __nv_bfloat16*)dout,
                                                                   (__nv_bfloat16*)grad, (int)n, (int)dim, rows, accumulate);
  return launch_status();
}

}  // extern "C"
