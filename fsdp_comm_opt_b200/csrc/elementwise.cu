// Memory-bound training ops for sm_100a: RMSNorm (+ residual add) forward/backward, RoPE, SwiGLU
// forward/backward, cross-entropy with in-place gradient and fused AdamW.  Every kernel moves 16-byte vectors, keeps fp32 math in registers and touches each
// HBM byte once per pass.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "launch_util.h"

namespace zc {

constexpr unsigned FULLM = 0xffffffffu;

struct alignas(16) BF8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const BF8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ BF8 pack8(const float (&f)[8]) {
  BF8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}
__device__ __forceinline__ BF8 ld8(const __nv_bfloat16* p) { return *reinterpret_cast<const BF8*>(p); }
__device__ __forceinline__ void st8(__nv_bfloat16* p, const BF8& v) { *reinterpret_cast<BF8*>(p) = v; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULLM, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(FULLM, v, o));
  return v;
}

// block-wide sum for up to 1024 threads; every thread gets the result
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  return warp_sum(t);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : -CUDART_INF_F;
  return warp_max(t);
}

// ---------------------------------------------------------------------------------------------
// RMSNorm (cols <= 8192, cols % 8 == 0).
//   h = x (+ residual, rounded to bf16);  rstd = rsqrt(mean(h^2) + eps);  y = h * rstd * w
// A CTA of NT threads, V vectors of eight columns each, walks its rows with the next row's operands on their way (kept as
// they are stored) and one barrier a row.  Bound by HBM: with the residual 4096 rows of 4096 columns take 24.9 us (the bytes
// 20.5; a warp a row 36.9, a CTA a row 29.8), of 5120 32.9 (25.6; 43.2), of 8192 46.7 (41.0; 62.8); 512 rows of 1024 columns 2.3.
// ---------------------------------------------------------------------------------------------
constexpr int RN_MAX_COLS = 8192;

template <int NT, int V, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) rmsnorm_fwd_kernel(
    const __nv_bfloat16* x, const __nv_bfloat16* res,
    const __nv_bfloat16* w, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
    float* __restrict__ rstd_out, int64_t rows, int cols, float eps) {
  chain();
  __shared__ float red[2][NT / 32];
  const int nvec = cols / 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  BF8 wv[V], a[V], b[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int v = threadIdx.x + i * NT;
    if (v < nvec) wv[i] = ld8(w + v * 8);
  }
  auto fetch = [&](int64_t row) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int v = threadIdx.x + i * NT;
      if (v < nvec) {
        a[i] = ld8(x + row * cols + v * 8);
        if (res) b[i] = ld8(res + row * cols + v * 8);
      }
    }
  };
  int64_t row = blockIdx.x;
  if (row < rows) fetch(row);
  for (int k = 0; row < rows; ++k) {
    const int64_t here = row;
    BF8 hv[V];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      hv[i] = a[i];
      if (res) {
        float f[8], r[8];
        unpack8(a[i], f);
        unpack8(b[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += r[j];
        hv[i] = pack8(f);  // the rounded sum is what gets normalised, as the unfused op order would
      }
    }
    row += gridDim.x;
    if (row < rows) fetch(row);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int v = threadIdx.x + i * NT;
      if (v < nvec) {
        if (res) st8(h_out + here * cols + v * 8, hv[i]);
        float f[8];
        unpack8(hv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) red[k & 1][warp] = ss;
    __syncthreads();  // the only one: a warp writes this half of `red` again after the next row's
    ss = warp_sum(lane < NT / 32 ? red[k & 1][lane] : 0.f);
    const float rstd = rsqrtf(ss / (float)cols + eps);
    if (threadIdx.x == 0) rstd_out[here] = rstd;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int v = threadIdx.x + i * NT;
      if (v < nvec) {
        float f[8], wf[8];
        unpack8(hv[i], f);
        unpack8(wv[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * wf[j];
        st8(y + here * cols + v * 8, pack8(f));
      }
    }
  }
}

// The sum of 32 W values, s[w] of lane l that of thread 32 w + l, in the order in which a CTA of W warps adds them up above: over the
// lanes of each warp, then over the warps.  A lane passes on half of its values at each of the first steps.
template <int W>
__device__ __forceinline__ float cta_sum(float (&s)[W]) {
  static_assert(W == 4 || W == 8, "the CTAs above");
  const int lane = threadIdx.x & 31;
  int step = 16;
#pragma unroll
  for (int n = W / 2; n > 0; n /= 2, step /= 2) {
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const bool hi = lane & step;
      const float mine = hi ? s[i + n] : s[i], other = hi ? s[i] : s[i + n];
      s[i] = mine + __shfl_xor_sync(FULLM, other, step);
    }
  }
  float v = s[0];
#pragma unroll
  for (int o = 16 / W; o > 0; o >>= 1) v += __shfl_xor_sync(FULLM, v, o);
#pragma unroll
  for (int o = 16; o >= 32 / W; o >>= 1) v += __shfl_xor_sync(FULLM, v, o);
  return v;
}

// The same as the kernel above, in the same bits, with a warp a row of up to NV vectors a lane, four rows a CTA: no barrier, a row's
// loads all in flight and the row kept as it is stored.  The next kernel's CTAs come up as these end: among many short CTAs they are in the
// way (recorded one behind the other, 4096 rows of 1024 columns take 6.7 us, 8.9 with the next one's on the chip from the start).
template <int NV>
__global__ void __launch_bounds__(128) rmsnorm_fwd_warp_kernel(
    const __nv_bfloat16* x, const __nv_bfloat16* res,
    const __nv_bfloat16* w, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
    float* __restrict__ rstd_out, int64_t rows, int cols, float eps) {
  chain_wait();
  const int lane = threadIdx.x & 31, nvec = cols / 8;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  BF8 hv[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) hv[i] = ld8(x + row * cols + v * 8);
  }
  if (res) {
    BF8 rv[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) rv[i] = ld8(res + row * cols + v * 8);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        float f[8], r[8];
        unpack8(hv[i], f);
        unpack8(rv[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += r[j];
        hv[i] = pack8(f);
        st8(h_out + row * cols + v * 8, hv[i]);
      }
    }
  }
  constexpr int W = NV > 4 ? 8 : 4;
  float part[W] = {};
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (lane + 32 * i < nvec) {
      float f[8];
      unpack8(hv[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) part[i % W] += f[j] * f[j];
    }
  }
  const float ss = cta_sum(part);
  const float rstd = rsqrtf(ss / (float)cols + eps);
  if (lane == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
      float f[8], wf[8];
      unpack8(hv[i], f);
      unpack8(ld8(w + v * 8), wf);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * wf[j];
      st8(y + row * cols + v * 8, pack8(f));
    }
  }
}

// dx = rstd * (g - xhat * mean(g * xhat)) (+ dh),  g = dy * w,  xhat = h * rstd
// dw = sum_rows dy * xhat: every CTA keeps partial sums in registers over its rows and writes them
// to its row of `partials` ([gridDim.x, cols] fp32), which rmsnorm_dw_reduce_kernel then sums
// (one fp32 atomic per column and CTA instead was 2.4 M atomics on 4096 addresses per call and
// took most of the kernel's time); with partials == nullptr the atomics into dw32 remain.
// A CTA of NT threads, V vectors of eight columns each, walks its rows with the next row's operands on their way (kept as
// they are stored, 16 bytes a vector) and one barrier a row.  Bound by HBM: 4096 rows of 4096 columns 41.6 -> 31.3 us (the
// bytes take 20.5), of 5120 91.8 -> 47.3, of 8192 120.5 -> 61.8 (41.0) against loads that begin after the row before.  Up to 2048
// columns smaller CTAs, four to an SM (65536 rows of 2048: 263 -> 176), or where an SM has ten rows at most one vector a thread, of
// fewer partial sums (1000 rows: 10.4 -> 9.1).
template <int NT, int V, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) rmsnorm_bwd_kernel(
    const __nv_bfloat16* dy, const __nv_bfloat16* h,
    const __nv_bfloat16* w, const float* rstd_in,
    const __nv_bfloat16* dh, __nv_bfloat16* __restrict__ dx, float* __restrict__ dw32,
    float* __restrict__ partials, int64_t rows, int cols) {
  chain();
  __shared__ float red[2][NT / 32];
  const int nvec = cols / 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  BF8 wv[V], d[V], x[V], e[V];  // e: the residual path's gradient
  float dwacc[V][8], rstd = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int v = threadIdx.x + i * NT;
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
    if (v < nvec) wv[i] = ld8(w + v * 8);
  }
  auto fetch = [&](int64_t row) {
    rstd = rstd_in[row];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int v = threadIdx.x + i * NT;
      if (v < nvec) {
        d[i] = ld8(dy + row * cols + v * 8);
        x[i] = ld8(h + row * cols + v * 8);
        if (dh) e[i] = ld8(dh + row * cols + v * 8);
      }
    }
  };
  int64_t row = blockIdx.x;
  if (row < rows) fetch(row);
  for (int k = 0; row < rows; ++k) {
    BF8 cd[V], cx[V], ce[V];
    const float r = rstd;
    const int64_t here = row;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      cd[i] = d[i];
      cx[i] = x[i];
      ce[i] = e[i];
    }
    row += gridDim.x;
    if (row < rows) fetch(row);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if ((int)threadIdx.x + i * NT < nvec) {
        float df[8], xh[8], wf[8];
        unpack8(cd[i], df);
        unpack8(cx[i], xh);
        unpack8(wv[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[j] *= r;
          dot += (df[j] * wf[j]) * xh[j];
          dwacc[i][j] += df[j] * xh[j];
        }
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) red[k & 1][warp] = dot;
    __syncthreads();  // the only one: a warp writes this half of `red` again after the next row's
    dot = warp_sum(lane < NT / 32 ? red[k & 1][lane] : 0.f) / (float)cols;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int v = threadIdx.x + i * NT;
      if (v < nvec) {
        float df[8], xh[8], wf[8], o[8];
        unpack8(cd[i], df);
        unpack8(cx[i], xh);
        unpack8(wv[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = r * (df[j] * wf[j] - xh[j] * r * dot);
        if (dh) {
          float ef[8];
          unpack8(ce[i], ef);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += ef[j];
        }
        st8(dx + here * cols + v * 8, pack8(o));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int v = threadIdx.x + i * NT;
    if (v < nvec) {
      if (partials) {
        float4* dst = reinterpret_cast<float4*>(partials + (int64_t)blockIdx.x * cols + v * 8);
        dst[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
        dst[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) atomicAdd(dw32 + v * 8 + j, dwacc[i][j]);
      }
    }
  }
}

// dw[c] = sum over the CTAs' partial rows; block (8, 128): 8 float4 columns (128 bytes of a row) x 128 row groups.  A
// latency: 1024 columns are 32 blocks of a few loads each (3.0 us; 8 blocks of 32 x 32 threads took 5.1).
__global__ void __launch_bounds__(1024) rmsnorm_dw_reduce_kernel(const float* partials, int nblocks,
                                                                int cols, float* __restrict__ dw) {
  chain();
  __shared__ float4 acc[8][33];
  const int c4 = blockIdx.x * 8 + threadIdx.x;  // float4 column
  const int lane = (threadIdx.y * 8 + threadIdx.x) & 31, warp = threadIdx.y >> 2;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c4 * 4 < cols) {
    for (int r = threadIdx.y; r < nblocks; r += 512) {  // four rows' loads in flight
      float4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (r + 128 * k < nblocks) v[k] = reinterpret_cast<const float4*>(partials + (int64_t)(r + 128 * k) * cols)[c4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (r + 128 * k < nblocks) { s.x += v[k].x; s.y += v[k].y; s.z += v[k].z; s.w += v[k].w; }
    }
  }
  auto add_lanes = [&](int k) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, k);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, k);
    s.z += __shfl_xor_sync(0xffffffffu, s.z, k);
    s.w += __shfl_xor_sync(0xffffffffu, s.w, k);
  };
  add_lanes(8);   // the warp's four row groups
  add_lanes(16);
  if (lane < 8) acc[lane][warp] = s;
  __syncthreads();
  if (warp >= 8) return;
  s = acc[warp][lane];  // warp w: column w of the 32 warps
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) add_lanes(k);
  if (lane == 0 && (blockIdx.x * 8 + warp) * 4 < cols) reinterpret_cast<float4*>(dw)[blockIdx.x * 8 + warp] = s;
}

// ---------------------------------------------------------------------------------------------
// RoPE in place on the first n_rot heads of a packed [T, total_heads * D] tensor
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) rope_kernel(__nv_bfloat16* __restrict__ qkv, const float* cosT,
                                                   const float* sinT, int64_t T, int S, int n_rot,
                                                   int total_heads, int D, float sign) {
  chain();
  const int vph = D / 16;  // 8-element vectors per half head
  const int64_t total = T * n_rot * vph;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int v = (int)(idx % vph);
    const int hd = (int)((idx / vph) % n_rot);
    const int64_t t = idx / ((int64_t)vph * n_rot);
    const int pos = (int)(t % S);
    __nv_bfloat16* p = qkv + (t * total_heads + hd) * D + v * 8;
    float a[8], b[8], oa[8], ob[8];
    unpack8(ld8(p), a);
    unpack8(ld8(p + D / 2), b);
    const float4* c4 = reinterpret_cast<const float4*>(cosT + (int64_t)pos * (D / 2) + v * 8);
    const float4* s4 = reinterpret_cast<const float4*>(sinT + (int64_t)pos * (D / 2) + v * 8);
    const float4 c0 = c4[0], c1 = c4[1], s0 = s4[0], s1 = s4[1];
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sj = s[j] * sign;
      oa[j] = a[j] * c[j] - b[j] * sj;
      ob[j] = b[j] * c[j] + a[j] * sj;
    }
    st8(p, pack8(oa));
    st8(p + D / 2, pack8(ob));
  }
}

// ---------------------------------------------------------------------------------------------
// SwiGLU on packed [T, 2F] = [gate | up]
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const __nv_bfloat16* gu,
                                                         __nv_bfloat16* __restrict__ out, int64_t T, int F) {
  chain();
  const int vpr = F / 8;
  const int64_t total = T * vpr;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / vpr;
    const int v = (int)(idx % vpr);
    float g[8], u[8], o[8];
    unpack8(ld8(gu + t * 2 * F + v * 8), g);
    unpack8(ld8(gu + t * 2 * F + F + v * 8), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    st8(out + t * F + v * 8, pack8(o));
  }
}

__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const __nv_bfloat16* gu,
                                                         const __nv_bfloat16* dy,
                                                         __nv_bfloat16* __restrict__ dgu, int64_t T, int F) {
  chain();
  const int vpr = F / 8;
  const int64_t total = T * vpr;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / vpr;
    const int v = (int)(idx % vpr);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(ld8(gu + t * 2 * F + v * 8), g);
    unpack8(ld8(gu + t * 2 * F + F + v * 8), u);
    unpack8(ld8(dy + t * F + v * 8), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      dg[j] = d[j] * u[j] * s * (1.f + g[j] * (1.f - s));
      du[j] = d[j] * g[j] * s;
    }
    st8(dgu + t * 2 * F + v * 8, pack8(dg));
    st8(dgu + t * 2 * F + F + v * 8, pack8(du));
  }
}

// ---------------------------------------------------------------------------------------------
// Cross-entropy with the row kept on the chip: one CTA, or a cluster of two, holds a row's 8-element vectors in
// shared memory between the two passes (maximum and sum; gradient); two CTAs exchange their maxima and sums
// through distributed shared memory.  A row is read once, and with at most CE_SMEM bytes a CTA three of them share
// an SM, so that one loads while another exponentiates.  Bound by HBM, the two exponentials a value close behind.
// 4096 x 32000: 216 -> 148 us, 1024 x 32768: 44 -> 30, 2048 x 50257 (two CTAs): 140 -> 120, against a second read from L2.
// Clusters of four lose (4096 x 128256: 717 us against 624): longer rows are read twice, by ce_kernel (564 with four loads in
// flight a thread).
// ---------------------------------------------------------------------------------------------
constexpr int CE_THREADS = 512, CE_SMEM = 72 * 1024;

// running maximum and sum of exponentials of eight more logits
__device__ __forceinline__ void ce_add8(const BF8& q, float& m, float& s) {
  float f[8];
  unpack8(q, f);
  float lm = f[0];
#pragma unroll
  for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
  if (lm > m) { s *= __expf(m - lm); m = lm; }
  const float ms = m == -CUDART_INF_F ? 0.f : m;  // masked logits only, so far: they add nothing
#pragma unroll
  for (int j = 0; j < 8; ++j) s += __expf(f[j] - ms);
}
// (softmax - onehot) * scale; `hot` is the label's place among the eight, if it is there
__device__ __forceinline__ BF8 ce_grad8(const BF8& q, float gm, float inv_s, float scale, int64_t hot) {
  float f[8];
  unpack8(q, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float p = __expf(f[j] - gm) * inv_s;
    if (j == hot) p -= 1.f;
    f[j] = p * scale;
  }
  return pack8(f);
}

template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CE_THREADS, 3)
    ce_row_kernel(__nv_bfloat16* __restrict__ logits, const int64_t* labels, float* __restrict__ row_loss,
                  const float* inv_count, int V, int64_t ld, int ignore_index) {
  chain();
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) uint8_t ce_smem[];
  BF8* part = reinterpret_cast<BF8*>(ce_smem);
  __shared__ float red[32];
  __shared__ float2 stat;  // this CTA's maximum and sum of exponentials
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CL == 1 ? 0 : (int)cluster.block_rank();
  const int64_t row = blockIdx.x / CL;
  __nv_bfloat16* lr = logits + row * ld;
  const int64_t label = labels[row];
  const int nvec = V / 8, per = (nvec + CL - 1) / CL, v0 = rank * per, v1 = min(nvec, v0 + per);
  const int tail0 = nvec * 8;  // the last V % 8 columns and the padding: the last CTA, one by one
  const bool tail = rank == CL - 1;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  if (label == ignore_index) {  // the whole cluster
    BF8 z;
#pragma unroll
    for (int i = 0; i < 4; ++i) z.v[i] = __floats2bfloat162_rn(0.f, 0.f);
    for (int v = v0 + threadIdx.x; v < v1; v += CE_THREADS) st8(lr + (int64_t)v * 8, z);
    if (tail)
      for (int64_t i = tail0 + threadIdx.x; i < ld; i += CE_THREADS) lr[i] = zero;
    if (rank == 0 && threadIdx.x == 0) row_loss[row] = 0.f;
    return;
  }
  float m = -CUDART_INF_F, s = 0.f;
  for (int v = v0 + threadIdx.x; v < v1; v += 4 * CE_THREADS) {
    BF8 q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (v + k * CE_THREADS < v1) q[k] = ld8(lr + (int64_t)(v + k * CE_THREADS) * 8);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (v + k * CE_THREADS < v1) {
        part[v - v0 + k * CE_THREADS] = q[k];
        ce_add8(q[k], m, s);
      }
  }
  if (tail)
    for (int i = tail0 + threadIdx.x; i < V; i += CE_THREADS) {
      const float f = __bfloat162float(lr[i]);
      if (f > m) { s *= __expf(m - f); m = f; }
      s += __expf(f - (m == -CUDART_INF_F ? 0.f : m));
    }
  float gm = block_max(m, red);
  s = (m == -CUDART_INF_F) ? s : s * __expf(m - gm);
  float gs = block_sum(s, red);
  if (CL > 1) {
    if (threadIdx.x == 0) stat = make_float2(gm, gs);
    cluster.sync();
    float2 st[CL];
#pragma unroll
    for (int k = 0; k < CL; ++k) st[k] = *cluster.map_shared_rank(&stat, k);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // waited for before leaving
    gm = st[0].x;
#pragma unroll
    for (int k = 1; k < CL; ++k) gm = fmaxf(gm, st[k].x);
    gs = 0.f;
#pragma unroll
    for (int k = 0; k < CL; ++k) gs += st[k].x == -CUDART_INF_F ? st[k].y : st[k].y * __expf(st[k].x - gm);
  }
  const float scale = inv_count[0], inv_s = 1.f / gs;
  // the CTA that holds the label's logit writes the loss (shared memory, or a tail column that this thread reads before
  // it overwrites any); a label that nobody holds, which the CPU path refuses, makes it NaN
  if (threadIdx.x == 0 && rank == 0 && (label < 0 || label >= V)) row_loss[row] = CUDART_NAN_F;
  if (threadIdx.x == (int)((label - tail0) & (CE_THREADS - 1)) && tail && label >= tail0 && label < V)
    row_loss[row] = gm + __logf(gs) - __bfloat162float(lr[label]);
  if (threadIdx.x == 0 && label >= (int64_t)v0 * 8 && label < (int64_t)v1 * 8)
    row_loss[row] = gm + __logf(gs) - __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(part)[label - (int64_t)v0 * 8]);
  for (int v = v0 + threadIdx.x; v < v1; v += CE_THREADS) {
    st8(lr + (int64_t)v * 8, ce_grad8(part[v - v0], gm, inv_s, scale, label - (int64_t)v * 8));
  }
  if (tail)
    for (int64_t i = tail0 + threadIdx.x; i < ld; i += CE_THREADS) {
      if (i < V) {
        float p = __expf(__bfloat162float(lr[i]) - gm) * inv_s;
        if (i == label) p -= 1.f;
        lr[i] = __float2bfloat16(p * scale);
      } else {
        lr[i] = zero;
      }
    }
  if (CL > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int CL>
static int ce_rows(__nv_bfloat16* logits, const int64_t* labels, float* row_loss, const float* inv_count, int64_t T, int V,
                   int64_t ld, int ignore_index, cudaStream_t st) {
  const int smem = ((V / 8 + CL - 1) / CL) * 16;
  if (cudaFuncSetAttribute(ce_row_kernel<CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, CE_SMEM) != cudaSuccess)
    return launch_status();
  zc::launch_chained(ce_row_kernel<CL>, (unsigned)(T * CL), CE_THREADS, smem, st, logits, labels, row_loss, inv_count, V, ld, ignore_index);
  return launch_status();
}

// ---------------------------------------------------------------------------------------------
// Cross-entropy of rows that are not aligned or too long for two CTAs' shared memory: one CTA per row; pass 1 online max / sum-exp, pass 2 writes the gradient over the
// logits.  row_loss = lse - logit[label];  grad = (softmax - onehot) * inv_count
// Rows are `ld` elements apart (ld >= V; ld > V for a vocabulary that is not a multiple of 8, whose
// logits the GEMM writes into rows padded to an aligned stride); the pad columns come out as zeros.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(CE_THREADS, 3) ce_kernel(__nv_bfloat16* __restrict__ logits,
                                                  const int64_t* labels,
                                                  float* __restrict__ row_loss, const float* inv_count,
                                                  int V, int64_t ld, int ignore_index) {
  chain();
  __shared__ float red[32];
  const int64_t row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const int64_t label = labels[row];
  // whole 8-element vectors when the row starts on 16 bytes; the last V % 8 columns one by one
  const int nvec = ((ld % 8 == 0) && ((reinterpret_cast<uintptr_t>(logits) & 15) == 0)) ? V / 8 : 0;
  const int tail0 = nvec * 8;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  if (label == ignore_index) {
    BF8 z;
#pragma unroll
    for (int i = 0; i < 4; ++i) z.v[i] = __floats2bfloat162_rn(0.f, 0.f);
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) st8(lr + v * 8, z);
    for (int64_t i = tail0 + threadIdx.x; i < ld; i += blockDim.x) lr[i] = zero;
    if (threadIdx.x == 0) row_loss[row] = 0.f;
    return;
  }
  float m = -CUDART_INF_F, s = 0.f;
  // four vectors in flight per thread and pass
  for (int v = threadIdx.x; v < nvec; v += 4 * CE_THREADS) {
    BF8 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * CE_THREADS < nvec) q[u] = ld8(lr + (int64_t)(v + u * CE_THREADS) * 8);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * CE_THREADS < nvec) ce_add8(q[u], m, s);
  }
  for (int i = tail0 + threadIdx.x; i < V; i += blockDim.x) {
    const float f = __bfloat162float(lr[i]);
    if (f > m) { s *= __expf(m - f); m = f; }
    s += __expf(f - (m == -CUDART_INF_F ? 0.f : m));
  }
  const float gm = block_max(m, red);
  s = (m == -CUDART_INF_F) ? s : s * __expf(m - gm);
  const float gs = block_sum(s, red);
  const float lse = gm + __logf(gs);
  const float scale = inv_count[0];
  const float picked = label >= 0 && label < V ? __bfloat162float(lr[label]) : CUDART_NAN_F;
  __syncthreads();  // everyone has read lr[label] before it is overwritten
  if (threadIdx.x == 0) row_loss[row] = lse - picked;
  const float inv_s = 1.f / gs;
  for (int v = threadIdx.x; v < nvec; v += 4 * CE_THREADS) {
    BF8 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * CE_THREADS < nvec) q[u] = ld8(lr + (int64_t)(v + u * CE_THREADS) * 8);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * CE_THREADS < nvec)
        st8(lr + (int64_t)(v + u * CE_THREADS) * 8, ce_grad8(q[u], gm, inv_s, scale, label - (int64_t)(v + u * CE_THREADS) * 8));
  }
  for (int64_t i = tail0 + threadIdx.x; i < ld; i += blockDim.x) {
    if (i < V) {
      float p = __expf(__bfloat162float(lr[i]) - gm) * inv_s;
      if (i == label) p -= 1.f;
      lr[i] = __float2bfloat16(p * scale);
    } else {
      lr[i] = zero;
    }
  }
}

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half(v); }

// ---------------------------------------------------------------------------------------------
// AdamW (decoupled weight decay), one launch per shard
// ---------------------------------------------------------------------------------------------
template <typename TP, typename TG, typename TS>
__global__ void __launch_bounds__(256) adamw_kernel(TP* __restrict__ p, TG* __restrict__ g, TS* __restrict__ m,
                                                    TS* __restrict__ v, int64_t n, float lr, float b1, float b2,
                                                    float eps, float wd, float bc1, float rsqrt_bc2, int zero_grad, const int* __restrict__ guard) {
  if (guard && *guard) return;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const float gf = to_f<TG>(g[i]);
    float pf = to_f<TP>(p[i]);
    float mf = to_f<TS>(m[i]) * b1 + (1.f - b1) * gf;
    float vf = to_f<TS>(v[i]) * b2 + (1.f - b2) * gf * gf;
    pf *= 1.f - lr * wd;
    const float denom = sqrtf(vf) * rsqrt_bc2 + eps;
    pf -= (lr / bc1) * mf / denom;
    p[i] = from_f<TP>(pf);
    m[i] = from_f<TS>(mf);
    v[i] = from_f<TS>(vf);
    if (zero_grad) g[i] = from_f<TG>(0.f);
  }
}

// eight elements per thread, 16-byte accesses (pointers 16-byte aligned, n % 8 == 0)
template <typename T> __device__ __forceinline__ void load8(const T* p, float (&f)[8]);
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&f)[8]) {
  unpack8(ld8(p), f);
}
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float (&f)[8]);
template <> __device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16* p, const float (&f)[8]) {
  st8(p, pack8(f));
}
template <> __device__ __forceinline__ void store8<float>(float* p, const float (&f)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}

template <typename TP, typename TG, typename TS>
__global__ void __launch_bounds__(256) adamw_vec_kernel(TP* __restrict__ p, TG* __restrict__ g, TS* __restrict__ m,
                                                        TS* __restrict__ v, int64_t nvec, float lr, float b1, float b2,
                                                        float eps, float wd, float bc1, float rsqrt_bc2,
                                                        int zero_grad, const int* guard) {
  chain();
  if (guard && *guard) return;  // a collective of this step gave up: leave parameters and moments alone
  const float decay = 1.f - lr * wd, step = lr / bc1;
  auto update = [&](float (&pf)[8], const float (&gf)[8], float (&mf)[8], float (&vf)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      mf[j] = mf[j] * b1 + (1.f - b1) * gf[j];
      vf[j] = vf[j] * b2 + (1.f - b2) * gf[j] * gf[j];
      pf[j] = pf[j] * decay - step * mf[j] / (sqrtf(vf[j]) * rsqrt_bc2 + eps);
    }
  };
  const float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // two vectors a thread, eight 16-byte loads (or more) in flight before the first use: 512 in a row a CTA, or half the buffer apart
  // where all four streams are 32 bits (below)
  constexpr bool APART = sizeof(TP) + sizeof(TG) + sizeof(TS) == 12;
  const int64_t i = (int64_t)blockIdx.x * (APART ? 256 : 512) + threadIdx.x, k = i + (APART ? (int64_t)gridDim.x * 256 : 256);
  if (k < nvec) {
    float pf[8], gf[8], mf[8], vf[8], pf2[8], gf2[8], mf2[8], vf2[8];
    load8<TP>(p + i * 8, pf);
    load8<TG>(g + i * 8, gf);
    load8<TS>(m + i * 8, mf);
    load8<TS>(v + i * 8, vf);
    load8<TP>(p + k * 8, pf2);
    load8<TG>(g + k * 8, gf2);
    load8<TS>(m + k * 8, mf2);
    load8<TS>(v + k * 8, vf2);
    update(pf, gf, mf, vf);
    update(pf2, gf2, mf2, vf2);
    store8<TP>(p + i * 8, pf);
    store8<TS>(m + i * 8, mf);
    store8<TS>(v + i * 8, vf);
    store8<TP>(p + k * 8, pf2);
    store8<TS>(m + k * 8, mf2);
    store8<TS>(v + k * 8, vf2);
    if (zero_grad) {
      store8<TG>(g + i * 8, z);
      store8<TG>(g + k * 8, z);
    }
  } else if (i < nvec) {
    float pf[8], gf[8], mf[8], vf[8];
    load8<TP>(p + i * 8, pf);
    load8<TG>(g + i * 8, gf);
    load8<TS>(m + i * 8, mf);
    load8<TS>(v + i * 8, vf);
    update(pf, gf, mf, vf);
    store8<TP>(p + i * 8, pf);
    store8<TS>(m + i * 8, mf);
    store8<TS>(v + i * 8, vf);
    if (zero_grad) store8<TG>(g + i * 8, z);
  }
}

template <typename TP, typename TG, typename TS>
int adamw_launch(void* p, void* g, void* m, void* v, int64_t n, float lr, float b1, float b2, float eps, float wd,
                 float bc1, float rs, int zg, const int* guard, cudaStream_t st) {
  const bool vec = (n % 8 == 0) && (((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) |
                                      reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15) == 0);
  if (vec) {
    const int64_t nvec = n / 8;
    // A CTA to 512 vectors in a row: 8 KB of every stream, and CTAs that follow one another in address order.  4 x 10^8
    // elements: 803 us (6.98 TB/s; a copy 6.48); CTAs that stride through the buffers, a few dozen per SM, with the
    // second vector of a trip a whole grid further, took 920, the same with 8 KB in a row 839.
    // All in 32 bits the second vector is a grid further: 5 x 10^7 elements 209 us, 213 with 16 KB in a row; 3.4 x 10^6 in L2 12.4 and 14.5.
    const int64_t grid = (nvec + 511) / 512;
    if (grid > 0x7fffffff) return ERR_BAD_ARG;
    zc::launch_chained(adamw_vec_kernel<TP, TG, TS>, (unsigned)grid, 256, 0, st, (TP*)p, (TG*)g, (TS*)m, (TS*)v, nvec, lr, b1, b2, eps, wd,
                                                        bc1, rs, zg, guard);
  } else {
    const int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)sm_count() * 16);
    adamw_kernel<TP, TG, TS><<<grid, 256, 0, st>>>((TP*)p, (TG*)g, (TS*)m, (TS*)v, n, lr, b1, b2, eps, wd, bc1, rs,
                                                    zg, guard);
  }
  return launch_status();
}

template <typename TP, typename TG>
int adamw_dispatch_s(void* p, void* g, void* m, void* v, int64_t n, int sdt, float lr, float b1, float b2, float eps,
                     float wd, float bc1, float bc2, int zg, const int* guard, cudaStream_t st) {
  const float rs = 1.f / sqrtf(bc2);
  if (sdt == 0) return adamw_launch<TP, TG, __nv_bfloat16>(p, g, m, v, n, lr, b1, b2, eps, wd, bc1, rs, zg, guard, st);
  if (sdt == 1) return adamw_launch<TP, TG, float>(p, g, m, v, n, lr, b1, b2, eps, wd, bc1, rs, zg, guard, st);
  return ERR_UNSUPPORTED;
}

}  // namespace zc

extern "C" {

using zc::ERR_BAD_ARG;
using zc::ERR_UNSUPPORTED;
typedef __nv_bfloat16 bf16;

int zc_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int64_t rows,
                   int cols, float eps, cudaStream_t st) {
  if (cols % 8 || cols > zc::RN_MAX_COLS) return ERR_UNSUPPORTED;
  if (rows == 0) return 0;
#define ZC_RN_FWD(kernel, grid, threads)                                                                               \
  zc::launch_chained(kernel, (unsigned)(grid), threads, 0, st, (const bf16*)x, (const bf16*)res, (const bf16*)w,       \
                     (bf16*)y, (bf16*)h_out, rstd, rows, cols, eps)
  const int64_t sms = zc::sm_count(), quads = (rows + 3) / 4;
  // From six rows an SM on, a warp a row where a lane holds it in few registers: (us, a CTA a row and a warp a row) 65536 rows of 64
  // columns 33.5 and 17.7, of 512 57 and 30, of 2048 152 and 110, with the residual 218 and 182; 1000 rows of 1024 3.1 and 2.8, 700 2.1 and
  // 2.7; without the residual 16384 of 3072 51.5 and 45.3, with it 76.0 and 77.4.
  if (rows > 6 * sms && (cols <= 2048 || (cols <= 3072 && !res))) {
    if (cols <= 1024) ZC_RN_FWD(zc::rmsnorm_fwd_warp_kernel<4>, quads, 128);
    else if (cols <= 2048) ZC_RN_FWD(zc::rmsnorm_fwd_warp_kernel<8>, quads, 128);
    else ZC_RN_FWD(zc::rmsnorm_fwd_warp_kernel<12>, quads, 128);
  } else if (cols <= 128 * 8) {
    ZC_RN_FWD((zc::rmsnorm_fwd_kernel<128, 1, 8>), std::min(rows, sms * 8), 128);
  } else if (cols <= 256 * 2 * 8) {
    ZC_RN_FWD((zc::rmsnorm_fwd_kernel<256, 2, 3>), std::min(rows, sms * 3), 256);
  } else {
    ZC_RN_FWD((zc::rmsnorm_fwd_kernel<512, 2, 2>), std::min(rows, sms * 2), 512);
  }
#undef ZC_RN_FWD
  return zc::launch_status();
}

// CTAs that the backward launches for `rows` rows at most: the number of rows `partials` must have
int zc_rmsnorm_bwd_ctas(int64_t rows) { return (int)std::min<int64_t>(rows, (int64_t)zc::sm_count() * 4); }

// dw32: [cols] fp32.  With partials ([zc_rmsnorm_bwd_ctas(rows), cols] fp32) it is overwritten with
// the column sums; with partials == nullptr it must be zero on entry and is accumulated with atomics.
int zc_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dh, void* dx,
                   float* dw32, float* partials, int64_t rows, int cols, cudaStream_t st) {
  if (cols % 8 || cols > zc::RN_MAX_COLS) return ERR_UNSUPPORTED;
  if (rows == 0) return 0;
  // as many CTAs as run at once; narrow rows do not hold a thread's loads long enough for that to matter
  int grid = 0;
#define ZC_RN_BWD(NT, V, PER_SM)                                                                                       \
  grid = (int)std::min<int64_t>(rows, (int64_t)zc::sm_count() * PER_SM);                                               \
  zc::launch_chained(zc::rmsnorm_bwd_kernel<NT, V, PER_SM>, grid, NT, 0, st, (const bf16*)dy, (const bf16*)h,          \
                     (const bf16*)w, rstd, (const bf16*)dh, (bf16*)dx, dw32, partials, rows, cols)
  if (cols <= 128 * 8) { ZC_RN_BWD(128, 1, 4); }
  else if (cols <= 256 * 8 && rows <= 10 * (int64_t)zc::sm_count()) { ZC_RN_BWD(256, 1, 2); }
  else if (cols <= 256 * 8) { ZC_RN_BWD(128, 2, 4); }
  else if (cols <= 256 * 2 * 8) { ZC_RN_BWD(256, 2, 2); }
  else { ZC_RN_BWD(512, 2, 1); }
#undef ZC_RN_BWD
  if (partials)
    zc::launch_chained(zc::rmsnorm_dw_reduce_kernel, (cols / 4 + 7) / 8, dim3(8, 128), 0, st, partials, grid, cols, dw32);
  return zc::launch_status();
}

int zc_rope_inplace(void* qkv, const float* cosT, const float* sinT, int64_t T, int S, int n_rot, int total_heads,
                    int D, float sign, cudaStream_t st) {
  if (D % 16 || n_rot > total_heads) return ERR_UNSUPPORTED;
  const int64_t total = T * n_rot * (D / 16);
  if (total == 0) return 0;
  const int grid = (int)std::min<int64_t>((total + 255) / 256, (int64_t)zc::sm_count() * 16);
  zc::launch_chained(zc::rope_kernel, grid, 256, 0, st, (bf16*)qkv, cosT, sinT, T, S, n_rot, total_heads, D, sign);
  return zc::launch_status();
}

int zc_swiglu_fwd(const void* gu, void* out, int64_t T, int F, cudaStream_t st) {
  if (F % 8) return ERR_UNSUPPORTED;
  const int64_t total = T * (F / 8);
  if (total == 0) return 0;
  const int grid = (int)std::min<int64_t>((total + 255) / 256, (int64_t)zc::sm_count() * 128);
  zc::launch_chained(zc::swiglu_fwd_kernel, grid, 256, 0, st, (const bf16*)gu, (bf16*)out, T, F);
  return zc::launch_status();
}

int zc_swiglu_bwd(const void* gu, const void* dy, void* dgu, int64_t T, int F, cudaStream_t st) {
  if (F % 8) return ERR_UNSUPPORTED;
  const int64_t total = T * (F / 8);
  if (total == 0) return 0;
  const int grid = (int)std::min<int64_t>((total + 255) / 256, (int64_t)zc::sm_count() * 128);
  zc::launch_chained(zc::swiglu_bwd_kernel, grid, 256, 0, st, (const bf16*)gu, (const bf16*)dy, (bf16*)dgu, T, F);
  return zc::launch_status();
}

int zc_ce_fwd_bwd_ld(void* logits, const int64_t* labels, float* row_loss, const float* inv_count, int64_t T, int V,
                     int64_t ld, int ignore_index, cudaStream_t st) {
  if (T == 0) return 0;
  if (V <= 0 || ld < V) return ERR_BAD_ARG;
  // the fewest CTAs whose shares fit; a row's vectors have to start on 16 bytes
  const int64_t bytes = (int64_t)(V / 8) * 16;
  if (ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && V >= 8 && bytes <= 2 * (zc::CE_SMEM - 16) &&
      T < (1 << 30)) {
    bf16* lg = (bf16*)logits;
    if (bytes <= zc::CE_SMEM) return zc::ce_rows<1>(lg, labels, row_loss, inv_count, T, V, ld, ignore_index, st);
    return zc::ce_rows<2>(lg, labels, row_loss, inv_count, T, V, ld, ignore_index, st);
  }
  zc::launch_chained(zc::ce_kernel, (unsigned)T, zc::CE_THREADS, 0, st, (bf16*)logits, labels, row_loss, inv_count, V, ld, ignore_index);
  return zc::launch_status();
}

int zc_ce_fwd_bwd(void* logits, const int64_t* labels, float* row_loss, const float* inv_count, int64_t T, int V,
                  int ignore_index, cudaStream_t st) {
  return zc_ce_fwd_bwd_ld(logits, labels, row_loss, inv_count, T, V, V, ignore_index, st);
}

// The library's health word of the current device (0 = healthy): set by a fused collective whose
// bounded wait ran out, read on the device by zc_adamw_guarded, read and cleared on the host by
// zc_health_read_and_clear.  Allocated on first use.
int* zc_health_word() {
  static int* words[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  if (!words[dev]) {
    if (cudaMalloc(&words[dev], sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(words[dev], 0, sizeof(int));
  }
  return words[dev];
}

int zc_health_read_and_clear() {
  int* w = zc_health_word();
  if (!w) return -1;
  int v = 0;
  cudaMemcpy(&v, w, sizeof(int), cudaMemcpyDeviceToHost);
  if (v) cudaMemset(w, 0, sizeof(int));
  return v;
}

// Host-side injection of a failure (tests, drills): what a collective that gave up would have written.
int zc_health_set(int value) {
  int* w = zc_health_word();
  if (!w) return -1;
  return cudaMemcpy(w, &value, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -1;
}

// `guard`: device pointer to a word that must be 0 for the update to happen (null: unconditional).
// With the health word there, an optimizer step that follows a collective which gave up leaves
// parameters and moments untouched, with no host synchronisation between the two.
int zc_adamw_guarded(void* p, void* g, void* m, void* v, int64_t n, int pdt, int gdt, int sdt, float lr, float b1,
                     float b2, float eps, float wd, float bc1, float bc2, int zero_grad, const int* guard,
                     cudaStream_t st) {
  if (n == 0) return 0;
  if (pdt == 0 && gdt == 0)
    return zc::adamw_dispatch_s<bf16, bf16>(p, g, m, v, n, sdt, lr, b1, b2, eps, wd, bc1, bc2, zero_grad, guard, st);
  if (pdt == 1 && gdt == 1)
    return zc::adamw_dispatch_s<float, float>(p, g, m, v, n, sdt, lr, b1, b2, eps, wd, bc1, bc2, zero_grad, guard, st);
  if (pdt == 0 && gdt == 1)
    return zc::adamw_dispatch_s<bf16, float>(p, g, m, v, n, sdt, lr, b1, b2, eps, wd, bc1, bc2, zero_grad, guard, st);
  if (pdt == 1 && gdt == 0)
    return zc::adamw_dispatch_s<float, bf16>(p, g, m, v, n, sdt, lr, b1, b2, eps, wd, bc1, bc2, zero_grad, guard, st);
  return ERR_UNSUPPORTED;
}

int zc_adamw(void* p, void* g, void* m, void* v, int64_t n, int pdt, int gdt, int sdt, float lr, float b1, float b2,
             float eps, float wd, float bc1, float bc2, int zero_grad, cudaStream_t st) {
  return zc_adamw_guarded(p, g, m, v, n, pdt, gdt, sdt, lr, b1, b2, eps, wd, bc1, bc2, zero_grad, nullptr, st);
}

}  // extern "C"
