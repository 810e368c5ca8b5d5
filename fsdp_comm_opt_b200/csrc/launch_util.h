// Host helpers shared by the launchers: cached device properties and launch error codes.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

namespace zc {

// Number of SMs of the current device (cached per device index).
inline int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cached[dev] = n > 0 ? n : 148;
  }
  return cached[dev];
}

// CTAs of `kernel` that are resident at once on the whole device: the grid of a persistent loop.  (A larger
// one runs its surplus CTAs after the others have finished their shares, a second wave of the same length.)
// The caller keeps the result: `cached` is one static array per kernel.
template <typename K>
inline int resident_ctas(K kernel, int threads, int dyn_smem, int (&cached)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, dyn_smem) != cudaSuccess || per_sm < 1) {
      cudaGetLastError();
      per_sm = 1;
    }
    cached[dev] = per_sm * sm_count();
  }
  return cached[dev];
}

// Clusters of `cluster` CTAs of `kernel` that run at once on the whole device: fewer than its SMs would hold one by one, since a
// cluster lies within a GPC (of 148, 74 clusters of two, 33 of four or 15 of eight CTAs an SM each).  Kept by the caller, as above.
template <typename K>
inline int clusters_at_once(K kernel, int cluster, int threads, int dyn_smem, int (&cached)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = dyn_smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 1;
    }
    cached[dev] = n;
  }
  return cached[dev];
}

// 0 on success, else the cudaError_t of the launch (configuration errors are reported here;
// execution errors surface at the next synchronisation).
inline int launch_status() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// Kernels of a recorded step that follow one another on a stream.  A kernel that begins with chain() (or calls chain_wait()
// before any thread's first access to global memory, and chain_next() once its CTA has what it needs of the SM) may be
// launched by launch_chained: in a launch that is being recorded its CTAs then come up while the kernel before it still runs and
// wait there until that has completed and its results are seen.  Not in launches that run at once: beside collectives, whose
// CTAs need the slots that the waiting ones would hold.  Step of the tiny model (110 kernels)
// 355 -> 334 us, of the small one (190) 1647 -> 1609.
// CTAs that wait have taken the first slots that came free, which may be many to an SM on a few SMs: a kernel of several waves of short
// CTAs does without chain_next(), and the next one's come up as its own end.
// Such a kernel is on the chip while its inputs are still written, so it reads them with ordinary loads, which stay behind the
// wait: the read-only path (__ldg, or a const __restrict__ parameter, of which the compiler makes the same) is for data that do
// not change while a kernel runs, and its loads may be moved ahead of the wait.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain() {
  chain_wait();
  chain_next();
}
// an ordinary load of what nobody reads again
__device__ __forceinline__ float4 ld_once(const float4* p) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
template <typename... P, typename... A>
inline void launch_chained_cluster(int cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                   A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int n = 0;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusActive) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = cluster;
    at[n].val.clusterDim.y = 1;
    at[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  launch_chained_cluster(1, kernel, grid, block, smem, st, args...);
}
#endif

constexpr int ERR_BAD_ARG = -1;
constexpr int ERR_UNSUPPORTED = -2;

}  // namespace zc
