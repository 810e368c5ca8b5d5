// What the default attention kernels (forward and backward) share: moving registers between warpgroups, two fp32
// operations an instruction, tcgen05.st, and a barrier that agrees on a failure.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace zc {

// Registers are moved between the warpgroups of a block; the shares have to add up to what it was launched with.
template <int N>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// pairs of fp32 values, one instruction for both
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// registers -> TMEM: 32 lanes x 32 columns of 32-bit values; thread t of the warp writes lane t
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// barrier over `nthreads` threads that also ORs a predicate: every participant gets the same answer,
// so all of them leave a loop at the same barrier when one of them timed out
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %3, 0;\n"
      "bar.red.or.pred q, %1, %2, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(id), "r"(nthreads), "r"((uint32_t)pred)
      : "memory");
  return r != 0;
}

// 64 columns of a warp's 32 rows, a row a lane (bf16 pairs), through `buf` (4 KB of shared memory of the warp's) to global
// memory: whole 128-byte lines, four rows an instruction.  `dst` is row 0's first column, rows lie `stride` elements apart;
// the first `rows` of them are stored.  (16 bytes of 32 rows an instruction, as the lanes hold them, take 60 clocks each.)
__device__ __forceinline__ void store_rows64(uint8_t* buf, const uint32_t (&pk)[32], __nv_bfloat16* dst, int64_t stride, int rows) {
  const int lane = threadIdx.x & 31, row = lane >> 3, chunk = lane & 7;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<uint4*>(buf + lane * 128 + ((q ^ (lane & 7)) << 4)) =
        make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
  __syncwarp();
  uint4 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = *reinterpret_cast<const uint4*>(buf + (4 * q + row) * 128 + ((chunk ^ ((4 * q + row) & 7)) << 4));
  __syncwarp();
  dst += row * stride + chunk * 8;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if (4 * q + row < rows) *reinterpret_cast<uint4*>(dst + (int64_t)(4 * q) * stride) = v[q];
}

}  // namespace zc
