// Causal GQA attention forward for sm_100a, head dimension 64 (the default forward path there).
//
// One CTA (256 threads, two CTAs per SM) owns 128 queries of one head and walks the key blocks of 128 keys at or below
// the diagonal.  Registers are moved from the first warpgroup to the second with setmaxnreg:
//   warpgroup 0   warp 0: TMA producer: the Q tile once, then K_0, V_0, K_1, V_1, ... into a ring of five slots;
//                 warp 1: MMA issuer, S = Q K^T (128 x 128, fp32 in TMEM) one block ahead, and O += P V
//   warpgroup 1   softmax, one thread per query row.  A thread holds its whole row of S (128 registers), so maximum,
//                 exponentials and row sum need no partner, and hands S back at once; P goes to tensor memory as bf16
//                 pairs and is the A operand of O += P V there.  It is handed over in two halves of 64 keys, so that
//                 the second is exponentiated while the tensor core works on the first.
// TMEM (256 columns, so that two CTAs share an SM): S 128 | O 64 | P 64.
// P is relative to the row's running maximum: raising it rescales the row of O in TMEM.  A maximum that may lag by up to
// 2^8, so that this almost never happens, rounds the largest probabilities to bf16 that are exact ones otherwise: 2 % more
// error against 64 bits (2-norm 0.00208 against 0.00204 at 3000 keys) for 4 % less time (8 x 1024 keys, 25 heads: 66.7
// against 69.7 us).
// What bounds it: the exponentials, 16 per clock and SM, twice the clocks of the matrix products; one CTA's
// set-up, MMAs and epilogue hide behind the other's exponentials.  25 heads: 8 x 1024 keys 137 -> 70 us, 2 x 8192 keys
// 1257 -> 621 (the exponentials alone: 417) against two threads a row and O in registers (attention_ws.cu).
// CTAs are numbered heaviest first (the last queries see the most keys).  Every wait is bounded; a timed-out role
// raises a CTA-wide abort flag, the CTA frees its TMEM and returns, and the launcher's status word reports it.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math_constants.h>

#include "attn_common.cuh"
#include "launch_util.h"

namespace zc {
namespace fwd64 {
using namespace attn;

constexpr int D = 64;
constexpr int THREADS = 256;
constexpr int SLOTS = 5;        // K / V ring
constexpr int TILE = 16384;     // bytes of the Q tile, a K block or a V block: one slab of [128 x 128 B]
constexpr int SMEM = (1 + SLOTS) * TILE + 1024;

struct Params {
  __nv_bfloat16* o;
  float* lse;
  int B, S, Hq, Hkv;
  float scale;
  int* status;
  int nqb;  // number of 128-query blocks
};

__global__ void __launch_bounds__(THREADS, 2) attn_fwd_d64_kernel(const __grid_constant__ CUtensorMap mapQ,
                                                                  const __grid_constant__ CUtensorMap mapK,
                                                                  const __grid_constant__ CUtensorMap mapV,
                                                                  const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + TILE;
  __shared__ uint64_t q_full, kv_full[SLOTS], kv_empty[SLOTS], s_full, s_empty, p_full[2], o_full;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_c = p.Hq * p.B;
  const int qb = p.nqb - 1 - (int)blockIdx.x / per_c;
  const int h = ((int)blockIdx.x % per_c) % p.Hq, b = ((int)blockIdx.x % per_c) / p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const int q0 = qb * 128;
  const int nb = qb + 1;  // key blocks up to the one on the diagonal
  if (tid == 0) {
    mbar_init(&q_full, 1);
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&s_empty, 4);  // one arrival per softmax warp
    mbar_init(&p_full[0], 4);
    mbar_init(&p_full[1], 4);
    mbar_init(&o_full, 1);
    mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base, 256);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm_s = tmem_base, tm_o = tm_s + 128, tm_p = tm_s + 192;
  chain_wait();
  if (warp == 1) chain_next();  // which has its TMEM

  if (warp < 4) {
    regs_dec<48>();  // 48 + 208 = the launch's 2 x 128
    if (warp == 0 && lane == 0) {
      mbar_expect_tx(&q_full, TILE);
      tma_load_4d(sQ, &mapQ, &q_full, 0, h, q0, b);
      for (int n = 0; n < 2 * nb; ++n) {
        const int s = n % SLOTS;
        if (!role_wait(&kv_empty[s], ((n / SLOTS) & 1) ^ 1, &s_abort)) { s_abort = 1; break; }
        mbar_expect_tx(&kv_full[s], TILE);
        tma_load_4d(sKV + s * TILE, (n & 1) ? &mapV : &mapK, &kv_full[s], 0, hk, (n >> 1) * 128, b);
      }
    } else if (warp == 1 && lane == 0) {
      const uint32_t id_s = idesc_bf16(128, 128, MAJOR_K, MAJOR_K);
      const uint32_t id_o = idesc_bf16(128, D, MAJOR_K, MAJOR_MN);
      // Descriptors at offset 0; an MMA adds a constant to their address field (byte offset >> 4; shared memory is below
      // 256 KB, the 14-bit field never carries)
      const uint64_t dQ = smem_desc(smem_u32(sQ), 16, 1024);
      const uint64_t dK0 = smem_desc(smem_u32(sKV), 16, 1024);      // K block in slot 0, K-major
      const uint64_t dV0 = smem_desc(smem_u32(sKV), 16384, 1024);   // V block in slot 0, MN-major
      bool ok = role_wait(&q_full, 0, &s_abort);
      auto issue_s = [&](int j) -> bool {
        const int s = (2 * j) % SLOTS;
        if (!role_wait(&kv_full[s], ((2 * j) / SLOTS) & 1, &s_abort)) return false;
        tc_fence_after_sync();
        const uint64_t dK = dK0 + (uint64_t)(s * (TILE >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          mma_bf16(tm_s, dQ + (uint64_t)((k * 32) >> 4), dK + (uint64_t)((k * 32) >> 4), id_s, k != 0);
        mma_commit(&s_full);
        mma_commit(&kv_empty[s]);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; j < nb && ok; ++j) {
        if (j + 1 < nb) {
          if (!(ok = role_wait(&s_empty, j & 1, &s_abort)) || !(ok = issue_s(j + 1))) break;
        }
        const int s = (2 * j + 1) % SLOTS;
        if (!(ok = role_wait(&kv_full[s], ((2 * j + 1) / SLOTS) & 1, &s_abort))) break;
        const uint64_t dV = dV0 + (uint64_t)(s * (TILE >> 4));
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (!(ok = role_wait(&p_full[half], j & 1, &s_abort))) break;
          tc_fence_after_sync();
          // O += P V: A = P [128 x 64 keys of this half] in tensor memory, B = V [64 keys x 64] MN-major
#pragma unroll
          for (int k = half * 4; k < half * 4 + 4; ++k)
            mma_bf16_tmem_a(tm_o, tm_p + (uint32_t)(k * 8), dV + (uint64_t)((k * 2048) >> 4), id_o, (j | k) != 0);
        }
        if (!ok) break;
        mma_commit(&o_full);
        mma_commit(&kv_empty[s]);
      }
      if (!ok) s_abort = 1;
    }
  } else {
    regs_inc<208>();
    const int quarter = warp & 3;          // TMEM lane quarter this warp may access
    const int r = quarter * 32 + lane;     // query row inside the tile == TMEM lane
    const int row = q0 + r;
    const uint32_t lane_base = (uint32_t)(quarter * 32);
    const float sl2 = p.scale * LOG2E;
    const uint64_t sl22 = pack2(sl2, sl2);
    float m_ref = -CUDART_INF_F, l = 0.f;
    bool fail = false;
    for (int j = 0; j < nb; ++j) {
      fail = !mbar_wait_parked(&s_full, j & 1, &s_abort);
      if (__any_sync(0xffffffffu, fail || s_abort)) { fail = true; break; }
      tc_fence_after_sync();
      uint32_t sc[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tmem_addr(tm_s, lane_base, c * 32), sc[c]);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty);  // the next block's scores may overwrite S now
      __syncwarp();
      if (j == nb - 1) {  // the block on the diagonal; keys past the end of the sequence lie right of it
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > r) sc[c][i] = __float_as_uint(-CUDART_INF_F);
      }
      // four independent chains: a single running maximum would serialise 128 dependent operations
      float mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int i = 0; i < 32; i += 2)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          mx4[c] = fmaxf(fmaxf(mx4[c], __uint_as_float(sc[c][i])), __uint_as_float(sc[c][i + 1]));
      const float m_cand = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
      const bool raise = m_cand > m_ref;  // also true for the first block (m_ref = -inf)
      float alpha = 1.f;
      if (raise) {
        alpha = exp2f(m_ref - m_cand);
        m_ref = m_cand;
        l *= alpha;
      }
      const float m_use = (m_ref == -CUDART_INF_F) ? 0.f : m_ref;
      if (j > 0) {
        // P V of the previous block: it has read the P that is about to be overwritten, and O may be rescaled
        fail = !mbar_wait_parked(&o_full, (j - 1) & 1, &s_abort);
        if (__any_sync(0xffffffffu, fail || s_abort)) { fail = true; break; }
        if (__any_sync(0xffffffffu, raise)) {
          tc_fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t rr[32];
            tmem_ld32(tmem_addr(tm_o, lane_base, c), rr);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) rr[i] = __float_as_uint(__uint_as_float(rr[i]) * alpha);
            tmem_st32(tmem_addr(tm_o, lane_base, c), rr);
          }
          tmem_st_wait();
        }
      }
      const uint64_t neg_m = pack2(-m_use, -m_use);
      uint64_t rs2[2] = {0ull, 0ull};  // pairs of fp32 partial sums
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t pk[32];  // 64 keys of the row of P as bf16 pairs: column c holds keys 2 c (low half) and 2 c + 1
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t* src = &sc[half * 2 + (i >> 4)][(i & 15) * 2];
          float a, b2;
          unpack2(fma2(pack2(__uint_as_float(src[0]), __uint_as_float(src[1])), sl22, neg_m), a, b2);
          a = exp2f(a);
          b2 = exp2f(b2);
          rs2[i & 1] = add2(rs2[i & 1], pack2(a, b2));
          pk[i] = pack_bf16(a, b2);
        }
        tmem_st32(tmem_addr(tm_p + (uint32_t)(half * 32), lane_base, 0), pk);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[half]);
        __syncwarp();
      }
      float e0, e1;
      unpack2(add2(rs2[0], rs2[1]), e0, e1);
      l += e0 + e1;
    }
    if (!fail) fail = !mbar_wait_parked(&o_full, (nb - 1) & 1, &s_abort);
    if (__any_sync(0xffffffffu, fail)) {
      s_abort = 1;
    } else {
      tc_fence_after_sync();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm_o, lane_base, c), rr);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          pk[c / 2 + i] = pack_bf16(__uint_as_float(rr[2 * i]) * inv, __uint_as_float(rr[2 * i + 1]) * inv);
      }
      // Q's place: the MMAs that read it have completed
      store_rows64(sQ + (warp & 3) * 4096, pk, p.o + ((int64_t)(b * p.S + row - lane) * p.Hq + h) * D, (int64_t)p.Hq * D,
                   p.S - (row - lane));
      if (row < p.S) p.lse[((int64_t)b * p.Hq + h) * p.S + row] = (l > 0.f) ? (m_ref + log2f(l)) * LN2 : -CUDART_INF_F;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(p.status, 10);
  if (warp == 1) tmem_dealloc(tm_s, 256);
}

}  // namespace fwd64

// Called by zc_attn_fwd_2q, which has checked the arguments and whose status word this kernel reports in.
int attn_fwd_d64(const void* q, const void* k, const void* v, void* o, float* lse, int B, int S, int Hq, int Hkv,
                 int64_t qs0, int64_t qs1, int64_t qs2, int64_t ks0, int64_t ks1, int64_t ks2, int64_t vs0, int64_t vs1,
                 int64_t vs2, float scale, int* status, cudaStream_t st) {
  using namespace fwd64;
  CUtensorMap mq, mk, mv;
  if (!make_map_bshd(&mq, q, D, Hq, S, B, qs0, qs1, qs2, 128) || !make_map_bshd(&mk, k, D, Hkv, S, B, ks0, ks1, ks2, 128) ||
      !make_map_bshd(&mv, v, D, Hkv, S, B, vs0, vs1, vs2, 128))
    return ERR_BAD_ARG;
  Params p;
  p.o = (__nv_bfloat16*)o; p.lse = lse; p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.status = status;
  p.nqb = (S + 127) / 128;
  if (cudaFuncSetAttribute(attn_fwd_d64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)
    return launch_status();
  zc::launch_chained(attn_fwd_d64_kernel, p.nqb * Hq * B, THREADS, SMEM, st, mq, mk, mv, p);
  return launch_status();
}

}  // namespace zc
