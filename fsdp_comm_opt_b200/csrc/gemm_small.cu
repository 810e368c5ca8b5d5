// bf16 GEMM for products that do not fill the chip with 256 x 256 tiles (layers of small models, few tokens):
// C[M,N] (+)= op(A) * op(B), fp32 accumulate, on one SM a tile.
//
// What such a product costs is not its arithmetic but the way from the launch to the last store, and the K blocks that one
// tile adds up one after the other.  So: 128 x 128 tiles, one a CTA (four times as many as the two-SM kernel has), no pair
// of SMs to bring together, the first loads issued by the warp that has initialised their barriers, before the others have
// met; and up to eight CTAs, a cluster, to the K blocks of a tile, whose fp32 sums meet in shared memory.
//   warp 0      barriers, TMA loads into a ring of `stages` buffers
//   warp 1      TMEM, MMA issue (M 128, N 128, K 16)
//   warps 2-5   alone: the accumulator through shared memory (over the ring, which is done with) into whole lines of C; in
//               a cluster: as fp32 into shared memory, from where every CTA is sent its rows (a bulk copy a CTA; reading them
//               from the others took 2 us more), sums them in the CTAs' order, adds bias and old values, rounds once, stores
// Every wait is bounded; on expiry the status word is set.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "gemm_common.cuh"
#include "launch_util.h"
#include "umma.cuh"

namespace zc {
namespace gs {
using namespace umma;

constexpr int BM = 128, BN = 128, BK = 64, THREADS = 192;
constexpr int A_BYTES = BM * BK * 2, STAGE = A_BYTES + BN * BK * 2;
constexpr int MAX_STAGES = 6;
constexpr int CLUSTER_STAGES = 4;  // and what the other CTAs send behind them
constexpr int TILE_BYTES = BM * BN * 4;
static_assert(CLUSTER_STAGES * STAGE + TILE_BYTES == MAX_STAGES * STAGE, "the same memory");
constexpr int MAX_PARTS = 8;
constexpr int EPI_ROW = 144;  // bytes between the rows of a warp's 32 x 64 bf16 block: the 16-byte accesses of a column do not meet

struct Params {
  __nv_bfloat16* C;
  const __nv_bfloat16* bias;
  int64_t M, N, ldc;
  int k_blocks, accumulate;
  int* status;
};
struct Shared {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full, received;
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// `bytes` of this CTA's shared memory to `dst` of CTA `rank` of the cluster, counted on that CTA's barrier `bar`
__device__ __forceinline__ void send(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar, uint32_t rank) {
  asm volatile(
      "{\n"
      ".reg .b32 d, m;\n"
      "mapa.shared::cluster.u32 d, %0, %4;\n"
      "mapa.shared::cluster.u32 m, %3, %4;\n"
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [d], [%1], %2, [m];\n"
      "}\n" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar), "r"(rank)
      : "memory");
}

template <int A_MAJOR, int B_MAJOR, int PARTS>
__global__ void __launch_bounds__(THREADS, 1)
    gemm_small_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {  // the same in all CTAs of a cluster
    if (threadIdx.x == 0) atomicExch(p.status, 9);
    return;
  }
  Shared& sh = *reinterpret_cast<Shared*>(smem + MAX_STAGES * STAGE);
  constexpr int STAGES = PARTS > 1 ? CLUSTER_STAGES : MAX_STAGES;
  constexpr int ROWS = BM / PARTS;                 // of the tile, which this CTA sums and stores
  constexpr int BLOCK = ROWS < 32 ? ROWS : 32;     // rows that are sent at a time, columns 4 c4 .. 4 c4 + 3 of them next to each other
  constexpr int SHARE = TILE_BYTES / PARTS, SENT = BLOCK * BN * 4;
  volatile int& s_abort = sh.abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part = blockIdx.x, m0 = blockIdx.y * BM, n0 = blockIdx.z * BN;
  const int kb0 = part * p.k_blocks / PARTS, kbs = (part + 1) * p.k_blocks / PARTS - kb0;  // at least one
  const uint32_t base = smem_u32(smem);
  auto load = [&](int i, int s) {  // the i-th K block of this CTA into stage s
    const uint32_t sa = base + s * STAGE, sb = sa + A_BYTES;
    const int k0 = (kb0 + i) * BK;
    mbar_expect_tx(&sh.full[s], STAGE);
    if (A_MAJOR == MAJOR_K) {
      tma_load(sa, &mapA, &sh.full[s], k0, m0);
    } else {
#pragma unroll
      for (int sl = 0; sl < BM / 64; ++sl) tma_load(sa + sl * 8192, &mapA, &sh.full[s], m0 + sl * 64, k0);
    }
    if (B_MAJOR == MAJOR_K) {
      tma_load(sb, &mapB, &sh.full[s], k0, n0);
    } else {
#pragma unroll
      for (int sl = 0; sl < BN / 64; ++sl) tma_load(sb + sl * 8192, &mapB, &sh.full[s], n0 + sl * 64, k0);
    }
  };
  if (warp == 0) {
    if (lane < 2 * MAX_STAGES + 2) mbar_init(&sh.full[lane], 1);
    mbar_fence_init();
    fence_proxy_async_smem();
    if (lane == 0) s_abort = 0;
    __syncwarp();
    chain_wait();
    if (lane == 0) {
      if (PARTS > 1) mbar_expect_tx(&sh.received, TILE_BYTES - SHARE);
      for (int i = 0; i < min(kbs, STAGES); ++i) load(i, i);
    }
    __syncwarp();
  } else if (warp == 1) {
    tmem_alloc(&sh.tmem_base, BN);
    tmem_relinquish();
  }
  if (PARTS > 1) cluster_arrive();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = sh.tmem_base;
  if (warp != 0) chain_wait();
  if (warp == 1) chain_next();  // which has its TMEM

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      for (int i = STAGES; i < kbs; ++i) {
        if (!mbar_wait(&sh.empty[s], ph)) { s_abort = 1; break; }
        load(i, s);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16(BM, BN, A_MAJOR, B_MAJOR);
      const uint64_t a0 = smem_desc(base, A_MAJOR == MAJOR_K ? 16 : 8192, 1024);
      const uint64_t b0 = smem_desc(base + A_BYTES, B_MAJOR == MAJOR_K ? 16 : 8192, 1024);
      constexpr uint64_t A_STEP = (A_MAJOR == MAJOR_K ? 32 : 2048) >> 4, B_STEP = (B_MAJOR == MAJOR_K ? 32 : 2048) >> 4;
      int s = 0;
      uint32_t ph = 0, accum = 0;
      bool ok = true;
      for (int i = 0; i < kbs; ++i) {
        if (!(ok = mbar_wait(&sh.full[s], ph))) break;
        const uint64_t da = a0 + (uint64_t)(s * (STAGE >> 4)), db = b0 + (uint64_t)(s * (STAGE >> 4));
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          mma_bf16(tm, da + k * A_STEP, db + k * B_STEP, idesc, accum);
          accum = 1;
        }
        mma_commit(&sh.empty[s]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (ok) mma_commit(&sh.acc_full);
      else s_abort = 1;
    }
  } else {
    if (PARTS > 1) cluster_wait();  // the others' barriers are initialised
    const bool ok = mbar_wait(&sh.acc_full, 0);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after_sync();
      const int quarter = warp & 3;
      if (PARTS > 1) {
        const int row = quarter * 32 + lane;
        float4* dst = reinterpret_cast<float4*>(smem) + (row / BLOCK) * (SENT / 16) + row % BLOCK;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          tmem_ld32(tmem_addr(tm, quarter * 32, c), r);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q)
            dst[(c / 4 + q) * BLOCK] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane < 32 / BLOCK) {
          const int block = quarter * (32 / BLOCK) + lane, to = block * BLOCK / ROWS;
          if (to != part)
            send(base + CLUSTER_STAGES * STAGE + part * SHARE + (block * SENT) % SHARE, base + block * SENT, SENT,
                 smem_u32(&sh.received), to);
        }
      } else {
        const int out_row = lane >> 3, out_chunk = lane & 7;
        const int rows_left = (int)min((int64_t)32, p.M - m0 - quarter * 32), cols_left = (int)min((int64_t)BN, p.N - n0);
        const int64_t row = m0 + quarter * 32;
        uint8_t* epi = smem + quarter * 32 * EPI_ROW;
        if (p.accumulate) {
          // the old values come in as they lie, 16 bytes of a row a thread
#pragma unroll 1
          for (int c = 0; c < BN; c += 32) {
            uint32_t r[32];
            tmem_ld32(tmem_addr(tm, quarter * 32, c), r);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (lane >= rows_left || c + q * 8 >= cols_left) continue;
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[q * 8 + j]);
              if (p.bias) add_bias8(p.bias, n0 + c + q * 8, p.N, f);
              uint4* dst = reinterpret_cast<uint4*>(p.C + (row + lane) * p.ldc + n0 + c + q * 8);
              add_old8(*dst, f);
              *dst = round8(f);
            }
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < BN; c += 64) {
            uint32_t r[2][32];
            tmem_ld32(tmem_addr(tm, quarter * 32, c), r[0]);
            tmem_ld32(tmem_addr(tm, quarter * 32, c + 32), r[1]);
            tmem_ld_wait();
            if (p.bias) {  // a column's value a lane
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int col = c + h * 32 + lane;
                const float mine = col < cols_left ? __bfloat162float(p.bias[n0 + col]) : 0.f;
#pragma unroll
                for (int j = 0; j < 32; ++j) r[h][j] = __float_as_uint(__uint_as_float(r[h][j]) + __shfl_sync(0xffffffffu, mine, j));
              }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[q >> 2][(q & 3) * 8 + j]);
              *reinterpret_cast<uint4*>(epi + lane * EPI_ROW + q * 16) = round8(f);
            }
            __syncwarp();
            uint4 v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = *reinterpret_cast<const uint4*>(epi + (4 * q + out_row) * EPI_ROW + out_chunk * 16);
            __syncwarp();
            if (c + out_chunk * 8 < cols_left) {
              __nv_bfloat16* dst = p.C + (row + out_row) * p.ldc + n0 + c + out_chunk * 8;
#pragma unroll
              for (int q = 0; q < 8; ++q)
                if (4 * q + out_row < rows_left) *reinterpret_cast<uint4*>(dst + (int64_t)(4 * q) * p.ldc) = v[q];
            }
          }
        }
      }
    } else {
      s_abort = 1;
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  if (PARTS > 1 && warp < 2) cluster_wait();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(p.status, 10);
  if (warp == 1) tmem_dealloc(tm, BN);
  if (PARTS > 1) {
    if (warp >= 2) {
      const bool ok = mbar_wait(&sh.received, 0);
      if (!__all_sync(0xffffffffu, ok) && lane == 0) atomicExch(p.status, 10);  // the flag's reader does not wait for this warp
      // a warp has 32 columns, eight rows a round: 128 bytes in a row of every load, 64 of every store
      const int c8 = (warp - 2) * 4 + (lane >> 3), cols_left = (int)min((int64_t)BN, p.N - n0);
      const int64_t row0 = m0 + part * ROWS + (lane & 7);
      __nv_bfloat16* dst = p.C + row0 * p.ldc + n0 + c8 * 8;
      float bias[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (p.bias && c8 * 8 < cols_left) add_bias8(p.bias, n0 + c8 * 8, p.N, bias);
#pragma unroll(PARTS == 2 ? 4 : 2)
      for (int r = 0; r < ROWS; r += 8) {
        const int at = (r / BLOCK) * (SENT / 16) + 2 * c8 * BLOCK + r % BLOCK + (lane & 7);
        float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < PARTS; ++c) {
          const float4* src = reinterpret_cast<const float4*>(smem + (c == part ? 0 : CLUSTER_STAGES * STAGE) + c * SHARE) + at;
          const float4 x = src[0], y = src[BLOCK];
          f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
          f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += bias[j];
        if (row0 + r < p.M && c8 * 8 < cols_left) {
          uint4* to = reinterpret_cast<uint4*>(dst + (int64_t)r * p.ldc);
          if (p.accumulate) add_old8(*to, f);
          *to = round8(f);
        }
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();  // the others have what this CTA sent them
  }
}

template <int A_MAJOR, int B_MAJOR, int PARTS>
static int launch(cudaLaunchConfig_t cfg, const CUtensorMap& mapA, const CUtensorMap& mapB, const Params& p) {
  const auto kernel = gemm_small_kernel<A_MAJOR, B_MAJOR, PARTS>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_STAGES * STAGE + (int)sizeof(Shared)) != cudaSuccess)
    return launch_status();
  launch_chained_cluster(PARTS, kernel, cfg.gridDim, cfg.blockDim, cfg.dynamicSmemBytes, cfg.stream, mapA, mapB, p);
  return launch_status();
}
template <int PARTS>
static int launch_forms(int a_major, int b_major, const cudaLaunchConfig_t& cfg, const CUtensorMap& mapA,
                        const CUtensorMap& mapB, const Params& p) {
  if (a_major == MAJOR_K && b_major == MAJOR_K) return launch<MAJOR_K, MAJOR_K, PARTS>(cfg, mapA, mapB, p);
  if (a_major == MAJOR_K) return launch<MAJOR_K, MAJOR_MN, PARTS>(cfg, mapA, mapB, p);
  return launch<MAJOR_MN, MAJOR_MN, PARTS>(cfg, mapA, mapB, p);
}

}  // namespace gs

// Tiles whose `parts` CTAs each, a cluster, run at once.
static int tiles_at_once(int parts) {
  using namespace gs;
  constexpr int SMEM = MAX_STAGES * STAGE + (int)sizeof(Shared);
  static int two[64], four[64], eight[64];
  switch (parts) {
    case 1: return sm_count();
    case 2: return clusters_at_once(gemm_small_kernel<MAJOR_K, MAJOR_K, 2>, 2, THREADS, SMEM, two);
    case 4: return clusters_at_once(gemm_small_kernel<MAJOR_K, MAJOR_K, 4>, 4, THREADS, SMEM, four);
    default: return clusters_at_once(gemm_small_kernel<MAJOR_K, MAJOR_K, 8>, 8, THREADS, SMEM, eight);
  }
}

// us that a product of these sizes is expected to take here, and in how many parts along K; 0 where there are more tiles than
// SMs.  Measured: 3.2 a launch and 0.27 a K block (500 clocks: the operands' way into shared memory and out of it), 1.9 to 2.8
// for what the CTAs of a cluster send each other.  512 x 256 x 256: 6.7 -> 4.3, 512 x 256 x 1024: 10.3 -> 7.0, 1024^3:
// 10.4 -> 7.4.  Only as many parts as let all clusters run at once (74 of two, 33 of four, 15 of eight on 148 SMs): with a second
// wave 16 tiles of K 1024 by eight took 11.8 us, 6.0 by four, and 36 tiles by four 11.2, 6.3 by two.
static double expected_us(int64_t M, int64_t N, int64_t K, bool cut_k, int& parts) {
  using namespace gs;
  const int64_t tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN), kbs = (K + BK - 1) / BK;
  static const double sent[4] = {0.0, 1.9, 2.5, 2.8};
  double least = 0;
  parts = 0;
  if (tiles > sm_count()) return 0;
  for (int i = 0; i < 4 && (i == 0 || (cut_k && tiles <= tiles_at_once(1 << i) && kbs >= 2LL << i)); ++i) {
    const double us = 3.2 + 0.27 * (double)((kbs + (1 << i) - 1) >> i) + sent[i];
    if (i == 0 || us < least) { least = us; parts = 1 << i; }
  }
  return least;
}
int gemm_small_parts(int64_t M, int64_t N, int64_t K, bool cut_k, double other_us) {
  int parts;
  return expected_us(M, N, K, cut_k, parts) <= other_us ? parts : 0;
}

int gemm_small_launch(const void* A, const void* B, void* C, const void* bias, int64_t M, int64_t N, int64_t K, int64_t lda,
                      int64_t ldb, int64_t ldc, int a_major, int b_major, int accumulate, int parts, int* status,
                      cudaStream_t st) {
  using namespace gs;
  CUtensorMap mapA, mapB;
  bool ok = a_major == MAJOR_K ? make_map(&mapA, A, M, K, lda, BK, BM) : make_map(&mapA, A, K, M, lda, 64, BK);
  ok = ok && (b_major == MAJOR_K ? make_map(&mapB, B, N, K, ldb, BK, BN) : make_map(&mapB, B, K, N, ldb, 64, BK));
  if (!ok) return ERR_BAD_ARG;
  Params p;
  p.C = (__nv_bfloat16*)C; p.bias = (const __nv_bfloat16*)bias;
  p.M = M; p.N = N; p.ldc = ldc;
  p.k_blocks = (int)((K + BK - 1) / BK);
  p.accumulate = accumulate; p.status = status;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(parts, (unsigned)((M + BM - 1) / BM), (unsigned)((N + BN - 1) / BN));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = MAX_STAGES * STAGE + sizeof(Shared);
  cfg.stream = st;
  if (parts == 1) return launch_forms<1>(a_major, b_major, cfg, mapA, mapB, p);
  if (parts == 2) return launch_forms<2>(a_major, b_major, cfg, mapA, mapB, p);
  if (parts == 4) return launch_forms<4>(a_major, b_major, cfg, mapA, mapB, p);
  return launch_forms<8>(a_major, b_major, cfg, mapA, mapB, p);
}

}  // namespace zc

// For a look at the rule: in how many parts along K the kernel of small products would take a product at best (0: more tiles
// than SMs), and how many tiles in so many parts run at once.
extern "C" int zc_gemm_small_best_parts(int64_t M, int64_t N, int64_t K) {
  int parts;
  zc::expected_us(M, N, K, true, parts);
  return parts;
}
extern "C" int zc_gemm_small_tiles_at_once(int parts) { return zc::tiles_at_once(parts); }
