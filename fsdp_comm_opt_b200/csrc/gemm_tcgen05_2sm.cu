// Two-SM (cta_group::2) persistent bf16 GEMM for sm_100a: C[M,N] (+)= op(A) * op(B), fp32 accumulate.
//
// A cluster of two CTAs owns a 256 x 256 output tile.  Each CTA stages its own 128 rows of A and its
// own 128 of the tile's 256 columns of B; one thread of the even CTA issues
// tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 16), which reads both CTAs' shared memory and
// accumulates each CTA's 128 rows into that CTA's TMEM.
//
//   warp 0      TMA producer (both CTAs): cp.async.bulk.tensor ... cta_group::2 loads into the CTA's
//               own stage buffers, transaction bytes counted on the even CTA's `full` barrier
//   warp 1      even CTA: MMA issuer; commits arrive on the `empty` / `acc_full` barriers of both CTAs
//   warps 2-5   epilogue (both CTAs): tcgen05.ld the CTA's 128 x 256 accumulator, convert, turn 64 columns of 32 rows
//               round in shared memory, store whole 128-byte lines; arrivals of both CTAs' epilogue warps free the
//               accumulator on the even CTA
// Every CTA fetches its own tiles with plain per-CTA TMA loads; no load is shared between CTAs.
//
// The issuing thread is the scarce resource: one thread has to launch a 128-clock MMA every 128
// clocks, so everything that can be is precomputed (stage-0 descriptors, remote barrier addresses)
// and the operand layouts are template parameters; per MMA the loop adds a constant to the
// descriptors and nothing else.
//
// Work is handed out dynamically.  The clusters take units from a global counter (the even CTA's
// producer thread fetches the next index and publishes it to every role of both CTAs through a small
// ring in shared memory), so a cluster that starts late, or not at all for a while, because another
// kernel (a collective running beside the GEMM) holds its SMs simply takes fewer units; with a
// static round-robin the whole GEMM would wait for that cluster's share.  (Launches recorded into a CUDA
// graph, which only a one-rank step makes, those with no second round, and those of streams beyond COUNTER_SLOTS use the
// static order.)
// Units: whole tiles first, then the tiles of the last, partial wave are split
// along K into `split` slices each, so that all clusters stay busy to the end.  A slice writes its
// fp32 partial sums to a workspace and a small second kernel adds the slices and rounds to bf16.
// What a small product costs is fixed: 256 x 256 x 64 took 7.5 us a launch in a graph, of which the epilogue, 16 bytes of 32
// rows a store, was 4.6, the pair's two barriers with release semantics 1.3, and an arrival with release behind the stores 0.6.
// It is 5.6 now: 0.45 to the pair's barrier, 0.4 to the first load, 0.4 for it, 0.4 for the MMAs, 2.0 for the epilogue (bound
// by the four warps' shared memory and store instructions; 32-column boxes stored by TMA took 2.6), 0.4 to leave.
// Every wait is bounded; on expiry the status word is set and both CTAs reach the teardown.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "gemm_common.cuh"
#include "launch_util.h"
#include "nvtx_util.h"
#include "umma.cuh"

namespace zc {
namespace g2 {
using namespace umma;

constexpr int BM_CTA = 128;   // rows of A per CTA (256 per cluster)
constexpr int BN_CTA = 128;   // columns of B staged per CTA (256 per cluster)
constexpr int BM = 256;
constexpr int BN = 256;       // accumulator columns
constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int THREADS = 192;
constexpr int A_BYTES = BM_CTA * BK * 2;  // 16 KB
constexpr int B_BYTES = BN_CTA * BK * 2;  // 16 KB
constexpr int STAGE = A_BYTES + B_BYTES;
constexpr int MAX_SPLIT = 4;          // slices of a tail tile
constexpr int MAX_SPLIT_SINGLE = 16;  // slices of a product that has fewer tiles than clusters
constexpr int SINGLE_MIN_KB = 8;      // K blocks of such a slice at least,
constexpr int SINGLE_MIN_SAVED = 20;  // and fewer K blocks one after the other than in the whole product
constexpr int SCHED = 4;       // slots of the unit-index ring
constexpr int EPI_COLS = 64;   // columns that an epilogue warp turns round in shared memory at a time: 32 rows x 128 bytes
constexpr int EPI_BYTES = 32 * EPI_COLS * 2;
constexpr int SHARED_OFF = STAGES * STAGE + 4 * EPI_BYTES;  // struct Shared behind the stages and the epilogue's buffers
constexpr int COUNTER_SLOTS = 256;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The pair's barrier in two halves.  Relaxed (with release the two barriers of a launch took 2400 clocks, so 400): at the start
// the other CTA has to see the initialised mbarriers, which fence.mbarrier_init publishes, and to come after the allocation
// of tensor memory, which has returned when its warp arrives; at the end every arrival at a CTA's mbarriers has been waited
// for there.  With release where a wait was given up, and arrivals may be on their way.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// shared::cluster address of `local_addr` (a shared::cta address) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same without waiting for this thread's earlier stores to be seen: where the arrival publishes nothing in memory, only
// that tcgen05.ld has read the accumulator (a release took 1100 clocks behind the epilogue's stores).
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 16 bytes of global memory into shared memory, and the wait for all of this thread's
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// TMA load into this CTA's shared memory; the bytes are counted on the barrier at `bar_cluster_addr`
// (the even CTA's `full` barrier)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(map), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void mma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at `cluster_addr` (either CTA of the pair) when all MMAs issued so far by this
// thread have completed
__device__ __forceinline__ void mma_commit_pair(uint32_t cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_addr)
               : "memory");
}
__device__ __forceinline__ uint32_t mbar_addr_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ uint32_t mbar_addr_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// the same wait with cluster-scope acquire: the arrival (and the data it publishes) came from the other CTA
__device__ __forceinline__ bool wait_bar_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_addr_try_wait_cluster(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (uint32_t it = 0;; ++it) {
    if (mbar_addr_try_wait_cluster(bar, parity)) return true;
    if ((it & 255u) == 255u && (*abort_flag || globaltimer_ns() - t0 > 2000000000ull)) return false;
  }
}
__device__ __forceinline__ void st_shared_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// bounded spin on a barrier given by its shared::cta address; the limit is only looked at on the slow path
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_addr_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (uint32_t it = 0;; ++it) {
    if (mbar_addr_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && (*abort_flag || globaltimer_ns() - t0 > 2000000000ull)) return false;
  }
}

// Everything is in dynamic shared memory, whose beginning is 1024-byte aligned when there is no static part: 208.2 KB in
// all, so that two 8 KB CTAs of a collective still fit beside this one.
struct Shared {
  uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  uint64_t sched_full[SCHED], sched_empty[SCHED];
  int sched_u[SCHED];
  uint32_t tmem_base;
  int abort;
};
constexpr int SMEM_BYTES = SHARED_OFF + (int)sizeof(Shared);
static_assert(SMEM_BYTES + 1024 + 2 * (8192 + 1024 + 128) <= 228 * 1024, "room for two CTAs of a collective");

struct Params {
  __nv_bfloat16* C;
  float* partial;      // [tail tiles][split] slabs of 256 x 256 fp32 (partial_off), or null when split == 1
  int64_t M, N;
  int m_tiles, n_tiles, k_blocks;
  float inv_band;      // 1 / (group_m * n_tiles)
  int64_t ldc;         // elements between rows of C (>= N rounded up to 8: whole 8-column groups are stored)
  const __nv_bfloat16* bias;  // [N] added to every row before rounding, or null
  int accumulate;
  int group_m;         // tiles are walked in bands of `group_m` m-tiles, n-major inside a band
  int full_tiles;      // tiles computed whole; the remaining tiles are split along K
  int split;           // K slices per tail tile (1: no tile is split)
  int* status;
  unsigned* counter;   // [0] units handed out beyond the first round, [1] clusters finished; both 0 at launch;
                       // null: unit i of cluster c is c + i * clusters
};

// Tile order.  The clusters running at one time work on consecutive tile indices; walking bands of
// `group_m` m-tiles keeps that set a compact block of the output, so the A rows and B columns it
// needs together stay in L2 however large K is (a full column of m-tiles does not once M * K
// outgrows the cache).
// (A division by a number whose reciprocal is known, for quotients below 2^24 right after one correction at most: the integer
// division's thirty instructions lie between two tiles, and before the first.)
__device__ __forceinline__ int div_by(int t, int d, float inv, int& rem) {
  int q = (int)((float)t * inv);
  rem = t - q * d;
  while (rem < 0) { --q; rem += d; }
  while (rem >= d) { ++q; rem -= d; }
  return q;
}
__device__ __forceinline__ void tile_coords(int t, const Params& p, int& mi, int& ni) {
  int r, in_col;
  const int band = div_by(t, p.group_m * p.n_tiles, p.inv_band, r);
  const int rows = min(p.group_m, p.m_tiles - band * p.group_m);
  ni = div_by(r, rows, __frcp_rn((float)rows), in_col);
  mi = band * p.group_m + in_col;
}

// One unit of work: a tile and a range of its K blocks.
struct Unit {
  int mi, ni;
  int kb0, kb1;
  int slice;  // index of the fp32 partial slab, or -1 for a whole tile
};
__device__ __forceinline__ Unit unit_of(int u, const Params& p) {
  Unit w;
  int t = u;
  w.kb0 = 0;
  w.kb1 = p.k_blocks;
  w.slice = -1;
  if (u >= p.full_tiles) {
    const int r = u - p.full_tiles;
    t = p.full_tiles + r / p.split;
    const int s = r % p.split;
    const int per = (p.k_blocks + p.split - 1) / p.split;
    w.kb0 = s * per;
    w.kb1 = min(p.k_blocks, w.kb0 + per);
    w.slice = r;
  }
  tile_coords(t, p, w.mi, w.ni);
  return w;
}

// Where a slab of partial sums keeps columns 4 c4 .. 4 c4 + 3 of a tile's row, in float4: the rows of a warp, which holds a
// row a thread, lie next to each other.
__device__ __forceinline__ int partial_off(int row, int c4) { return ((row >> 5) * (BN / 4) + c4) * 32 + (row & 31); }

// ADD: to the old values of C.
// Shared memory allows one CTA to an SM; the registers are bounded as for three, which is 96 a thread, so that a collective's CTAs fit
// beside it.
template <int A_MAJOR, int B_MAJOR, bool ADD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 3)
    gemm_2sm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {  // the same in both CTAs of a pair
    if (threadIdx.x == 0) atomicExch(p.status, 9);
    return;
  }
  Shared& sh = *reinterpret_cast<Shared*>(smem + SHARED_OFF);
  uint64_t *full = sh.full, *empty = sh.empty, *acc_full = sh.acc_full, *acc_empty = sh.acc_empty;
  uint64_t *sched_full = sh.sched_full, *sched_empty = sh.sched_empty;
  volatile int* sched_u = sh.sched_u;
  volatile int& s_abort = sh.abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();  // 0: even CTA (issues the MMAs), 1: odd CTA
  if (warp == 0) {
    // A thread per barrier: full (used on the even CTA: its producer's arrive.expect_tx), empty (one commit per use, on
    // both CTAs), acc_full (one commit per unit, on both CTAs), acc_empty (on the even CTA: four epilogue warps of each CTA),
    // sched_full (the even CTA's producer publishes a unit index in both CTAs), sched_empty (on the even CTA: every other
    // role of both CTAs has read it)
    constexpr int ACC_EMPTY = 2 * STAGES + 2, SCHED_FULL = ACC_EMPTY + 2, SCHED_EMPTY = SCHED_FULL + SCHED;
    if (lane < SCHED_EMPTY + SCHED)
      mbar_init(&full[lane], lane >= SCHED_EMPTY ? 10 : lane >= ACC_EMPTY && lane < SCHED_FULL ? 8 : 1);
    mbar_fence_init();
    if (lane == 0) s_abort = 0;
    __syncwarp();
  }
  if (warp == 1) {
    // each CTA allocates its own SM's whole TMEM (512 columns, so the base is column 0 in both), and arrives at the pair's
    // barrier behind that: the even CTA's MMAs write the odd one's tensor memory
    tmem_alloc(&sh.tmem_base, 2 * BN);
    tmem_relinquish();
    tc_fence_before_sync();
  } else if (warp == 2 && lane < 2) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(lane ? &mapB : &mapA) : "memory");
  }
  __syncwarp();
  cluster_arrive();
  // edge tiles: rows / columns / K blocks past the matrix read as zeros (TMA fill) and are not stored
  const int units = p.full_tiles + (p.m_tiles * p.n_tiles - p.full_tiles) * p.split;
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const Unit first = unit_of(cluster_id, p);
  // This CTA's abort flag is clear and its accumulators' address known.  The producer, which cleared the one and has no use for
  // the other, does not wait here.
  if (warp == 0) {
    asm volatile("bar.arrive 1, 192;" ::: "memory");
  } else {
    tc_fence_before_sync();
    asm volatile("bar.sync 1, 192;" ::: "memory");
    tc_fence_after_sync();
  }
  cluster_wait();  // both CTAs have their barriers, before any remote arrival, and their tensor memory
  tc_fence_after_sync();
  chain_wait();
  if (warp == 1) chain_next();  // which has its TMEM
  const uint32_t tm = sh.tmem_base;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t full_base = smem_u32(&full[0]), empty_base = smem_u32(&empty[0]);
  const uint32_t sfull_base = smem_u32(&sched_full[0]);
  const uint32_t sempty_c0 = map_to_cta(smem_u32(&sched_empty[0]), 0);  // the even CTA's sched_empty[0]
  bool ok = true;
  // Every role walks the same sequence of units, i = 0, 1, ... (an index >= units ends it).  The first is the cluster's
  // number, known without waiting for another CTA; with counters slot (i - 1) % SCHED of the ring holds the i-th.
  auto from_ring = [&](uint32_t i) { return p.counter && i > 0; };
  auto next_unit = [&](uint32_t i, bool& good) -> int {
    if (!from_ring(i)) return cluster_id + (int)i * n_clusters;
    const uint32_t slot = (i - 1) & (SCHED - 1), sph = ((i - 1) / SCHED) & 1;
    good = rank == 0 ? wait_bar(sfull_base + 8 * slot, sph, &s_abort)
                     : wait_bar_cluster(sfull_base + 8 * slot, sph, &s_abort);
    return good ? sched_u[slot] : 0x7fffffff;
  };
  auto release_unit = [&](uint32_t i) {
    if (from_ring(i)) mbar_arrive_cluster(sempty_c0 + 8 * ((i - 1) & (SCHED - 1)));
  };

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t full0 = map_to_cta(full_base, 0);  // the even CTA's full[0]; full[s] is 8 s bytes on
      const uint32_t sfull_c1 = map_to_cta(sfull_base, 1);
      const uint32_t su_c1 = map_to_cta(smem_u32(sh.sched_u), 1);
      uint32_t s = 0, ph = 0, i = 0;
      for (; ok; ++i) {
        int u;
        if (rank == 0 && from_ring(i)) {
          // fetch the i-th unit and publish it to both CTAs
          const uint32_t slot = (i - 1) & (SCHED - 1), sph = ((i - 1) / SCHED) & 1;
          if (!(ok = wait_bar_cluster(smem_u32(&sched_empty[slot]), sph ^ 1, &s_abort))) break;
          u = n_clusters + (int)atomicAdd(p.counter, 1u);
          sched_u[slot] = u;
          st_shared_cluster_u32(su_c1 + 4 * slot, (uint32_t)u);
          mbar_arrive(&sched_full[slot]);
          mbar_arrive_cluster(sfull_c1 + 8 * slot);  // release.cluster: orders the store above
        } else {
          u = next_unit(i, ok);
          if (!ok) break;
          release_unit(i);
        }
        if (u >= units) break;
        const Unit w = i == 0 ? first : unit_of(u, p);
        const int m0 = w.mi * BM + (int)rank * BM_CTA;
        const int n0 = w.ni * BN + (int)rank * BN_CTA;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!(ok = wait_bar(empty_base + 8 * s, ph ^ 1, &s_abort))) break;
          const uint32_t sa = smem_base + s * STAGE, sb = sa + A_BYTES;
          const uint32_t fb = full0 + 8 * s;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE);  // both CTAs' bytes land on this barrier
          const int k0 = kb * BK;
          if (A_MAJOR == MAJOR_K) {
            tma_load_2d_pair(sa, &mapA, fb, k0, m0);
          } else {
#pragma unroll
            for (int sl = 0; sl < BM_CTA / 64; ++sl) tma_load_2d_pair(sa + sl * 8192, &mapA, fb, m0 + sl * 64, k0);
          }
          if (B_MAJOR == MAJOR_K) {
            tma_load_2d_pair(sb, &mapB, fb, k0, n0);
          } else {
#pragma unroll
            for (int sl = 0; sl < BN_CTA / 64; ++sl) tma_load_2d_pair(sb + sl * 8192, &mapB, fb, n0 + sl * 64, k0);
          }
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      // What the other CTA still sends to this one's barriers: the releases of the last slots, i of which have been published
      // (here on the even CTA), and the commits of the last stages.
      if (rank == 0 && p.counter)
        for (uint32_t k = i > SCHED ? i - SCHED : 0; ok && k < i; ++k)
          ok = wait_bar_cluster(smem_u32(&sched_empty[k & (SCHED - 1)]), (k / SCHED) & 1, &s_abort);
      for (int k = 0; ok && k < STAGES; ++k) {
        ok = wait_bar(empty_base + 8 * s, ph ^ 1, &s_abort);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (!ok) s_abort = 1;
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_bf16(BM, BN, A_MAJOR, B_MAJOR);
      // descriptors of stage 0, K step 0; a stage adds STAGE >> 4, a K = 16 step adds KSTEP >> 4 to the
      // start-address field (shared memory is below 256 KB, so the 14-bit field never carries)
      const uint64_t a0 = (A_MAJOR == MAJOR_K) ? smem_desc(smem_base, 16, 1024) : smem_desc(smem_base, 8192, 1024);
      const uint64_t b0 = (B_MAJOR == MAJOR_K) ? smem_desc(smem_base + A_BYTES, 16, 1024)
                                               : smem_desc(smem_base + A_BYTES, 8192, 1024);
      constexpr uint64_t A_KSTEP = ((A_MAJOR == MAJOR_K) ? 32 : 2048) >> 4;
      constexpr uint64_t B_KSTEP = ((B_MAJOR == MAJOR_K) ? 32 : 2048) >> 4;
      constexpr uint64_t STAGE_STEP = STAGE >> 4;
      const uint32_t empty_c0 = map_to_cta(empty_base, 0), empty_c1 = map_to_cta(empty_base, 1);
      const uint32_t accf_c0 = map_to_cta(smem_u32(&acc_full[0]), 0), accf_c1 = map_to_cta(smem_u32(&acc_full[0]), 1);
      const uint32_t acce = smem_u32(&acc_empty[0]);
      uint32_t s = 0, ph = 0, unit_it = 0;
      for (; ok; ++unit_it) {
        const int u = next_unit(unit_it, ok);
        if (!ok) break;
        release_unit(unit_it);
        if (u >= units) break;
        const Unit w = unit_it == 0 ? first : unit_of(u, p);
        const uint32_t acc = unit_it & 1, acc_ph = (unit_it >> 1) & 1;
        if (!(ok = wait_bar_cluster(acce + 8 * acc, acc_ph ^ 1, &s_abort))) break;
        tc_fence_after_sync();
        const uint32_t d = tm + acc * BN;
        uint32_t accum = 0;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!(ok = wait_bar(full_base + 8 * s, ph, &s_abort))) break;
          const uint64_t da = a0 + s * STAGE_STEP, db = b0 + s * STAGE_STEP;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            mma_bf16_pair(d, da + k * A_KSTEP, db + k * B_KSTEP, idesc, accum);
            accum = 1;
          }
          // the stage is reusable in both CTAs once these MMAs have read it
          mma_commit_pair(empty_c0 + 8 * s);
          mma_commit_pair(empty_c1 + 8 * s);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) {
          mma_commit_pair(accf_c0 + 8 * acc);
          mma_commit_pair(accf_c1 + 8 * acc);
        }
      }
      // both CTAs' epilogue warps have let go of the last accumulators
      for (uint32_t k = unit_it > 2 ? unit_it - 2 : 0; ok && k < unit_it; ++k)
        ok = wait_bar_cluster(acce + 8 * (k & 1), (k >> 1) & 1, &s_abort);
      if (!ok) s_abort = 1;
    }
  } else {
    const int quarter = warp & 3;
    const uint32_t accf = smem_u32(&acc_full[0]);
    const uint32_t acce_c0 = map_to_cta(smem_u32(&acc_empty[0]), 0);
    // This warp's buffer: row `lane`, 128 bytes, its 16-byte chunk j at position j ^ lane % 8.  Written a row a thread, read
    // (and stored) four rows an instruction.
    uint8_t* epi = smem + STAGES * STAGE + quarter * EPI_BYTES;
    const int out_row = lane >> 3, out_chunk = lane & 7;
    for (uint32_t unit_it = 0; ok; ++unit_it) {
      const int u = next_unit(unit_it, ok);
      if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
      __syncwarp();
      if (lane == 0) release_unit(unit_it);
      if (u >= units) break;
      const Unit w = unit_it == 0 ? first : unit_of(u, p);
      const uint32_t acc = unit_it & 1, acc_ph = (unit_it >> 1) & 1;
      const int64_t warp_row = (int64_t)w.mi * BM + rank * BM_CTA + quarter * 32, col0 = (int64_t)w.ni * BN;
      const int rows_left = (int)min((int64_t)32, p.M - warp_row) - out_row;  // from this thread's first on
      const int cols_left = (int)min((int64_t)BN, p.N - col0);
      __nv_bfloat16* dst = p.C + (warp_row + out_row) * p.ldc + col0 + out_chunk * 8;
      auto whole = [&](int q) { return reinterpret_cast<uint4*>(epi + (4 * q + out_row) * 128 + ((out_chunk ^ ((4 * q + out_row) & 7)) << 4)); };
      // Old values come into the buffer as new ones go out, in whole lines, the first while the products are still computed (16 bytes
      // of 32 rows a load, behind them: 7424 x 1536 x 320 took 59 us, 19 now).
      auto fetch_old = [&](int c) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (c + out_chunk * 8 < cols_left && 4 * q < rows_left) copy16_async(whole(q), dst + c + (int64_t)(4 * q) * p.ldc);
      };
      if (ADD && w.slice < 0) fetch_old(0);
      ok = wait_bar_cluster(accf + 8 * acc, acc_ph, &s_abort);
      if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
      tc_fence_after_sync();
      if (w.slice < 0) {
        // No branch in this loop but those on whole chunks: one at every group of eight columns, bias or not, old values
        // or not, cost more than the work.  32 columns at a time in registers: with 64 some were kept in local memory.
#pragma unroll 1
        for (int c = 0; c < BN; c += EPI_COLS) {
          if (ADD) {
            copies_done();
            __syncwarp();
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld32(tmem_addr(tm + acc * BN, quarter * 32, c + h * 32), r);
            tmem_ld_wait();
            if (h == 1 && c == BN - EPI_COLS) {  // the accumulator is free
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster_relaxed(acce_c0 + 8 * acc);
            }
            if (p.bias) {  // a column's value a lane
              const int col = c + h * 32 + lane;
              const float mine = col < cols_left ? __bfloat162float(p.bias[col0 + col]) : 0.f;
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __shfl_sync(0xffffffffu, mine, j));
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4* at = reinterpret_cast<uint4*>(epi + lane * 128 + (((4 * h + q) ^ (lane & 7)) << 4));
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[q * 8 + j]);
              if (ADD) add_old8(*at, f);
              *at = round8(f);
            }
          }
          __syncwarp();
          uint4 v[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) v[q] = *whole(q);
          __syncwarp();
          if (ADD && c + EPI_COLS < BN) fetch_old(c + EPI_COLS);
          if (c + out_chunk * 8 < cols_left) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (4 * q < rows_left) *reinterpret_cast<uint4*>(dst + c + (int64_t)(4 * q) * p.ldc) = v[q];
          }
        }
      } else {
        // K slice of a tail tile: fp32 partial sums, added up by gemm_2sm_fixup_kernel; a warp's store is 512 bytes in a row
        float4* prow = reinterpret_cast<float4*>(p.partial + (int64_t)w.slice * (BM * BN)) + partial_off((int)rank * BM_CTA + quarter * 32 + lane, 0);
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          tmem_ld32(tmem_addr(tm + acc * BN, quarter * 32, c), r);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q)
            prow[(c / 4 + q) * 32] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                 __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(acce_c0 + 8 * acc);
      }
    }
    if (!ok) s_abort = 1;
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(p.status, 8);
  // Neither CTA may leave (or free its TMEM) while the pair's MMAs or the other CTA's arrivals can still touch its memory.  Both
  // have come by now (the producers and the MMA issuer have waited for the last of them) unless a wait was given up.
  __syncwarp();
  if (s_abort) cluster_arrive_release();
  else cluster_arrive();
  cluster_wait();
  if (warp == 1) tmem_dealloc(tm, 2 * BN);
  if (tid == 0 && rank == 0 && p.counter) {
    // the last cluster to finish puts the counters back to zero for the next launch that uses this slot
    if (atomicAdd(p.counter + 1, 1u) == (unsigned)n_clusters - 1u) {
      p.counter[0] = 0u;
      p.counter[1] = 0u;
    }
  }
}

// C tile (+)= sum over the K slices of its fp32 partials, rounded once to bf16.
__global__ void __launch_bounds__(256) gemm_2sm_fixup_kernel(const Params p) {
  chain();
  const int tail = blockIdx.y;  // index among the split tiles
  int mi, ni;
  tile_coords(p.full_tiles + tail, p, mi, ni);
  const float4* base = reinterpret_cast<const float4*>(p.partial) + (int64_t)tail * p.split * (BM * BN / 4);
  // a warp takes eight rows x 32 columns: 128 bytes in a row of every load, 64 of every store
  for (int i = blockIdx.x * 256 + threadIdx.x; i < BM * BN / 8; i += gridDim.x * 256) {
    const int wi = i >> 5, lane = i & 31;
    const int row = (wi / (BN / 32)) * 8 + (lane & 7), c8 = (wi % (BN / 32)) * 4 + (lane >> 3);
    if ((int64_t)mi * BM + row >= p.M || (int64_t)ni * BN + c8 * 8 >= p.N) continue;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < p.split; ++s) {
      const float4* src = base + (int64_t)s * (BM * BN / 4);
      const float4 x = src[partial_off(row, 2 * c8)], y = src[partial_off(row, 2 * c8 + 1)];
      f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
      f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
    }
    if (p.bias) add_bias8(p.bias, (int64_t)ni * BN + c8 * 8, p.N, f);
    uint4* dst = reinterpret_cast<uint4*>(p.C + ((int64_t)mi * BM + row) * p.ldc + (int64_t)ni * BN + c8 * 8);
    if (p.accumulate) add_old8(*dst, f);
    *dst = round8(f);
  }
}

// Per-device launch state: how many clusters of two the device runs at once, and the tile counters.
struct DeviceState {
  bool ready = false;
  int clusters = 0;
  unsigned* counters = nullptr;  // COUNTER_SLOTS pairs, all zero between launches
  cudaStream_t owner[COUNTER_SLOTS];  // a stream's launches, which follow one another, share a pair
  int owners = 0;
};
static DeviceState g_state[64];
static std::mutex g_mutex;
// The counters.  Zero from the module's load: a cleared allocation would have to be waited for by the first launch on every
// stream, which the legacy stream's memset is not ordered with.
static __device__ unsigned g_counters[2 * COUNTER_SLOTS];

template <int A_MAJOR, int B_MAJOR, bool ADD>
static int max_clusters(int smem) {
  cudaFuncSetAttribute(gemm_2sm_kernel<A_MAJOR, B_MAJOR, ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (sm_count() / 2));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_2sm_kernel<A_MAJOR, B_MAJOR, ADD>, &cfg) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = sm_count() / 2;
  }
  return std::min(n, sm_count() / 2);
}

// K slices of a product whose tiles leave at least half of the clusters idle (a layer of a small model, or few
// tokens): it is cut along K altogether, so that about every cluster has a slice.  A K block
// takes 0.25 to 0.3 us there, the fp32 partials and the pass that adds them 4 to 5 us: SINGLE_MIN_SAVED.
static int single_split(int64_t tiles, int64_t k_blocks, int clusters) {
  if (tiles <= 0 || tiles * 2 > clusters) return 1;
  const int64_t want = std::min<int64_t>(std::min<int64_t>(clusters / tiles, MAX_SPLIT_SINGLE), k_blocks / SINGLE_MIN_KB);
  if (want < 2) return 1;
  const int64_t per = (k_blocks + want - 1) / want;
  if (k_blocks - per < SINGLE_MIN_SAVED) return 1;
  return (int)((k_blocks + per - 1) / per);  // no empty slice
}

// How a product's tiles are cut along K: the last `split_tiles` of them into `split` slices each.
struct Cut {
  int64_t tiles;
  int split = 1, split_tiles = 0, grid_clusters;
  int64_t bytes() const { return split > 1 ? (int64_t)split_tiles * split * BM * BN * sizeof(float) : 0; }
};
static Cut cut_of(int64_t M, int64_t N, int64_t K, int device_clusters) {
  static const int forced_split = getenv("ZC_GEMM_SPLIT") ? atoi(getenv("ZC_GEMM_SPLIT")) : -1;
  Cut c;
  c.tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int64_t k_blocks = (K + BK - 1) / BK;
  const int clusters = c.grid_clusters = (int)std::min<int64_t>(c.tiles, device_clusters);
  // Tail: the tiles of the last, partial wave are cut into K slices so that every cluster has one
  // unit of about the same length to finish with.
  const int64_t rem = c.tiles % clusters;
  if (rem > 0 && c.tiles > clusters) {
    int split = (int)std::min<int64_t>(std::min<int64_t>(clusters / rem, MAX_SPLIT), k_blocks / 8);
    if (forced_split >= 0) split = std::min(forced_split, MAX_SPLIT);
    if (split >= 2 && rem * 10 <= (int64_t)clusters * 8) {  // a nearly full last wave is left alone
      c.split = split;
      c.split_tiles = (int)rem;
    }
    return c;
  }
  const int single = single_split(c.tiles, k_blocks, device_clusters);
  if (single > 1) {
    c.split = single;
    c.split_tiles = (int)c.tiles;
    c.grid_clusters = (int)c.tiles * single;
  }
  return c;
}

// In how many parts along K the kernel of small products takes a product, 0 where this kernel is expected to be faster: with
// many tiles, or where K is so long that 256 x 256 tiles, which read half as much an FMA, cut into more slices win.  In us: what
// a launch costs beside its K blocks, a K block, the fix-up.
static int small_parts(int64_t M, int64_t N, int64_t K, bool cut_k, int clusters) {
  const Cut cut = cut_of(M, N, K, clusters);
  const int split = cut_k ? cut.split : 1;
  return gemm_small_parts(M, N, K, cut_k, 5.6 + 0.28 * (double)((K + BK - 1) / BK) / split + (split > 1 ? 4.0 : 0.0));
}

static int init_state(DeviceState& ds, int smem) {
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!ds.ready) {
    int c = std::min(max_clusters<MAJOR_K, MAJOR_K, false>(smem), max_clusters<MAJOR_K, MAJOR_K, true>(smem));
    c = std::min({c, max_clusters<MAJOR_K, MAJOR_MN, false>(smem), max_clusters<MAJOR_K, MAJOR_MN, true>(smem)});
    c = std::min({c, max_clusters<MAJOR_MN, MAJOR_MN, false>(smem), max_clusters<MAJOR_MN, MAJOR_MN, true>(smem)});
    ds.clusters = c;
    if (cudaGetSymbolAddress((void**)&ds.counters, g_counters) != cudaSuccess) return ERR_BAD_ARG;
    ds.ready = true;
  }
  return 0;
}

}  // namespace g2
}  // namespace zc

extern "C" {

int* zc_gemm_status_word();  // gemm_tcgen05.cu: the current device's GEMM status word

// Same contract as zc_gemm_bf16 with explicit leading dimensions: lda / ldb / ldc are the distances in
// elements between consecutive rows of the STORED A, B and C ([M,K] or [K,M]; [N,K] or [K,N]; [M,N]).
// M, N and K are free; every leading dimension must be a multiple of 8 (16 bytes) and ldc at least N
// rounded up to 8, because C is stored in whole 8-column groups (the up to 7 padding columns after
// column N of a row are written too: with zeros, since the operand columns they multiply are outside the
// tensor map and load as zeros).  Edge tiles are zero-filled on load and masked on store.  Shares zc_gemm_bf16's status word
// (zc_gemm_status_read_and_clear; code 8 = a bounded wait of this kernel expired).
// `bias`: null, or N bf16 values (16-byte aligned) added to every row of the product before it is rounded
// (and before the old C is added when `accumulate` is set).
// `ws`: null, or `ws_bytes` of device memory (16-byte aligned) of the caller's, that no other stream uses meanwhile, for the
// fp32 partial sums of a product that zc_gemm_2sm_split_bytes names a size for; without it such a product is not split.
static int gemm_2sm(const void* A, const void* B, void* C, const void* bias, int64_t M, int64_t N, int64_t K, int64_t lda,
                    int64_t ldb, int64_t ldc, int trans_a, int trans_b, int accumulate, bool cut_k, void* ws, int64_t ws_bytes,
                    cudaStream_t st) {
  ZC_NVTX_RANGE("zc_gemm_bf16_2sm");
  if (reinterpret_cast<uintptr_t>(bias) & 15) return zc::ERR_UNSUPPORTED;
  using namespace zc;
  using namespace zc::g2;
  if (M <= 0 || N <= 0 || K <= 0) return ERR_UNSUPPORTED;
  if (lda % 8 || ldb % 8 || ldc % 8 || ldc < ((N + 7) / 8) * 8) return ERR_UNSUPPORTED;
  if (lda < (trans_a ? M : K) || ldb < (trans_b ? K : N)) return ERR_BAD_ARG;
  const int64_t m_tiles = (M + BM - 1) / BM, n_tiles = (N + BN - 1) / BN;
  if (m_tiles * n_tiles > (1 << 28)) return ERR_UNSUPPORTED;
  int* status = zc_gemm_status_word();
  if (!status) return ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15)
    return ERR_UNSUPPORTED;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaSetDevice(dev);
  if (dev < 0 || dev >= 64) return ERR_BAD_ARG;
  const int a_major = trans_a ? MAJOR_MN : MAJOR_K;
  const int b_major = trans_b ? MAJOR_K : MAJOR_MN;
  if (a_major == MAJOR_MN && b_major == MAJOR_K) return ERR_UNSUPPORTED;  // no layer GEMM has this form
  const int smem = SMEM_BYTES;
  DeviceState& ds = g_state[dev];
  if (const int rc = init_state(ds, smem)) return rc;
  if (const int parts = small_parts(M, N, K, cut_k, ds.clusters))
    return gemm_small_launch(A, B, C, bias, M, N, K, lda, ldb, ldc, a_major, b_major, accumulate, parts, status, st);
  CUtensorMap mapA, mapB;
  bool ok;
  if (a_major == MAJOR_K) ok = make_map(&mapA, A, M, K, lda, BK, BM_CTA);
  else ok = make_map(&mapA, A, K, M, lda, 64, BK);
  if (b_major == MAJOR_K) ok = ok && make_map(&mapB, B, N, K, ldb, BK, BN_CTA);
  else ok = ok && make_map(&mapB, B, K, N, ldb, 64, BK);
  if (!ok) return ERR_BAD_ARG;
  Params p;
  p.C = (__nv_bfloat16*)C; p.M = M; p.N = N; p.ldc = ldc;
  p.m_tiles = (int)m_tiles; p.n_tiles = (int)n_tiles; p.k_blocks = (int)((K + BK - 1) / BK);
  p.bias = (const __nv_bfloat16*)bias;
  p.accumulate = accumulate;
  static const int forced_gm = getenv("ZC_GEMM_GROUP_M") ? atoi(getenv("ZC_GEMM_GROUP_M")) : 0;
  p.group_m = forced_gm > 0 ? forced_gm : 8;
  p.inv_band = 1.f / (float)((int64_t)p.group_m * p.n_tiles);
  p.status = status;
  Cut cut = cut_of(M, N, K, ds.clusters);
  if (!ws || ws_bytes < cut.bytes()) {
    cut.split = 1;
    cut.grid_clusters = (int)std::min<int64_t>(cut.tiles, ds.clusters);
  }
  p.split = cut.split;
  p.full_tiles = (int)(cut.split > 1 ? cut.tiles - cut.split_tiles : cut.tiles);
  p.partial = cut.split > 1 ? (float*)ws : nullptr;
  // Counters only where a second round is handed out, and not in a launch that is being recorded, which may be
  // replayed on any stream, nor on a stream beyond the first COUNTER_SLOTS or one of several under one handle.
  p.counter = nullptr;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cut.tiles > ds.clusters && st != cudaStreamPerThread && cudaStreamIsCapturing(st, &capture) == cudaSuccess &&
      capture == cudaStreamCaptureStatusNone) {
    std::lock_guard<std::mutex> lock(g_mutex);
    int slot = 0;
    while (slot < ds.owners && ds.owner[slot] != st) ++slot;
    if (slot == ds.owners && slot < COUNTER_SLOTS) ds.owner[ds.owners++] = st;
    if (slot < COUNTER_SLOTS) p.counter = ds.counters + 2 * slot;
  }
  const dim3 grid(2 * cut.grid_clusters);
  const auto launch = [&](auto kernel) { zc::launch_chained(kernel, grid, THREADS, smem, st, mapA, mapB, p); };
  if (a_major == MAJOR_K && b_major == MAJOR_K) launch(accumulate ? gemm_2sm_kernel<MAJOR_K, MAJOR_K, true> : gemm_2sm_kernel<MAJOR_K, MAJOR_K, false>);
  else if (a_major == MAJOR_K) launch(accumulate ? gemm_2sm_kernel<MAJOR_K, MAJOR_MN, true> : gemm_2sm_kernel<MAJOR_K, MAJOR_MN, false>);
  else launch(accumulate ? gemm_2sm_kernel<MAJOR_MN, MAJOR_MN, true> : gemm_2sm_kernel<MAJOR_MN, MAJOR_MN, false>);
  int rc = launch_status();
  if (rc == 0 && p.split > 1) {
    zc::launch_chained(gemm_2sm_fixup_kernel, dim3(BM * BN / 8 / 256, (unsigned)cut.split_tiles), 256, 0, st, p);
    rc = launch_status();
  }
  return rc;
}

int zc_gemm_bf16_2sm_ws(const void* A, const void* B, void* C, const void* bias, int64_t M, int64_t N, int64_t K,
                        int64_t lda, int64_t ldb, int64_t ldc, int trans_a, int trans_b, int accumulate, void* ws,
                        int64_t ws_bytes, cudaStream_t st) {
  return gemm_2sm(A, B, C, bias, M, N, K, lda, ldb, ldc, trans_a, trans_b, accumulate, true, ws, ws_bytes, st);
}

// The same with every sum along K in one piece.
int zc_gemm_bf16_2sm_bias(const void* A, const void* B, void* C, const void* bias, int64_t M, int64_t N, int64_t K,
                          int64_t lda, int64_t ldb, int64_t ldc, int trans_a, int trans_b, int accumulate,
                          cudaStream_t st) {
  return gemm_2sm(A, B, C, bias, M, N, K, lda, ldb, ldc, trans_a, trans_b, accumulate, false, nullptr, 0, st);
}

// Bytes of the workspace with which zc_gemm_bf16_2sm_ws splits an M x N x K product along K; 0 when it does not.
int64_t zc_gemm_2sm_split_bytes(int64_t M, int64_t N, int64_t K) {
  using namespace zc;
  using namespace zc::g2;
  int dev = 0;
  cudaGetDevice(&dev);
  if (M <= 0 || N <= 0 || K <= 0 || dev < 0 || dev >= 64 || init_state(g_state[dev], SMEM_BYTES)) return 0;
  return cut_of(M, N, K, g_state[dev].clusters).bytes();
}

// Bytes of the workspace that zc_gemm_bf16_2sm_ws wants for an M x N x K product: those, or 0 for one that the kernel of
// small products takes.
int64_t zc_gemm_ws_bytes(int64_t M, int64_t N, int64_t K) {
  using namespace zc::g2;
  const int64_t bytes = zc_gemm_2sm_split_bytes(M, N, K);  // (makes the device's state)
  int dev = 0;
  cudaGetDevice(&dev);
  return bytes && small_parts(M, N, K, true, g_state[dev].clusters) ? 0 : bytes;
}

int zc_gemm_bf16_2sm_ld(const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K, int64_t lda,
                        int64_t ldb, int64_t ldc, int trans_a, int trans_b, int accumulate, cudaStream_t st) {
  return zc_gemm_bf16_2sm_bias(A, B, C, nullptr, M, N, K, lda, ldb, ldc, trans_a, trans_b, accumulate, st);
}

// Contiguous operands: M, N and K multiples of 8.
int zc_gemm_bf16_2sm(const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K, int trans_a, int trans_b,
                     int accumulate, cudaStream_t st) {
  if (M % 8 || N % 8 || K % 8) return zc::ERR_UNSUPPORTED;
  return zc_gemm_bf16_2sm_ld(A, B, C, M, N, K, trans_a ? M : K, trans_b ? K : N, N, trans_a, trans_b, accumulate, st);
}

}  // extern "C"
