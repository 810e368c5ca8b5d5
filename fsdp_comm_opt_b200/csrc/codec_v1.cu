// v1 (window-7) codec kernels for sm_100a: the wire format of the reference's hopper_fastzip2
// streams (reference: zipccl/hopper_zip.cu), produced and consumed by new kernels.
//
// Differences in how the work is done (the bytes on the wire are the same fields):
//   * bit planes, codes and sign/mantissa bytes are built four elements at a time on packed bytes
//     (codec_dev.cuh) instead of 32-iteration scalar loops, straight from registers;
//   * a CTA owns a range of consecutive chunks (1024 elements) of one work, each of its four warps a part of
//     it, and a warp keeps its outliers packed while it goes (no atomics, no block-wide synchronisation); a
//     second pass turns the parts' totals into offsets and moves every part's bytes to their place, so the
//     outlier stream is in element order and the result is deterministic;
//   * one decode kernel serves the fused/split x plain/unpad/unpad_v variants;
//   * sizes and offsets are 64-bit; ragged tails and unaligned outputs take a scalar path.
//
// Encode = 2 launches (encode, place); decode = 1 launch.  No host sync, no allocation.
//
// Why ranges: one CTA per 4096-element block spent a microsecond of dependent loads on finding its work
// before its first input load, synchronised to place its outliers, and needed a scan launch over all blocks
// between encode and compaction.  A part finds its work once and has the next chunk's input in flight while
// it codes the current one.
#include "codec_dev.cuh"
#include "launch_util.h"

namespace zc {

enum : int { LAYOUT_SPLIT = 0, LAYOUT_FUSED = 1 };

// The works' ranges are numbered one work after the other; range r covers `cnt` chunks from `c0` on, `part`
// of them per warp.
constexpr int V1_CHUNK = 1024;
// Chunks of a work: of its whole blocks, which are what the stream has offsets for (a size that is not a multiple of a
// block loses its rest, as it always has).
__device__ __forceinline__ int v1_chunks(long long n) { return (int)(n / V1_BLOCK_ELEMS) * (V1_BLOCK_ELEMS / V1_CHUNK); }
struct V1Range {
  int work;          // -1: no such range
  int c0, cnt;       // chunks inside the work
  int first;         // number of the work's first range
  int last;          // whether this is the work's last range
  long long n;       // padded elements of the work
  long long det_off; // byte offset of the work's stream (split: det stream, fused: scratch/final)
  long long aux_off; // split: offset into the outlier scratch / compacted stream; fused: unused
  long long in_off;  // element offset of the work in the dense input
  long long valid;   // valid elements of the work
  long long pad_off; // sum of padded sizes of the previous works
};

// Fused scratch layout of one work (stride 4*n): [0, det) det fields, [S, S+n) staged outliers.
__device__ __host__ inline long long fused_stage_off(long long n) { return align128(v1_det_bytes(n) + n); }

// Locate range `r` of 4 * `part` chunks.  Thread 0 walks the (few) works; the result is broadcast through
// shared memory.  Blocks past `total_blocks` (the size that the host was told) are left out.
__device__ __forceinline__ void v1_locate(int r, int part, long long total_blocks, const int* n_8, const int* orig_n,
                                          const int* nbytes_8, int n_works, int layout, bool decode, long long total_n,
                                          V1Range& w) {
  const long long total = total_blocks * (V1_BLOCK_ELEMS / V1_CHUNK);
  const int per = 4 * part;
  long long chunk = 0, det = 0, aux = 0, in_off = 0, pad = 0;
  int first = 0;
  w.work = -1;
  for (int i = 0; i < n_works; ++i) {
    const int n = __ldg(n_8 + i);
    const int nc = v1_chunks(n), nr = (nc + per - 1) / per;
    if (r < first + nr) {
      const int c0 = (r - first) * per;
      long long cnt = min(per, nc - c0);
      if (cnt > total - (chunk + c0)) cnt = total - (chunk + c0);
      if (cnt <= 0) return;
      w.work = i; w.c0 = c0; w.cnt = (int)cnt; w.first = first; w.last = r == first + nr - 1;
      w.n = n; w.det_off = det; w.aux_off = aux; w.in_off = in_off; w.pad_off = pad;
      if (orig_n) {
        w.valid = __ldg(orig_n + i);
      } else {
        const long long v = total_n - in_off;
        w.valid = v < 0 ? 0 : (v > n ? n : v);
      }
      return;
    }
    first += nr;
    chunk += nc;
    pad += n;
    in_off += orig_n ? __ldg(orig_n + i) : n;
    if (layout == LAYOUT_SPLIT) {
      det += n ? align128(v1_det_bytes(n)) : 0;
      aux += decode ? align128((long long)__ldg(nbytes_8 + i)) : n;
    } else {
      det += decode ? (long long)__ldg(nbytes_8 + i) : 4ll * n;
    }
  }
}

struct V1Fields {
  uint8_t* sm;
  uint32_t* b0;
  uint32_t* b1;
  uint32_t* b2;
  int* boff;
};

__device__ __forceinline__ V1Fields v1_fields(uint8_t* stream, long long n) {
  V1Fields f;
  f.sm = stream;
  f.b0 = reinterpret_cast<uint32_t*>(stream + n);
  f.b1 = f.b0 + n / 32;
  f.b2 = f.b1 + n / 32;
  f.boff = reinterpret_cast<int*>(f.b2 + n / 32);
  return f;
}

// ---------------------------------------------------------------------------------------------
// encode: one CTA of four warps per range, every warp on its own part of it
// ---------------------------------------------------------------------------------------------
// Outliers of a chunk go to shared memory at their place in the part's packed stream modulo 16, and leave
// for the staging area in whole 16-byte pieces; the bytes of an unfinished piece stay for the next chunk.
// boff holds offsets inside the part and totals[range] the counts of its four parts until the place kernel
// has run.
__global__ void __launch_bounds__(128, 8) v1_encode_kernel(
    const uint16_t* __restrict__ in, long long total_n, const int* __restrict__ n_8,
    const int* __restrict__ orig_n, int n_works, const int* __restrict__ bases, int layout,
    uint8_t* __restrict__ stream, uint8_t* __restrict__ stage, int* __restrict__ totals, int part, long long total_blocks) {
  __shared__ V1Range sw;
  __shared__ __align__(16) uint8_t pack_all[4][V1_CHUNK + 32];
  __shared__ __align__(16) uint8_t rows[128 * 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0)
    v1_locate(blockIdx.x, part, total_blocks, n_8, orig_n, nullptr, n_works, layout, false, total_n, sw);
  __syncthreads();
  if (sw.work < 0) return;
  const long long n = sw.n, valid = sw.valid;
  const int c0 = sw.c0 + warp * part, c1 = sw.c0 + min(sw.cnt, (warp + 1) * part);
  const int base = __ldg(bases);
  uint8_t* wstream = stream + sw.det_off;
  const V1Fields f = v1_fields(wstream, n);
  const uint16_t* src = in + sw.in_off;
  const int al = align_of(src);
  const bool sm32 = (reinterpret_cast<uintptr_t>(f.sm) & 31) == 0;
  uint8_t* st = ((layout == LAYOUT_SPLIT) ? stage + sw.aux_off : wstream + fused_stage_off(n)) + (long long)c0 * V1_CHUNK;
  const bool st16 = (reinterpret_cast<uintptr_t>(st) & 15) == 0;
  uint8_t* pack = pack_all[warp];
  if (tid == 0 && sw.c0 == 0) f.boff[n / V1_BLOCK_ELEMS] = base;
  int run = 0;  // outliers of the part so far
  LaneIn next;
  long long e0 = (long long)c0 * V1_CHUNK + lane * 32;
  if (c0 < c1) load_lane_v(src + e0, valid - e0, al, next);
  for (int c = c0; c < c1; ++c, e0 += V1_CHUNK) {
    LaneSplit s;
    split_lane(next, s);
    if (c + 1 < c1) load_lane_v(src + e0 + V1_CHUNK, valid - (e0 + V1_CHUNK), al, next);
    uint32_t code[8];
    codes_lane(s, base, 7u, code);
    if (base > 249) {
      // window would wrap past exponent 255: codes above 256-base do not exist
      const uint32_t lim = 256u - (uint32_t)base;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        uint32_t c8 = code[k], r = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t v = (c8 >> (8 * j)) & 0xFFu;
          r |= (v <= lim ? v : 0u) << (8 * j);
        }
        code[k] = r;
      }
    }
    uint32_t planes[4];
    const uint32_t zm = code_planes(code, planes);
    int total;
    const int pos = warp_excl_scan(__popc(zm), lane, total);
    if (sm32) {
      st32(f.sm + e0, s.sm);
    } else {
      uint4* smp = reinterpret_cast<uint4*>(f.sm + e0);
      smp[0] = make_uint4(s.sm[0], s.sm[1], s.sm[2], s.sm[3]);
      smp[1] = make_uint4(s.sm[4], s.sm[5], s.sm[6], s.sm[7]);
    }
    const long long widx = (long long)c * 32 + lane;
    f.b0[widx] = planes[0];
    f.b1[widx] = planes[1];
    f.b2[widx] = planes[2];
    if (lane == 0 && (c & 3) == 0) f.boff[c >> 2] = run;
    if (total == 0) continue;
    const int carry = run & 15;  // bytes of the unfinished piece, already at the front of pack
    scatter_escapes(pack + carry + pos, s, zm, rows + tid * 32);
    __syncwarp();
    const int have = carry + total, whole = have & ~15, full = st16 ? whole : 0;
    uint8_t* dst = st + (run - carry);
    for (int i = lane * 16; i < full; i += 512)
      *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(pack + i);
    // the unfinished piece is written too, and once more as a whole by the next chunk with outliers
    for (int i = full + lane; i < have; i += 32) dst[i] = pack[i];
    // Only the bytes of that piece move to the front: the next chunk's outliers are stored right behind them, by other
    // lanes and with nothing in between that orders the two.
    const uint8_t v = pack[whole + (lane & 15)];
    __syncwarp();
    if (lane < have - whole) pack[lane] = v;
    run += total;
  }
  if (lane == 0) totals[blockIdx.x * 4 + warp] = run;
}

// ---------------------------------------------------------------------------------------------
// place: ranges' totals -> offsets; staged outliers (and, for the fused layout, the det fields) -> final
// streams.  Every CTA adds up the totals before its own range (at most a few thousand words).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void copy_bytes(uint8_t* dst, const uint8_t* src, long long nbytes, int tid, int nthr) {
  if (dst == src || nbytes <= 0) return;
  if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0) {
    const long long nv = nbytes / 16;
    for (long long k = tid; k < nv; k += nthr)
      reinterpret_cast<uint4*>(dst)[k] = reinterpret_cast<const uint4*>(src)[k];
    for (long long k = nv * 16 + tid; k < nbytes; k += nthr) dst[k] = src[k];
  } else {
    for (long long k = tid; k < nbytes; k += nthr) dst[k] = src[k];
  }
}

// dst at any byte, src on a word: whole destination words cut out of two source words
__device__ __forceinline__ void copy_shifted(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, int nbytes,
                                             int tid, int nthr) {
  const int head = min(nbytes, (int)(-(intptr_t)dst & 3));
  if (tid < head) dst[tid] = src[tid];
  const int nw = (nbytes - head) >> 2, tail = head + 4 * nw;
  const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
  const uint32_t sh = (uint32_t)head * 8;
  uint32_t* d = reinterpret_cast<uint32_t*>(dst + head);
  int k = tid;
  for (; k + 3 * nthr < nw; k += 4 * nthr) {  // four words' loads in flight
    uint32_t a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      a[u] = w[k + u * nthr];
      b[u] = head ? w[k + u * nthr + 1] : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) d[k + u * nthr] = __funnelshift_r(a[u], b[u], sh);
  }
  for (; k < nw; k += nthr) d[k] = __funnelshift_r(w[k], head ? w[k + 1] : 0u, sh);
  if (tid < nbytes - tail) dst[tail + tid] = src[tail + tid];
}

__device__ __forceinline__ int sum4(const int4& v) { return v.x + v.y + v.z + v.w; }

__global__ void __launch_bounds__(128) v1_place_kernel(
    const int* __restrict__ n_8, int n_works, int layout, int* __restrict__ counts,
    int* __restrict__ nbytes_8, uint8_t* __restrict__ stream, const uint8_t* __restrict__ stage,
    uint8_t* __restrict__ final_out, const int4* __restrict__ totals, int part, long long total_blocks) {
  __shared__ V1Range sw;
  __shared__ int s_before[4];
  __shared__ unsigned long long s_final;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    v1_locate(blockIdx.x, part, total_blocks, n_8, nullptr, nullptr, n_works, layout, false, 0x7fffffffffffffffLL, sw);
    s_final = 0;
  }
  if (blockIdx.x == 0)
    for (int i = tid; i < n_works; i += 128)
      if (v1_chunks(n_8[i]) == 0) {
        counts[i] = 0;
        if (nbytes_8) nbytes_8[i] = n_8[i] ? (int)align128(v1_det_bytes(n_8[i])) : 0;
      }
  __syncthreads();
  if (sw.work < 0) return;
  // outliers of this work in earlier ranges: all warps; the streams of earlier works: one work per warp
  const int4 mine4 = __ldg(totals + blockIdx.x);
  int before = 0;
#pragma unroll 4
  for (int r = sw.first + tid; r < (int)blockIdx.x; r += 128) before += sum4(__ldg(totals + r));
  before = __reduce_add_sync(FULL, before);
  if (lane == 0) s_before[warp] = before;
  int first = 0;
  for (int j = 0; j < sw.work; ++j) {
    const long long n = n_8[j];
    const int nr = (v1_chunks(n) + 4 * part - 1) / (4 * part);
    if ((j & 3) == warp) {
      int t = 0;
#pragma unroll 4
      for (int r = lane; r < nr; r += 32) t += sum4(__ldg(totals + first + r));
      t = __reduce_add_sync(FULL, t);
      if (lane == 0 && n > 0)
        atomicAdd(&s_final, (unsigned long long)(layout == LAYOUT_SPLIT ? align128(t) : align128(v1_det_bytes(n) + t)));
    }
    first += nr;
  }
  __syncthreads();
  before = s_before[0] + s_before[1] + s_before[2] + s_before[3];
  const long long n = sw.n, nb = n / V1_BLOCK_ELEMS;
  if (sw.last && tid == 0) {
    counts[sw.work] = before + sum4(mine4);
    if (nbytes_8) nbytes_8[sw.work] = (int)align128(v1_det_bytes(n) + before + sum4(mine4));
  }
  // this warp's part
  const int mine = warp == 0 ? mine4.x : warp == 1 ? mine4.y : warp == 2 ? mine4.z : mine4.w;
  before += (warp > 0 ? mine4.x : 0) + (warp > 1 ? mine4.y : 0) + (warp > 2 ? mine4.z : 0);
  const int c0 = sw.c0 + warp * part, c1 = sw.c0 + min(sw.cnt, (warp + 1) * part);
  uint8_t* wstream = stream + sw.det_off;
  const V1Fields f = v1_fields(wstream, n);
  const uint8_t* st = ((layout == LAYOUT_SPLIT) ? stage + sw.aux_off : wstream + fused_stage_off(n)) + (long long)c0 * V1_CHUNK;
  uint8_t* fstream = final_out + s_final;
  const V1Fields g = v1_fields(fstream, n);
  uint8_t* dst = (layout == LAYOUT_SPLIT ? fstream : reinterpret_cast<uint8_t*>(g.boff + nb + 1)) + before;
  if ((reinterpret_cast<uintptr_t>(st) & 3) == 0) copy_shifted(dst, st, mine, lane, 32);
  else copy_bytes(dst, st, mine, lane, 32);
  const bool copy_det = layout == LAYOUT_FUSED && fstream != wstream;
  for (int b = ((c0 + 3) >> 2) + lane; b < (c1 + 3) >> 2; b += 32) {
    const int off = f.boff[b] + before;
    f.boff[b] = off;
    if (copy_det) g.boff[b] = off;
  }
  if (copy_det && c0 < c1) {
    const long long e0 = (long long)c0 * V1_CHUNK;
    copy_bytes(g.sm + e0, f.sm + e0, (long long)(c1 - c0) * V1_CHUNK, lane, 32);
    for (long long k = (long long)c0 * 32 + lane; k < (long long)c1 * 32; k += 32) {
      g.b0[k] = f.b0[k];
      g.b1[k] = f.b1[k];
      g.b2[k] = f.b2[k];
    }
    if (tid == 0 && sw.c0 == 0) g.boff[nb] = f.boff[nb];
  }
}

// ---------------------------------------------------------------------------------------------
// decode: every variant; one CTA per range, every warp on its own part with the next chunk's planes and
// bytes in flight.  The outlier stream of a work has no gaps, so a warp needs its place in it once.  A
// chunk's outliers are fetched together into shared memory (one latency for all of them).
// ---------------------------------------------------------------------------------------------
struct V1Regs {
  uint32_t sm[8], pl[3];
};
__device__ __forceinline__ void v1_fetch(const V1Fields& f, int c, int lane, bool sm32, V1Regs& r) {
  const long long e0 = (long long)c * V1_CHUNK + lane * 32, widx = (long long)c * 32 + lane;
  r.pl[0] = __ldg(f.b0 + widx);
  r.pl[1] = __ldg(f.b1 + widx);
  r.pl[2] = __ldg(f.b2 + widx);
  if (sm32) {
    ld32(f.sm + e0, r.sm);
  } else {
    const uint4* smp = reinterpret_cast<const uint4*>(f.sm + e0);
    const uint4 a = __ldg(smp), b = __ldg(smp + 1);
    r.sm[0] = a.x; r.sm[1] = a.y; r.sm[2] = a.z; r.sm[3] = a.w;
    r.sm[4] = b.x; r.sm[5] = b.y; r.sm[6] = b.z; r.sm[7] = b.w;
  }
}

__global__ void __launch_bounds__(128, 8) v1_decode_kernel(
    const uint8_t* __restrict__ stream, const uint8_t* __restrict__ esc_stream, const int* __restrict__ n_8,
    const int* __restrict__ nbytes_8, int n_works, int layout, long long orig_each,
    const int* __restrict__ out_off, const int* __restrict__ orig_n, uint16_t* __restrict__ out,
    long long out_numel, int part, long long total_blocks) {
  __shared__ V1Range sw;
  __shared__ __align__(16) uint8_t esc_all[4][V1_CHUNK + 32];
  __shared__ __align__(16) uint8_t rows[128 * 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0)
    v1_locate(blockIdx.x, part, total_blocks, n_8, orig_n, nbytes_8, n_works, layout, true, 0x7fffffffffffffffLL, sw);
  __syncthreads();
  if (sw.work < 0) return;
  const long long n = sw.n, nb = n / V1_BLOCK_ELEMS;
  const int c0 = sw.c0 + warp * part, c1 = sw.c0 + min(sw.cnt, (warp + 1) * part);
  if (c0 >= c1) return;
  const V1Fields f = v1_fields(const_cast<uint8_t*>(stream) + sw.det_off, n);
  const bool sm32 = (reinterpret_cast<uintptr_t>(f.sm) & 31) == 0;
  V1Regs cur;
  v1_fetch(f, c0, lane, sm32, cur);
  const int base = __ldg(f.boff + nb);
  // the part's place in the outlier stream: its block's offset and the outliers of the block's earlier chunks
  int skip = 0;
  for (int c = c0 & ~3; c < c0; ++c) {
    const long long widx = (long long)c * 32 + lane;
    skip += __popc(~(__ldg(f.b0 + widx) | __ldg(f.b1 + widx) | __ldg(f.b2 + widx)));
  }
  const uint8_t* esc = ((layout == LAYOUT_SPLIT) ? esc_stream + sw.aux_off
                                                 : reinterpret_cast<const uint8_t*>(f.boff + nb + 1)) +
                       __ldg(f.boff + (c0 >> 2)) + __reduce_add_sync(FULL, skip);
  long long valid_work = orig_n ? sw.valid : (orig_each >= 0 ? orig_each : n);
  const long long ooff = out_off ? (long long)out_off[sw.work]
                                 : (orig_each >= 0 ? (long long)sw.work * orig_each : sw.pad_off);
  if (valid_work > out_numel - ooff) valid_work = out_numel - ooff;
  uint16_t* dst = out + ooff;
  const int al = align_of(dst);
  uint8_t* es = esc_all[warp];
  long long e0 = (long long)c0 * V1_CHUNK + lane * 32;
  for (int c = c0; c < c1; ++c, e0 += V1_CHUNK) {
    V1Regs next;
    if (c + 1 < c1) v1_fetch(f, c + 1, lane, sm32, next);
    const uint32_t zm = ~(cur.pl[0] | cur.pl[1] | cur.pl[2]);
    int total;
    const int pos = warp_excl_scan(__popc(zm), lane, total);
    const int mis = (int)(reinterpret_cast<uintptr_t>(esc) & 15);
    const uint4* ev = reinterpret_cast<const uint4*>(esc - mis);
    if (total > 0)
      for (int i = lane; i * 16 < mis + total; i += 32) reinterpret_cast<uint4*>(es)[i] = __ldg(ev + i);
    esc += total;
    LaneSplit s;
#pragma unroll
    for (int k = 0; k < 8; ++k) s.sm[k] = cur.sm[k];
    uint32_t nib[4] = {cur.pl[0], cur.pl[1], cur.pl[2], 0u}, code[8];
    planes_to_nibbles(nib);
    unpack_nibbles(nib, code);
    exponents_lane(code, base, s.ex);
    if (total > 0) {
      __syncwarp();
      insert_escapes(es + mis + pos, zm, s.ex, rows + tid * 32);
      __syncwarp();
    }
    LaneIn o;
    join_lane(s, o);
    store_lane_v(dst + e0, valid_work - e0, al, o);
    cur = next;
  }
}

// Ranges: one per resident CTA, so the launch is one wave and every part's chunks follow one another, and up
// to four waves once a part still has a dozen chunks then: their CTAs sweep the buffers more closely in address
// order (218 112 000 elements: encode 160 -> 149 us, decode 141 -> 127; at 27 M elements the waves' set-up costs
// more than they give).  Works end their last range early, hence the surplus of one range per work.
template <typename K>
static int v1_split(K kernel, int (&cached)[64], long long total_blocks, int n_works, int& part) {
  const long long ctas = resident_ctas(kernel, 128, 0, cached);
  const long long waves = std::min<long long>(4, std::max<long long>(1, total_blocks / (12 * ctas)));
  part = (int)((total_blocks + waves * ctas - 1) / (waves * ctas));  // four chunks a block, four warps a CTA
  return (int)std::min<long long>(total_blocks, (total_blocks + part - 1) / part + n_works);
}

// ---------------------------------------------------------------------------------------------
// base statistic: bases[0] = clamp(floor(log2(max(std,1e-30)) - 5.35 + 127), 0, 255)
// (reference rule: main/zipccl_comm.py:56-64).  One launch, no host sync: one CTA per SM adds up its
// moments in double, eight elements per load, and the last CTA to finish adds the partial sums and
// evaluates the rule.  (Atomic adds of all CTAs into one pair of doubles took as long as the reading.)
// ---------------------------------------------------------------------------------------------
constexpr int MOMENT_CTAS = 256, MOMENT_THREADS = 1024;
struct Moments {
  double2 part[MOMENT_CTAS];
  unsigned done, pad[3];
};
__device__ __forceinline__ double2 block_sum2(double s, double q) {  // result in warp 0
  __shared__ double2 red[MOMENT_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(FULL, s, o);
    q += __shfl_xor_sync(FULL, q, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_double2(s, q);
  __syncthreads();
  const double2 v = red[threadIdx.x & 31];
  s = v.x;
  q = v.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(FULL, s, o);
    q += __shfl_xor_sync(FULL, q, o);
  }
  return make_double2(s, q);
}

__global__ void __launch_bounds__(MOMENT_THREADS) v1_base_kernel(const uint16_t* __restrict__ x, long long n,
                                                                 Moments* __restrict__ acc, int* __restrict__ bases) {
  double s = 0.0, q = 0.0;
  auto add2 = [&](uint32_t w) {
    const float a = __uint_as_float(w << 16), b = __uint_as_float(w & 0xFFFF0000u);
    s += a;
    s += b;
    q += (double)a * a;
    q += (double)b * b;
  };
  const long long t = (long long)blockIdx.x * MOMENT_THREADS + threadIdx.x, nt = (long long)gridDim.x * MOMENT_THREADS;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const long long nv = vec ? n / 8 : 0;
  const uint4* xv = reinterpret_cast<const uint4*>(x);
  // The next trip's loads are in flight while this one's values are added, the last trip's together like the others'
  // (an encode of 27 264 000 elements with its statistic: 53.5 -> 51.5 us).
  uint4 v[4];
  auto fetch = [&](long long i) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * nt < nv) v[k] = __ldg(xv + i + k * nt);
  };
  fetch(t);
  long long i = t;
  for (; i + 7 * nt < nv; i += 4 * nt) {  // all of the next trip is there: no checks (27 264 000 elements in L2 15.7 -> 14.6 us, 2 x 10^8 78 -> 64)
    uint4 c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = v[k];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __ldg(xv + i + (4 + k) * nt);
#pragma unroll
    for (int k = 0; k < 4; ++k) { add2(c[k].x); add2(c[k].y); add2(c[k].z); add2(c[k].w); }
  }
  for (; i < nv; i += 4 * nt) {
    uint4 c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = v[k];
    fetch(i + 4 * nt);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * nt < nv) { add2(c[k].x); add2(c[k].y); add2(c[k].z); add2(c[k].w); }
  }
  for (i = nv * 8 + t; i < n; i += nt) add2((uint32_t)__ldg(x + i));
  __shared__ bool last;
  double2 t2 = block_sum2(s, q);
  if (threadIdx.x == 0) {
    acc->part[blockIdx.x] = t2;
    __threadfence();
    last = atomicAdd(&acc->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  t2 = make_double2(0.0, 0.0);
  if (threadIdx.x < gridDim.x) {
    t2.x = __ldcg(&acc->part[threadIdx.x].x);
    t2.y = __ldcg(&acc->part[threadIdx.x].y);
  }
  t2 = block_sum2(t2.x, t2.y);
  if (threadIdx.x != 0) return;
  s = t2.x;
  q = t2.y;
  const double mean = s / (double)n;
  double var = n > 1 ? (q - (double)n * mean * mean) / (double)(n - 1) : 0.0;
  if (!(var > 0.0)) var = 0.0;
  double sd = sqrt(var);
  if (sd < 1e-30) sd = 1e-30;
  double b = floor(log2(sd) - 5.35 + 127.0);
  b = b < 0.0 ? 0.0 : (b > 255.0 ? 255.0 : b);
  bases[0] = (int)b;
  acc->done = 0u;
}

}  // namespace zc

extern "C" {

// Words of `totals` (16-byte aligned) that an encode of `total_blocks` blocks in `n_works` works may use.
long long zc_v1_totals_words(long long total_blocks, int n_works) {
  return 4 * std::min<long long>(total_blocks, 4 * 16ll * zc::sm_count() + n_works);
}

static int v1_encode(const void* in, long long total_n, const int* n_8, const int* orig_n, int n_works, const int* bases,
                     int layout, void* stream, void* stage, void* final_out, int* nbytes_8, int* counts, int* totals,
                     long long total_blocks, cudaStream_t st) {
  using namespace zc;
  if (total_blocks <= 0) return 0;
  if (n_works <= 0) return ERR_BAD_ARG;
  static int cached[64];
  int part;
  const int grid = v1_split(v1_encode_kernel, cached, total_blocks, n_works, part);
  v1_encode_kernel<<<grid, 128, 0, st>>>((const uint16_t*)in, total_n, n_8, orig_n, n_works, bases, layout,
                                         (uint8_t*)stream, (uint8_t*)stage, totals, part, total_blocks);
  v1_place_kernel<<<grid, 128, 0, st>>>(n_8, n_works, layout, counts, nbytes_8, (uint8_t*)stream, (const uint8_t*)stage,
                                        (uint8_t*)final_out, (const int4*)totals, part, total_blocks);
  return launch_status();
}

int zc_v1_encode_split(const void* in, long long total_n, const int* n_8, const int* orig_n, int n_works,
                       const int* bases, void* det, void* scratch, void* esc_final, int* counts, int* totals,
                       long long total_blocks, cudaStream_t st) {
  return v1_encode(in, total_n, n_8, orig_n, n_works, bases, zc::LAYOUT_SPLIT, det, scratch, esc_final, nullptr, counts,
                   totals, total_blocks, st);
}

int zc_v1_encode_fused(const void* in, long long total_n, const int* n_8, int n_works, const int* bases,
                       void* scratch, void* out_final, long long out_final_bytes, int* nbytes_8, int* counts, int* totals,
                       long long total_blocks, cudaStream_t st) {
  (void)out_final_bytes;
  return v1_encode(in, total_n, n_8, nullptr, n_works, bases, zc::LAYOUT_FUSED, scratch, nullptr, out_final, nbytes_8,
                   counts, totals, total_blocks, st);
}

static int v1_decode(const void* stream, const void* esc, const int* n_8, const int* nbytes_8, int n_works, int layout,
                     long long orig_each, const int* out_off, const int* orig_n, void* out, long long out_numel,
                     long long total_blocks, cudaStream_t st) {
  using namespace zc;
  if (total_blocks <= 0) return 0;
  static int cached[64];
  int part;
  const int grid = v1_split(v1_decode_kernel, cached, total_blocks, n_works, part);
  v1_decode_kernel<<<grid, 128, 0, st>>>((const uint8_t*)stream, (const uint8_t*)esc, n_8, nbytes_8, n_works, layout,
                                         orig_each, out_off, orig_n, (uint16_t*)out, out_numel, part, total_blocks);
  return launch_status();
}

int zc_v1_decode_split(const void* det, const void* esc, const int* n_8, const int* nbytes_8, int n_works,
                       long long orig_each, const int* out_off, const int* orig_n, void* out,
                       long long out_numel, long long total_blocks, cudaStream_t st) {
  return v1_decode(det, esc, n_8, nbytes_8, n_works, zc::LAYOUT_SPLIT, orig_each, out_off, orig_n, out, out_numel,
                   total_blocks, st);
}

int zc_v1_decode_fused(const void* comp, const int* n_8, const int* nbytes_8, int n_works, long long orig_each,
                       void* out, long long out_numel, long long total_blocks, cudaStream_t st) {
  return v1_decode(comp, nullptr, n_8, nbytes_8, n_works, zc::LAYOUT_FUSED, orig_each, nullptr, nullptr, out, out_numel,
                   total_blocks, st);
}

// Bytes of the workspace (16-byte aligned) of a base statistic.
long long zc_v1_moments_bytes() { return sizeof(zc::Moments); }

// `ws`: zero before its first use and left so by every launch; launches that share it have to follow one another.
int zc_v1_base_from_std(const void* x, long long n, int* bases, void* ws, cudaStream_t st) {
  using namespace zc;
  if (n <= 0) return 0;
  const int grid = (int)std::min<long long>(n / 8 / MOMENT_THREADS + 1, std::min(sm_count(), MOMENT_CTAS));
  v1_base_kernel<<<grid, MOMENT_THREADS, 0, st>>>((const uint16_t*)x, n, (Moments*)ws, bases);
  return launch_status();
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Allocation-free variant (see zc_noalloc.h): the outlier staging area is a static device array.
// ---------------------------------------------------------------------------------------------
#include <cstdio>
#include <mutex>

#include "zc_noalloc.h"

static __device__ __align__(256) unsigned char g_noalloc_scratch[ZC_NOALLOC_MAX_ELEMS];
// the ranges' outlier totals (a range has at least one block)
static __device__ int4 g_noalloc_totals[ZC_NOALLOC_MAX_ELEMS / zc::V1_BLOCK_ELEMS];

namespace {
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_ptr[64] = {nullptr};  // device addresses of the arrays, per device
int* g_noalloc_totals_ptr[64] = {nullptr};

// In host code `g_noalloc_scratch` is only a handle for the runtime, not a device address; the
// address is looked up once per device, with that device current.
int noalloc_scratch(unsigned char** out, int** totals) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ZC_ERR_SYMBOL;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    unsigned char* p = nullptr;
    int* q = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
    if (e == cudaSuccess) e = cudaGetSymbolAddress((void**)&q, g_noalloc_totals);
    if (e != cudaSuccess || p == nullptr || q == nullptr) {
      fprintf(stderr, "[zc_noalloc] cudaGetSymbolAddress failed on device %d: %s\n", dev, cudaGetErrorString(e));
      return ZC_ERR_SYMBOL;
    }
    g_noalloc_ptr[dev] = p;
    g_noalloc_totals_ptr[dev] = q;
  }
  *out = g_noalloc_ptr[dev];
  *totals = g_noalloc_totals_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int zc_v1_encode_split_noalloc(const void* in, long long total_n, const int* n_8, const int* orig_n,
                                          int n_works, const int* bases, void* det, void* esc_final, int* counts,
                                          long long total_blocks, cudaStream_t st) {
  using namespace zc;
  if (total_blocks <= 0) return 0;
  if (n_works <= 0) return ERR_BAD_ARG;
  if (total_blocks * V1_BLOCK_ELEMS > ZC_NOALLOC_MAX_ELEMS) {
    fprintf(stderr,
            "[zc_noalloc] request of %lld padded elements exceeds the built-in scratch of %lld; "
            "use zc_v1_encode_split with your own scratch buffer\n",
            total_blocks * V1_BLOCK_ELEMS, (long long)ZC_NOALLOC_MAX_ELEMS);
    return ZC_ERR_TOO_LARGE;
  }
  unsigned char* scratch = nullptr;
  int* totals = nullptr;
  const int rc = noalloc_scratch(&scratch, &totals);
  if (rc != 0) return rc;
  return zc_v1_encode_split(in, total_n, n_8, orig_n, n_works, bases, det, scratch, esc_final, counts, totals,
                            total_blocks, st);
}
