// v2 codec device functions shared by the standalone kernels (codec_v2.cu) and the fused
// collective kernels (symm_collectives.cu): window choice, chunk encode, chunk decode.
// `rec` may point to global or shared memory (generic address).
#pragma once
#include "codec_dev.cuh"

namespace zc {


// Largest / smallest exponent of the lane's 32: a comparison of byte pairs orders by the upper byte, so
// the words as they are give the odd bytes and the words shifted by one byte the even ones.
__device__ __forceinline__ uint32_t lane_max(const LaneSplit& s) {
  uint32_t m = __vmaxu2(s.ex[0], s.ex[0] << 8);
#pragma unroll
  for (int k = 1; k < 8; ++k) m = __vmaxu2(__vmaxu2(m, s.ex[k]), s.ex[k] << 8);
  return max(m >> 24, (m >> 8) & 0xFFu);
}
__device__ __forceinline__ uint32_t lane_min(const LaneSplit& s) {
  uint32_t m = __vminu2(s.ex[0], s.ex[0] << 8);
#pragma unroll
  for (int k = 1; k < 8; ++k) m = __vminu2(__vminu2(m, s.ex[k]), s.ex[k] << 8);
  return min(m >> 24, (m >> 8) & 0xFFu);
}
// 1 << sh, zero for sh outside 0..31
__device__ __forceinline__ uint32_t bit_or_zero(uint32_t sh) {
  uint32_t r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(sh));
  return r;
}

// What a lane brings to the window choice, the same for every chunk: its 0 / 1 weights for the prefix sum,
// and for its two candidates the prefixes it needs and the key of a window that holds no sample.
struct V2Lane {
  uint32_t wt[4];
  int key[2];
  uint32_t cand[2];  // width | first bin << 8 | end bin << 16
  __device__ __forceinline__ explicit V2Lane(int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      wt[i] = (i < lane ? 1u : 0u) | (i + 4 < lane ? 1u << 8 : 0u) | (i + 8 < lane ? 1u << 16 : 0u) |
              (i + 12 < lane ? 1u << 24 : 0u);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int idx = lane + 32 * r;
      int w = 1, d0 = 0;
      if (idx < V2_NUM_CAND) v2_candidate(idx, w, d0);
      cand[r] = (uint32_t)w | (uint32_t)d0 << 8 | (uint32_t)(d0 + (1 << w) - 1) << 16;
      key[r] = idx < V2_NUM_CAND ? ((128 * w + 4 * 256) << 6) | idx : 0x3fffffff;
    }
  }
};

// Window choice for one chunk.  Every lane passes its 8 exponent words; the result (header with
// n_esc = 0, or a raw header) is uniform across the warp.
__device__ __forceinline__ uint32_t v2_choose_warp(const LaneSplit& s, const V2Lane& k) {
  const int emax = (int)__reduce_max_sync(FULL, lane_max(s));
  const uint32_t all = rep4((uint32_t)emax);
  uint32_t diff = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) diff |= s.ex[i] ^ all;
  if (!__any_sync(FULL, diff != 0)) return v2_header(emax, 0, 0);
  const int anchor = emax > 15 ? emax - 15 : 0;
  // Sample histogram: byte 0 of every word (elements with index % 4 == 0).  Eight samples fit four bits,
  // so bins 0..7 and 8..15 are two words of nibble counters; a sample below the window shifts out of both.
  uint32_t h0 = 0, h1 = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t sh = ((s.ex[i] & 0xFFu) - (uint32_t)anchor) * 4u;
    h0 += bit_or_zero(sh);
    h1 += bit_or_zero(sh - 32u);
  }
  // Sum over the warp in 16-bit fields: word i has bins i and i + 4, word 4 + i bins 8 + i and 12 + i.
  // Lane k then keeps prefix[k], the sum of the bins below k, as dot products with its own 0 / 1 weights.
  int mine = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t ta = __reduce_add_sync(FULL, (h0 >> (4 * i)) & 0x000F000Fu);
    const uint32_t tb = __reduce_add_sync(FULL, (h1 >> (4 * i)) & 0x000F000Fu);
    mine = (int)__dp2a_hi(tb, k.wt[i], __dp2a_lo(ta, k.wt[i], (uint32_t)mine));
  }
  // estimated cost 128 w + 4 (256 - samples inside), ties to the smaller index
  int best = 0x7fffffff;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int hi = __shfl_sync(FULL, mine, (k.cand[r] >> 16) & 31);
    const int lo = __shfl_sync(FULL, mine, (k.cand[r] >> 8) & 31);
    best = min(best, k.key[r] - ((hi - lo) << 8));
  }
  best = __reduce_min_sync(FULL, best);
  if ((best >> 6) > V2_CHUNK_ELEMS) return v2_header(0, V2_RAW_WIDTH, 0);
  const uint32_t c0 = __shfl_sync(FULL, k.cand[0], best & 31), c1 = __shfl_sync(FULL, k.cand[1], best & 31);
  const uint32_t c = (best & 32) ? c1 : c0;
  return v2_header(anchor + (int)((c >> 8) & 0xFF), (int)(c & 0xFF), 0);
}

// Encode the chunk whose split fields are in `s` into `rec`; returns the final header.
// STORE_SM = false leaves out the first 1024 bytes of the record (the sign+mantissa bytes, which a
// caller that pushes them straight from registers does not need staged): only rec[1024 ...) is
// written, so `rec` may then point 1024 bytes before a buffer that holds just the record's tail.
// `row`: 32 bytes of shared memory of this lane, or null (scatter_escapes).
template <bool STORE_SM = true>
__device__ __forceinline__ uint32_t v2_encode_chunk(const LaneSplit& s, uint8_t* rec, int lane, const V2Lane& vl,
                                                    uint8_t* row = nullptr) {
  uint32_t hdr = v2_choose_warp(s, vl);
  int w = v2_hdr_width(hdr);
  const int base = v2_hdr_base(hdr);
  if (STORE_SM) {
    uint4* smp = reinterpret_cast<uint4*>(rec + lane * 32);
    smp[0] = make_uint4(s.sm[0], s.sm[1], s.sm[2], s.sm[3]);
    smp[1] = make_uint4(s.sm[4], s.sm[5], s.sm[6], s.sm[7]);
  }
  if (w != V2_RAW_WIDTH && w > 0) {
    uint32_t code[8], planes[4];
    codes_lane(s, base, (1u << w) - 1u, code);
    const uint32_t zm = code_planes(code, planes);
    int n_esc;
    const int pos = warp_excl_scan(__popc(zm), lane, n_esc);
    if (128 * w + n_esc > V2_CHUNK_ELEMS) {
      w = V2_RAW_WIDTH;
      hdr = v2_header(0, V2_RAW_WIDTH, 0);
    } else {
      hdr = v2_header(base, w, n_esc);
      uint32_t* pl = reinterpret_cast<uint32_t*>(rec + 1024) + lane;
      pl[0] = planes[0];
      if (w > 1) pl[32] = planes[1];
      if (w > 2) pl[64] = planes[2];
      if (w > 3) pl[96] = planes[3];
      if (n_esc > 0) {
        if (row) scatter_escapes(rec + 1024 + 128 * w + pos, s, zm, row);
        else scatter_escapes(rec + 1024 + 128 * w + pos, s, zm);
      }
    }
  }
  if (w == V2_RAW_WIDTH) {
    uint4* ep = reinterpret_cast<uint4*>(rec + 1024 + lane * 32);
    ep[0] = make_uint4(s.ex[0], s.ex[1], s.ex[2], s.ex[3]);
    ep[1] = make_uint4(s.ex[4], s.ex[5], s.ex[6], s.ex[7]);
  }
  return hdr;
}

// Encode with a window carried over from the previous chunk of the same stream ("hint", a header
// with width 1..4, or 0xFFFFFFFF for none).  The hint is kept while its exact escape count stays
// close to the count it had when it was chosen; otherwise the window is chosen afresh.  Any valid
// choice decodes correctly, so this only trades a little compression for skipping the histogram.
// Returns the header; `hint` / `hint_esc` are updated for the next chunk.
template <bool STORE_SM = true>
__device__ __forceinline__ uint32_t v2_encode_chunk_hint(const LaneSplit& s, uint8_t* rec, int lane, const V2Lane& vl,
                                                         uint32_t& hint, int& hint_esc) {
  if (hint != 0xFFFFFFFFu) {
    const int w = v2_hdr_width(hint), base = v2_hdr_base(hint);
    uint32_t code[8], planes[4];
    codes_lane(s, base, (1u << w) - 1u, code);
    const uint32_t zm = code_planes(code, planes);
    int n_esc;
    const int pos = warp_excl_scan(__popc(zm), lane, n_esc);
    if (n_esc <= hint_esc + (hint_esc >> 1) + 16 && 128 * w + n_esc <= V2_CHUNK_ELEMS) {
      if (STORE_SM) {
        uint4* smp = reinterpret_cast<uint4*>(rec + lane * 32);
        smp[0] = make_uint4(s.sm[0], s.sm[1], s.sm[2], s.sm[3]);
        smp[1] = make_uint4(s.sm[4], s.sm[5], s.sm[6], s.sm[7]);
      }
      uint32_t* pl = reinterpret_cast<uint32_t*>(rec + 1024) + lane;
      pl[0] = planes[0];
      if (w > 1) pl[32] = planes[1];
      if (w > 2) pl[64] = planes[2];
      if (w > 3) pl[96] = planes[3];
      scatter_escapes(rec + 1024 + 128 * w + pos, s, zm);
      return v2_header(base, w, n_esc);
    }
  }
  const uint32_t hdr = v2_encode_chunk<STORE_SM>(s, rec, lane, vl);
  const int w = v2_hdr_width(hdr);
  if (w >= 1 && w <= 4) {
    hint = hdr & 0xFFFFu;
    hint_esc = v2_hdr_nesc(hdr);
  } else {
    hint = 0xFFFFFFFFu;
  }
  return hdr;
}

// ---------------------------------------------------------------------------------------------
// Nibble mode: the cheap variant of the same idea, used by the fused collectives when the links are
// not the bottleneck.  Always four code bits with the window anchored at the chunk's largest
// exponent (base = max(emax - 14, 0): no histogram, no candidate search), and the 4-bit codes
// packed two per byte instead of sliced into four bit planes: byte 4 k + j of a lane's 16 code bytes
// holds element 8 k + j in its low nibble and element 8 k + 4 + j in its high one, so that encode is
// one shift-or per eight elements and decode two masks.  Same header word (base | 4 << 8 |
// n_esc << 16), same record size (1024 + 512 + n_esc bytes), same escape rule and raw fallback as
// width 4 of the plane format; which of the two layouts a width-4 record has is a property of the
// stream (the caller's choice), not of the record.  About 1.50 bytes per element on weights and
// gradients against 1.40 for the plane format, for roughly half the instructions.
// Writes only rec[1024 ...) (the sign+mantissa bytes are the caller's).  Returns the header.
__device__ __forceinline__ uint32_t v2_encode_chunk_nibble(const LaneSplit& s, uint8_t* rec, int lane,
                                                           uint8_t* row = nullptr) {
  const int emax = (int)__reduce_max_sync(FULL, lane_max(s));
  const int emin = (int)__reduce_min_sync(FULL, lane_min(s));
  if (emin == emax) return v2_header(emax, 0, 0);
  const int base = emax > 14 ? emax - 14 : 0;
  uint32_t code[8], nib[4];
  codes_lane(s, base, 15u, code);
  pack_nibbles(code, nib);
  int n_esc = 0, pos = 0;
  uint32_t zm = 0;
  if (emin < base) {  // warp-uniform: only then can an element fall below the window
    uint32_t planes[4] = {nib[0], nib[1], nib[2], nib[3]};
    nibbles_to_planes(planes);
    zm = ~(planes[0] | planes[1] | planes[2] | planes[3]);
    pos = warp_excl_scan(__popc(zm), lane, n_esc);
    if (512 + n_esc > V2_CHUNK_ELEMS) {
      uint4* ep = reinterpret_cast<uint4*>(rec + 1024 + lane * 32);
      ep[0] = make_uint4(s.ex[0], s.ex[1], s.ex[2], s.ex[3]);
      ep[1] = make_uint4(s.ex[4], s.ex[5], s.ex[6], s.ex[7]);
      return v2_header(0, V2_RAW_WIDTH, 0);
    }
  }
  reinterpret_cast<uint4*>(rec + 1024)[lane] = make_uint4(nib[0], nib[1], nib[2], nib[3]);
  if (n_esc > 0) {
    if (row) scatter_escapes(rec + 1024 + 512 + pos, s, zm, row);
    else scatter_escapes(rec + 1024 + 512 + pos, s, zm);
  }
  return v2_header(base, 4, n_esc);
}

// ---------------------------------------------------------------------------------------------
// Two-phase decode: `v2_prefetch` issues every global load a lane needs of one record (32 sign +
// mantissa bytes, its word of up to four planes, its share of the escape bytes) without using the
// values, `v2_decode_regs` turns them into exponents later.  A decoder that prefetches record i+1
// before it decodes record i keeps one record's loads in flight per warp at all times, which is what
// hides the memory latency when few warps per SM are available (inside the fused collectives, next
// to a GEMM).  Escapes go through 1 KB of shared memory per warp: the lanes store the 16-byte pieces
// they fetched, then every lane picks its own bytes by prefix position (no serial global loads).
// Loads use ld.global.cg: records may have been written by another GPU.
// ---------------------------------------------------------------------------------------------
struct RecRegs {
  uint32_t hdr;
  uint4 sm0, sm1;   // sign+mantissa bytes of this lane (raw mode: e0/e1 hold its exponent bytes)
  uint32_t pl[4];
  uint4 e0, e1;     // bytes [16 lane, 16 lane + 16) and [512 + 16 lane, ...) of the escape area
};

// SM_SPLIT: the sign+mantissa section is stored as two 512-byte halves (lane l's bytes 0..15 at 16 l,
// bytes 16..31 at 512 + 16 l) instead of 32 consecutive bytes per lane.  The fused collectives stage
// their records that way: each of a warp's two stores then covers 512 contiguous bytes of the peer's
// memory instead of 32 half-used 32-byte sectors.  Records in the documented format use SM_SPLIT = false.
// NIBBLE: width-4 records of this stream carry nibble-packed codes (v2_encode_chunk_nibble): a lane's
// 16 code bytes are one load and land in pl[0..3].
// `a32`: the record starts on a 32-byte boundary (documented format only): 32-byte sections are one access.
template <bool SM_SPLIT = false, bool NIBBLE = false>
__device__ __forceinline__ void v2_prefetch(const uint8_t* rec, uint32_t hdr, int lane, RecRegs& r, bool a32 = false) {
  r.hdr = hdr;
  if (!SM_SPLIT && a32) {
    uint32_t t[8];
    ld32(rec + lane * 32, t);
    r.sm0 = make_uint4(t[0], t[1], t[2], t[3]);
    r.sm1 = make_uint4(t[4], t[5], t[6], t[7]);
  } else if (SM_SPLIT) {
    const uint4* smp = reinterpret_cast<const uint4*>(rec) + lane;
    r.sm0 = __ldcg(smp);
    r.sm1 = __ldcg(smp + 32);
  } else {
    const uint4* smp = reinterpret_cast<const uint4*>(rec + lane * 32);
    r.sm0 = __ldcg(smp);
    r.sm1 = __ldcg(smp + 1);
  }
  const int w = v2_hdr_width(hdr);
  if (w == V2_RAW_WIDTH) {
    const uint4* ep = reinterpret_cast<const uint4*>(rec + 1024 + lane * 32);
    r.e0 = __ldcg(ep);
    r.e1 = __ldcg(ep + 1);
    return;
  }
  if (w == 0) return;
  if (NIBBLE) {
    const uint4 nb = __ldcg(reinterpret_cast<const uint4*>(rec + 1024) + lane);
    r.pl[0] = nb.x; r.pl[1] = nb.y; r.pl[2] = nb.z; r.pl[3] = nb.w;
  } else {
    const uint32_t* pl = reinterpret_cast<const uint32_t*>(rec + 1024) + lane;
    r.pl[0] = __ldcg(pl);
    r.pl[1] = w > 1 ? __ldcg(pl + 32) : 0u;
    r.pl[2] = w > 2 ? __ldcg(pl + 64) : 0u;
    r.pl[3] = w > 3 ? __ldcg(pl + 96) : 0u;
  }
  const int n_esc = v2_hdr_nesc(hdr);
  const uint4* eb = reinterpret_cast<const uint4*>(rec + 1024 + 128 * w);
  if (16 * lane < n_esc) r.e0 = __ldcg(eb + lane);
  if (512 + 16 * lane < n_esc) r.e1 = __ldcg(eb + 32 + lane);
}

// `esc_smem`: 1024 bytes of shared memory owned by this warp (16-byte aligned); `row`: 32 more of this lane, or
// null (insert_escapes).
template <bool NIBBLE = false>
__device__ __forceinline__ void v2_decode_regs(const RecRegs& r, uint8_t* esc_smem, int lane, LaneSplit& s,
                                               uint8_t* row = nullptr) {
  s.sm[0] = r.sm0.x; s.sm[1] = r.sm0.y; s.sm[2] = r.sm0.z; s.sm[3] = r.sm0.w;
  s.sm[4] = r.sm1.x; s.sm[5] = r.sm1.y; s.sm[6] = r.sm1.z; s.sm[7] = r.sm1.w;
  const int w = v2_hdr_width(r.hdr);
  const int base = v2_hdr_base(r.hdr);
  if (w == V2_RAW_WIDTH) {
    s.ex[0] = r.e0.x; s.ex[1] = r.e0.y; s.ex[2] = r.e0.z; s.ex[3] = r.e0.w;
    s.ex[4] = r.e1.x; s.ex[5] = r.e1.y; s.ex[6] = r.e1.z; s.ex[7] = r.e1.w;
    return;
  }
  if (w == 0) {
    const uint32_t e4 = rep4((uint32_t)base);
#pragma unroll
    for (int k = 0; k < 8; ++k) s.ex[k] = e4;
    return;
  }
  const int n_esc = v2_hdr_nesc(r.hdr);
  uint32_t nib[4] = {r.pl[0], r.pl[1], r.pl[2], r.pl[3]}, planes[4] = {r.pl[0], r.pl[1], r.pl[2], r.pl[3]};
  if (!NIBBLE) planes_to_nibbles(nib);
  uint32_t code[8];
  unpack_nibbles(nib, code);
  exponents_lane(code, base, s.ex);
  if (n_esc > 0) {  // warp-uniform
    if (NIBBLE) nibbles_to_planes(planes);
    const uint32_t zm = ~(planes[0] | planes[1] | planes[2] | planes[3]);
    uint4* es = reinterpret_cast<uint4*>(esc_smem);
    if (16 * lane < n_esc) es[lane] = r.e0;
    if (512 + 16 * lane < n_esc) es[32 + lane] = r.e1;
    int total;
    const int pos = warp_excl_scan(__popc(zm), lane, total);
    __syncwarp();
    if (row) insert_escapes(esc_smem + pos, zm, s.ex, row);
    else insert_escapes(esc_smem + pos, zm, s.ex);
    __syncwarp();  // the next record's escapes overwrite esc_smem
  }
}
}  // namespace zc
