// v2 codec kernels (per-chunk base and width) for sm_100a: standalone encode and decode.
//
// One warp per 1024-element chunk, eight warps per CTA, persistent grid-stride loop sized to the
// SM count.  No shared memory, no atomics, no cross-chunk dependency: chunk c lives at the fixed
// offset c*2048 of the record buffer, so encode and decode are embarrassingly parallel and the
// same device functions are reused inside the fused collective kernels.
#include "codec_v2_dev.cuh"
#include "launch_util.h"
#include "nvtx_util.h"

namespace zc {


// NIBBLE: records in nibble mode (codec_format.h): fixed four code bits, codes packed two per byte.
// The plane encoder is bound by its integer work (window choice, codes, planes), the others by memory.
template <bool NIBBLE>
__global__ void __launch_bounds__(256) v2_encode_kernel(const uint16_t* __restrict__ in, int64_t n,
                                                        uint8_t* __restrict__ records,
                                                        uint32_t* __restrict__ headers, int64_t nc) {
  __shared__ __align__(16) uint8_t rows[256 * 32];
  const int lane = threadIdx.x & 31;
  const V2Lane vl(lane);
  uint8_t* row = rows + threadIdx.x * 32;
  const int64_t warp0 = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t stride = (int64_t)gridDim.x * 8;
  const int al = align_of(in);
  const bool ral = align_of(records) == 32;
  // the next chunk's elements are in flight while this chunk is coded
  LaneIn li;
  auto fetch = [&](int64_t c) {
    const int64_t e0 = c * V2_CHUNK_ELEMS + lane * 32;
    load_lane_v(in + e0, n - e0, al, li);
  };
  if (warp0 < nc) fetch(warp0);
  for (int64_t c = warp0; c < nc; c += stride) {
    LaneSplit s;
    split_lane(li, s);
    if (c + stride < nc) fetch(c + stride);
    uint8_t* rec = records + c * V2_SLOT_BYTES;
    if (ral) {
      st32(rec + lane * 32, s.sm);
    } else {
      uint4* smp = reinterpret_cast<uint4*>(rec + lane * 32);
      smp[0] = make_uint4(s.sm[0], s.sm[1], s.sm[2], s.sm[3]);
      smp[1] = make_uint4(s.sm[4], s.sm[5], s.sm[6], s.sm[7]);
    }
    const uint32_t hdr = NIBBLE ? v2_encode_chunk_nibble(s, rec, lane, row) : v2_encode_chunk<false>(s, rec, lane, vl, row);
    if (lane == 0) headers[c] = hdr;
  }
}

template <bool NIBBLE>
__global__ void __launch_bounds__(256) v2_decode_kernel(const uint8_t* __restrict__ records,
                                                        const uint32_t* __restrict__ headers, int64_t n,
                                                        uint16_t* __restrict__ out, int64_t nc) {
  __shared__ __align__(16) uint8_t esc[8][1024];
  __shared__ __align__(16) uint8_t rows[256 * 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t warp0 = (int64_t)blockIdx.x * 8 + warp;
  const int64_t stride = (int64_t)gridDim.x * 8;
  const int al = align_of(out);
  const bool ral = align_of(records) == 32;
  // software pipeline: record c + stride is in flight while record c is decoded and stored
  RecRegs cur, nxt;
  int64_t c = warp0;
  if (c < nc) v2_prefetch<false, NIBBLE>(records + c * V2_SLOT_BYTES, __ldcg(headers + c), lane, cur, ral);
  uint32_t hdr_next = (c + stride < nc) ? __ldcg(headers + c + stride) : 0u;
  for (; c < nc; c += stride) {
    const int64_t cn = c + stride;
    if (cn < nc) {
      v2_prefetch<false, NIBBLE>(records + cn * V2_SLOT_BYTES, hdr_next, lane, nxt, ral);
      if (cn + stride < nc) hdr_next = __ldcg(headers + cn + stride);
    }
    LaneSplit s;
    v2_decode_regs<NIBBLE>(cur, esc[warp], lane, s, rows + threadIdx.x * 32);
    LaneIn o;
    join_lane(s, o);
    const int64_t e0 = c * V2_CHUNK_ELEMS + lane * 32;
    store_lane_v(out + e0, n - e0, al, o);
    cur = nxt;
  }
}

// Waves of CTAs per launch.  One wave that strides through the whole buffer lets its warps drift apart, and
// DRAM then serves more open pages than it keeps: 200 M elements in nibble mode took 132 us to encode
// and 127 to decode, with 16 waves (a warp codes two or three chunks, the CTAs follow one another in address
// order) 107 and 107; the bytes need 108 at the copy bandwidth.  The plane coder has more registers and set-up
// per CTA: 4 waves (140 / 127 -> 123 / 113 us), 16 are slower again.
static int v2_grid(int64_t nc, int64_t resident, bool nibble) {
  // three chunks per warp at least, so that a warp has one to fetch ahead (20 M elements decoded in one
  // wave 14.4 us, in shorter ones 17)
  const int64_t waves = std::min<int64_t>(nibble ? 16 : 4, std::max<int64_t>(1, nc / (resident * 8 * 3)));
  return (int)std::min<int64_t>((nc + 7) / 8, waves * resident);
}

template <bool NIBBLE>
int v2_encode_launch(const void* in, int64_t n, void* records, void* headers, cudaStream_t stream) {
  const int64_t nc = (n + V2_CHUNK_ELEMS - 1) / V2_CHUNK_ELEMS;
  if (nc == 0) return 0;
  static int cached[64];
  const int grid = v2_grid(nc, resident_ctas(v2_encode_kernel<NIBBLE>, 256, 0, cached), NIBBLE);
  v2_encode_kernel<NIBBLE><<<grid, 256, 0, stream>>>((const uint16_t*)in, n, (uint8_t*)records, (uint32_t*)headers, nc);
  return launch_status();
}

template <bool NIBBLE>
int v2_decode_launch(const void* records, const void* headers, int64_t n, void* out, int max_ctas, cudaStream_t stream) {
  const int64_t nc = (n + V2_CHUNK_ELEMS - 1) / V2_CHUNK_ELEMS;
  if (nc == 0) return 0;
  static int cached[64];
  int grid = v2_grid(nc, resident_ctas(v2_decode_kernel<NIBBLE>, 256, 0, cached), NIBBLE);
  if (max_ctas > 0) grid = std::min(grid, max_ctas);
  v2_decode_kernel<NIBBLE><<<grid, 256, 0, stream>>>((const uint8_t*)records, (const uint32_t*)headers, n,
                                                     (uint16_t*)out, nc);
  return launch_status();
}

}  // namespace zc

extern "C" {

int zc_v2_encode(const void* in, int64_t n, void* records, void* headers, cudaStream_t stream) {
  ZC_NVTX_RANGE("zc_v2_encode");
  return zc::v2_encode_launch<false>(in, n, records, headers, stream);
}

// `max_ctas` > 0 caps the grid (how the decoder behaves with the SM budget it has inside a fused
// collective); 0 sizes it to the device.
int zc_v2_decode_ctas(const void* records, const void* headers, int64_t n, void* out, int max_ctas,
                      cudaStream_t stream) {
  return zc::v2_decode_launch<false>(records, headers, n, out, max_ctas, stream);
}

int zc_v2_decode(const void* records, const void* headers, int64_t n, void* out, cudaStream_t stream) {
  ZC_NVTX_RANGE("zc_v2_decode");
  return zc::v2_decode_launch<false>(records, headers, n, out, 0, stream);
}

// The same two entry points for records in nibble mode (the records the fused collectives stage by
// default, here with the documented 32-consecutive-bytes-per-lane sign+mantissa section).
int zc_v2_encode_nibble(const void* in, int64_t n, void* records, void* headers, cudaStream_t stream) {
  ZC_NVTX_RANGE("zc_v2_encode_nibble");
  return zc::v2_encode_launch<true>(in, n, records, headers, stream);
}

int zc_v2_decode_nibble(const void* records, const void* headers, int64_t n, void* out, cudaStream_t stream) {
  ZC_NVTX_RANGE("zc_v2_decode_nibble");
  return zc::v2_decode_launch<true>(records, headers, n, out, 0, stream);
}

}  // extern "C"
