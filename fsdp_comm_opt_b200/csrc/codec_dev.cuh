// Warp-level building blocks of the BF16 exponent codec for sm_100a.
//
// One warp handles 1024 consecutive elements; lane l owns elements l*32 .. l*32+31 (64 bytes),
// which is the ownership both wire formats prescribe (v1: thread t of a 128-thread block, v2: lane
// l of a chunk).  Everything is done four elements at a time on packed bytes (SWAR), with no
// shared memory and no per-element branches:
//   split      16 u32 (32 bf16) -> 8 u32 of sign+mantissa bytes, 8 u32 of exponent bytes
//   codes      per-byte  c = e - (base-1);  code = (1 <= c <= span) ? c : 0
//   planes     bit p of every code gathered into one 32-bit word per plane: the 32 four-bit codes are
//              an 4 x 32 bit matrix in four words, transposed in place by two exchanges of index bits
//              (24 instructions for all planes; gathering bit by bit took 40 per plane)
//   escapes    exponent bytes whose code is 0, compacted in element order
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "codec_format.h"

namespace zc {

constexpr unsigned FULL = 0xffffffffu;
constexpr uint32_t H4 = 0x80808080u;
constexpr uint32_t L4 = 0x7f7f7f7fu;

__device__ __forceinline__ uint32_t rep4(uint32_t b) { return (b & 0xFFu) * 0x01010101u; }

// per-byte x - y (mod 256), y given as  yl = y & 0x7f7f7f7f  and  yn = ~y & 0x80808080
__device__ __forceinline__ uint32_t sub4(uint32_t x, uint32_t yl, uint32_t yn) {
  return ((x | H4) - yl) ^ ((x & H4) ^ yn);
}

// 0xFF in every byte of m that is non-zero, 0x00 elsewhere (prmt's sign mode spreads bit 7 of a byte)
__device__ __forceinline__ uint32_t nzmask4(uint32_t m) {
  const uint32_t hb = ((m & L4) + L4) | m;
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(r) : "r"(hb));
  return r;
}
// a where mask is set, b elsewhere
__device__ __forceinline__ uint32_t sel4(uint32_t mask, uint32_t a, uint32_t b) { return (a & mask) | (b & ~mask); }

// 32 bf16 values of one lane, as loaded (two elements per word, low half first)
struct LaneIn {
  uint32_t w[16];
};

// sign+mantissa bytes and exponent bytes of one lane, four elements per word
struct LaneSplit {
  uint32_t sm[8];
  uint32_t ex[8];
};

__device__ __forceinline__ void split_lane(const LaneIn& in, LaneSplit& s) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    // high bytes: sign and exponent bits 7..1; low bytes: exponent bit 0 and mantissa
    const uint32_t a = in.w[2 * k], b = in.w[2 * k + 1];
    const uint32_t hi = __byte_perm(a, b, 0x7531), lo = __byte_perm(a, b, 0x6420);
    s.sm[k] = sel4(H4, hi, lo);
    s.ex[k] = sel4(0xFEFEFEFEu, hi << 1, lo >> 7);
  }
}

__device__ __forceinline__ void join_lane(const LaneSplit& s, LaneIn& out) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t sm = s.sm[k], ex = s.ex[k];
    const uint32_t hi = sel4(H4, sm, ex >> 1), lo = sel4(L4, sm, ex << 7);
    out.w[2 * k] = __byte_perm(lo, hi, 0x5140);
    out.w[2 * k + 1] = __byte_perm(lo, hi, 0x7362);
  }
}

// thirty-two bytes at a 32-byte boundary in one access
__device__ __forceinline__ void ld32(const void* p, uint32_t* r) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p));
}
__device__ __forceinline__ void st32(void* p, const uint32_t* r) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Loads.  `aligned`: pointer is 16-byte aligned and all 32 elements are in range.
__device__ __forceinline__ void load_lane(const uint16_t* p, int64_t valid, bool aligned, LaneIn& in) {
  if (aligned && valid >= 32) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2), d = __ldg(q + 3);
    in.w[0] = a.x; in.w[1] = a.y; in.w[2] = a.z; in.w[3] = a.w;
    in.w[4] = b.x; in.w[5] = b.y; in.w[6] = b.z; in.w[7] = b.w;
    in.w[8] = c.x; in.w[9] = c.y; in.w[10] = c.z; in.w[11] = c.w;
    in.w[12] = d.x; in.w[13] = d.y; in.w[14] = d.z; in.w[15] = d.w;
  } else {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t lo = (2 * k < valid) ? (uint32_t)__ldg(p + 2 * k) : 0u;
      const uint32_t hi = (2 * k + 1 < valid) ? (uint32_t)__ldg(p + 2 * k + 1) : 0u;
      in.w[k] = lo | (hi << 16);
    }
  }
}

__device__ __forceinline__ void store_lane(uint16_t* p, int64_t valid, bool aligned, const LaneIn& o) {
  if (aligned && valid >= 32) {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(o.w[0], o.w[1], o.w[2], o.w[3]);
    q[1] = make_uint4(o.w[4], o.w[5], o.w[6], o.w[7]);
    q[2] = make_uint4(o.w[8], o.w[9], o.w[10], o.w[11]);
    q[3] = make_uint4(o.w[12], o.w[13], o.w[14], o.w[15]);
  } else {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (2 * k < valid) p[2 * k] = (uint16_t)(o.w[k] & 0xFFFFu);
      if (2 * k + 1 < valid) p[2 * k + 1] = (uint16_t)(o.w[k] >> 16);
    }
  }
}

// out[i] = the word at byte 4 i + off of e, off even and below 16 (uniform over the warp)
__device__ __forceinline__ void shift_words(const uint32_t (&e)[20], int off, uint32_t (&out)[16]) {
  const uint32_t sh = (uint32_t)(off & 3) * 8;
  switch (off >> 2) {
#define ZC_SHIFT(D)                                                                     \
  _Pragma("unroll") for (int i = 0; i < 16; ++i) out[i] = __funnelshift_r(e[i + D], e[i + D + 1 < 20 ? i + D + 1 : 19], sh);
    case 0: ZC_SHIFT(0) break;
    case 1: ZC_SHIFT(1) break;
    case 2: ZC_SHIFT(2) break;
    default: ZC_SHIFT(3) break;
#undef ZC_SHIFT
  }
}
// The same loads and stores with whole 32-byte sectors per access where the base is on such a boundary (a
// lane's 64 bytes are then two accesses instead of four that each use half a sector), and whole 16-byte
// pieces where it is on none at all: the odd start of a work inside a packed buffer.  `align` is the
// base's (align_of), equal for the whole warp, whose lanes hold consecutive groups of 32 elements; a warp
// with an incomplete lane goes element by element.
__device__ __forceinline__ void load_lane_v(const uint16_t* p, int64_t valid, int align, LaneIn& in) {
  if (align == 32 && valid >= 32) {
    ld32(p, in.w);
    ld32(p + 16, in.w + 8);
  } else if (align == 0 && __all_sync(FULL, valid >= 32)) {
    // five pieces cover the lane's bytes, and each of them holds at least one of these bytes
    const int mis = (int)(reinterpret_cast<uintptr_t>(p) & 15);
    const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<uintptr_t>(p) - mis);
    uint32_t e[20];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const uint4 v = __ldg(q + k);
      e[4 * k] = v.x; e[4 * k + 1] = v.y; e[4 * k + 2] = v.z; e[4 * k + 3] = v.w;
    }
    shift_words(e, mis, in.w);
  } else {
    load_lane(p, valid, align >= 16, in);
  }
}
__device__ __forceinline__ void store_lane_v(uint16_t* p, int64_t valid, int align, const LaneIn& o) {
  if (align == 32 && valid >= 32) {
    st32(p, o.w);
    st32(p + 16, o.w + 8);
  } else if (align == 0 && __activemask() == FULL && __all_sync(FULL, valid >= 32)) {
    // every lane stores the four pieces that start in its bytes rounded down: the first of them begins with
    // the previous lane's last bytes.  The warp's first and last bytes share their pieces with others.
    const int lane = threadIdx.x & 31;
    const int mis = (int)(reinterpret_cast<uintptr_t>(p) & 15);
    uint32_t e[20], w[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = __shfl_up_sync(FULL, o.w[12 + k], 1);
#pragma unroll
    for (int k = 0; k < 16; ++k) e[4 + k] = o.w[k];
    shift_words(e, 16 - mis, w);
    uint4* q = reinterpret_cast<uint4*>(reinterpret_cast<uintptr_t>(p) - mis);
    if (lane > 0) q[0] = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int k = 1; k < 4; ++k) q[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 7; ++i)
        if (2 * i < 16 - mis) p[i] = (uint16_t)(o.w[i >> 1] >> (16 * (i & 1)));
    } else if (lane == 31) {
#pragma unroll
      for (int i = 25; i < 32; ++i)
        if (2 * (32 - i) <= mis) p[i] = (uint16_t)(o.w[i >> 1] >> (16 * (i & 1)));
    }
  } else {
    store_lane(p, valid, align >= 16, o);
  }
}
__host__ __device__ __forceinline__ int align_of(const void* p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  return (a & 31) == 0 ? 32 : (a & 15) == 0 ? 16 : (a & 1) == 0 ? 0 : -1;
}

// codes for a window [base, base+span), span + 1 a power of two: per-byte codes (0 = escape), four per word
__device__ __forceinline__ void codes_lane(const LaneSplit& s, int base, uint32_t span, uint32_t (&code)[8]) {
  const uint32_t y = rep4((uint32_t)(base - 1));
  const uint32_t yl = y & L4, yn = ~y & H4;
  const uint32_t ns = rep4(~span);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t c = sub4(s.ex[k], yl, yn);
    code[k] = c & ~nzmask4(c & ns);
  }
}

// Codes <-> nibbles: byte j of word i holds the code of element 8 i + j in its low nibble and of element
// 8 i + 4 + j in its high one (the nibble records' layout).
__device__ __forceinline__ void pack_nibbles(const uint32_t (&code)[8], uint32_t (&n)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) n[i] = code[2 * i] + (code[2 * i + 1] << 4);
}
__device__ __forceinline__ void unpack_nibbles(const uint32_t (&n)[4], uint32_t (&code)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    code[2 * i] = n[i] & 0x0F0F0F0Fu;
    code[2 * i + 1] = (n[i] >> 4) & 0x0F0F0F0Fu;
  }
}

// 4 x 4 byte transpose: byte i of word j <-> byte j of word i
__device__ __forceinline__ void transpose_bytes(uint32_t (&t)[4]) {
  const uint32_t a = __byte_perm(t[0], t[1], 0x5140), b = __byte_perm(t[2], t[3], 0x5140);
  const uint32_t c = __byte_perm(t[0], t[1], 0x7362), d = __byte_perm(t[2], t[3], 0x7362);
  t[0] = __byte_perm(a, b, 0x5410);
  t[1] = __byte_perm(a, b, 0x7632);
  t[2] = __byte_perm(c, d, 0x5410);
  t[3] = __byte_perm(c, d, 0x7632);
}
// exchange the two bits of the word index with the two low bits of the bit position
__device__ __forceinline__ void exchange_bits(uint32_t (&t)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const uint32_t a = t[i], b = t[i + 1];
    t[i] = sel4(0x55555555u, a, b << 1);
    t[i + 1] = sel4(0x55555555u, a >> 1, b);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t a = t[i], b = t[i + 2];
    t[i] = sel4(0x33333333u, a, b << 2);
    t[i + 2] = sel4(0x33333333u, a >> 2, b);
  }
}
// Nibbles -> planes: bit p of element j's code becomes bit j of word p.  With an element's index bits
// written e4..e0, word i = e4 e3 holds byte e1 e0, nibble e2; the byte transpose makes that word e1 e0,
// byte e4 e3, and exchanging the word index with the bit-in-nibble leaves word p, bit e4 e3 e2 e1 e0.
// Both steps are their own inverses.
__device__ __forceinline__ void nibbles_to_planes(uint32_t (&t)[4]) {
  transpose_bytes(t);
  exchange_bits(t);
}
__device__ __forceinline__ void planes_to_nibbles(uint32_t (&t)[4]) {
  exchange_bits(t);
  transpose_bytes(t);
}
// planes of the codes, and the mask of elements whose code is zero
__device__ __forceinline__ uint32_t code_planes(const uint32_t (&code)[8], uint32_t (&pl)[4]) {
  pack_nibbles(code, pl);
  nibbles_to_planes(pl);
  return ~(pl[0] | pl[1] | pl[2] | pl[3]);
}

// exclusive prefix of v over the warp; total returned through `total`
__device__ __forceinline__ int warp_excl_scan(int v, int lane, int& total) {
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += t;
  }
  total = __shfl_sync(FULL, x, 31);
  return x - v;
}

// The exponents of the elements in zmask, at dst[0..popc(zmask)).  `row`: 32 bytes of shared memory of this
// lane (16-byte aligned), through which a byte is picked by its index; one trip per escape, so a warp makes
// as many trips as its fullest lane has escapes (walking the eight register words instead took eight tests
// per lane and two to three times the instructions).
__device__ __forceinline__ void scatter_escapes(uint8_t* dst, const LaneSplit& s, uint32_t zmask, uint8_t* row) {
  uint4* r = reinterpret_cast<uint4*>(row);
  r[0] = make_uint4(s.ex[0], s.ex[1], s.ex[2], s.ex[3]);
  r[1] = make_uint4(s.ex[4], s.ex[5], s.ex[6], s.ex[7]);
  uint8_t* d = dst + __popc(zmask);
  while (zmask) {
    const int i = 31 - __clz(zmask);
    zmask ^= 1u << i;
    *--d = row[i];
  }
}
// Overwrite the exponents of the elements in zmask with the bytes at esc[0..popc(zmask)), in the same way.
__device__ __forceinline__ void insert_escapes(const uint8_t* esc, uint32_t zmask, uint32_t (&ex)[8], uint8_t* row) {
  uint4* r = reinterpret_cast<uint4*>(row);
  r[0] = make_uint4(ex[0], ex[1], ex[2], ex[3]);
  r[1] = make_uint4(ex[4], ex[5], ex[6], ex[7]);
  const uint8_t* e = esc + __popc(zmask);
  while (zmask) {
    const int i = 31 - __clz(zmask);
    zmask ^= 1u << i;
    row[i] = *--e;
  }
  const uint4 a = r[0], b = r[1];
  ex[0] = a.x; ex[1] = a.y; ex[2] = a.z; ex[3] = a.w;
  ex[4] = b.x; ex[5] = b.y; ex[6] = b.z; ex[7] = b.w;
}

// The same two without shared memory beyond the escapes themselves (the fused collectives, whose CTAs have
// to fit beside a GEMM).
// write this lane's escapes (exponents of zero-coded elements) at dst[0..popc(zmask))
__device__ __forceinline__ void scatter_escapes(uint8_t* dst, const LaneSplit& s, uint32_t zmask) {
  if (zmask == 0) return;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    uint32_t m = (zmask >> (4 * k)) & 0xFu;
    while (m) {
      const int j = __ffs(m) - 1;
      *dst++ = (uint8_t)((s.ex[k] >> (j * 8)) & 0xFFu);
      m &= m - 1;
    }
  }
}

// exponent bytes of coded elements, e = base + code - 1: a per-byte sum modulo 256 (codes are below 16, so
// nothing carries out of a byte once bit 7 is added by exclusive or).  Escapes come out as base - 1.
__device__ __forceinline__ void exponents_lane(const uint32_t (&code)[8], int base, uint32_t (&ex)[8]) {
  const uint32_t y = rep4((uint32_t)(base - 1));
  const uint32_t yl = y & L4, yh = y & H4;
#pragma unroll
  for (int k = 0; k < 8; ++k) ex[k] = (code[k] + yl) ^ yh;
}
// overwrite the exponents of the elements in zmask with the bytes at esc[0..popc(zmask))
__device__ __forceinline__ void insert_escapes(const uint8_t* esc, uint32_t zmask, uint32_t (&ex)[8]) {
  if (zmask == 0) return;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    uint32_t m = (zmask >> (4 * k)) & 0xFu;
    while (m) {
      const int j = (__ffs(m) - 1) * 8;
      ex[k] = (ex[k] & ~(0xFFu << j)) | ((uint32_t)(*esc++) << j);
      m &= m - 1;
    }
  }
}

}  // namespace zc
