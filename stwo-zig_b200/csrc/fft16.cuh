// Register radix-16 circle-FFT building blocks (used by fft.cu for domains of
// 2^16 .. 2^22 words).
//
// A thread holds 16 elements whose indices differ only in a 4-bit window of
// the transform index, applies up to 4 butterfly layers of that window in
// registers, and exchanges elements with other threads through shared memory
// between windows. Twiddles of one window come from one to two vector loads
// per layer (the elements of a window share consecutive twiddle blocks), read
// from the doubled balanced tower (TwiddleView::tower2): t2 = 2t for the
// representative t of the twiddle in [-(p-1)/2, (p-1)/2].
//
// Products and ranges. A signed product of |a| <= p and t2 reduces to [-p, p-1]
// with one shift-and-add and no conditional subtraction (smul2), and the
// butterflies keep their values in whatever range the next step accepts, so a
// butterfly takes six instructions where canonical values in and out take
// seven, of which five instead of six hold the ALU pipe:
//   S: signed in [-p, p-1]   (canonical: min of v, v + p as unsigned words)
//   U: unsigned in [0, 2p-1] (canonical: min of v, v - p)
// In registers, 10.7 cycles per butterfly, warp and scheduler before, 8.6
// (inverse) and 9.5 (forward, both outputs S) now. Interpolation and blow-up-2
// extension of 100 columns of 2^20: 260 + 497 + 500 us before (low inverse,
// high, low forward pass), 234 + 463 + 477 us now.
//
// Shared-memory positions are swizzled by swz(i) = i ^ (16*parity(i>>5) ^ ((i>>5)&15)).
// swz is linear over GF(2), so the position of element k of a thread is
// swz(base) ^ swz(k << W) with the second term a per-k constant, and every
// window mapping used here puts the 32 threads of a warp on 32 distinct banks.
#pragma once
#include "circle.cuh"
#include "field.cuh"

namespace sb {
namespace fft16 {

__host__ __device__ __forceinline__ uint32_t swz(uint32_t i) {
  uint32_t v = i >> 5;
#if defined(__CUDA_ARCH__)
  uint32_t par = __popc(v) & 1;
#else
  uint32_t par = __builtin_popcount(v) & 1;
#endif
  return i ^ ((par << 4) ^ (v & 15));
}

// a * t mod p in [-p, p-1] for an S value (or a difference of two canonical ones) a and t2 = 2t, |t| <= (p-1)/2.
// With 2at + 2^31 = H 2^32 + L (L even), at = H 2^31 + L / 2 - 2^30 = H + L / 2 - 2^30 (mod p); |2at| <= p (p-1)
// gives 1 - 2^30 <= H <= 2^30 - 1, so the sum lies in [1 - 2^31, 2^31 - 2]. The bias -2^62 takes 2^30 off H.
__device__ __forceinline__ uint32_t smul2(uint32_t a, uint32_t t2) {
  const int64_t x = (int64_t)(int32_t)a * (int32_t)t2 + ((1ll << 31) - (1ll << 62));
  return (uint32_t)((uint64_t)x >> 32) + ((uint32_t)x >> 1);
}
__device__ __forceinline__ uint32_t canon_s(uint32_t v) { return umin32(v, v + P); }
__device__ __forceinline__ uint32_t canon_u(uint32_t v) { return umin32(v, v - P); }
// Negation of a doubled balanced twiddle.
__device__ __forceinline__ uint32_t mneg2(uint32_t t2) { return 0u - t2; }

enum Range { RANGE_CANON, RANGE_S, RANGE_U };
template <Range R>
__device__ __forceinline__ uint32_t to_canon(uint32_t v) {
  return R == RANGE_S ? canon_s(v) : R == RANGE_U ? canon_u(v) : v;
}

// Forward butterfly: v0 in range IN, v1 canonical or S. OUT: both results canonical, both S, or v0 S and v1 U (one
// instruction less where the next layer multiplies neither).
template <Range IN, Range OUT>
__device__ __forceinline__ void butterfly2(uint32_t& v0, uint32_t& v1, uint32_t t2) {
  const uint32_t m = smul2(v1, t2), u = to_canon<IN>(v0);
  if (OUT == RANGE_CANON) {
    const uint32_t c = canon_s(m);
    v1 = msub(u, c);
    v0 = madd(u, c);
  } else if (OUT == RANGE_S) {
    const uint32_t c = canon_s(m);
    v1 = u - c;
    v0 = u + c - P;
  } else {
    const uint32_t n = m > m - P ? m : m - P;  // the representative in [-p, -1]
    v1 = u - n;
    v0 = u + n;
  }
}
// Inverse butterfly, canonical in and out.
__device__ __forceinline__ void ibutterfly2(uint32_t& v0, uint32_t& v1, uint32_t it2) {
  const uint32_t a = v0;
  v0 = madd(a, v1);
  v1 = canon_s(smul2(a - v1, it2));
}

// `n` consecutive doubled twiddles of line layer s (s >= 1) starting at block h0
// (h0 is a multiple of n, the layer offset a multiple of 16 bytes).
template <int N>
__device__ __forceinline__ void load_line(const TwiddleView& tv, uint32_t s, uint64_t h0, uint32_t (&tw)[8]) {
  const uint32_t* p = tv.tower2 + ((1u << tv.root_log) - (1u << (tv.line_log - s + 1))) + h0;
  if (N == 8) {
    uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    tw[0] = a.x; tw[1] = a.y; tw[2] = a.z; tw[3] = a.w; tw[4] = b.x; tw[5] = b.y; tw[6] = b.z; tw[7] = b.w;
  } else if (N == 4) {
    uint4 a = __ldg(reinterpret_cast<const uint4*>(p));
    tw[0] = a.x; tw[1] = a.y; tw[2] = a.z; tw[3] = a.w;
  } else if (N == 2) {
    uint2 a = __ldg(reinterpret_cast<const uint2*>(p));
    tw[0] = a.x; tw[1] = a.y;
  } else {
    tw[0] = __ldg(p);
  }
}

// Doubled circle-layer twiddles of 8 consecutive pairs h0 .. h0+7 (h0 a multiple of 8):
// pattern [y, -y, -x, x] over the (x, y) pairs of line layer 0.
__device__ __forceinline__ void load_circle8(const TwiddleView& tv, uint64_t h0, uint32_t (&tw)[8]) {
  const uint32_t* l0 = tv.tower2 + ((1u << tv.root_log) - (1u << tv.line_log));
  uint4 q = __ldg(reinterpret_cast<const uint4*>(l0 + (h0 >> 1)));
  tw[0] = q.y; tw[1] = mneg2(q.y); tw[2] = mneg2(q.x); tw[3] = q.x;
  tw[4] = q.w; tw[5] = mneg2(q.w); tw[6] = mneg2(q.z); tw[7] = q.z;
}

// Applies window layers j in [JLO, JHI) to x (element k at transform index
// base + (k << w0) in the window's index space). Layer j is global layer
// s = sbase + w0 + j; its pair (k, k + 2^j) uses twiddle block
// (hb >> (w0 + j + 1)) + (k >> (j + 1)), hb being the index of element 0 in the
// space where twiddle blocks are counted.
//
// Forward ranges: the window's inputs are in range IN, its outputs in range OUT (canonical or S). Between its
// layers, both results of a pair are the same operand of the next layer (bit J - 1 of k): where they are its v0,
// the second one stays U, where they are its v1 (a factor), both are S.
template <bool INV, int J, int JLO, int JHI, Range IN, Range OUT>
__device__ __forceinline__ void layer16(uint32_t (&x)[16], const TwiddleView& tv, uint32_t sbase, uint32_t w0,
                                        uint64_t hb) {
  const uint32_t s = sbase + w0 + J;
  uint32_t tw[8];
  const uint64_t h0 = hb >> (w0 + J + 1);
  if (s == 0) {
    load_circle8(tv, h0, tw);
  } else {
    load_line<(8 >> J)>(tv, s, h0, tw);
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (k & (1 << J)) continue;
    const uint32_t t = tw[k >> (J + 1)];
    uint32_t &v0 = x[k], &v1 = x[k | (1 << J)];
    if (INV) {
      ibutterfly2(v0, v1, t);
      continue;
    }
    constexpr bool first = J == JHI - 1, last = J == JLO;
    const bool second = (k >> (J + 1)) & 1;               // v0 was the second result of the layer before
    const bool factor = J > 0 && ((k >> (J - 1)) & 1);    // the next layer multiplies both results
    if (last) {
      if (first) butterfly2<IN, OUT>(v0, v1, t);
      else if (second) butterfly2<RANGE_U, OUT>(v0, v1, t);
      else butterfly2<RANGE_S, OUT>(v0, v1, t);
    } else if (factor) {
      if (first) butterfly2<IN, RANGE_S>(v0, v1, t);
      else if (second) butterfly2<RANGE_U, RANGE_S>(v0, v1, t);
      else butterfly2<RANGE_S, RANGE_S>(v0, v1, t);
    } else {
      if (first) butterfly2<IN, RANGE_U>(v0, v1, t);
      else if (second) butterfly2<RANGE_U, RANGE_U>(v0, v1, t);
      else butterfly2<RANGE_S, RANGE_U>(v0, v1, t);
    }
  }
}

template <bool INV, int J, int JLO, int JHI, Range IN, Range OUT>
__device__ __forceinline__ void radix16_from(uint32_t (&x)[16], const TwiddleView& tv, uint32_t sbase, uint32_t w0,
                                             uint64_t hb) {
  if constexpr (J >= JLO && J < JHI) {
    layer16<INV, J, JLO, JHI, IN, OUT>(x, tv, sbase, w0, hb);
    radix16_from<INV, INV ? J + 1 : J - 1, JLO, JHI, IN, OUT>(x, tv, sbase, w0, hb);
  }
}

// Inverse windows take and give canonical values.
template <bool INV, int JLO, int JHI, Range IN = INV ? RANGE_CANON : RANGE_S, Range OUT = INV ? RANGE_CANON : RANGE_S>
__device__ __forceinline__ void radix16(uint32_t (&x)[16], const TwiddleView& tv, uint32_t sbase, uint32_t w0,
                                        uint64_t hb) {
  radix16_from<INV, INV ? JLO : JHI - 1, JLO, JHI, IN, OUT>(x, tv, sbase, w0, hb);
}

template <bool INV>
__device__ __forceinline__ void radix16_dyn(uint32_t (&x)[16], const TwiddleView& tv, uint32_t sbase, uint32_t w0,
                                            uint64_t hb, uint32_t nl) {
  switch (nl) {
    case 4: radix16<INV, 0, 4>(x, tv, sbase, w0, hb); break;
    case 3: radix16<INV, 0, 3>(x, tv, sbase, w0, hb); break;
    case 2: radix16<INV, 0, 2>(x, tv, sbase, w0, hb); break;
    default: radix16<INV, 0, 1>(x, tv, sbase, w0, hb); break;
  }
}

// Inserts 4 zero bits at position w0 of q.
__device__ __forceinline__ uint32_t spread(uint32_t q, uint32_t w0) {
  return ((q >> w0) << (w0 + 4)) | (q & ((1u << w0) - 1));
}

}  // namespace fft16
}  // namespace sb
