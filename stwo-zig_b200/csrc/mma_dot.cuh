// Sums of M31 x QM31 products on the tensor cores, exact.
//
// sum_e v_e * q_e (v_e a 32-bit word of column e, q_e a QM31 coefficient) is a contraction over e with
// the same coefficients for every row. Each word is four byte limbs, so with u8 x u8 -> s32 products
// sum_e v_e q_e[j] = sum_s 2^(8 s) S[j][s], S[j][s] = sum_e sum_{a + b = s} limb_a(v_e) limb_b(q_e[j]):
// per coordinate j seven sums S[j][0..6], each below 8256 columns x 4 x 255^2 < 2^31.
//
// mma.sync.m16n8k32 (u8): a thread's A register holds four consecutive k bytes of one row, which is one
// word of one column when k = (column, limb) - a word is an operand as it lies, with no shuffle or
// conversion. Lane (g, t) = (lane / 4, lane % 4) takes, for m tile m of 64 rows and a group of eight
// columns, rows 16 m + 2 g and + 1 of column t (registers a0, a1: row slots g and g + 8) and of column
// 4 + t (a2, a3): two 8-byte reads that fill the operand's four registers without a move. The
// B register of (column c, n) holds, over limb a = 0..3 of v, limb s - a of q_c[j]: the byte-reversed
// coordinate shifted by s - 3 bytes. Column n = 8 i + 2 j + b of the product is (j, s = 2 i + b), which
// leaves all seven sums of coordinate t in lane (g, t): no exchange between lanes afterwards.
//
// Per eight columns and 64 rows a warp issues 8 reads, 8 shifts and 16 mma (1131 T operations/s measured
// for this shape) where lazily accumulated 64-bit multiply-adds take ten instructions per word and lane:
// the kernels built on it wait for HBM instead of the integer pipes.
#pragma once
#include <cstdint>

#include "field.cuh"

namespace sb {
namespace mmadot {

__device__ __forceinline__ void mma_u8(int32_t (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t byte_reverse(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

// B registers of the four n tiles for a byte-reversed coordinate: lane parity b = g & 1 picks s = 2 i + b.
// shl.b32 gives 0 for a shift by 32 (s = 7, unused).
struct LaneShifts { uint32_t r0, r1, l2, l3; };
__device__ __forceinline__ LaneShifts lane_shifts(uint32_t b) { return {24 - 8 * b, 8 - 8 * b, 8 + 8 * b, 24 + 8 * b}; }
__device__ __forceinline__ uint32_t shl32(uint32_t v, uint32_t n) {
  uint32_t r;
  asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
  return r;
}
__device__ __forceinline__ void expand(uint32_t w, const LaneShifts& s, uint32_t (&b)[4]) {
  b[0] = w >> s.r0;
  b[1] = w >> s.r1;
  b[2] = shl32(w, s.l2);
  b[3] = shl32(w, s.l3);
}

// The words of this lane for a step: a[m] = rows 16 m + 2 g, + 1 of columns t (x, y) and 4 + t (z, w).
struct Words { uint4 a[4]; };

// Sums of 64 rows x this lane's coordinate: c[m][i][slot * 2 + b]; the tiles share a step's B registers.
struct Acc {
  int32_t c[4][4][4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < 64; ++k) c[k >> 4][(k >> 2) & 3][k & 3] = 0;
  }
  // wlo, whi: byte-reversed coordinates g / 2 of columns t and 4 + t.
  __device__ __forceinline__ void step(const Words& w, uint32_t wlo, uint32_t whi, const LaneShifts& s) {
    uint32_t b0[4], b1[4];
    expand(wlo, s, b0);
    expand(whi, s, b1);
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int i = 0; i < 4; ++i) mma_u8(c[m][i], w.a[m].x, w.a[m].y, w.a[m].z, w.a[m].w, b0[i], b1[i]);
  }
};

// sum_s 2^(8 s) S[s] mod p: 2^32, 2^40 and 2^48 are 2, 2^9 and 2^17 mod p.
__device__ __forceinline__ uint32_t combine(const int32_t (&c)[4][4], int slot) {
  auto u = [&](int i, int b) { return (uint64_t)(uint32_t)c[i][2 * slot + b]; };
  const uint64_t x = u(0, 0) + (u(0, 1) << 8) + (u(1, 0) << 16) + (u(1, 1) << 24) + (u(2, 0) << 1) + (u(2, 1) << 9) +
                     (u(3, 0) << 17);
  return mreduce64(x);
}
// This lane's coordinate of row 16 m + 2 g + s.
__device__ __forceinline__ uint32_t row_sum(const Acc& a, int m, int s) { return combine(a.c[m], s); }

}  // namespace mmadot
}  // namespace sb
