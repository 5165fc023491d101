// LogUp interaction columns: per-row fractions of a relation's uses, running
// sums across a row's columns, and the row scan of the last column.
//
// Reference behaviour:
//  - fractions and the per-row accumulation across columns: stwo_zig_relation_fused,
//    src/backends/metal/shaders/core/relation.metal:131-158 (a column with two uses is
//    (n_a d_b + n_b d_a) / (d_a d_b), relation.metal:77-90; the pair batching of
//    src/frontends/riscv/air/logup.zig:76-105);
//  - coset-order scan with the total/N shift: relation.metal:160-237, scalar law
//    src/tests/metal/backend/commitment_test.zig:73-154 (scan index s visits circle index
//    s/2 for even s and N-1-s/2 for odd s, stored at its bit reverse; value(s) =
//    sum_{s' <= s} v(s') - total (s+1)/N; claimed = total);
//  - storage-order scan without shift: cumulativeColumn, src/frontends/riscv/air/logup.zig:83-105.
//
// Kernels: k_logup_fractions (one thread per row, one QM31 inversion per row by
// the suffix-product trick), then a three-pass scan over 1024-position blocks:
// block sums, a one-CTA scan of the block sums (which also writes the claimed
// sum), and the finalising rescan that writes the last column in place.
#include <algorithm>

#include "kernels.cuh"

namespace sb {

namespace {

constexpr int LU_THREADS = 256;
constexpr int SCAN_PER_THREAD = 4;
constexpr int SCAN_BLOCK = LU_THREADS * SCAN_PER_THREAD;  // positions per scan block

// sum_j alphas[j] word_j - z. LAZY: accumulated per coordinate in 64 bits, folded every third product; else each
// product is reduced (logup_interaction says where).
template <bool LAZY>
__device__ __forceinline__ QM31 use_denominator(const LogupParams& p, const LogupUse& u, uint64_t row) {
  const QM31 nz = qneg(p.z);
  if (!LAZY) {
    QM31 acc = nz;
    for (uint32_t j = 0; j < u.n_words; ++j) {
      const uint32_t w = u.words[j] ? u.words[j][row] : u.constants[j];
      acc = qadd(acc, qmulm(p.alphas[j], w));
    }
    return acc;
  }
  uint64_t a0 = nz.c0.a, a1 = nz.c0.b, a2 = nz.c1.a, a3 = nz.c1.b;
  for (uint32_t j = 0; j < u.n_words; ++j) {
    const uint32_t w = u.words[j] ? __ldg(u.words[j] + row) : u.constants[j];
    const QM31 al = p.alphas[j];
    a0 += (uint64_t)al.c0.a * w; a1 += (uint64_t)al.c0.b * w;
    a2 += (uint64_t)al.c1.a * w; a3 += (uint64_t)al.c1.b * w;
    if (j % 3 == 2) { a0 = mfold64(a0); a1 = mfold64(a1); a2 = mfold64(a2); a3 = mfold64(a3); }
  }
  return qmake(mreduce64(a0), mreduce64(a1), mreduce64(a2), mreduce64(a3));
}

__device__ __forceinline__ uint32_t use_numerator(const LogupUse& u, uint64_t row) {
  uint32_t m = u.multiplicity ? u.multiplicity[row] : 1u;
  return u.negate ? mneg(m) : m;
}

// Numerator and denominator of interaction column c at `row`.
template <bool LAZY>
__device__ __forceinline__ void column_fraction(const LogupParams& p, uint32_t c, uint64_t row, QM31& num,
                                                QM31& den) {
  uint32_t u0 = c * p.batch;
  QM31 da = use_denominator<LAZY>(p, p.uses[u0], row);
  uint32_t ma = use_numerator(p.uses[u0], row);
  if (p.batch == 2 && u0 + 1 < p.n_uses) {
    QM31 db = use_denominator<LAZY>(p, p.uses[u0 + 1], row);
    uint32_t mb = use_numerator(p.uses[u0 + 1], row);
    num = qadd(qmulm(da, mb), qmulm(db, ma));
    den = qmul(da, db);
  } else {
    num = qbase(ma);
    den = da;
  }
}

__device__ __forceinline__ QM31 col_load(const uint32_t* out, uint64_t stride, uint32_t c, uint64_t row) {
  const uint32_t* b = out + 4ull * c * stride + row;
  return qmake(b[0], b[stride], b[2 * stride], b[3 * stride]);
}
__device__ __forceinline__ void col_store(uint32_t* out, uint64_t stride, uint32_t c, uint64_t row, QM31 v) {
  uint32_t* b = out + 4ull * c * stride + row;
  b[0] = v.c0.a;
  b[stride] = v.c0.b;
  b[2 * stride] = v.c1.a;
  b[3 * stride] = v.c1.b;
}

template <bool LAZY>
__global__ void __launch_bounds__(LU_THREADS) k_logup_fractions(const __grid_constant__ LogupParams p, uint32_t* out,
                                                                uint64_t stride, uint32_t* zero_flag) {
  uint64_t row = (uint64_t)blockIdx.x * LU_THREADS + threadIdx.x;
  if (row >= (1ull << p.log_rows)) return;
  const uint32_t n_cols = logup_n_cols(p.n_uses, p.batch);
  // Backward: out[c] = n_c * prod_{c' > c} d_c', suffix = prod of all denominators.
  QM31 suffix = qone();
  for (uint32_t c = n_cols; c-- > 0;) {
    QM31 num, den;
    column_fraction<LAZY>(p, c, row, num, den);
    col_store(out, stride, c, row, qmul(num, suffix));
    suffix = qmul(suffix, den);
  }
  if (qiszero(suffix)) {
    atomicOr(zero_flag, 1u);
    return;
  }
  // Forward: running = (prod_{c' < c} d_c') / prod_all, so out[c] * running = n_c / d_c.
  QM31 running = qinv(suffix), acc = qzero();
  for (uint32_t c = 0; c < n_cols; ++c) {
    QM31 num, den;
    column_fraction<LAZY>(p, c, row, num, den);
    acc = qadd(acc, qmul(col_load(out, stride, c, row), running));
    col_store(out, stride, c, row, acc);
    running = qmul(running, den);
  }
}

// Up to four interaction columns (LOGUP_REG_COLS): every fraction of the row stays in registers, so the words are
// read once, each denominator is formed once and each column written once (the general kernel above keeps
// n_c times the later denominators in the output and forms the denominators again on the way back). One
// inversion per row over the prefix products. Bound by the field products, about 1500 instructions a row for five
// uses in three columns: 2^20 rows 174 us with the general kernel, 123 us here.
constexpr uint32_t LOGUP_REG_COLS = 4;
template <int C>
__global__ void __launch_bounds__(LU_THREADS) k_logup_fractions_reg(const __grid_constant__ LogupParams p, uint32_t* out,
                                                                    uint64_t stride, uint32_t* zero_flag) {
  const uint64_t row = (uint64_t)blockIdx.x * LU_THREADS + threadIdx.x;
  if (row >= (1ull << p.log_rows)) return;
  QM31 num[C], den[C], pre[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    column_fraction<true>(p, c, row, num[c], den[c]);
    pre[c] = c == 0 ? den[0] : qmul(pre[c - 1], den[c]);
  }
  if (qiszero(pre[C - 1])) {
    atomicOr(zero_flag, 1u);
    return;
  }
  QM31 inv = qinv(pre[C - 1]);  // of the first c + 1 denominators' product on the way down
#pragma unroll
  for (int c = C - 1; c > 0; --c) {
    num[c] = qmul(num[c], qmul(inv, pre[c - 1]));
    inv = qmul(inv, den[c]);
  }
  num[0] = qmul(num[0], inv);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    if (c) num[c] = qadd(num[c], num[c - 1]);
    col_store(out, stride, c, row, num[c]);
  }
}

__device__ __forceinline__ uint64_t scan_row(uint64_t s, uint32_t log_rows, uint32_t order) {
  if (order == 0 || log_rows == 0) return s;
  uint64_t rows = 1ull << log_rows;
  uint64_t ci = (s & 1) == 0 ? s >> 1 : rows - 1 - (s >> 1);
  return __brevll(ci) >> (64 - log_rows);
}

__device__ __forceinline__ QM31 shfl_up_q(QM31 v, int d) {
  return qmake(__shfl_up_sync(0xffffffffu, v.c0.a, d), __shfl_up_sync(0xffffffffu, v.c0.b, d),
               __shfl_up_sync(0xffffffffu, v.c1.a, d), __shfl_up_sync(0xffffffffu, v.c1.b, d));
}

// Inclusive scan over a warp.
__device__ __forceinline__ QM31 warp_inclusive_scan(QM31 v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const QM31 o = shfl_up_q(v, d);
    if (lane >= d) v = qadd(v, o);
  }
  return v;
}

// Inclusive scan of one QM31 per thread over a CTA of THREADS threads; also returns the CTA total.
template <int THREADS>
__device__ __forceinline__ QM31 block_inclusive_scan(QM31 v, QM31& total) {
  constexpr int WARPS = THREADS / 32;
  __shared__ QM31 warp_sums[WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_inclusive_scan(v);
  if (lane == 31) warp_sums[warp] = v;
  __syncthreads();
  if (warp == 0) {
    const QM31 w = warp_inclusive_scan(lane < WARPS ? warp_sums[lane] : qzero());
    if (lane < WARPS) warp_sums[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v = qadd(v, warp_sums[warp - 1]);
  total = warp_sums[WARPS - 1];
  return v;
}

__global__ void __launch_bounds__(LU_THREADS) k_logup_block_sums(const uint32_t* col, uint64_t stride,
                                                                 uint32_t log_rows, uint32_t order, QM31* block_sums) {
  const uint64_t rows = 1ull << log_rows;
  const uint64_t s0 = (uint64_t)blockIdx.x * SCAN_BLOCK + (uint64_t)threadIdx.x * SCAN_PER_THREAD;
  QM31 sum = qzero();
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k)
    if (s0 + k < rows) sum = qadd(sum, col_load(col, stride, 0, scan_row(s0 + k, log_rows, order)));
  QM31 total;
  block_inclusive_scan<LU_THREADS>(sum, total);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// One CTA: block_sums[b] <- sum of blocks before b; *claimed <- sum of all. 1024 sums at a time, contiguous
// across the threads, the next ones fetched while these are scanned (each thread summing a run of its own
// took 55 us for 8192 sums).
constexpr int SCAN_THREADS = 1024;
__global__ void __launch_bounds__(SCAN_THREADS) k_logup_scan_blocks(QM31* block_sums, uint32_t n_blocks,
                                                                    QM31* claimed) {
  QM31 carry = qzero();
  QM31 v = threadIdx.x < n_blocks ? block_sums[threadIdx.x] : qzero();
  for (uint32_t b = threadIdx.x, base = 0; base < n_blocks; base += SCAN_THREADS, b += SCAN_THREADS) {
    const QM31 next = (uint64_t)b + SCAN_THREADS < n_blocks ? block_sums[b + SCAN_THREADS] : qzero();
    QM31 total;
    const QM31 incl = block_inclusive_scan<SCAN_THREADS>(v, total);
    if (b < n_blocks) block_sums[b] = qadd(carry, qsub(incl, v));
    carry = qadd(carry, total);
    v = next;
    __syncthreads();  // the scan's shared words are written again
  }
  if (threadIdx.x == 0) *claimed = carry;
}

__global__ void __launch_bounds__(LU_THREADS) k_logup_finalize(uint32_t* col, uint64_t stride, uint32_t log_rows,
                                                               uint32_t order, const QM31* block_prefix,
                                                               const QM31* claimed) {
  const uint64_t rows = 1ull << log_rows;
  const uint64_t s0 = (uint64_t)blockIdx.x * SCAN_BLOCK + (uint64_t)threadIdx.x * SCAN_PER_THREAD;
  QM31 v[SCAN_PER_THREAD];
  QM31 sum = qzero();
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    v[k] = s0 + k < rows ? col_load(col, stride, 0, scan_row(s0 + k, log_rows, order)) : qzero();
    sum = qadd(sum, v[k]);
  }
  QM31 total_block;
  QM31 incl = block_inclusive_scan<LU_THREADS>(sum, total_block);
  QM31 run = qadd(block_prefix[blockIdx.x], qsub(incl, sum));
  const QM31 total = *claimed;
  // 1/N = 2^(31 - log_rows) in M31 (2^31 = 1).
  const uint32_t inv_rows = log_rows == 0 ? 1u : (1u << (31 - log_rows)) % P;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    uint64_t s = s0 + k;
    if (s >= rows) break;
    run = qadd(run, v[k]);
    QM31 out = run;
    if (order == 1) out = qsub(out, qmulm(total, mmul(inv_rows, (uint32_t)((s + 1) % P))));
    col_store(col, stride, 0, scan_row(s, log_rows, order), out);
  }
}

// ---- The coset-order scan by whole memory sectors (2^10 rows or more, 16-byte aligned columns) ------------------
// Coset positions 2j and 2j + 1 (j < N / 2) are rows r = 2 bitrev(j) and N - 1 - r, so consecutive positions lie
// a large power of two apart and a row-by-row gather fetches a 32-byte sector for every word (2^20 rows: 20 us for
// the block sums, 58 us for the final pass). With j = (a, m, l), a its top two bits and l its lowest six, the
// sector of eight rows at (bitrev l, bitrev m, 000) holds the even positions of (a, m, l) for the four a and, by
// the complement, the odd ones of (a, ~m, ~l): a CTA that takes m and ~m with every a and l reads 128 whole
// sectors of each coordinate and owns eight segments of 128 consecutive positions, one per warp. The segments'
// sums are scanned as the blocks' are. Now 9 and 15 us.
constexpr uint32_t SEG = 128;           // positions of a segment
constexpr uint32_t COSET_MIN_LOG = 10;  // at least one bit of m

struct CosetTile {
  uint32_t log, mid_bits, m;  // log rows, bits of m, this CTA's m (its complement is the other one)
  __device__ __forceinline__ explicit CosetTile(uint32_t log_rows) : log(log_rows), mid_bits(log_rows - 9), m(blockIdx.x) {}
  // First row of this thread's four (half a sector).
  __device__ __forceinline__ uint64_t row() const {
    const uint32_t q = threadIdx.x >> 1, l = q & 63;
    return ((uint64_t)(__brev(l) >> 26) << (log - 6)) | ((uint64_t)(__brev(mid(q >> 6)) >> (32 - mid_bits)) << 3) |
           (4 * (threadIdx.x & 1));
  }
  __device__ __forceinline__ uint32_t mid(uint32_t sel) const { return sel ? (1u << mid_bits) - 1 - m : m; }
  // Place (segment * SEG + position in it) of the thread's i-th word.
  __device__ __forceinline__ static uint32_t place(int i) {
    const uint32_t q = threadIdx.x >> 1, l = q & 63, sel = q >> 6, w = 4 * (threadIdx.x & 1) + i;
    const uint32_t k = (w & 1 ? 7 - w : w) >> 1, a = ((k & 1) << 1) | (k >> 1);
    return w & 1 ? ((1 - sel) * 4 + a) * SEG + 2 * (63 - l) + 1 : (sel * 4 + a) * SEG + 2 * l;
  }
  // Number of segment `seg` (0..7) of this CTA among all of the scan's.
  __device__ __forceinline__ uint32_t segment(uint32_t seg) const { return ((seg & 3) << mid_bits) | mid(seg >> 2); }
};

// The CTA's rows, by coordinate and place.
__device__ __forceinline__ void coset_load(const CosetTile& t, const uint32_t* col, uint64_t stride, uint32_t (&v)[4][8 * SEG]) {
  const uint64_t row = t.row();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint4 x = *reinterpret_cast<const uint4*>(col + c * stride + row);
    v[c][t.place(0)] = x.x; v[c][t.place(1)] = x.y; v[c][t.place(2)] = x.z; v[c][t.place(3)] = x.w;
  }
  __syncthreads();
}
// Lane's four consecutive positions of its warp's segment.
__device__ __forceinline__ void coset_lane(const uint32_t (&v)[4][8 * SEG], QM31 (&x)[4]) {
  const uint32_t at = threadIdx.x * 4;
  uint4 c[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) c[k] = *reinterpret_cast<const uint4*>(&v[k][at]);
  x[0] = qmake(c[0].x, c[1].x, c[2].x, c[3].x);
  x[1] = qmake(c[0].y, c[1].y, c[2].y, c[3].y);
  x[2] = qmake(c[0].z, c[1].z, c[2].z, c[3].z);
  x[3] = qmake(c[0].w, c[1].w, c[2].w, c[3].w);
}

__global__ void __launch_bounds__(LU_THREADS) k_logup_coset_sums(const uint32_t* col, uint64_t stride, uint32_t log_rows,
                                                                 QM31* seg_sums) {
  __shared__ __align__(16) uint32_t v[4][8 * SEG];
  const CosetTile t(log_rows);
  coset_load(t, col, stride, v);
  QM31 x[4];
  coset_lane(v, x);
  const QM31 incl = warp_inclusive_scan(qadd(qadd(x[0], x[1]), qadd(x[2], x[3])));
  if ((threadIdx.x & 31) == 31) seg_sums[t.segment(threadIdx.x >> 5)] = incl;
}

__global__ void __launch_bounds__(LU_THREADS) k_logup_coset_finalize(uint32_t* col, uint64_t stride, uint32_t log_rows,
                                                                     const QM31* seg_prefix, const QM31* claimed) {
  __shared__ __align__(16) uint32_t v[4][8 * SEG];
  const CosetTile t(log_rows);
  coset_load(t, col, stride, v);
  QM31 x[4];
  coset_lane(v, x);
  const QM31 sum = qadd(qadd(x[0], x[1]), qadd(x[2], x[3]));
  const uint32_t seg = t.segment(threadIdx.x >> 5);
  QM31 run = qadd(seg_prefix[seg], qsub(warp_inclusive_scan(sum), sum));
  const QM31 step = qmulm(*claimed, 1u << (31 - log_rows));  // total / N: 1 / N = 2^(31 - log_rows) in M31
  const uint64_t s0 = (uint64_t)seg * SEG + 4 * (threadIdx.x & 31);
  const uint32_t at = threadIdx.x * 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    run = qadd(run, x[k]);
    const QM31 o = qsub(run, qmulm(step, (uint32_t)((s0 + k + 1) % P)));
    v[0][at + k] = o.c0.a; v[1][at + k] = o.c0.b; v[2][at + k] = o.c1.a; v[3][at + k] = o.c1.b;
  }
  __syncthreads();
  const uint64_t row = t.row();
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(col + c * stride + row) =
        make_uint4(v[c][t.place(0)], v[c][t.place(1)], v[c][t.place(2)], v[c][t.place(3)]);
}

uint32_t scan_blocks(uint32_t log_rows) {
  uint64_t rows = 1ull << log_rows;
  return (uint32_t)((rows + SCAN_BLOCK - 1) / SCAN_BLOCK);
}

// XOR-lookup trace: seeded uniform u8 pairs, their XOR, the 2^16-row XOR table
// in the layout of the reference's bitwise table (row a * 256 + b holds (a, b, a ^ b),
// src/frontends/riscv/air/preprocessed/bitwise.zig:17-35) and the multiplicity of
// every table row in the trace.
__device__ __forceinline__ uint64_t xor_splitmix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void k_xor_trace(uint32_t log_n, uint64_t seed, uint32_t* main_cols, uint32_t* mult) {
  const uint64_t rows = 1ull << log_n;
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t x = xor_splitmix(seed ^ (0xD6E8FEB86659FD93ull * (r + 1)));
    uint32_t a = (uint32_t)x & 255u, b = (uint32_t)(x >> 8) & 255u;
    main_cols[r] = a;
    main_cols[rows + r] = b;
    main_cols[2 * rows + r] = a ^ b;
    atomicAdd(mult + (a << 8 | b), 1u);
  }
}

__global__ void k_xor_table(uint32_t* table) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 65536) return;
  const uint32_t a = i >> 8, b = i & 255u;
  table[i] = a;
  table[65536 + i] = b;
  table[2 * 65536 + i] = a ^ b;
}

}  // namespace

size_t logup_scratch_count(uint32_t log_rows) {
  return log_rows >= COSET_MIN_LOG ? (1ull << log_rows) / SEG : scan_blocks(log_rows);
}

cudaError_t logup_interaction(const LogupParams& p, uint32_t* out, uint64_t out_stride, QM31* claimed,
                              QM31* scratch, uint32_t* zero_flag, cudaStream_t stream) {
  if (p.n_uses == 0 || p.n_uses > LOGUP_MAX_USES || (p.batch != 1 && p.batch != 2) || p.log_rows > 28 ||
      p.order > 1)
    return cudaErrorInvalidValue;
  const uint64_t rows = 1ull << p.log_rows;
  const uint32_t n_cols = logup_n_cols(p.n_uses, p.batch);
  // Above the register kernels' four columns the denominators are formed twice, and reducing each product keeps the
  // chain of a use shorter: sixteen uses of two words at 2^14 rows 25.1 us, lazily 26.6, and 385 against 394 at
  // 2^20. Uses of many words over rows enough to hide the chain gain from fewer instructions instead: six of eight
  // words at 2^20 rows 279 us, else 300 (at 2^16 29.1 against 27.7).
  uint32_t max_words = 0;
  for (uint32_t u = 0; u < p.n_uses; ++u) max_words = std::max(max_words, p.uses[u].n_words);
  const bool lazy = p.log_rows >= 18 && max_words > 4;
  auto fractions = n_cols == 1 ? k_logup_fractions_reg<1> : n_cols == 2 ? k_logup_fractions_reg<2>
                 : n_cols == 3 ? k_logup_fractions_reg<3> : n_cols == LOGUP_REG_COLS ? k_logup_fractions_reg<LOGUP_REG_COLS>
                 : lazy ? k_logup_fractions<true> : k_logup_fractions<false>;
  fractions<<<(unsigned)((rows + LU_THREADS - 1) / LU_THREADS), LU_THREADS, 0, stream>>>(p, out, out_stride, zero_flag);
  note_launch();
  uint32_t* last = out + 4ull * (n_cols - 1) * out_stride;
  const bool sectors = p.order == 1 && p.log_rows >= COSET_MIN_LOG && (reinterpret_cast<uintptr_t>(last) & 15) == 0 &&
                       out_stride % 4 == 0;
  const uint32_t nb = sectors ? (uint32_t)(rows / SEG) : scan_blocks(p.log_rows);
  if (sectors) k_logup_coset_sums<<<(unsigned)(rows / (8 * SEG)), LU_THREADS, 0, stream>>>(last, out_stride, p.log_rows, scratch);
  else k_logup_block_sums<<<nb, LU_THREADS, 0, stream>>>(last, out_stride, p.log_rows, p.order, scratch);
  note_launch();
  k_logup_scan_blocks<<<1, SCAN_THREADS, 0, stream>>>(scratch, nb, claimed);
  note_launch();
  if (sectors)
    k_logup_coset_finalize<<<(unsigned)(rows / (8 * SEG)), LU_THREADS, 0, stream>>>(last, out_stride, p.log_rows, scratch, claimed);
  else k_logup_finalize<<<nb, LU_THREADS, 0, stream>>>(last, out_stride, p.log_rows, p.order, scratch, claimed);
  note_launch();
  return cudaGetLastError();
}

cudaError_t xor_lookup_trace(uint32_t log_n, uint64_t seed, uint32_t* main_cols, uint32_t* table, uint32_t* mult,
                             cudaStream_t stream) {
  if (log_n > 28) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(mult, 0, 65536 * 4, stream);
  if (e != cudaSuccess) return e;
  const uint64_t rows = 1ull << log_n;
  const uint32_t grid = (uint32_t)std::min<uint64_t>((rows + 255) / 256, 148 * 16);
  k_xor_trace<<<grid, 256, 0, stream>>>(log_n, seed, main_cols, mult);
  note_launch();
  k_xor_table<<<256, 256, 0, stream>>>(table);
  note_launch();
  return cudaGetLastError();
}

}  // namespace sb
