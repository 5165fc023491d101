// Per-stage kernels of the wide-Fibonacci proof: trace generation, constraint
// (composition) evaluation, OODS point evaluation, DEEP quotients, FRI folds and
// decommitment gathers.
//
// Sums of QM31 x M31 products are accumulated lazily per coordinate in 64-bit
// registers (each product < 2^62, folded every third term) and reduced once,
// which gives the same canonical result as the reference's term-by-term adds.
#include <atomic>

#include "blake2s.cuh"
#include "kernels.cuh"
#include "mma_dot.cuh"
#include "tuner.hpp"

namespace sb {

namespace {

// ---------------------------------------------------------------------------
// Trace generation (src/examples/wide_fibonacci/trace.zig:34-162). Storage
// position s holds logical row circleDomainIndexToCosetIndex(bitReverse(s)).
// kind 0: (1, row) seeds of the reference; kind 1: seeded uniform col0/col1 in
// [0, p-1): SplitMix64 keyed by seed ^ (0xD1B54A32D192ED03 * (2 row + col + 1)),
// top 31 bits, values >= p-1 rejected.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t splitmix64(uint64_t& state) {
  state += 0x9E3779B97F4A7C15ull;
  uint64_t z = state;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ uint32_t seeded_value(uint64_t seed, uint32_t column, uint64_t row) {
  uint64_t state = seed ^ (0xD1B54A32D192ED03ull * (2 * row + column + 1));
  for (int guard = 0; guard < 64; ++guard) {
    uint32_t v = (uint32_t)(splitmix64(state) >> 33);
    if (v < P - 1) return v;
  }
  return 0;  // probability 2^-1984: unreachable in practice
}

// Wide-Fibonacci trace in bit-reversed circle order: col0/col1 are the reference's (1, row) for
// kind 0, seeded uniform for kind 1, or already in `out` for kind 2; col_k = col_{k-2}^2 + col_{k-1}^2.
__global__ void k_wide_fib_trace(uint32_t log_n, uint32_t W, int kind, uint64_t seed, uint32_t* out, uint64_t stride) {
  const uint32_t n = 1u << log_n;
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    uint32_t ci = bitrev(s, log_n);
    uint32_t row = ci < n / 2 ? ci * 2 : (n - 1 - ci) * 2 + 1;
    uint32_t a, b;
    if (kind == 2) {  // the first two columns are given: derive the rest
      a = out[s];
      b = out[stride + s];
    } else {
      if (kind == 0) { a = 1; b = row % P; }
      else { a = seeded_value(seed, 0, row); b = seeded_value(seed, 1, row); }
      out[s] = a;
      out[stride + s] = b;
    }
    for (uint32_t k = 2; k < W; ++k) {
      uint32_t c = madd(mmul(a, a), mmul(b, b));
      out[k * stride + s] = c;
      a = b; b = c;
    }
  }
}

// Quadratic-recurrence trace of a seven-word recipe (the fillQuadraticRecurrenceTrace column
// source, src/examples/wide_fibonacci/trace.zig:13-16): for the logical row k of each storage
// position, col0 = r0 + r1 k, col1 = r2 + r3 k, col_j = r4 col_{j-2}^2 + r5 col_{j-1}^2 + r6 (M31).
struct QuadRecipe { uint32_t r[7]; };
__global__ void k_quadratic_trace(uint32_t log_n, uint32_t W, QuadRecipe q, uint32_t* out, uint64_t stride) {
  const uint32_t n = 1u << log_n;
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const uint32_t ci = bitrev(s, log_n);
    const uint32_t row = ci < n / 2 ? ci * 2 : (n - 1 - ci) * 2 + 1;
    uint32_t a = madd(q.r[0], mmul(q.r[1], row)), b = madd(q.r[2], mmul(q.r[3], row));
    out[s] = a;
    out[stride + s] = b;
    for (uint32_t k = 2; k < W; ++k) {
      const uint32_t c = madd(madd(mmul(q.r[4], mmul(a, a)), mmul(q.r[5], mmul(b, b))), q.r[6]);
      out[k * stride + s] = c;
      a = b;
      b = c;
    }
  }
}

// ---------------------------------------------------------------------------
// Composition (src/examples/wide_fibonacci/component.zig:138-236): per row of
// CanonicCoset(n+1), sum_k coeff_k * (c_k - a_k^2 - b_k^2), times the inverse
// coset vanishing value den_inv[row >> n]. coeff_k = random_coeff^(W-3-k).
// ---------------------------------------------------------------------------
// R consecutive rows per thread, U columns loaded before they are used (a multiple of three: the sums are folded
// after every third product), each column squared once (its square is b^2 of one constraint and a^2 of the next).
// R = 2 needs columns and output aligned to two words (eval, stride, out, out_stride).
// Bound by the field products where rows are many, by the latency of the loads where they are few: 1000 columns on
// 16 rows took 116 us a column at a time and 75 us six at a time, 39 us with 24 columns in flight.

template <int R>
__device__ __forceinline__ void load_rows(const uint32_t* p, uint32_t (&v)[R]) {
  if (R == 2) {
    const uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
    v[0] = x.x; v[R - 1] = x.y;
  } else {
    v[0] = __ldg(p);
  }
}

template <int R, uint32_t U>
__global__ void __launch_bounds__(256, U > 6 ? 2 : 4) k_composition(uint32_t log_n, uint32_t W, const uint32_t* __restrict__ eval,
                                                        uint64_t stride, const QM31* __restrict__ coeffs,
                                                        uint32_t den0, uint32_t den1, uint32_t* out, uint64_t out_stride) {
  extern __shared__ uint4 sco[];  // W - 2 coefficients
  const uint32_t n_cons = W - 2;
  for (uint32_t i = threadIdx.x; i < n_cons; i += blockDim.x) {
    const QM31 c = coeffs[i];
    sco[i] = make_uint4(c.c0.a, c.c0.b, c.c1.a, c.c1.b);
  }
  __syncthreads();
  const uint32_t groups = (2u << log_n) / R;
  for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi < groups; gi += gridDim.x * blockDim.x) {
    const uint32_t row0 = gi * R;
    const uint32_t* p = eval + row0;
    uint32_t a[R], b[R];  // squares of the two columns before
    load_rows<R>(p, a);
    load_rows<R>(p + stride, b);
    p += 2 * stride;
    uint64_t acc[R][4];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      a[j] = mmul(a[j], a[j]);
      b[j] = mmul(b[j], b[j]);
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j][c] = 0;
    }
    // `count` columns from constraint k on, all of them loaded first.
    auto batch = [&](uint32_t k, uint32_t count) {
      uint32_t v[U][R];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u)
        if (u < count) load_rows<R>(p + (uint64_t)(k + u) * stride, v[u]);
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
        if (u >= count) break;
        const uint4 q = sco[k + u];
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const uint32_t w = v[u][j], cons = msub(w, madd(a[j], b[j]));
          a[j] = b[j];
          b[j] = mmul(w, w);
          acc[j][0] += (uint64_t)q.x * cons; acc[j][1] += (uint64_t)q.y * cons;
          acc[j][2] += (uint64_t)q.z * cons; acc[j][3] += (uint64_t)q.w * cons;
          if (u % 3 == 2) {
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[j][c] = mfold64(acc[j][c]);
          }
        }
      }
    };
    uint32_t k = 0;
    for (; k + U <= n_cons; k += U) batch(k, U);
    if (k < n_cons) batch(k, n_cons - k);
    const uint32_t d = (row0 >> log_n) ? den1 : den0;  // the R rows share row >> log_n
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t* o = out + (uint64_t)c * out_stride + row0;
      if (R == 2) *reinterpret_cast<uint2*>(o) = make_uint2(mmul(mreduce64(acc[0][c]), d), mmul(mreduce64(acc[R - 1][c]), d));
      else *o = mmul(mreduce64(acc[0][c]), d);
    }
  }
}

// The same sums on the tensor cores (mma_dot.cuh). A constraint is linear in the columns and their
// squares, so sum_k coeff_k (c_{k+2} - c_k^2 - c_{k+1}^2) = sum_c (alpha_c v_c + beta_c v_c^2) with
// alpha_c = coeff_{c-2} and beta_c = -(coeff_c + coeff_{c-1}) (a coefficient outside 0 .. W-3 is zero):
// two products per column with coefficients that are the same for every row. The square enters as any
// 32-bit word congruent to it, so it is folded once and not made canonical.
//
// Bound by HBM and the integer mma rate: 2^21 rows x 100 columns 207 us, 4.2 TB/s (the kernel with
// lazily accumulated 64-bit multiply-adds, two rows per thread, 243 us).
constexpr int MMA_THREADS = 128;

// The words of a step (64 rows of eight columns), STAGES steps ahead: each warp copies them
// asynchronously into a ring of its own in shared memory, so that it keeps 2 KB a stage in flight across steps
// and row blocks without block barriers and without registers for them. The copies' lanes follow memory
// (sixteen lanes a column, 256 bytes; two columns per instruction) and the operand lanes read back
// theirs; columns lie 288 bytes apart, which puts the sixteen lanes of a read phase on distinct banks.
// A read-only probe of this walk (108 columns of 2^21 rows) runs at 6.9 TB/s; with each lane copying its
// own operand words (neighbour lanes on four different columns) it stays at 3.9 TB/s at any depth, and
// with the same depth in registers the quotients took 325 us.
// Stages of the composition and of the quotients (four CTAs per SM each).
constexpr int COMP_STAGES = 4, QUOT_STAGES = 5;
constexpr uint32_t MMA_ROWS = 64;           // rows of a warp's block
constexpr uint32_t MMA_COL = 4 * MMA_ROWS + 32;   // bytes between a stage's columns
constexpr uint32_t MMA_STAGE = 8 * MMA_COL;       // bytes of a warp's stage
constexpr uint32_t mma_ring_bytes(int stages) { return (MMA_THREADS / 32) * stages * MMA_STAGE; }
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <int STAGES>
class WordRing {
 public:
  __device__ __forceinline__ explicit WordRing(const void* ring) : in_(0), out_(0) {
    const uint32_t lane = threadIdx.x & 31;
    const char* warp = static_cast<const char*>(ring) + (threadIdx.x >> 5) * (STAGES * MMA_STAGE);
    put_ = smem_u32(warp) + (lane >> 4) * MMA_COL + (lane & 15) * 16;
    get_ = warp + (lane & 3) * MMA_COL + (lane >> 2) * 8;
  }
  // Column of a step (before the pair's number) and row of the block that this lane copies.
  __device__ __forceinline__ static uint32_t column() { return (threadIdx.x & 31) >> 4; }
  __device__ __forceinline__ static uint32_t row() { return 4 * (threadIdx.x & 15); }
  // Starts the copy of this lane's four rows of column 2 u + column() of the step (16-byte aligned when ALIGNED).
  template <bool ALIGNED>
  __device__ __forceinline__ void fetch(int u, const uint32_t* src) {
    const uint32_t d = put_ + in_ + u * 2 * MMA_COL;
    if (ALIGNED) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * k), "l"(src + k) : "memory");
    }
  }
  // Ends a step's copies (also of none): one per step, in order.
  __device__ __forceinline__ void commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    in_ = in_ + MMA_STAGE == STAGES * MMA_STAGE ? 0 : in_ + MMA_STAGE;
  }
  // This lane's words of the oldest step not yet taken; its slots are then free for the next fetch.
  __device__ __forceinline__ void take(mmadot::Words& w) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
    __syncwarp();  // every lane's copies of the step have landed
    const char* s = get_ + out_;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint2 lo = *reinterpret_cast<const uint2*>(s + 64 * m), hi = *reinterpret_cast<const uint2*>(s + 4 * MMA_COL + 64 * m);
      w.a[m] = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
    out_ = out_ + MMA_STAGE == STAGES * MMA_STAGE ? 0 : out_ + MMA_STAGE;
    __syncwarp();  // every lane has read its words
  }

 private:
  uint32_t put_, in_, out_;
  const char* get_;
};

template <bool ALIGNED>
__device__ __forceinline__ void store_rows2(uint32_t* p, uint2 v) {
  if (ALIGNED) { *reinterpret_cast<uint2*>(p) = v; return; }
  p[0] = v.x; p[1] = v.y;
}

// A word below 2^32 congruent to a^2 (a < p): 2 a^2 = hi 2^32 + lo gives a^2 = hi + lo / 2 (mod p).
__device__ __forceinline__ uint32_t square_word(uint32_t a) {
  const uint64_t x = (uint64_t)a * (a + a);
  return (uint32_t)(x >> 32) + ((uint32_t)x >> 1);
}
__device__ __forceinline__ uint4 square_word4(uint4 v) {
  return make_uint4(square_word(v.x), square_word(v.y), square_word(v.z), square_word(v.w));
}

// Byte-reversed coordinate words of a coefficient.
__device__ __forceinline__ void put_reversed(uint32_t* d, QM31 c) {
  d[0] = mmadot::byte_reverse(c.c0.a); d[1] = mmadot::byte_reverse(c.c0.b);
  d[2] = mmadot::byte_reverse(c.c1.a); d[3] = mmadot::byte_reverse(c.c1.b);
}

// Needs 2^(log_n+1) >= 64 rows; ALIGNED: columns and output 16-byte aligned with strides of a multiple
// of four words.
template <bool ALIGNED>
__global__ void __launch_bounds__(MMA_THREADS, 4) k_composition_mma(uint32_t log_n, uint32_t W,
                                                                    const uint32_t* __restrict__ eval, uint64_t stride,
                                                                    const QM31* __restrict__ coeffs, uint32_t den0,
                                                                    uint32_t den1, uint32_t* out, uint64_t out_stride) {
  extern __shared__ uint4 scm[];  // the ring, then alpha, then beta, of the columns padded to a multiple of 8
  const uint32_t steps = (W + 7) / 8, n_cons = W - 2;
  uint32_t* alpha = reinterpret_cast<uint32_t*>(scm + mma_ring_bytes(COMP_STAGES) / 16);
  uint32_t* beta = alpha + 32 * steps;
  for (uint32_t c = threadIdx.x; c < 8 * steps; c += MMA_THREADS) {
    auto coeff = [&](uint32_t k) { return k < n_cons ? coeffs[k] : qzero(); };  // k wraps above for c < 2
    put_reversed(alpha + 4 * c, c < W ? coeff(c - 2) : qzero());
    put_reversed(beta + 4 * c, c < W ? qneg(qadd(coeff(c), coeff(c - 1))) : qzero());
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const mmadot::LaneShifts shifts = mmadot::lane_shifts(g & 1);
  const uint32_t n_blocks = (2u << log_n) / MMA_ROWS, warps = gridDim.x * (MMA_THREADS / 32);
  const uint32_t first_blk = blockIdx.x * (MMA_THREADS / 32) + (threadIdx.x >> 5);
  WordRing<COMP_STAGES> ring(scm);
  uint32_t p_blk = first_blk, p_step = 0;  // next step to load
  auto fetch = [&]() {
    if (p_blk < n_blocks) {
      // Padding columns (zero coefficients) read the last column.
      const uint32_t* rows = eval + MMA_ROWS * p_blk + ring.row();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        ring.fetch<ALIGNED>(u, rows + (uint64_t)min(8 * p_step + 2 * u + ring.column(), W - 1) * stride);
      if (++p_step == steps) { p_step = 0; p_blk += warps; }
    }
    ring.commit();
  };
  for (int d = 0; d < COMP_STAGES; ++d) fetch();
  for (uint32_t blk = first_blk; blk < n_blocks; blk += warps) {
    const uint32_t row0 = MMA_ROWS * blk + 2 * g;
    mmadot::Acc acc;
    acc.clear();
    const uint32_t* qa = alpha + 4 * t + (g >> 1);
    const uint32_t* qb = beta + 4 * t + (g >> 1);
    for (uint32_t s = 0; s < steps; ++s, qa += 32, qb += 32) {
      mmadot::Words w;
      ring.take(w);
      acc.step(w, qa[0], qa[16], shifts);
      fetch();
#pragma unroll
      for (int m = 0; m < 4; ++m) w.a[m] = square_word4(w.a[m]);
      acc.step(w, qb[0], qb[16], shifts);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint32_t row = row0 + 16 * m, den = (row >> log_n) ? den1 : den0;  // both rows share row >> log_n
      store_rows2<ALIGNED>(out + t * out_stride + row,
                           make_uint2(mmul(mmadot::row_sum(acc, m, 0), den), mmul(mmadot::row_sum(acc, m, 1), den)));
    }
  }
}

// ---------------------------------------------------------------------------
// OODS evaluation (src/prover/poly/circle/poly.zig:62-230): value = sum_j c_j *
// prod_{bit b of j} F_b with F_0 = y, F_1 = x, F_b = pi^{b-1}(x).
// ---------------------------------------------------------------------------
constexpr uint32_t OODS_CHUNK_BITS = 12;
constexpr uint32_t OODS_THREADS = 256;

struct OodsFactors { QM31 f[32]; uint32_t log_size; };

__device__ QM31 subset_product(const OodsFactors& F, uint32_t bits, uint32_t first) {
  QM31 r = qone();
  for (uint32_t b = 0; bits; ++b, bits >>= 1)
    if (bits & 1) r = qmul(r, F.f[first + b]);
  return r;
}

__device__ __forceinline__ QM31 shfl_down_q(QM31 v, int d) {
  return qmake(__shfl_down_sync(0xffffffffu, v.c0.a, d), __shfl_down_sync(0xffffffffu, v.c0.b, d),
               __shfl_down_sync(0xffffffffu, v.c1.a, d), __shfl_down_sync(0xffffffffu, v.c1.b, d));
}

// Columns of fewer than 2^12 coefficients: one CTA a column, thread t sums its 16 coefficients against
// the subset products of F_0..F_3 and multiplies by its own (F_4.. by the bits of t).
__global__ void __launch_bounds__(OODS_THREADS) k_oods_small(OodsFactors F, const uint32_t* __restrict__ coeffs,
                                                             uint64_t stride, QM31* out) {
  __shared__ QM31 b4[3][16];
  __shared__ QM31 wsum[OODS_THREADS / 32];
  const uint32_t col = blockIdx.x, log = F.log_size, t = threadIdx.x;
  if (t < 48) {
    const uint32_t lvl = t / 16, r = t % 16, first = 4 * lvl;
    // factors beyond log_size do not exist; mask them out
    const uint32_t valid_bits = first >= log ? 0 : (log - first >= 4 ? 4 : log - first);
    b4[lvl][r] = (r >> valid_bits) ? qzero() : subset_product(F, r, first);
  }
  __syncthreads();
  const uint32_t n_in = 1u << log;
  const uint32_t nw = 16 * t < n_in ? (n_in - 16 * t < 16 ? n_in - 16 * t : 16) : 0;
  const uint32_t* c = coeffs + col * stride + 16 * t;
  uint64_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
  for (uint32_t r = 0; r < nw; ++r) {
    const QM31 bb = b4[0][r];
    const uint32_t w = c[r];
    a0 = mfold64(a0) + (uint64_t)bb.c0.a * w; a1 = mfold64(a1) + (uint64_t)bb.c0.b * w;
    a2 = mfold64(a2) + (uint64_t)bb.c1.a * w; a3 = mfold64(a3) + (uint64_t)bb.c1.b * w;
  }
  QM31 acc = qmake(mreduce64(a0), mreduce64(a1), mreduce64(a2), mreduce64(a3));
  acc = qmul(acc, qmul(b4[1][t & 15], b4[2][t >> 4]));
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) acc = qadd(acc, shfl_down_q(acc, d));
  if ((t & 31) == 0) wsum[t >> 5] = acc;
  __syncthreads();
  if (t == 0) {
    QM31 sum = qzero();
    for (int i = 0; i < OODS_THREADS / 32; ++i) sum = qadd(sum, wsum[i]);
    out[col] = sum;
  }
}

// Columns of 2^12 coefficients or more, the sums on the tensor cores (mma_dot.cuh's limb products). A warp
// takes chunks of 4096 coefficients, chunk = w + k G with G the column's warps (a power of two), so that a
// chunk's product of F_12.. splits over disjoint bits into the warp's part (the bits of w, multiplied in
// once at the end) and k's part (a table hk[k] in shared memory). In a chunk, the coefficients' bits 4..7
// are the sixteen rows of a product and the other eight bits (lo = 0..3, h = 8..11) its contraction
// with F_lo F_h, the same 256 coefficients for every chunk and column: one row of 16 coefficients is 64
// contiguous bytes, so a lane's 16-byte load holds its operand words of two mma steps, and a step h
// reads 1 KB in a row. The chunk's sixteen sums are multiplied by hk[k] and accumulated per row; the
// row's own factor (F_4..F_7) comes at the end. HN: the steps of a chunk that one warp takes. All sixteen
// when there are chunks for every scheduler; otherwise four warps share a chunk (four columns of 2^18:
// 13 us with whole chunks, 6.2 us with quarters).
// 100 columns of 2^20: 89 us, 4.7 TB/s (16 coefficients a thread with 64-bit multiply-adds: 145 us).
constexpr uint32_t OODS_SMEM_CHUNKS = 1024;  // chunk-factor table entries kept in shared memory
constexpr uint32_t OODS_WARPS = 4;

template <int HN>
__global__ void __launch_bounds__(32 * OODS_WARPS) k_oods_mma(OodsFactors F, const uint32_t* __restrict__ coeffs,
                                                              uint64_t stride, QM31* partial, uint32_t n_chunks) {
  __shared__ QM31 f_lo[16], f_row[16], f_h[16];
  __shared__ uint32_t tab[16][4][4][4];  // [h][lo & 3][lo >> 2][coordinate], byte-reversed
  __shared__ QM31 hk[OODS_SMEM_CHUNKS];
  __shared__ QM31 wsum[OODS_WARPS];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, col = blockIdx.y;
  constexpr uint32_t PARTS = 16 / HN;  // warps per chunk
  const uint32_t n_warps = gridDim.x * OODS_WARPS / PARTS, unit = blockIdx.x * OODS_WARPS + warp, w = unit / PARTS;
  const uint32_t h_first = unit % PARTS * HN;
  const uint32_t k_first = OODS_CHUNK_BITS + __ffs(n_warps) - 1;  // factor index of k's bit 0
  if (threadIdx.x < 48) {
    const uint32_t lvl = threadIdx.x / 16, r = threadIdx.x % 16;
    (lvl == 0 ? f_lo : lvl == 1 ? f_row : f_h)[r] = subset_product(F, r, 4 * lvl);
  }
  const uint32_t n_k = (n_chunks + n_warps - 1) / n_warps;  // of the CTA's first warp, the most
  for (uint32_t k = threadIdx.x; k < n_k && k < OODS_SMEM_CHUNKS; k += 32 * OODS_WARPS) hk[k] = subset_product(F, k, k_first);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 256; i += 32 * OODS_WARPS)
    put_reversed(tab[i >> 4][i & 3][(i >> 2) & 3], qmul(f_lo[i & 15], f_h[i >> 4]));
  __syncthreads();
  const mmadot::LaneShifts shifts = mmadot::lane_shifts(g & 1);
  const uint32_t* b = &tab[h_first][0][t][g >> 1];
  QM31 acc = qzero();  // lanes t = 0 and 1: rows g and g + 8
  for (uint32_t k = 0, chunk = w; chunk < n_chunks; ++k, chunk += n_warps) {
    const uint4* c = reinterpret_cast<const uint4*>(coeffs + col * stride + ((uint64_t)chunk << OODS_CHUNK_BITS)) +
                     h_first * 64 + lane;
    int32_t s[4][4];
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i >> 2][i & 3] = 0;
    constexpr int HALF = HN < 8 ? HN : 8;  // h steps loaded together
#pragma unroll 1
    for (int h0 = 0; h0 < HN; h0 += HALF) {
      uint4 x[HALF], y[HALF];
#pragma unroll
      for (int h = 0; h < HALF; ++h) {
        x[h] = __ldg(c + (h0 + h) * 64);
        y[h] = __ldg(c + (h0 + h) * 64 + 32);
      }
#pragma unroll
      for (int h = 0; h < HALF; ++h) {
        const uint32_t* bh = b + (h0 + h) * 64;
        uint32_t e0[4], e1[4];
        mmadot::expand(bh[0], shifts, e0);
        mmadot::expand(bh[16], shifts, e1);
#pragma unroll
        for (int i = 0; i < 4; ++i) mmadot::mma_u8(s[i], x[h].x, y[h].x, x[h].y, y[h].y, e0[i], e1[i]);
        mmadot::expand(bh[32], shifts, e0);
        mmadot::expand(bh[48], shifts, e1);
#pragma unroll
        for (int i = 0; i < 4; ++i) mmadot::mma_u8(s[i], x[h].z, y[h].z, x[h].w, y[h].w, e0[i], e1[i]);
      }
    }
    const uint32_t v0 = mmadot::combine(s, 0), v1 = mmadot::combine(s, 1);
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t a = __shfl_sync(0xffffffffu, v0, j, 4), d = __shfl_sync(0xffffffffu, v1, j, 4);
      v[j] = t & 1 ? d : a;
    }
    QM31 f = hk[k & (OODS_SMEM_CHUNKS - 1)];
    if (k >= OODS_SMEM_CHUNKS) {  // beyond the table: the rest of k's bits multiplied in
      uint32_t bits = k / OODS_SMEM_CHUNKS;
      for (uint32_t i = k_first + 10; bits; ++i, bits >>= 1)
        if (bits & 1) f = qmul(f, F.f[i]);
    }
    acc = qadd(acc, qmul(qload4(v), f));
  }
  acc = t < 2 ? qmul(acc, qmul(f_row[g + 8 * t], subset_product(F, w, OODS_CHUNK_BITS))) : qzero();
  __syncwarp();
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) acc = qadd(acc, shfl_down_q(acc, d));
  if (lane == 0) wsum[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    QM31 sum = qzero();
    for (uint32_t i = 0; i < OODS_WARPS; ++i) sum = qadd(sum, wsum[i]);
    partial[(uint64_t)col * gridDim.x + blockIdx.x] = sum;
  }
}

// One warp per column: the lanes sum every 32nd partial, then a shuffle
// reduction (M31 addition is associative and commutative, so the order does not
// change the value). A thread per column summing up to 1184 partials in turn
// took 18-33 us for the few-column evaluations.
__global__ void k_oods_sum(const QM31* partial, uint32_t n_chunks, uint32_t n_cols, QM31* out) {
  const uint32_t col = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (col >= n_cols) return;  // warp-uniform
  const QM31* p = partial + (uint64_t)col * n_chunks;
  QM31 acc = qzero();
  for (uint32_t i = lane; i < n_chunks; i += 32) acc = qadd(acc, p[i]);
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) acc = qadd(acc, shfl_down_q(acc, d));
  if (lane == 0) out[col] = acc;
}

// ---------------------------------------------------------------------------
// DEEP quotients (src/core/pcs/quotients/row_evaluation.zig:101-140,400-521):
// row value = sum_batches (sum_i c_i v_i(row) - (sum_a * y + sum_b)) / den,
// den = (Re(Px) - x) Im(Py) - (Re(Py) - y) Im(Px) at the lifting-domain point of
// the row (bit-reversed circle-domain order).
// ---------------------------------------------------------------------------
constexpr uint32_t QUOT_MAX_ENTRIES = 1024;

// One row per thread, for domains of fewer than 64 rows: few threads that wait for memory, so QUOT_U entries are
// loaded before they are used (1024 columns on 16 rows: 260 us an entry at a time, 67 us now).
constexpr uint32_t QUOT_U = 24;  // a multiple of three: the sums are folded after every third product

__global__ void __launch_bounds__(256) k_quotients(PointTable pts, uint32_t log_size, uint32_t n_batches,
                                                   const QuotientBatchDev* batches,
                                                   const __grid_constant__ QuotientBatchDev one,
                                                   const uint32_t* const* __restrict__ col_ptrs,
                                                   const QM31* __restrict__ coeff_c, uint32_t* out, uint64_t out_stride) {
  extern __shared__ uint32_t sq[];  // 4 words per entry
  if (!batches) batches = &one;
  uint32_t n_entries = 0;
  for (uint32_t b = 0; b < n_batches; ++b) n_entries = max(n_entries, batches[b].first + batches[b].count);
  for (uint32_t i = threadIdx.x; i < n_entries; i += blockDim.x) qstore4(coeff_c[i], sq + 4 * i);
  __syncthreads();
  const uint32_t rows = 1u << log_size;
  const CircleDomain dom = canonic_domain(log_size);
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x) {
    PointM dp = pts.at(dom.index_at(bitrev(row, log_size)));
    QM31 acc = qzero();
    for (uint32_t b = 0; b < n_batches; ++b) {
      const QuotientBatchDev bt = batches[b];
      uint64_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
      // `count` entries from e on, all of their words loaded first.
      auto take = [&](uint32_t e, uint32_t count) {
        uint32_t v[QUOT_U];
#pragma unroll
        for (uint32_t u = 0; u < QUOT_U; ++u)
          if (u < count) v[u] = __ldg(col_ptrs[e + u] + row);
#pragma unroll
        for (uint32_t u = 0; u < QUOT_U; ++u) {
          if (u >= count) break;
          const uint32_t* q = sq + 4 * (e + u);
          a0 += (uint64_t)q[0] * v[u]; a1 += (uint64_t)q[1] * v[u];
          a2 += (uint64_t)q[2] * v[u]; a3 += (uint64_t)q[3] * v[u];
          if (u % 3 == 2) { a0 = mfold64(a0); a1 = mfold64(a1); a2 = mfold64(a2); a3 = mfold64(a3); }
        }
      };
      uint32_t i = 0;
      for (; i + QUOT_U <= bt.count; i += QUOT_U) take(bt.first + i, QUOT_U);
      if (i < bt.count) take(bt.first + i, bt.count - i);
      QM31 num = qmake(mreduce64(a0), mreduce64(a1), mreduce64(a2), mreduce64(a3));
      num = qsub(num, qadd(qmulm(bt.sum_a, dp.y), bt.sum_b));
      CM31 prx = bt.point.x.c0, pry = bt.point.y.c0, pix = bt.point.x.c1, piy = bt.point.y.c1;
      CM31 den = csub(cmul(csub(prx, CM31{dp.x, 0}), piy), cmul(csub(pry, CM31{dp.y, 0}), pix));
      acc = qadd(acc, qmulc(num, cinv(den)));
    }
    out[row] = acc.c0.a;
    out[out_stride + row] = acc.c0.b;
    out[2 * out_stride + row] = acc.c1.a;
    out[3 * out_stride + row] = acc.c1.b;
  }
}

// Adds one batch's quotient to R rows: the numerators accumulated in `a` (lazy 64-bit sums of
// c_i v_i(row)) minus the batch's linear term, times the inverse denominators, the R rows'
// denominators inverted together.
template <int R>
__device__ __forceinline__ void quot_batch_finish(const QuotientBatchDev& bt, const PointM (&dp)[R],
                                                  const uint64_t (&a)[R][4], QM31 (&acc)[R]) {
  CM31 prx = bt.point.x.c0, pry = bt.point.y.c0, pix = bt.point.x.c1, piy = bt.point.y.c1;
  CM31 den[R], pre[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    den[j] = csub(cmul(csub(prx, CM31{dp[j].x, 0}), piy), cmul(csub(pry, CM31{dp[j].y, 0}), pix));
    pre[j] = j == 0 ? den[0] : cmul(pre[j - 1], den[j]);
  }
  CM31 inv[R];
  if (pre[R - 1].a == 0 && pre[R - 1].b == 0) {
#pragma unroll
    for (int j = 0; j < R; ++j) inv[j] = cinv(den[j]);
  } else {
    CM31 t = cinv(pre[R - 1]);
#pragma unroll
    for (int j = R - 1; j >= 1; --j) {
      inv[j] = cmul(t, pre[j - 1]);
      t = cmul(t, den[j]);
    }
    inv[0] = t;
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
    QM31 num = qmake(mreduce64(a[j][0]), mreduce64(a[j][1]), mreduce64(a[j][2]), mreduce64(a[j][3]));
    num = qsub(num, qadd(qmulm(bt.sum_a, dp[j].y), bt.sum_b));
    acc[j] = qadd(acc[j], qmulc(num, inv[j]));
  }
}

// The quotients of 64 rows per warp, the numerators' sums on the tensor cores (mma_dot.cuh): lane (g, t)
// ends with coordinate t of rows 16m + 2g and + 1 for m = 0..3. A batch's entries are taken eight columns a step, padded
// with zero coefficients. Lane t inverts the denominators of tile t's two rows, whose points are
// conjugates, with one inversion, and the four lanes exchange them. ALIGNED: columns and output 16-byte aligned, with strides of a multiple of four words.
//
// Bound by HBM: 2^21 rows x 108 columns 162 us, 5.8 TB/s, and 175 us where the kernel looks at the pointers (64-bit
// multiply-adds, ten instructions per word, 265 us; the bulk-staged kernel 258 us).
template <bool ALIGNED>
__device__ __forceinline__ void quotients_mma_rows(const PointTable& pts, uint32_t log_size, uint32_t n_batches,
                                                   const QuotientBatchDev* batches, uint4* qmma, const uint32_t* sq,
                                                   const uint32_t* const* sptr, uint32_t total, uint32_t* out,
                                                   uint64_t out_stride) {
  const uint32_t lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const mmadot::LaneShifts shifts = mmadot::lane_shifts(g & 1);
  const uint32_t n_blocks = (1u << log_size) / MMA_ROWS, warps = gridDim.x * (MMA_THREADS / 32);
  const uint32_t first_blk = blockIdx.x * (MMA_THREADS / 32) + (threadIdx.x >> 5);
  const CircleDomain dom = canonic_domain(log_size);
  WordRing<QUOT_STAGES> ring(qmma);
  uint32_t p_blk = first_blk, p_step = 0;  // next step to load
  auto fetch = [&]() {
    if (p_blk < n_blocks && total) {
      const uint32_t* const* ptr = sptr + 8 * p_step + ring.column();
#pragma unroll
      for (int u = 0; u < 4; ++u) ring.fetch<ALIGNED>(u, ptr[2 * u] + MMA_ROWS * p_blk + ring.row());
      if (++p_step == total) { p_step = 0; p_blk += warps; }
    }
    ring.commit();
  };
  for (int d = 0; d < QUOT_STAGES; ++d) fetch();
  for (uint32_t blk = first_blk; blk < n_blocks; blk += warps) {
    const uint32_t row0 = MMA_ROWS * blk + 2 * g;
    uint32_t num[4][2] = {};  // this lane's coordinate of the eight rows
    // The point of the even row of tile t (the odd row's is its conjugate), added up after the loop.
    const uint32_t idx = dom.index_at(bitrev(row0 + 16 * t, log_size));
    const PointM plo = pts.lo(idx), phi = pts.hi(idx);
    const uint32_t* q = sq + 4 * t + (g >> 1);
    for (uint32_t b = 0; b < n_batches; ++b) {
      mmadot::Acc acc;
      acc.clear();
      for (uint32_t s = (batches[b].count + 7) / 8; s > 0; --s, q += 32) {
        mmadot::Words w;
        ring.take(w);
        acc.step(w, q[0], q[16], shifts);
        fetch();
      }
      uint32_t sum[4][2];  // before the denominators: it ends the accumulators' registers
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int s = 0; s < 2; ++s) sum[m][s] = mmadot::row_sum(acc, m, s);
      const PointM at = padd(plo, phi);
      CM31 inv[2];
      {
        const PointQ pq = batches[b].point;
        // (Re Px - x) Im Py - (Re Py - y) Im Px at (x, y) and (x, -y).
        const CM31 u = cmul(csub(pq.x.c0, CM31{at.x, 0}), pq.y.c1);
        const CM31 den0 = csub(u, cmul(csub(pq.y.c0, CM31{at.y, 0}), pq.x.c1));
        const CM31 den1 = csub(u, cmul(cadd(pq.y.c0, CM31{at.y, 0}), pq.x.c1));
        const CM31 both = cmul(den0, den1);
        if (both.a == 0 && both.b == 0) {  // a zero denominator gives a zero quotient term
          inv[0] = cinv(den0);
          inv[1] = cinv(den1);
        } else {
          const CM31 r = cinv(both);
          inv[0] = cmul(r, den1);
          inv[1] = cmul(r, den0);
        }
        __syncwarp();
      }
      const uint32_t sum_a = reinterpret_cast<const uint32_t*>(&batches[b].sum_a)[t];
      const uint32_t sum_b = reinterpret_cast<const uint32_t*>(&batches[b].sum_b)[t];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t ay = mmul(sum_a, __shfl_sync(0xffffffffu, at.y, m, 4));
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const CM31 iv = {__shfl_sync(0xffffffffu, inv[s].a, m, 4), __shfl_sync(0xffffffffu, inv[s].b, m, 4)};
          const uint32_t line = s ? msub(sum_b, ay) : madd(sum_b, ay);
          const uint32_t v = msub(sum[m][s], line);
          // (v0 + v1 i)(a + b i): lane t holds v0 (even) or v1 (odd) of its half and keeps that coordinate.
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 1);
          const uint32_t va = mmul(v, iv.a), ob = mmul(o, iv.b);
          num[m][s] = madd(num[m][s], t & 1 ? madd(va, ob) : msub(va, ob));
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
      store_rows2<ALIGNED>(out + t * out_stride + row0 + 16 * m, make_uint2(num[m][0], num[m][1]));
  }
}

// batches == nullptr: the one batch `one`. CHECK: the kernel looks at the column pointers itself (a caller that
// vouches for their alignment takes the other).
template <bool CHECK>
__global__ void __launch_bounds__(MMA_THREADS, 4) k_quotients_mma(PointTable pts, uint32_t log_size, uint32_t n_batches,
                                                                  const QuotientBatchDev* batches,
                                                                  const __grid_constant__ QuotientBatchDev one,
                                                                  const uint32_t* const* __restrict__ col_ptrs,
                                                                  const QM31* __restrict__ coeff_c, uint32_t padded,
                                                                  uint32_t* out, uint64_t out_stride) {
  extern __shared__ uint4 qmma[];
  __shared__ int s_bad;
  if (!batches) batches = &one;
  uint32_t* sq = reinterpret_cast<uint32_t*>(qmma + mma_ring_bytes(QUOT_STAGES) / 16);  // byte-reversed coefficients
  const uint32_t** sptr = reinterpret_cast<const uint32_t**>(sq + 4 * padded);  // column pointers
  if (CHECK) {
    if (threadIdx.x == 0) s_bad = (reinterpret_cast<uintptr_t>(out) & 15) != 0 || out_stride % 4 != 0;
    __syncthreads();
  }
  uint32_t total = 0;  // steps of eight entries of all batches
  for (uint32_t b = 0; b < n_batches; ++b) {
    const uint32_t first = batches[b].first, count = batches[b].count, room = (count + 7) / 8 * 8;
    for (uint32_t i = threadIdx.x; i < room; i += MMA_THREADS) {
      const uint32_t e = first + (i < count ? i : 0);
      put_reversed(sq + 4 * (8 * total + i), i < count ? coeff_c[e] : qzero());
      const uint32_t* p = col_ptrs[e];
      sptr[8 * total + i] = p;
      if (CHECK && (reinterpret_cast<uintptr_t>(p) & 15)) s_bad = 1;
    }
    total += room / 8;
  }
  __syncthreads();
  if (CHECK && s_bad) quotients_mma_rows<false>(pts, log_size, n_batches, batches, qmma, sq, sptr, total, out, out_stride);
  else quotients_mma_rows<true>(pts, log_size, n_batches, batches, qmma, sq, sptr, total, out, out_stride);
}

// ---- Quotients with the column words staged in shared memory by bulk async copies ----------
// Warp-specialized: eight consumer warps own a tile of QB_ROWS rows (two per thread); a ninth,
// producer warp streams the tile's column chunks (2 KB each) into a ring of QB_STAGES stages of
// QB_GROUP columns with 1-D bulk copies (cp.async.bulk global -> shared, one chunk per lane,
// completing on the stage's `full` mbarrier with the stage's byte count). A consumer warp waits on
// `full`, reads its threads' two words of each column, and arrives on the stage's `empty` mbarrier;
// the producer refills a stage once all eight consumer warps have arrived. The loads of the stages
// ahead stay in flight while one is consumed without taking registers, and the producer never holds the
// consumers at a block barrier. Items run batch by
// batch (a batch's entries in groups of at most QB_GROUP); the last group of a batch adds the
// batch's quotient. Each wait is bounded (about a second of the global timer): a side that runs out
// sets QUOT_STATUS_TIMEOUT in *status and a shared abort flag that ends the other side's loop; the
// producer then waits (again bounded) for the copies it issued. Batches that reach past the
// n_entries columns, or more groups than the item table holds, set QUOT_STATUS_LAYOUT before any
// copy is issued.
constexpr uint32_t QB_ROWS = 512, QB_GROUP = 8, QB_STAGES = 4, QB_MAX_BATCHES = 64;
constexpr uint32_t QB_CONSUMER_WARPS = QB_ROWS / 2 / 32, QB_THREADS = (QB_CONSUMER_WARPS + 1) * 32;
constexpr uint64_t QB_WAIT_NS = 1000000000ull;
// A test hook: the next bulk quotient launch issues no copy for its first item, so that every wait
// on that stage runs out.
std::atomic<bool> g_quot_skip_first_item{false};

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 1-D bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) into this CTA's shared
// memory; its completion counts against the barrier's expected bytes.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// Waits for the completion of phase `parity` of the barrier for at most QB_WAIT_NS, or until *abort
// is set; false unless the phase completed.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, const volatile int* abort) {
  const uint32_t a = smem_u32(bar);
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0;; ++it) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(a), "r"(parity) : "memory");
    if (done) return true;
    // The clock and the abort flag are looked at every 64th try only (try_wait itself suspends).
    if ((it & 63) == 63 && ((abort && *abort) || global_ns() - t0 > QB_WAIT_NS)) return false;
  }
}

struct QbItem {
  uint32_t e0;     // first entry of the group
  uint16_t ne;     // entries in the group (0 .. QB_GROUP; 0 only for a batch without entries)
  uint16_t batch;  // 1 + the batch index when the group is its batch's last, else 0
};

template <int MINB>
__global__ void __launch_bounds__(QB_THREADS, MINB) k_quotients_bulk(PointTable pts, uint32_t log_size,
                                                                     uint32_t n_batches,
                                                                     const QuotientBatchDev* __restrict__ batches,
                                                                     const uint32_t* const* __restrict__ col_ptrs,
                                                                     const QM31* __restrict__ coeff_c,
                                                                     uint32_t n_entries, uint32_t item_cap,
                                                                     uint32_t* out, uint64_t out_stride,
                                                                     uint32_t* status, int skip_first_item) {
  constexpr int R = 2;
  extern __shared__ __align__(16) uint8_t qsm[];
  uint32_t* ring = reinterpret_cast<uint32_t*>(qsm);                     // QB_STAGES x QB_GROUP x QB_ROWS words
  uint4* sq = reinterpret_cast<uint4*>(ring + QB_STAGES * QB_GROUP * QB_ROWS);  // n_entries coefficients
  const uint32_t** sptr = reinterpret_cast<const uint32_t**>(sq + n_entries);  // n_entries column pointers
  QbItem* items = reinterpret_cast<QbItem*>(sptr + n_entries);                 // item_cap groups of one tile
  __shared__ uint64_t full[QB_STAGES], empty[QB_STAGES];
  __shared__ QuotientBatchDev sbt[QB_MAX_BATCHES];
  __shared__ int s_abort;
  __shared__ uint32_t s_items;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (uint32_t i = tid; i < n_entries; i += blockDim.x) {
    const QM31 c = coeff_c[i];
    sq[i] = make_uint4(c.c0.a, c.c0.b, c.c1.a, c.c1.b);
    sptr[i] = col_ptrs[i];
  }
  for (uint32_t b = tid; b < n_batches; b += blockDim.x) sbt[b] = batches[b];
  if (tid == 0) {
    uint32_t k = 0;
    bool bad = n_batches > QB_MAX_BATCHES;
    for (uint32_t b = 0; b < n_batches && !bad; ++b) {
      const uint32_t first = batches[b].first, count = batches[b].count;
      if (first > n_entries || count > n_entries - first) {
        bad = true;
        break;
      }
      // A batch without entries still adds its linear term: one empty group.
      for (uint32_t g = 0; g < count || (count == 0 && g == 0); g += QB_GROUP) {
        if (k == item_cap) {
          bad = true;
          break;
        }
        const uint32_t ne = min(QB_GROUP, count - g);
        items[k++] = QbItem{first + g, (uint16_t)ne, (uint16_t)(g + ne == count ? b + 1 : 0)};
      }
    }
    for (uint32_t s = 0; s < QB_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], QB_CONSUMER_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_items = k;
    s_abort = bad ? 1 : 0;
    if (bad) atomicOr(status, QUOT_STATUS_LAYOUT);
  }
  __syncthreads();
  if (s_abort) return;  // nothing issued
  const uint32_t n_items = s_items;
  const uint32_t n_tiles = (1u << log_size) / QB_ROWS;
  const uint32_t my_tiles = blockIdx.x < n_tiles ? (n_tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const uint64_t total = (uint64_t)my_tiles * n_items;
  volatile int* abort = &s_abort;

  if (warp == QB_CONSUMER_WARPS) {
    // Producer warp: item i (tile-major, groups minor) into stage i % QB_STAGES, lane k copying the
    // group's k-th column chunk.
    uint64_t i = 0;
    bool ok = true;
    for (; i < total; ++i) {
      const uint32_t s = (uint32_t)(i % QB_STAGES);
      // Every lane waits (each acquires the consumers' release); the warp decides together.
      const bool got = i < QB_STAGES || mbar_wait_bounded(&empty[s], (uint32_t)(i / QB_STAGES - 1) & 1, abort);
      if (!__all_sync(0xffffffffu, got)) {
        ok = false;
        break;
      }
      if (skip_first_item && i == 0) continue;
      const uint32_t tile = blockIdx.x + (uint32_t)(i / n_items) * gridDim.x;
      const QbItem it = items[i % n_items];
      uint32_t* dst = ring + s * (QB_GROUP * QB_ROWS);
      // The stage's words were last read through the generic proxy; every lane that issues a copy
      // orders those reads before the async-proxy writes of its refill.
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (lane == 0) mbar_arrive_expect_tx(&full[s], it.ne * QB_ROWS * 4);
      __syncwarp();
      if (lane < it.ne)
        bulk_load(dst + lane * QB_ROWS, sptr[it.e0 + lane] + (uint64_t)tile * QB_ROWS, QB_ROWS * 4, &full[s]);
    }
    if (lane == 0) {
      if (!ok) {
        *abort = 1;
        atomicOr(status, QUOT_STATUS_TIMEOUT);
      }
      // Items i - QB_STAGES .. i - 1 are the last ones issued (earlier ones were consumed before
      // their stages were refilled): let their copies land before the CTA's shared memory is
      // released, also when the consumers stopped early (bounded, the abort flag ignored).
      const uint64_t from = i > QB_STAGES ? i - QB_STAGES : 0;
      for (uint64_t j = from; j < i; ++j)
        if (!(skip_first_item && j == 0)) mbar_wait_bounded(&full[j % QB_STAGES], (uint32_t)(j / QB_STAGES) & 1, nullptr);
    }
  } else {
    const CircleDomain dom = canonic_domain(log_size);
    uint64_t item = 0;
    bool ok = true;
    for (uint32_t q = 0; q < my_tiles && ok; ++q) {
      const uint32_t row0 = (blockIdx.x + q * gridDim.x) * QB_ROWS + R * tid;
      PointM dp[R];
#pragma unroll
      for (int j = 0; j < R; ++j) dp[j] = pts.at(dom.index_at(bitrev(row0 + j, log_size)));
      QM31 acc[R];
#pragma unroll
      for (int j = 0; j < R; ++j) acc[j] = qzero();
      uint64_t a[R][4];
#pragma unroll
      for (int j = 0; j < R; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) a[j][c] = 0;
      for (uint32_t g = 0; g < n_items; ++g, ++item) {
        const uint32_t s = (uint32_t)(item % QB_STAGES);
        // Every lane waits (each acquires the copies' completion); the warp decides together.
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[s], (uint32_t)(item / QB_STAGES) & 1, abort))) {
          ok = false;
          break;
        }
        const QbItem it = items[g];
        const uint32_t* col = ring + s * (QB_GROUP * QB_ROWS) + R * tid;
        const uint4* cq = sq + it.e0;
        // Terms of a group are folded after its entries 2, 5 and 7 (and after its last): at most
        // three products (< 2^62 each) on top of a folded value (< 2^34) between folds.
        auto term = [&](uint32_t k) {
          const uint2 v = *reinterpret_cast<const uint2*>(col + k * QB_ROWS);
          const uint4 c = cq[k];
          a[0][0] += (uint64_t)c.x * v.x; a[0][1] += (uint64_t)c.y * v.x;
          a[0][2] += (uint64_t)c.z * v.x; a[0][3] += (uint64_t)c.w * v.x;
          a[1][0] += (uint64_t)c.x * v.y; a[1][1] += (uint64_t)c.y * v.y;
          a[1][2] += (uint64_t)c.z * v.y; a[1][3] += (uint64_t)c.w * v.y;
        };
        auto fold = [&]() {
#pragma unroll
          for (int j = 0; j < R; ++j)
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) a[j][c4] = mfold64(a[j][c4]);
        };
        if (it.ne == QB_GROUP) {
#pragma unroll
          for (uint32_t k = 0; k < QB_GROUP; ++k) {
            term(k);
            if (k == 2 || k == 5 || k == 7) fold();
          }
        } else {
          for (uint32_t k = 0; k < it.ne; ++k) {
            term(k);
            if (k == 2 || k == 5 || k + 1 == it.ne) fold();
          }
        }
        // This warp is done with the stage's words.
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (it.batch) {
          quot_batch_finish<R>(sbt[it.batch - 1], dp, a, acc);
#pragma unroll
          for (int j = 0; j < R; ++j)
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) a[j][c4] = 0;
        }
      }
      if (!ok) break;
      const uint32_t w0[4] = {acc[0].c0.a, acc[0].c0.b, acc[0].c1.a, acc[0].c1.b};
      const uint32_t w1[4] = {acc[1].c0.a, acc[1].c0.b, acc[1].c1.a, acc[1].c1.b};
#pragma unroll
      for (int c4 = 0; c4 < 4; ++c4)
        *reinterpret_cast<uint2*>(out + c4 * out_stride + row0) = make_uint2(w0[c4], w1[c4]);
    }
    if (!ok) {
      *abort = 1;
      if (lane == 0) atomicOr(status, QUOT_STATUS_TIMEOUT);
    }
  }
  // The producer's bounded wait for its own copies ends before any thread of the CTA exits.
  __syncthreads();
}

// ---------------------------------------------------------------------------
// FRI folds (src/core/fri/folding.zig:352-384, 558-602). The inverse twiddles
// of the fold are the inverse FFT twiddles of the source domain: 1/py of the
// circle layer for fold_circle_into_line, 1/x of line layer 0 for fold_line.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void qibfly(QM31& f0, QM31& f1, uint32_t it) {
  QM31 a = f0;
  f0 = qadd(a, f1);
  f1 = qmulm(qsub(a, f1), it);
}

__global__ void k_fold_circle(TwiddleView itv, uint32_t dst_log, const uint32_t* __restrict__ src, uint64_t ss,
                              QM31 alpha, QM31 alpha_sq, uint32_t* dst, uint64_t ds, int accumulate) {
  const uint32_t n = 1u << dst_log;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint2 w0 = *reinterpret_cast<const uint2*>(src + 2 * i);
    uint2 w1 = *reinterpret_cast<const uint2*>(src + ss + 2 * i);
    uint2 w2 = *reinterpret_cast<const uint2*>(src + 2 * ss + 2 * i);
    uint2 w3 = *reinterpret_cast<const uint2*>(src + 3 * ss + 2 * i);
    QM31 f0 = qmake(w0.x, w1.x, w2.x, w3.x), f1 = qmake(w0.y, w1.y, w2.y, w3.y);
    qibfly(f0, f1, itv.circ(i));
    QM31 r = qadd(qmul(alpha, f1), f0);
    if (accumulate) r = qadd(qmul(qmake(dst[i], dst[ds + i], dst[2 * ds + i], dst[3 * ds + i]), alpha_sq), r);
    dst[i] = r.c0.a; dst[ds + i] = r.c0.b; dst[2 * ds + i] = r.c1.a; dst[3 * ds + i] = r.c1.b;
  }
}

__global__ void k_fold_line(TwiddleView itv, uint32_t dst_log, const uint32_t* __restrict__ src, uint64_t ss,
                            QM31 alpha, uint32_t* dst, uint64_t ds) {
  const uint32_t n = 1u << dst_log;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint2 w0 = *reinterpret_cast<const uint2*>(src + 2 * i);
    uint2 w1 = *reinterpret_cast<const uint2*>(src + ss + 2 * i);
    uint2 w2 = *reinterpret_cast<const uint2*>(src + 2 * ss + 2 * i);
    uint2 w3 = *reinterpret_cast<const uint2*>(src + 3 * ss + 2 * i);
    QM31 f0 = qmake(w0.x, w1.x, w2.x, w3.x), f1 = qmake(w0.y, w1.y, w2.y, w3.y);
    qibfly(f0, f1, itv.line(1, i));
    QM31 r = qadd(f0, qmul(alpha, f1));
    dst[i] = r.c0.a; dst[ds + i] = r.c0.b; dst[2 * ds + i] = r.c1.a; dst[3 * ds + i] = r.c1.b;
  }
}

__global__ void k_gather_words(const GatherItem* items, uint32_t n, uint32_t* out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = items[i].src[items[i].index];
}

__global__ void k_gather_hashes(const HashGatherItem* items, uint32_t n, uint8_t* out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint4* s = reinterpret_cast<const uint4*>(items[i].layers + items[i].node * 32);
  uint4* d = reinterpret_cast<uint4*>(out + (uint64_t)i * 32);
  d[0] = s[0];
  d[1] = s[1];
}

inline uint32_t grid_for(uint64_t n, uint32_t threads, uint32_t cap = 148 * 32) {
  uint64_t g = (n + threads - 1) / threads;
  if (g > cap) g = cap;
  return g == 0 ? 1 : (uint32_t)g;
}

// Largest dynamic shared memory of the kernels that take more than the 48 KB a launch has without asking.
constexpr size_t COMP_SMEM_MAX = mma_ring_bytes(COMP_STAGES) + 3008 * 32;  // W <= 3000
constexpr size_t QUOT_SMEM_MAX = 200 * 1024;
constexpr size_t QB_SMEM_MAX = (size_t)QB_STAGES * QB_GROUP * QB_ROWS * 4 +
                               (size_t)QUOT_MAX_ENTRIES * (16 + sizeof(void*)) +
                               (size_t)(QUOT_MAX_ENTRIES / QB_GROUP + QB_MAX_BATCHES) * sizeof(QbItem);

}  // namespace

cudaError_t prover_smem_limits(const SetSmemLimit& set) {
  struct { const void* kernel; size_t bytes; } const limits[] = {
      {(const void*)k_composition_mma<true>, COMP_SMEM_MAX},  {(const void*)k_composition_mma<false>, COMP_SMEM_MAX},
      {(const void*)k_quotients_mma<true>, QUOT_SMEM_MAX},    {(const void*)k_quotients_mma<false>, QUOT_SMEM_MAX},
      {(const void*)k_quotients_bulk<2>, QB_SMEM_MAX},        {(const void*)k_quotients_bulk<3>, QB_SMEM_MAX}};
  for (const auto& l : limits) {
    const cudaError_t e = set(l.kernel, (int)l.bytes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t quadratic_trace(uint32_t log_n, uint32_t W, const uint32_t recipe[7], uint32_t* out, uint64_t stride,
                            cudaStream_t stream) {
  QuadRecipe q;
  for (int i = 0; i < 7; ++i) q.r[i] = recipe[i] % P;
  k_quadratic_trace<<<grid_for(1ull << log_n, 256), 256, 0, stream>>>(log_n, W, q, out, stride); note_launch();
  return cudaGetLastError();
}

cudaError_t wide_fib_trace(uint32_t log_n, uint32_t W, int kind, uint64_t seed, uint32_t* out, uint64_t stride,
                           cudaStream_t stream) {
  k_wide_fib_trace<<<grid_for(1ull << log_n, 256), 256, 0, stream>>>(log_n, W, kind, seed, out, stride); note_launch();
  return cudaGetLastError();
}

cudaError_t wide_fib_composition(uint32_t log_n, uint32_t W, const uint32_t* eval, uint64_t stride,
                                 const QM31* coeffs_dev, uint32_t den_inv0, uint32_t den_inv1, uint32_t* out,
                                 uint64_t out_stride, cudaStream_t stream) {
  // Fewer rows than a warp's block of the tensor-core kernel, or so few columns that padding them to steps of eight
  // costs it more than its products save (2^21 rows: 3 columns 17 us here, 32 there; 9: 35, 46; 14: 46, 47; 16: 54,
  // 47; 17: 54, 60; 20: 60, 60; 24: 74, 60).
  const bool few_rows = (2u << log_n) < MMA_ROWS;
  if (few_rows || W < 16 || (W > 16 && W <= 20)) {
    const bool pairs = ((reinterpret_cast<uintptr_t>(eval) | reinterpret_cast<uintptr_t>(out)) & 7) == 0 &&
                       stride % 2 == 0 && out_stride % 2 == 0;
    auto kernel = few_rows ? k_composition<1, 24> : pairs ? k_composition<2, 6> : k_composition<1, 6>;
    kernel<<<grid_for(2ull << log_n, pairs ? 512 : 256), 256, (size_t)(W - 2) * 16, stream>>>(
        log_n, W, eval, stride, coeffs_dev, den_inv0, den_inv1, out, out_stride);
    note_launch();
    return cudaGetLastError();
  }
  const bool aligned = ((reinterpret_cast<uintptr_t>(eval) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                       stride % 4 == 0 && out_stride % 4 == 0;
  // Persistent: four CTAs per SM (fewer where W's coefficients fill the shared memory), 64 rows per warp at a time.
  const uint32_t blocks = (2u << log_n) / MMA_ROWS, per_cta = MMA_THREADS / 32;
  const uint32_t grid = std::min<uint32_t>((blocks + per_cta - 1) / per_cta, 148 * 4);
  const size_t smem_m = (size_t)mma_ring_bytes(COMP_STAGES) + (size_t)((W + 7) / 8) * 8 * 32;
  auto kernel = aligned ? k_composition_mma<true> : k_composition_mma<false>;
  kernel<<<grid, MMA_THREADS, smem_m, stream>>>(log_n, W, eval, stride, coeffs_dev, den_inv0, den_inv1, out, out_stride);
  note_launch();
  return cudaGetLastError();
}

namespace {
// dst[i] += coeff * src[lifted i] over 4 coordinate columns (src of 2^src_log <= 2^dst_log rows).
__global__ void k_accumulate_lifted(uint32_t dst_log, uint32_t* dst, uint64_t ds, uint32_t src_log,
                                    const uint32_t* __restrict__ src, uint64_t ss, QM31 coeff) {
  const uint64_t n = 1ull << dst_log;
  const uint32_t sh = dst_log - src_log + 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t j = src_log == dst_log ? i : (((i >> sh) << 1) | (i & 1));
    const QM31 v = qmul(coeff, qmake(src[j], src[ss + j], src[2 * ss + j], src[3 * ss + j]));
    dst[i] = madd(dst[i], v.c0.a);
    dst[ds + i] = madd(dst[ds + i], v.c0.b);
    dst[2 * ds + i] = madd(dst[2 * ds + i], v.c1.a);
    dst[3 * ds + i] = madd(dst[3 * ds + i], v.c1.b);
  }
}

}  // namespace

cudaError_t accumulate_lifted(uint32_t dst_log, uint32_t* dst, uint64_t dst_stride, uint32_t src_log,
                              const uint32_t* src, uint64_t src_stride, QM31 coeff, cudaStream_t stream) {
  if (src_log > dst_log) return cudaErrorInvalidValue;
  k_accumulate_lifted<<<grid_for(1ull << dst_log, 256), 256, 0, stream>>>(dst_log, dst, dst_stride, src_log, src,
                                                                           src_stride, coeff);
  note_launch();
  return cudaGetLastError();
}

size_t eval_at_point_partial_count(uint32_t log_size, uint32_t n_cols) {
  uint32_t chunk_bits = log_size < OODS_CHUNK_BITS ? log_size : OODS_CHUNK_BITS;
  return (size_t)n_cols << (log_size - chunk_bits);
}

cudaError_t eval_at_point(const DeviceTables&, uint32_t log_size, uint32_t n_cols, const uint32_t* coeffs,
                          uint64_t stride, PointQ p, QM31*, QM31* partial, QM31* out, cudaStream_t stream) {
  if (log_size > 31) return cudaErrorInvalidValue;
  OodsFactors F{};
  F.log_size = log_size;
  if (log_size > 0) {
    F.f[0] = p.y;
    QM31 x = p.x;
    for (uint32_t b = 1; b < log_size; ++b) { F.f[b] = x; x = qdouble_x(x); }
  }
  if (log_size < OODS_CHUNK_BITS) {
    k_oods_small<<<n_cols, OODS_THREADS, 0, stream>>>(F, coeffs, stride, out); note_launch();
    return cudaGetLastError();
  }
  const uint32_t n_chunks = 1u << (log_size - OODS_CHUNK_BITS);
  // A power of two of CTAs per column (the chunk factor splits over the warp's bits): about twenty CTAs of
  // four warps per SM over all columns, no more than give every warp work. Fewer chunks than four warps per
  // scheduler: a chunk per CTA instead of per warp.
  const bool quarters = (uint64_t)n_chunks * n_cols < 148ull * 16;
  const uint32_t per_cta = quarters ? 1 : OODS_WARPS;  // chunks
  uint32_t per_col = 1;
  while (per_col * per_cta < n_chunks && (uint64_t)per_col * n_cols < 148ull * 20) per_col <<= 1;
  (quarters ? k_oods_mma<4> : k_oods_mma<16>)<<<dim3(per_col, n_cols), 32 * OODS_WARPS, 0, stream>>>(F, coeffs, stride, partial, n_chunks); note_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_oods_sum<<<(n_cols + 3) / 4, 128, 0, stream>>>(partial, per_col, n_cols, out); note_launch();
  return cudaGetLastError();
}

void arm_quotient_stage_timeout_for_testing() { g_quot_skip_first_item.store(true); }

cudaError_t accumulate_quotients(const DeviceTables& t, uint32_t log_size, uint32_t n_batches, uint32_t n_entries,
                                 const QuotientBatchDev* batches, const uint32_t* const* col_ptrs, const QM31* coeff_c,
                                 uint32_t* out, uint64_t out_stride, cudaStream_t stream, uint32_t* status,
                                 const QuotientBatchDev* one) {
  const size_t smem = QUOT_MAX_ENTRIES * 16;
  // Tensor-core kernel: every batch padded to a multiple of eight entries.
  const uint32_t padded = n_entries + 7 * n_batches;
  const size_t smem_m = (size_t)mma_ring_bytes(QUOT_STAGES) + (size_t)padded * (16 + sizeof(void*));
  // Bulk-staged kernel: the ring, the coefficients and pointers, and the item table (every batch
  // adds at most one partial group).
  const uint32_t item_cap = (n_entries + QB_GROUP - 1) / QB_GROUP + n_batches;
  const size_t smem_b = (size_t)QB_STAGES * QB_GROUP * QB_ROWS * 4 + (size_t)n_entries * (16 + sizeof(void*)) +
                        (size_t)item_cap * sizeof(QbItem);
  // The tensor-core kernel takes whole blocks of 64 rows.
  if ((1ull << log_size) < MMA_ROWS || smem_m > QUOT_SMEM_MAX) {
    k_quotients<<<grid_for(1ull << log_size, 256), 256, smem, stream>>>(PointTable{t.points}, log_size, n_batches, batches,
                                                                        one ? *one : QuotientBatchDev{}, col_ptrs,
                                                                        coeff_c, out, out_stride);
    note_launch();
    return cudaGetLastError();
  }
  // The bulk-staged kernel takes whole 512-row tiles of 16-byte aligned columns (the caller vouches
  // for the pointers by passing `status`) and stores two words at a time. It runs when a caller forces the
  // last variant.
  const bool bulk = status != nullptr && log_size >= 16 && n_batches <= QB_MAX_BATCHES &&
                    n_entries <= QUOT_MAX_ENTRIES && (reinterpret_cast<uintptr_t>(out) & 7) == 0 && out_stride % 2 == 0;
  auto run = [&](int variant) -> cudaError_t {
    const PointTable pts{t.points};
    if (variant == 3 && bulk) {
      // Persistent: as many CTAs as stay resident (three per SM while the shared memory allows).
      const int minb = smem_b <= 70 * 1024 ? 3 : 2;
      const uint32_t n_tiles = (uint32_t)((1ull << log_size) / QB_ROWS);
      const uint32_t g = std::min<uint32_t>(n_tiles, t.sm_count * (uint32_t)minb);
      const int skip = g_quot_skip_first_item.exchange(false) ? 1 : 0;
      if (minb == 3)
        k_quotients_bulk<3><<<g, QB_THREADS, smem_b, stream>>>(pts, log_size, n_batches, batches, col_ptrs, coeff_c, n_entries,
                                                        item_cap, out, out_stride, status, skip);
      else
        k_quotients_bulk<2><<<g, QB_THREADS, smem_b, stream>>>(pts, log_size, n_batches, batches, col_ptrs, coeff_c, n_entries,
                                                        item_cap, out, out_stride, status, skip);
    } else {
      // Persistent: four CTAs per SM, each warp 64 rows at a time. Sixteen-byte copies where the caller
      // vouches for the columns and the output allows them, or the kernel finds them aligned.
      const uint32_t blocks = (uint32_t)((1ull << log_size) / MMA_ROWS), per_cta = MMA_THREADS / 32;
      const uint32_t g = std::min<uint32_t>((blocks + per_cta - 1) / per_cta, t.sm_count * 4);
      const bool aligned = status != nullptr && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && out_stride % 4 == 0;
      (aligned ? k_quotients_mma<false> : k_quotients_mma<true>)<<<g, MMA_THREADS, smem_m, stream>>>(
          pts, log_size, n_batches, batches, one ? *one : QuotientBatchDev{}, col_ptrs, coeff_c, padded, out, out_stride);
    }
    note_launch();
    return cudaGetLastError();
  };
  // The tensor-core kernel is the fastest variant at every size, so nothing is tuned: variants 1 and 2
  // are the same kernel, the last one the bulk-staged kernel when forced.
  return tuned_run(TUNE_QUOTIENTS, log_size, n_entries, log_size >= 16 ? 4 : 1, false, stream, run);
}

cudaError_t fold_circle_into_line(const DeviceTables& t, uint32_t src_log, const uint32_t* src, uint64_t src_stride,
                                  QM31 alpha, uint32_t* dst, uint64_t dst_stride, bool accumulate,
                                  cudaStream_t stream) {
  TwiddleView itv = t.view(src_log, true);
  k_fold_circle<<<grid_for(1ull << (src_log - 1), 256), 256, 0, stream>>>(itv, src_log - 1, src, src_stride, alpha,
                                                                          qsq(alpha), dst, dst_stride, accumulate); note_launch();
  return cudaGetLastError();
}

cudaError_t fold_line(const DeviceTables& t, uint32_t src_log, const uint32_t* src, uint64_t src_stride, QM31 alpha,
                      uint32_t* dst, uint64_t dst_stride, cudaStream_t stream) {
  // Source line domain halfOdds(src_log): its tower layer is the line layer 0 of
  // the circle domain of log src_log + 1.
  TwiddleView itv = t.view(src_log + 1, true);
  k_fold_line<<<grid_for(1ull << (src_log - 1), 256), 256, 0, stream>>>(itv, src_log - 1, src, src_stride, alpha, dst,
                                                                        dst_stride); note_launch();
  return cudaGetLastError();
}

cudaError_t gather_words(const GatherItem* items, uint32_t n, uint32_t* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_gather_words<<<(n + 255) / 256, 256, 0, stream>>>(items, n, out); note_launch();
  return cudaGetLastError();
}

cudaError_t gather_hashes(const HashGatherItem* items, uint32_t n, uint8_t* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_gather_hashes<<<(n + 255) / 256, 256, 0, stream>>>(items, n, out); note_launch();
  return cudaGetLastError();
}

}  // namespace sb
