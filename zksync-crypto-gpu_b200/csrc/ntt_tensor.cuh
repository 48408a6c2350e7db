// NTT passes whose radix rounds run on the tensor cores (included by ntt.cu).
//
// A radix-2^r round is, for every group of 2^r values, r butterfly stages whose twiddles are, for
// block m of the round's first stage, the powers g^(2^u) of one element g = g_m times constant
// roots of unity.  So the round is a diagonal and a constant matrix:
//   n2b:  out = F (g^j v_j)      b2n:  out_j = g^j (F' v)_j
// with F the stages at block 0 (a 2^r-point DFT in the stages' order; F' the b2n stages).  F is the
// byte contraction of tcgen.cuh: a row of 2^r words (K = 8 * 2^r bytes) gives 8 * 2^r digit sums.
// What is left for the integer pipes is, per value and round, one carry-and-reduce and one twiddle
// product, where radix-2 butterflies need r/2 products and r additions with their corrections.
// Round 0 of a pass has one block per tile, so its g and N^-1 go into the tile's own matrix and
// cost nothing per value.
//
// One CTA of two warpgroups owns tiles of 2^12 elements: 256 threads, 16 values each.  Tile index e
// = (mid, w): the pass's k stages act on mid, w are the 2^log_w = 2^(12-k) contiguous elements of a
// strided pass.  A round on the bits [p, p + r) reads the tile as 2^(12-r) rows; a row is one TMEM
// lane of one 128-row product, so a thread gets its rows' values from TMEM, multiplies by the next
// round's twiddles and stores them straight into the next round's operand rows: one CTA barrier a
// round.  The next column's elements are copied into the operand rows while the last round's values
// are reduced and written.
//
// Bound: latency between the rounds of the two CTAs an SM holds (TMEM: 256 of 512 columns each), then
// the integer pipes (ALU and fmaheavy 41-48%, DRAM 21-37%, tensor 10-17% of peak); the waits for the
// products cost 15%.  About 45 thread instructions per value and round of 4 stages, where the
// radix-16 register rounds (ntt_tile.cuh) take 104.  Measured on B200, us, register rounds -> this:
// inverse 2^20 x 128: 2731 -> 1610; 2^22 x 176: 16547 -> 10900; forward coset 2^20 x 128: 2672 -> 1645.
// 512 threads with 8 values each instead: 14% slower (12.9 ms at 2^22 x 176): a thread's share of
// the addresses and waits does not shrink with its values.
#pragma once
#include "ntt_tile.cuh"
#include "tcgen.cuh"

namespace glc {

static constexpr uint32_t TT_LOG = 12;  // log2 of a tile's elements
static constexpr uint32_t TT_THREADS = 256;
static constexpr uint32_t TT_COLUMNS = 256;  // TMEM: 2^(12-r) / 128 products of 8 * 2^r columns
static constexpr uint32_t TT_MAX_ROUNDS = 4;
static constexpr uint32_t TT_MAX_COLS = 16;  // columns that share a CTA's matrix and twiddles
// F of radix 4, 8 and 16 as operand B, then its coefficients
__host__ __device__ constexpr uint32_t dft_bytes(uint32_t r) { return 64u << (2 * r); }
__host__ __device__ constexpr uint32_t dft_offset(uint32_t r) { return r == 2 ? 0 : r == 3 ? dft_bytes(2) : dft_bytes(2) + dft_bytes(3); }
static constexpr uint32_t DFT_MATRICES = dft_bytes(2) + dft_bytes(3) + dft_bytes(4);
static constexpr uint32_t DFT_BYTES = DFT_MATRICES + DFT_MATRICES / 8;
// the largest digit sum: 128 products of bytes
static_assert(128u * 255 * 255 <= tc::digit_limit, "a digit sum is too large");
// Operand rows: 16-byte chunk c (values 2c, 2c+1) of row x at c * lbo(r) + x * 16.  The 16 bytes of
// padding a chunk keep a half-warp that writes 8 chunks of one row on different banks.
__host__ __device__ constexpr uint32_t tt_lbo(uint32_t r) { return (16u << (TT_LOG - r)) + 16; }
static constexpr uint32_t TT_A_BYTES = tt_lbo(4) * 8;
static constexpr uint32_t TT_B0 = TT_A_BYTES, TT_B = TT_B0 + dft_bytes(4), TT_TABLES = TT_B + DFT_MATRICES;

struct TensorPass {
  const uint64_t *in;
  uint64_t *out;
  uint64_t in_stride, out_stride;
  uint32_t num_cols, cols_per_cta;
  uint32_t log_n, s0, k, log_w, log_m;
  uint32_t rounds;
  uint32_t r[TT_MAX_ROUNDS], t[TT_MAX_ROUNDS];  // round q covers stages s0 + t[q] .. + r[q] - 1
  uint32_t table[TT_MAX_ROUNDS];                // its twiddles' place in shared memory (words), q >= 1
  uint32_t plain_first;  // round 0 is F itself
  uint32_t radices;      // bit r: some round uses F of radix 2^r
  uint32_t last;         // canonical output
  uint32_t staged;       // contiguous n2b pass whose output is not 32-byte aligned: a thread's 16
                         // consecutive values go out through shared memory instead of 32-byte stores
  uint32_t smem_bar;     // mbarrier, TMEM address, the barrier of tc::finish: 8 bytes each
  unsigned long long *expired;  // counts the waits that gave up
  const uint64_t *tw;
  const uint8_t *dft;
  uint64_t scale;        // N^-1 on an inverse's last pass, else 1
  PassArgs coset;        // fold: the coset factors ride on the twiddles
};

// Twiddle j of block m of a round with nblk blocks: word j * (nblk + 2) + m of its table (two words
// of padding a row: a half-warp reading 8 rows hits different banks).
__host__ __device__ constexpr uint32_t tt_table_words(uint32_t r, uint32_t nblk) { return (nblk + 2) << r; }

// g of block m (of the round's first stage) of round q
__device__ __forceinline__ uint64_t tt_twiddle(const TensorPass &a, uint32_t q, uint64_t m) {
  const uint64_t g = a.tw[m << (a.r[q] - 1)];
  return a.coset.fold ? mul(g, coset_power(a.coset, 1u << (a.log_n - a.s0 - a.t[q] - a.r[q]))) : g;
}

// The twiddles of round q >= 1 for the tile's blocks.
__device__ __forceinline__ void tt_build_table(const TensorPass &a, uint32_t q, uint64_t hi, uint64_t *table) {
  const uint32_t r = a.r[q], t = a.t[q], nblk = 1u << t, row = nblk + 2;
  for (uint32_t m = threadIdx.x; m < nblk; m += TT_THREADS) {
    uint64_t pw[16];
    pw[0] = 1;
    pw[1] = tt_twiddle(a, q, (hi << t) + m);
    pw[2] = sqr(pw[1]);
    pw[3] = mul(pw[1], pw[2]);
    if (r >= 3) {
      pw[4] = sqr(pw[2]);
#pragma unroll
      for (int j = 1; j < 4; j++) pw[4 + j] = mul(pw[j], pw[4]);
      if (r >= 4) {
        pw[8] = sqr(pw[4]);
#pragma unroll
        for (int j = 1; j < 8; j++) pw[8 + j] = mul(pw[j], pw[8]);
      }
    }
#pragma unroll
    for (uint32_t j = 0; j < 16; j++)
      if (j < (1u << r)) table[j * row + m] = pw[j];
  }
}

// Round 0's matrix for this tile: F's coefficients times g^j (n2b: of input j, b2n: of output j)
// and the scale, spread into digits.
template <bool DIF>
__device__ __forceinline__ void tt_build_first(const TensorPass &a, uint64_t hi, uint8_t *matrix) {
  const uint32_t r = a.r[0], n = 1u << r;
  if (threadIdx.x >= n * n) return;
  const uint32_t o = threadIdx.x >> r, i = threadIdx.x & (n - 1);
  uint64_t c = reinterpret_cast<const uint64_t *>(a.dft + DFT_MATRICES + dft_offset(r) / 8)[threadIdx.x];
  c = mul(c, a.scale);
  uint64_t g = tt_twiddle(a, 0, hi);
#pragma unroll 1
  for (uint32_t e = DIF ? o : i; e; e >>= 1, g = sqr(g))
    if (e & 1) c = mul(c, g);
  // digit d of c * 2^(8b), b = 0..7, is byte b of the 8 bytes at row 8 o + d
  uint64_t digits[8] = {};
#pragma unroll
  for (int b = 0; b < 8; b++) {
    c = canon(c);
#pragma unroll
    for (int d = 0; d < 8; d++) digits[d] |= (uint64_t)((c >> (8 * d)) & 255) << (8 * b);
    c = add(c << 8, (c >> 56) * EPS);
  }
#pragma unroll
  for (uint32_t d = 0; d < 8; d++)
    *reinterpret_cast<uint64_t *>(matrix + (i >> 1) * (128u << r) + (8 * o + d) * 16 + (i & 1) * 8) = digits[d];
}

__device__ __forceinline__ void tt_store(uint32_t addr, uint64_t v) {
  asm volatile("st.shared.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

// One round of the column's tile after its products are done: 16 values a thread, four at a time,
// the next four loading from TMEM meanwhile.  The next round (n2b: q + 1, b2n: q - 1) has r2 bits;
// the last one writes the column's results instead.
template <uint32_t R, bool DIF, bool FINAL>
__device__ __forceinline__ void tt_round(const TensorPass &a, uint32_t q, uint32_t tmem, uint32_t smem_a,
                                         const uint64_t *smem, uint64_t *dst) {
  const uint32_t lane = threadIdx.x & 127, first_product = (threadIdx.x >> 7) * (16u >> R);
  const uint32_t p = a.k - a.t[q] - R + a.log_w;
  const uint32_t r2 = FINAL ? 0 : a.r[DIF ? q - 1 : q + 1];
  const uint32_t p2 = DIF ? p + R : p - r2;
  const uint32_t columns = tmem + first_product * (8u << R);  // this thread's values in order
  uint32_t to = 0, step = 0, tw_row = 0;
  const uint64_t *tw = nullptr;
  uint64_t *out = nullptr;
  uint64_t out_step = 0;
  // place the results of row `product * 128 + lane`
  auto locate = [&](uint32_t product) {
    const uint32_t row = product * 128 + lane;
    const uint32_t low = row & ((1u << p) - 1), high = row >> p;
    if (!FINAL) {
      // value i goes to row row0 + (i << step) of the next round's operand, as value j2 of the row
      uint32_t j2, row0;
      if (DIF) {
        j2 = high & ((1u << r2) - 1);
        row0 = ((high >> r2) << p2) | low;
      } else {
        j2 = low >> p2;
        row0 = (high << (R + p2)) | (low & ((1u << p2) - 1));
      }
      step = 16u << (DIF ? p : p2);
      to = smem_a + (j2 >> 1) * tt_lbo(r2) + (j2 & 1) * 8 + row0 * 16;
      // n2b multiplies by the next round's twiddles (block (high, i), power j2), b2n by this one's
      // (block high, power i)
      tw = DIF ? smem + a.table[q] + high : smem + a.table[q + 1] + j2 * ((1u << (a.t[q] + R)) + 2) + (high << R);
      tw_row = (1u << a.t[q]) + 2;
    } else {
      out = dst + ((uint64_t)(((high << (p + R)) | low) >> a.log_w) << a.log_m) + (low & ((1u << a.log_w) - 1));
      out_step = 1ull << (p - a.log_w + a.log_m);
    }
  };
  auto emit = [&](const uint32_t (&d)[32], uint32_t c) {
    const uint32_t i = 4 * c & ((1u << R) - 1);
    if (i == 0) locate(first_product + (4 * c >> R));
    uint64_t v[4];
#pragma unroll
    for (uint32_t x = 0; x < 4; x++) v[x] = tc::reduce_digits(d + 8 * x);
    if (!FINAL) {
      if (DIF) {
#pragma unroll
        for (uint32_t x = 0; x < 4; x++, tw += tw_row)
          if (i + x > 0) v[x] = mul(v[x], *tw);
      } else {
#pragma unroll
        for (uint32_t x = 0; x < 4; x += 2) {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(tw + i + x);
          v[x] = mul(v[x], w.x);
          v[x + 1] = mul(v[x + 1], w.y);
        }
      }
#pragma unroll
      for (uint32_t x = 0; x < 4; x++, to += step) tt_store(to, v[x]);
    } else {
      if (a.last) {
#pragma unroll
        for (uint32_t x = 0; x < 4; x++) v[x] = canon(v[x]);
      }
      if (!DIF && a.staged) {
        // value i of row x in slot 16 x + (i ^ x mod 16): no bank conflicts either way
#pragma unroll
        for (uint32_t x = 0; x < 4; x++) tt_store(smem_a + (lane + first_product * 128) * 128 + (((i + x) ^ (lane & 15)) * 8), v[x]);
      } else if (!DIF && a.log_m == 0) {
        asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(out + i), "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3])
                     : "memory");
      } else {
#pragma unroll
        for (uint32_t x = 0; x < 4; x++, out += out_step) *out = v[x];
      }
    }
  };
  uint32_t x[32], y[32];
  tc::ld32(x, columns);
  tc::ld_wait(x);
  tc::ld32(y, columns + 32);
  emit(x, 0);
  tc::ld_wait(y);
  tc::ld32(x, columns + 64);
  emit(y, 1);
  tc::ld_wait(x);
  tc::ld32(y, columns + 96);
  emit(x, 2);
  tc::ld_wait(y);
  emit(y, 3);
}

template <bool DIF, bool FINAL>
__device__ __forceinline__ void tt_round_any(const TensorPass &a, uint32_t q, uint32_t tmem, uint32_t smem_a,
                                             const uint64_t *smem, uint64_t *dst) {
  if (a.r[q] == 4)
    tt_round<4, DIF, FINAL>(a, q, tmem, smem_a, smem, dst);
  else if (a.r[q] == 3)
    tt_round<3, DIF, FINAL>(a, q, tmem, smem_a, smem, dst);
  else
    tt_round<2, DIF, FINAL>(a, q, tmem, smem_a, smem, dst);
}

template <bool DIF>
__global__ void __launch_bounds__(TT_THREADS, 2) ntt_tensor_kernel(const __grid_constant__ TensorPass a) {
  extern __shared__ __align__(128) uint8_t tt_smem[];
  uint64_t *const words = reinterpret_cast<uint64_t *>(tt_smem);
  const uint32_t smem_a = tc::smem_addr(tt_smem);
  const uint32_t group = threadIdx.x >> 7;
  const uint32_t bar = smem_a + a.smem_bar, slot = bar + 8;
  const uint32_t log_tiles = a.log_m - a.log_w;  // strided pass: tiles of one hi
  const uint64_t hi = blockIdx.x >> log_tiles;
  const uint64_t base_i = (hi << (a.log_n - a.s0)) + ((uint64_t)(blockIdx.x & ((1u << log_tiles) - 1)) << a.log_w);
  const uint32_t col0 = blockIdx.y * a.cols_per_cta, col1 = min(col0 + a.cols_per_cta, a.num_cols);

  // copies a column's tile into the rows of the first round executed
  const uint32_t first = DIF ? a.rounds - 1 : 0;
  const uint32_t r0 = a.r[first], p0 = a.k - a.t[first] - r0 + a.log_w;
  auto row_addr = [&](uint32_t e) {  // additive over disjoint bits of e
    const uint32_t j = (e >> p0) & ((1u << r0) - 1);
    return (j >> 1) * tt_lbo(r0) + (j & 1) * 8 + (((e >> (p0 + r0)) << p0) | (e & ((1u << p0) - 1))) * 16;
  };
  auto column_index = [&](uint32_t e) { return ((uint64_t)(e >> a.log_w) << a.log_m) + (e & ((1u << a.log_w) - 1)); };
  const uint32_t my_row = smem_a + row_addr(threadIdx.x);
  const uint64_t *const my_src = a.in + base_i + column_index(threadIdx.x);
  // elements threadIdx.x + 256 u: equally far apart in the column (log_w <= 8), and the bits of u
  // add their distances in the rows
  const uint64_t src_step = (uint64_t)(TT_THREADS >> a.log_w) << a.log_m;
  const uint32_t row1 = row_addr(TT_THREADS), row2 = row_addr(2 * TT_THREADS), row4 = row_addr(4 * TT_THREADS),
                 row8 = row_addr(8 * TT_THREADS);
  auto copy_column = [&](uint32_t col) {
    const uint64_t *src = my_src + (uint64_t)col * a.in_stride;
#pragma unroll
    for (uint32_t u = 0; u < 16; u++, src += src_step) {
      const uint32_t row = my_row + (u & 1 ? row1 : 0) + (u & 2 ? row2 : 0) + (u & 4 ? row4 : 0) + (u & 8 ? row8 : 0);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(row), "l"(src) : "memory");
    }
  };
  if (col0 < col1) copy_column(col0);

  for (uint32_t r = 2; r <= 4; r++)
    if (a.radices >> r & 1)
      for (uint32_t i = threadIdx.x; i < dft_bytes(r) / 16; i += TT_THREADS)
        reinterpret_cast<uint4 *>(tt_smem + TT_B + dft_offset(r))[i] = reinterpret_cast<const uint4 *>(a.dft + dft_offset(r))[i];
  if (!a.plain_first) tt_build_first<DIF>(a, hi, tt_smem + TT_B0);
  for (uint32_t q = 1; q < a.rounds; q++) tt_build_table(a, q, hi, words + a.table[q]);
  if (threadIdx.x < 32) tc::tmem_alloc<TT_COLUMNS>(slot);
  if (threadIdx.x == 0) tc::mbar_init(bar, 2);  // both groups' products: either group overwrites any row
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(slot) : "memory");
  const uint32_t tmem_lanes = tmem + ((threadIdx.x & 96) << 16);  // this warp's quarter of the lanes
  uint32_t phase = 0;
  for (uint32_t col = col0; col < col1; col++) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (uint32_t n = 0; n < a.rounds; n++) {
      const uint32_t q = DIF ? a.rounds - 1 - n : n;
      const uint32_t r = a.r[q];
      tc::fence_smem();
      tc::fence_before();
      __syncthreads();
      if ((threadIdx.x & 127) == 0) {
        tc::fence_after();
        const uint32_t cols = 8u << r, lbo = tt_lbo(r);
        const uint64_t db = tc::operand(smem_a + (q || a.plain_first ? TT_B + dft_offset(r) : TT_B0), cols * 16);
        for (uint32_t h = 0; h < (16u >> r); h++) {
          const uint32_t product = group * (16u >> r) + h;
          const uint64_t da = tc::operand(smem_a + product * 2048, lbo);
          for (uint32_t kk = 0; kk < (1u << r) / 4; kk++)
            tc::mma(tmem + product * cols, da + 2 * kk * (lbo >> 4), db + 2 * kk * cols, tc::idesc(cols), kk > 0);
        }
        tc::commit(bar);
      }
      __syncwarp();
      tc::mbar_wait(bar, phase, a.expired);
      if (n + 1 < a.rounds) {
        tt_round_any<DIF, false>(a, q, tmem_lanes, smem_a, words, nullptr);
      } else {
        // the rows are free: every product is done
        uint64_t *const dst = a.out + (uint64_t)col * a.out_stride + base_i;
        if (!a.staged && col + 1 < col1) copy_column(col + 1);
        tt_round_any<DIF, true>(a, q, tmem_lanes, smem_a, words, dst);
        if (a.staged) {
          __syncthreads();
#pragma unroll
          for (uint32_t e = threadIdx.x; e < (1u << TT_LOG); e += TT_THREADS) dst[e] = words[e ^ ((e >> 4) & 15)];
          __syncthreads();
          if (col + 1 < col1) copy_column(col + 1);
        }
      }
    }
  }
  tc::finish<TT_COLUMNS>(tmem, phase, bar + 16, (threadIdx.x & 127) == 0, 2, a.expired);
}

// ---- host side ----

// F (n2b) or F' (b2n) of radix 2^r for the transform whose 16th root of unity is w16, as operand B:
// digit d of output o is row n = 8 o + d; byte b of input i is column k = 8 i + b, in chunk k / 16.  coefs[o 2^r + i] are the coefficients themselves.
inline void build_dft_matrix(uint8_t *out, uint64_t *coefs, uint32_t r, bool b2n, uint64_t w16) {
  const uint32_t n = 1u << r;
  for (uint32_t i = 0; i < n; i++) {
    uint64_t v[16] = {};
    v[i] = 1;
    for (uint32_t uu = 0; uu < r; uu++) {
      const uint32_t u = b2n ? r - 1 - uu : uu, bit = r - 1 - u;
      for (uint32_t j = 0; j < n; j++) {
        if (j & (1u << bit)) continue;
        // block jj's twiddle w_{2^(u+1)}^bitrev_u(jj)
        const uint32_t jj = j >> (r - u);
        uint32_t rev = 0;
        for (uint32_t x = 0; x < u; x++) rev |= ((jj >> x) & 1u) << (u - 1 - x);
        const uint64_t w = h_pow(w16, (uint64_t)rev << (3 - u));
        const uint64_t x = v[j], y = v[j | (1u << bit)];
        if (!b2n) {
          const uint64_t yw = h_mul(y, w);
          v[j] = (uint64_t)(((unsigned __int128)x + yw) % P);
          v[j | (1u << bit)] = (uint64_t)(((unsigned __int128)x + P - yw) % P);
        } else {
          v[j] = (uint64_t)(((unsigned __int128)x + y) % P);
          v[j | (1u << bit)] = h_mul((uint64_t)(((unsigned __int128)x + P - y) % P), w);
        }
      }
    }
    for (uint32_t o = 0; o < n; o++) {
      uint64_t coef = v[o];
      coefs[o * n + i] = coef;
      for (uint32_t b = 0; b < 8; b++, coef = h_mul(coef, 256)) {
        const uint32_t k = 8 * i + b;
        for (uint32_t d = 0; d < 8; d++) out[(k >> 4) * (8 * n * 16) + (8 * o + d) * 16 + (k & 15)] = (uint8_t)(coef >> (8 * d));
      }
    }
  }
}
// The stages of a pass as rounds of 4, 3 and 2 stages (k >= 2).
inline uint32_t tt_split(uint32_t k, uint32_t *r) {
  uint32_t n = (k + 3) / 4;
  for (uint32_t q = 0; q < n; q++) r[q] = k / n + (q < k % n ? 1 : 0);
  return n;
}

// The pass over stages s0 .. s0 + k - 1 of a batch of `cols` NTTs on the tensor cores: all 12 stages
// left (contiguous tiles) or the first k (strided).
inline int tt_launch_pass(const DeviceTables *t, uint32_t s0, uint32_t k, bool first, bool last, const uint64_t *in,
                          uint64_t *out, uint64_t in_stride, uint64_t out_stride, uint32_t cols, uint32_t log_n,
                          bool bitrev_inputs, bool inverse, uint32_t log_ext, uint32_t coset_idx,
                          cudaStream_t stream) {
  TensorPass a{};
  a.in = first ? in : out;
  a.in_stride = first ? in_stride : out_stride;
  a.out = out;
  a.out_stride = out_stride;
  a.num_cols = cols;
  a.log_n = log_n;
  a.s0 = s0;
  a.k = k;
  a.log_m = log_n - s0 - k;
  a.log_w = a.log_m ? TT_LOG - k : 0;
  a.rounds = tt_split(k, a.r);
  a.coset.dif = bitrev_inputs;
  a.coset.log_n = log_n;
  a.coset.fold = log_ext > 0;
  a.coset.log_ext = log_ext;
  a.coset.coset = coset_idx;
  a.coset.g_lo = t->g_lo;
  a.coset.g_hi = t->g_hi;
  a.coset.w_lo = t->w_lo;
  a.coset.w_hi = t->w_hi;
  a.last = last;
  a.scale = inverse && last ? t->inv_sizes[log_n] : 1;
  // round 0 at stage 0 has the twiddles w^0
  a.plain_first = s0 == 0 && !a.coset.fold && a.scale == 1;
  uint32_t words = TT_TABLES / 8;
  for (uint32_t q = 0, st = 0; q < a.rounds; st += a.r[q++]) {
    a.t[q] = st;
    a.table[q] = words;
    if (q) words += tt_table_words(a.r[q], 1u << st);
    if (q || a.plain_first) a.radices |= 1u << a.r[q];
  }
  a.smem_bar = words * 8;
  const size_t smem = (size_t)a.smem_bar + 24;
  a.expired = t->expired;
  a.staged = !bitrev_inputs && a.log_m == 0 && ((reinterpret_cast<uintptr_t>(out) & 31) || (out_stride & 3));
  a.tw = inverse ? t->tw_inv : t->tw_fwd;
  a.dft = t->dft + ((inverse ? 2 : 0) + (bitrev_inputs ? 1 : 0)) * DFT_BYTES;
  const uint32_t tiles = 1u << (log_n - TT_LOG);
  a.cols_per_cta = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(TT_MAX_COLS, ((uint64_t)tiles * cols + 295) / 296));
  const uint32_t groups = (cols + a.cols_per_cta - 1) / a.cols_per_cta;
  for (uint32_t y0 = 0; y0 < groups; y0 += 65535) {
    TensorPass b = a;
    const uint32_t n = std::min<uint32_t>(65535, groups - y0);
    b.in += (uint64_t)y0 * a.cols_per_cta * a.in_stride;
    b.out += (uint64_t)y0 * a.cols_per_cta * a.out_stride;
    b.num_cols = std::min<uint32_t>(cols - y0 * a.cols_per_cta, n * a.cols_per_cta);
    if (bitrev_inputs)
      ntt_tensor_kernel<true><<<dim3(tiles, n), TT_THREADS, smem, stream>>>(b);
    else
      ntt_tensor_kernel<false><<<dim3(tiles, n), TT_THREADS, smem, stream>>>(b);
    const int e = last_launch_error();
    if (e) return e;
  }
  return 0;
}

}  // namespace glc
