// The 22 partial rounds of the Poseidon2 permutation on the fifth-generation tensor cores.
// Included by poseidon2.cu, whose S-box, 96-bit sums and round constants it uses.
//
// In a partial round only element 0 goes through the S-box, so the rounds are linear in the state
// on entry v and the 22 S-box outputs x_0 .. x_21.  With M = M_I, N = M with column 0 cleared and
// u = M e_0, the input of S-box k and the state after the last round are
//   y_k = e_0^T N^k v + sum_{i<k} (e_0^T N^(k-1-i) u) x_i + rc[4+k][0]        (k >= 1)
//   out = N^22 v + sum_i N^(21-i) u x_i + rc[26],
// and v[0] itself only enters through x_0 (N e_0 = 0).  These constant matrices over the field
// become matrices of bytes: the byte b of an input word w, times 2^(8b) times the coefficient,
// reduced mod p, is 8 bytes of the output word.  A row of 8-bit integers (11 state words, the
// S-box outputs, and a constant 1 whose coefficient is the round constant) times such a matrix is
// one exact u8 x u8 -> s32 tensor-core contraction (kind::i8), whose 8 result columns per output
// word are the word's base-256 digits before carries, each below 2^24 (checked when the matrix is
// built).
//
// A warpgroup holds 128 permutations, one per thread and TMEM lane.  Each thread writes its row of
// bytes (a uint64_t is its own digit string) to shared memory; one thread issues the products;
// every thread reads its digits back with tcgen05.ld and carries them into a 96-bit sum.  Rounds 0
// and 1 are computed directly, rounds 2 .. 21 in five blocks of four: the tensor cores give each
// block's four S-box inputs from everything before the block, and the terms inside the block have
// small coefficients (17, 11, 31718: e_0^T N^m u) and are added directly.
//
// Bound: the integer pipes (leaves: fmaheavy 67%, ALU 56%) with five warpgroups an SM, as many as the
// operand rows leave room for in shared memory and one 96-column result each in TMEM; tensor pipe 4%.  A
// permutation takes 12.2 K instructions, 14.2 K without (the 22 internal layers were 3 K).  Measured
// on B200: 2^22 nodes 2532 -> 2365 us, leaves of 176 columns at 2^22 54.6 -> 52.8 ms, registers' worth
// of addresses kept out of the full rounds included (1.69 -> 1.71 G permutations/s).  Four groups with
// 128 registers each: 1.68 against 1.78 G permutations/s with five (permutations alone).
#pragma once
#include "tcgen.cuh"

namespace glc {
namespace tc {

static constexpr uint32_t TILE = 128;      // permutations of a warpgroup
static constexpr uint32_t GROUPS = 5;      // warpgroups of a CTA
static constexpr uint32_t BLOCKS = 5;      // blocks of four rounds
// A row is 17 chunks of 16 bytes (two words each): 1, v1..v11 | x0, x1 | x2..x21.  A K step covers
// two chunks: steps 0..2 the state, step 3 x0, x1 and a chunk whose coefficients are zero, step
// 4 + b block b's four S-box outputs.
static constexpr uint32_t CHUNKS = 17;
static constexpr uint32_t A_BYTES = TILE * CHUNKS * 16;
static constexpr uint32_t Y_COLS = 32, OUT_COLS = 96;  // TMEM columns: 4 and 12 words of 8 digits
// matrix of block b: (7 + 2b) chunks x 32 rows; of the output: 17 chunks x 96 rows; zeros for step 3
__host__ __device__ constexpr uint32_t y_offset(uint32_t b) { return Y_COLS * 16 * (7 * b + b * (b - 1)); }
static constexpr uint32_t OUT_OFFSET = Y_COLS * 16 * (7 * BLOCKS + BLOCKS * (BLOCKS - 1));
static constexpr uint32_t ZERO_OFFSET = OUT_OFFSET + OUT_COLS * 16 * CHUNKS;
static constexpr uint32_t B_BYTES = ZERO_OFFSET + OUT_COLS * 16;
static constexpr uint32_t SMEM_TAIL = B_BYTES + GROUPS * A_BYTES;  // mbarriers, TMEM address, finish()'s barrier
static constexpr uint32_t SMEM_DRAIN = SMEM_TAIL + 8 * GROUPS + 8;
static constexpr uint32_t SMEM_BYTES = SMEM_DRAIN + 8;

struct Matrices {
  alignas(16) uint8_t b[B_BYTES];
};

constexpr uint64_t c_mul(uint64_t a, uint64_t b) {
  return (uint64_t)((unsigned __int128)a * b % P);
}

// The byte matrices for round constants rc.  Row n of a block's matrix (n = 8 * output + digit)
// at chunk c: bytes b + c * rows * 16 + n * 16.
constexpr Matrices make_matrices(const uint64_t (&rc)[ROUNDS][WIDTH]) {
  constexpr int LOG_MU_MINUS_ONE[WIDTH] = {4, 14, 11, 8, 0, 5, 2, 9, 13, 6, 3, 12};
  Matrices m{};
  uint64_t alpha[22][WIDTH] = {};  // alpha[k] = e_0^T N^k (columns 1..11; column 0 stays 0 for k >= 1)
  uint64_t beta[22] = {};          // beta[m] = e_0^T N^m u
  uint64_t col[22][WIDTH] = {};    // col[m] = N^m u
  uint64_t full[WIDTH][WIDTH] = {};  // N^22, column by column (columns 1..11)
  // v <- N v: the sum of elements 1..11 plus 2^e_i v_i on i >= 1
  auto step = [&](uint64_t (&v)[WIDTH]) {
    unsigned __int128 sum = 0;
    for (uint32_t i = 1; i < WIDTH; i++) sum += v[i];
    const uint64_t s = (uint64_t)(sum % P);
    for (uint32_t i = 0; i < WIDTH; i++)
      v[i] = (uint64_t)((s + (i ? (unsigned __int128)v[i] << LOG_MU_MINUS_ONE[i] : 0)) % P);
  };
  uint64_t u[WIDTH] = {};
  for (uint32_t i = 0; i < WIDTH; i++) u[i] = i ? 1 : 1 + (1ull << LOG_MU_MINUS_ONE[0]);
  for (uint32_t k = 0; k < 22; k++) {
    for (uint32_t i = 0; i < WIDTH; i++) col[k][i] = u[i];
    beta[k] = u[0];
    step(u);
  }
  for (uint32_t j = 1; j < WIDTH; j++) {
    uint64_t v[WIDTH] = {};
    v[j] = 1;
    for (uint32_t k = 0; k < 22; k++) {
      alpha[k][j] = v[0];
      step(v);
    }
    for (uint32_t i = 0; i < WIDTH; i++) full[j][i] = v[i];
  }
  // word w of the row times coefficient `coef` into output word o of the matrix at `off`
  auto put = [&](uint32_t off, uint32_t rows, uint32_t o, uint32_t w, uint64_t coef) {
    for (uint32_t byte = 0; byte < 8; byte++) {
      const uint32_t k = w * 8 + byte;
      for (uint32_t d = 0; d < 8; d++)
        m.b[off + (k >> 4) * rows * 16 + (8 * o + d) * 16 + (k & 15)] = (uint8_t)(coef >> (8 * d));
      coef = c_mul(coef, 256);
    }
  };
  auto put_one = [&](uint32_t off, uint32_t rows, uint32_t o, uint64_t value) {  // the constant 1 is byte 0
    for (uint32_t d = 0; d < 8; d++) m.b[off + (8 * o + d) * 16] = (uint8_t)((value % P) >> (8 * d));
  };
  auto x_word = [](uint32_t i) { return 12 + i; };
  for (uint32_t b = 0; b < BLOCKS; b++)
    for (uint32_t o = 0; o < 4; o++) {
      const uint32_t k = 2 + 4 * b + o, first = 2 + 4 * b;
      put_one(y_offset(b), Y_COLS, o, rc[4 + k][0]);
      for (uint32_t j = 1; j < WIDTH; j++) put(y_offset(b), Y_COLS, o, j, alpha[k][j]);
      for (uint32_t i = 0; i < first; i++) put(y_offset(b), Y_COLS, o, x_word(i), beta[k - 1 - i]);
    }
  for (uint32_t o = 0; o < WIDTH; o++) {
    put_one(OUT_OFFSET, OUT_COLS, o, rc[26][o]);
    for (uint32_t j = 1; j < WIDTH; j++) put(OUT_OFFSET, OUT_COLS, o, j, full[j][o]);
    for (uint32_t i = 0; i < 22; i++) put(OUT_OFFSET, OUT_COLS, o, x_word(i), col[21 - i][o]);
  }
  return m;
}

// The digit sums of every output are at most digit_limit: the sum of a matrix row times 255 is the
// largest.
// (Round constants add at most 255 to a row, which the bound leaves room for.)
constexpr bool digits_fit(const Matrices &m) {
  auto fits = [&](uint32_t off, uint32_t rows, uint32_t chunks) {
    for (uint32_t n = 0; n < rows; n++) {
      uint32_t sum = 0;
      for (uint32_t c = 0; c < chunks; c++)
        for (uint32_t k = 0; k < 16; k++) sum += m.b[off + c * rows * 16 + n * 16 + k];
      if ((sum + 255) * 255 > digit_limit) return false;
    }
    return true;
  };
  for (uint32_t b = 0; b < BLOCKS; b++)
    if (!fits(y_offset(b), Y_COLS, 7 + 2 * b)) return false;
  return fits(OUT_OFFSET, OUT_COLS, CHUNKS);
}

// For the placeholder constants; replaced when constants are installed.
static constexpr Matrices k_matrices = make_matrices(k_placeholder_rc);
static_assert(digits_fit(k_matrices), "a digit sum is too large");
__device__ Matrices d_matrices = k_matrices;

// One warpgroup's share of the CTA's tensor-core resources.  Only the phase is kept; the addresses
// are cheap to compute again (thread() keeps the compiler from holding them in registers, which the
// full rounds need).
extern __shared__ __align__(128) uint8_t smem[];
__device__ __forceinline__ uint32_t thread() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
struct Group {
  uint32_t phase;
  __device__ __forceinline__ static uint32_t index() { return thread() / TILE; }
  __device__ __forceinline__ static bool leader() { return thread() % TILE == 0; }
  __device__ __forceinline__ static uint32_t matrices() { return smem_addr(smem); }
  __device__ __forceinline__ static uint32_t tile() { return smem_addr(smem) + B_BYTES + index() * A_BYTES; }
  // this thread's row in the operand tile (chunk c at row + c * 2048)
  __device__ __forceinline__ static uint32_t row() {
    const uint32_t t = thread();
    return smem_addr(smem) + B_BYTES + (t / TILE) * A_BYTES + (t % TILE) * 16;
  }
  __device__ __forceinline__ static uint32_t bar() { return smem_addr(smem) + SMEM_TAIL + 8 * index(); }
  // the CTA's TMEM, all 512 columns, and the first column of the group, at lane 0 (where the products go)
  __device__ __forceinline__ static uint32_t base() {
    uint32_t base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(base) : "r"(smem_addr(smem) + SMEM_TAIL + 8 * GROUPS) : "memory");
    return base;
  }
  __device__ __forceinline__ static uint32_t tmem() { return base() + index() * OUT_COLS; }
  // the same column at this warp's quarter of the lanes (what it may read)
  __device__ __forceinline__ static uint32_t lanes() { return tmem() + ((thread() % TILE & ~31u) << 16); }
};

// Every thread of the group waits until the products issued so far are done.
__device__ __forceinline__ void wait(Group &g) { mbar_wait(g.bar(), g.phase, &d_expired); }

// Makes the group's shared-memory rows visible to the tensor cores and orders its TMEM reads
// before the products issued next.
__device__ __forceinline__ void publish(const Group &g) {
  asm volatile("fence.proxy.async.shared::cta;\n\ttcgen05.fence::before_thread_sync;\n\tbar.sync %0, 128;" ::"r"(1 + g.index())
               : "memory");
}

__device__ __forceinline__ void store_words(uint32_t row, uint32_t chunk, uint64_t x, uint64_t y) {
  asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(row + chunk * (TILE * 16)), "l"(x), "l"(y) : "memory");
}

// 8 digits (each below 2^24) carried into a 96-bit sum
__device__ __forceinline__ w96 carry_digits(const uint32_t *v) {
  const uint32_t p0 = v[0] + (v[1] << 8), p1 = v[2] + (v[3] << 8), p2 = v[4] + (v[5] << 8), p3 = v[6] + (v[7] << 8);
  w96 r;
  asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;"
      : "=&r"(r.l0), "=&r"(r.l1), "=&r"(r.h)
      : "r"(p0), "r"(p1 << 16), "r"(p2), "r"(__byte_perm(p1, p3, 0x5432)), "r"(p3 >> 16));
  return r;
}
// a + x * m for small m
__device__ __forceinline__ w96 mad_small(w96 a, uint64_t x, uint32_t m) {
  const uint64_t t0 = madw(lo32(x), m, (uint64_t)a.l0);
  const uint64_t t1 = madw(hi32(x), m, (uint64_t)a.l1 + hi32(t0));
  return {lo32(t0), lo32(t1), a.h + hi32(t1)};
}

// D = A B over `steps` K steps with the matrix at `b` (n rows), by one thread
__device__ __forceinline__ void multiply(const Group &g, uint32_t b, uint32_t n, uint32_t steps) {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint64_t da = operand(g.tile(), TILE * 16), db = operand(b, n * 16);
  const uint32_t tmem = g.tmem();
  const uint32_t a_chunk = TILE * 16 >> 4, b_chunk = n * 16 >> 4;
#pragma unroll
  for (uint32_t k = 0; k < 3; k++) mma(tmem, da + 2 * k * a_chunk, db + 2 * k * b_chunk, idesc(n), k > 0);
  mma(tmem, da + 6 * a_chunk, operand(b + 6 * n * 16, g.matrices() + ZERO_OFFSET - (b + 6 * n * 16)), idesc(n), true);
  for (uint32_t k = 4; k < steps; k++)
    mma(tmem, da + (2 * k - 1) * a_chunk, db + (2 * k - 1) * b_chunk, idesc(n), true);
  commit(g.bar());
}

// The partial rounds of the group's 128 permutations; s[0] carries round 4's constant.  Every
// thread of the group calls it.
__device__ __forceinline__ void partial_rounds(uint64_t s[WIDTH], Group &g) {
  uint32_t row = g.row();
  store_words(row, 0, 1, s[1]);
#pragma unroll
  for (int c = 1; c < 6; c++) store_words(row, c, s[2 * c], s[2 * c + 1]);
  // round 5's S-box input directly: N's row 0 is all ones on elements 1..11
  {
    const w96 a = w_add(w_add64(s[1], s[2]), w_add64(s[3], s[4])), b = w_add(w_add64(s[5], s[6]), w_add64(s[7], s[8]));
    const w96 c = w_add(w_add64(s[9], s[10]), w_add64(s[11], c_rc[5][0]));
    const uint64_t x0 = sbox(s[0]);
    const uint64_t x1 = sbox(w_red(mad_small(w_add(w_add(a, b), c), x0, 17)));
    store_words(row, 6, x0, x1);
  }
#pragma unroll 1
  for (uint32_t b = 0; b < BLOCKS; b++) {
    publish(g);
    if (g.leader()) multiply(g, g.matrices() + y_offset(b), Y_COLS, 4 + b);
    __syncwarp();
    wait(g);
    uint32_t v[32];
    ld32(v, g.lanes());
    ld_wait(v);
    const uint64_t xa = sbox(w_red(carry_digits(v)));
    const uint64_t xb = sbox(w_red(mad_small(carry_digits(v + 8), xa, 17)));
    const uint64_t xc = sbox(w_red(mad_small(mad_small(carry_digits(v + 16), xa, 11), xb, 17)));
    const uint64_t xd =
        sbox(w_red(mad_small(mad_small(mad_small(carry_digits(v + 24), xa, 31718), xb, 11), xc, 17)));
    row = g.row();
    store_words(row, 7 + 2 * b, xa, xb);
    store_words(row, 8 + 2 * b, xc, xd);
  }
  publish(g);
  if (g.leader()) multiply(g, g.matrices() + OUT_OFFSET, OUT_COLS, 4 + BLOCKS);
  __syncwarp();
  wait(g);
#pragma unroll
  for (int q = 0; q < 3; q++) {
    uint32_t v[32];
    ld32(v, g.lanes() + 32 * q);
    ld_wait(v);
#pragma unroll
    for (int i = 0; i < 4; i++) s[4 * q + i] = w_red(carry_digits(v + 8 * i));
  }
}

__device__ __forceinline__ void permutation(uint64_t s[WIDTH], Group &g) {
  external_layer<true>(s, 0);
#pragma unroll 1
  for (int q = 0; q < 8; q++) {
#pragma unroll
    for (int i = 0; i < WIDTH; i++) s[i] = sbox(s[i]);
    const int r = q < 4 ? q : q + 22;
    external_layer<true>(s, q == 7 ? RC_ROW_NONE : (q == 3 ? RC_ROW_PARTIAL_ENTRY : (uint32_t)(r + 1)));
    if (q == 3) partial_rounds(s, g);
  }
#pragma unroll
  for (int i = 0; i < WIDTH; i++) s[i] = canon(s[i]);
}

// CTA prologue: matrices to shared memory, TMEM for the groups, mbarriers.
__device__ __forceinline__ Group setup() {
  const uint4 *src = reinterpret_cast<const uint4 *>(d_matrices.b);
  for (uint32_t i = threadIdx.x; i < B_BYTES / 16; i += blockDim.x) reinterpret_cast<uint4 *>(smem)[i] = src[i];
  if (threadIdx.x < 32) tmem_alloc<512>(smem_addr(smem) + SMEM_TAIL + 8 * GROUPS);
  if (Group::leader()) mbar_init(Group::bar(), 1);
  fence_smem();
  fence_before();
  __syncthreads();
  fence_after();
  return {0};
}
__device__ __forceinline__ void teardown(const Group &g) {
  finish<512>(Group::base(), g.phase, smem_addr(smem) + SMEM_DRAIN, Group::leader(), GROUPS, &d_expired);
}

// One CTA whose wait runs out: a product is issued, and nothing completes the barrier waited on.
__global__ void __launch_bounds__(TILE) expired_wait_kernel(uint32_t polls) {
  __shared__ __align__(128) uint8_t rows[TILE * 32 + Y_COLS * 32];
  __shared__ __align__(8) uint64_t words[3];  // the barrier, the TMEM address, finish()'s barrier
  for (uint32_t i = threadIdx.x; i < sizeof(rows) / 8; i += TILE) reinterpret_cast<uint64_t *>(rows)[i] = 0;
  const uint32_t bar = smem_addr(words);
  if (threadIdx.x < 32) tmem_alloc<32>(bar + 8);
  if (threadIdx.x == 0) mbar_init(bar, 1);
  fence_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&words[1]);
  if (threadIdx.x == 0)
    mma(tmem, operand(smem_addr(rows), TILE * 16), operand(smem_addr(rows) + TILE * 32, Y_COLS * 16), idesc(Y_COLS), false);
  __syncwarp();
  uint32_t phase = 0;
  mbar_wait(bar, phase, &d_expired, polls);
  finish<32>(tmem, phase, bar + 16, threadIdx.x == 0, 1, &d_expired);
}

}  // namespace tc
}  // namespace glc
