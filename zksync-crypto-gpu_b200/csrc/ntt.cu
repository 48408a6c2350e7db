// Batched Goldilocks NTT / coset LDE and bit reversal for sm_100a.
//
// Replaces boojum-cuda's ntt:: and ops_complex::bit_reverse (crates/boojum-cuda/src/ntt.rs,
// native/ntt*.cu*, native/ops_complex.cu:88-156) with a B200 design of its own:
//
//  * An NTT of size N = 2^L runs as one pass (L <= 12) or two passes (L <= 24).  A pass covers
//    k consecutive radix-2 stages.  Writing a position as i = hi*2^(L-s0) + mid*M + lo
//    (M = 2^(L-s0-k)), the pass transforms the 2^k values of every (hi, lo) group.  One CTA
//    owns a tile of W consecutive lo values of one hi (W*8 bytes contiguous per row: coalesced
//    128-bit loads), stages it in shared memory and runs the k stages as radix-4..16 register
//    rounds with shared-memory exchanges in a padded layout.  The CTA walks several columns with
//    the same twiddles, which it builds once in shared memory.
//  * Batches that fill the GPU run their rounds on the tensor cores instead (ntt_tensor.cuh, chosen
//    by tt_usable): 2^22 x 176 in 10.9 ms where the register rounds take 16.5 ms.
//  * n2b (natural -> bit-reversed) runs the stages in increasing order with DIT butterflies,
//    b2n (bit-reversed -> natural) is its transpose: decreasing order, DIF butterflies.  Both
//    use the twiddle T[b] = w^bitrev(b) of block b at each stage; T is one flat table.
//  * Coset scaling (forward LDE: x s^j on load) and N^-1 s^-j (inverse: on store) are fused
//    into the first / last pass, so an LDE costs no extra HBM pass.
//  * Optionally (tuning), batches larger than an L2-sized chunk of columns run pass 1 and pass 2
//    chunk by chunk, so the second pass reads the first pass's output from the 126 MB L2.  The
//    NTT is integer-bound, and small chunks cost more in per-CTA twiddle tables than they save
//    in HBM traffic, so the default is one chunk.
#include <algorithm>
#include <vector>

#include "glc_field.cuh"
#include "glc_internal.h"
#include "launch.cuh"
#include "ntt_tensor.cuh"
#include "ntt_tile.cuh"

namespace glc {

template <uint32_t RB>
__global__ void __launch_bounds__(pass_threads(RB), pass_min_blocks(RB)) ntt_pass_kernel(const PassArgs a) {
  extern __shared__ uint64_t smem[];
  ntt_pass_tile<RB>(a, blockIdx.x, blockIdx.y, smem);
}

// ---- bit reversal (ops_complex.cu:88-156 semantics) ----

__global__ void bitrev_naive_kernel(const uint64_t *src, uint64_t src_stride, uint64_t *dst, uint64_t dst_stride,
                                    uint32_t log_rows) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  dependency_wait();
  if (i >= (1u << log_rows)) return;
  const uint32_t r = log_rows ? __brev(i) >> (32 - log_rows) : 0;
  if (i > r) return;
  const uint64_t col = blockIdx.y;
  const uint64_t vi = src[col * src_stride + i], vr = src[col * src_stride + r];
  dst[col * dst_stride + i] = vr;
  dst[col * dst_stride + r] = vi;
}

// log_rows = 2h + odd, h >= 5.  Position i = a*2^(h+odd) + m*2^h + b.  Tile (A, B, m) holds
// a = x*2^(h-5) + A, b = B*32 + y (x, y < 32); its image is tile (rev(B), rev(A), m) with
// (x, y) -> (rev5(y), rev5(x)).  One CTA moves a tile and its image, so in place is safe.
__global__ void __launch_bounds__(256) bitrev_tiled_kernel(const uint64_t *src, uint64_t src_stride, uint64_t *dst,
                                                           uint64_t dst_stride, uint32_t log_rows) {
  __shared__ uint64_t t0[32][33];
  __shared__ uint64_t t1[32][33];
  const uint32_t h = log_rows >> 1;
  const uint32_t odd = log_rows & 1;
  const uint32_t hb = h - 5;
  const uint32_t A = blockIdx.x >> hb, B = blockIdx.x & ((1u << hb) - 1);
  const uint32_t As = hb ? __brev(B) >> (32 - hb) : 0, Bs = hb ? __brev(A) >> (32 - hb) : 0;
  dependency_wait();
  if (A > As || (A == As && B > Bs)) return;  // the image tile's CTA moves this pair
  const uint32_t m = blockIdx.z;
  const uint64_t col = blockIdx.y;
  const uint64_t *s = src + col * src_stride;
  uint64_t *d = dst + col * dst_stride;
  const bool self = (A == As && B == Bs);
  auto pos = [&](uint32_t TA, uint32_t TB, uint32_t x, uint32_t y) -> uint64_t {
    const uint64_t a = ((uint64_t)x << hb) + TA, b = ((uint64_t)TB << 5) + y;
    return (a << (h + odd)) + ((uint64_t)m << h) + b;
  };
  const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 8 rows per sweep
  for (uint32_t x = ty; x < 32; x += 8) {
    t0[x][tx] = s[pos(A, B, x, tx)];
    if (!self) t1[x][tx] = s[pos(As, Bs, x, tx)];
  }
  __syncthreads();
  // element (x, y) of tile (A, B) goes to (rev5(y), rev5(x)) of tile (As, Bs); store row-wise
  for (uint32_t xr = ty; xr < 32; xr += 8) {
    const uint32_t y = __brev(xr) >> 27, x = __brev(tx) >> 27;
    d[pos(As, Bs, xr, tx)] = t0[x][y];
    if (!self) d[pos(A, B, xr, tx)] = t1[x][y];
  }
}

int ntt_init_device() {
  cudaError_t e = cudaFuncSetAttribute(ntt_pass_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, NTT_SMEM_MAX);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(ntt_pass_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, NTT_SMEM_MAX);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(ntt_pass_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, NTT_SMEM_MAX);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(ntt_tensor_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, NTT_SMEM_MAX);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(ntt_tensor_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, NTT_SMEM_MAX);
  return (int)e;
}

int ntt_dft_create(uint8_t **out) {
  std::vector<uint8_t> m(4 * DFT_BYTES);
  for (uint32_t v = 0; v < 4; v++)
    for (uint32_t r = 2; r <= 4; r++) {
      uint8_t *p = m.data() + v * DFT_BYTES + dft_offset(r);
      const uint64_t w16 = h_root_of_unity(4);
      uint64_t *coefs = reinterpret_cast<uint64_t *>(m.data() + v * DFT_BYTES + DFT_MATRICES + dft_offset(r) / 8);
      build_dft_matrix(p, coefs, r, v & 1, v & 2 ? h_inv(w16) : w16);
    }
  cudaError_t e = cudaMalloc(out, m.size());
  if (e == cudaSuccess) e = cudaMemcpy(*out, m.data(), m.size(), cudaMemcpyHostToDevice);
  return (int)e;
}

int bitrev_launch(const uint64_t *src, uint64_t src_stride, uint64_t *dst, uint64_t dst_stride, uint32_t log_rows,
                  uint32_t cols, cudaStream_t stream) {
  if (cols == 0) return 0;
  if (cols > 65535) {
    for (uint32_t c = 0; c < cols; c += 65535) {
      const int e = bitrev_launch(src + c * src_stride, src_stride, dst + c * dst_stride, dst_stride, log_rows,
                                  std::min<uint32_t>(65535, cols - c), stream);
      if (e) return e;
    }
    return 0;
  }
  if (log_rows < 10) {
    const uint32_t n = 1u << log_rows;
    const uint32_t threads = std::min<uint32_t>(n, 256);
    launch(bitrev_naive_kernel, dim3((n + threads - 1) / threads, cols), threads, 0, stream, src, src_stride, dst, dst_stride,
           log_rows);
  } else {
    const uint32_t h = log_rows >> 1;
    const uint32_t tiles = 1u << (2 * (h - 5));
    launch(bitrev_tiled_kernel, dim3(tiles, cols, 1u << (log_rows & 1)), 256, 0, stream, src, src_stride, dst, dst_stride,
           log_rows);
  }
  return last_launch_error();
}

// ---- NTT planner ----

NttTuning g_ntt_tuning[MAX_DEVICES][MAX_LOG_N + 1];

NttTuning &ntt_tuning(uint32_t log_n) {
  int dev = 0;
  cudaGetDevice(&dev);
  return g_ntt_tuning[(dev >= 0 && dev < MAX_DEVICES) ? dev : 0][std::min(log_n, MAX_LOG_N)];
}

// Whether a batch runs its passes on the tensor cores (ntt_tensor.cuh).  Needed: whole tiles (2^12
// rows, or at least 4 strided stages before 12 contiguous ones), and no per-element coset factor
// (a coset on the b2n side or in an inverse).  Worth it when the tiles fill the GPU, since a tile's
// rounds are a longer chain of latencies than the small tiles of ntt_pass_kernel, and a coset's
// matrices and twiddles cost more to build.  Measured on B200, us, tensor cores / radix passes:
//   no coset: 16 x 2^16 (256 tiles) 30 / 30, 4 x 2^18 33 / 36, 1 x 2^20 34 / 40; 8 x 2^16 (128) 23 / 22
//   coset:    32 x 2^16 (512 tiles) 47 / 53, 8 x 2^18 52 / 61; 16 x 2^16 (256) 36 / 32, 4 x 2^18 39 / 38
//   2^24, whose strided rows hold one element: 1 column 636 / 565, 16 columns 7761 / 8482; of two: 2^23 on a
//   coset, 1 column 280 / 257, 2 columns 408 / 457
// More tiles than the 296 CTAs of a wave take two columns a CTA, and the time of a second column before
// there are enough of them.  2^16 and 2^17 rows, whose radix passes are the quickest, wait for that:
//   n2b: 19 x 2^16 (304 tiles) 31 / 33, 20 x 2^16 39 / 34, 25 x 2^16 (400) 39 / 39, 26 x 2^16 39 / 43,
//        10 x 2^17 (320) 45 / 37, 13 x 2^17 (416) 45 / 43, 14 x 2^17 (448) 45 / 47
//   b2n inverse: 10 x 2^17 41 / 38, 20 x 2^16 36 / 35, 21 x 2^16 (336) 36 / 38
//   exactly 256 tiles, n2b forward: 16 x 2^16 28.8 / 26.8, 8 x 2^17 30.9 / 29.4 (the other way no slower)
//   but 5 and 7 x 2^18 (320, 448) 35 / 43, 45 / 55
static bool tt_usable(uint32_t log_n, uint32_t num_ntts, bool bitrev_inputs, bool inverse, uint32_t log_ext) {
  if (log_n < TT_LOG || (log_n > TT_LOG && log_n < TT_LOG + 4) || (log_ext && (inverse || bitrev_inputs))) return false;
  if ((log_n == 24 && num_ntts < 16) || (log_n == 23 && log_ext && num_ntts < 2)) return false;
  const uint64_t tiles = (uint64_t)num_ntts << (log_n - TT_LOG);
  if ((log_n == 16 || log_n == 17) && !log_ext) {
    if (tiles > 304 && tiles < (bitrev_inputs ? 336 : log_n == 16 ? 416 : 432)) return false;
    if (tiles == 256 && !bitrev_inputs && !inverse) return false;
  }
  return tiles >= (log_ext ? 512 : 256);
}

int ntt_launch(const uint64_t *in, uint64_t *out, uint32_t log_n, uint32_t num_ntts, uint64_t in_stride,
               uint64_t out_stride, bool bitrev_inputs, bool inverse, uint32_t log_ext, uint32_t coset_idx,
               cudaStream_t stream, uint32_t l2_chunk_cols, bool registers_only) {
  const DeviceTables *t = current_tables();
  if (!t) return fail("NTT: glc_context_create has not been called on this device");
  if (num_ntts == 0) return 0;
  const NttTuning &tu = ntt_tuning(log_n);
  Pass passes[2];
  const uint32_t np = make_plan(log_n, bitrev_inputs, tu, passes);
  if (!registers_only && tt_usable(log_n, num_ntts, bitrev_inputs, inverse, log_ext)) {
    const uint32_t k0 = log_n - TT_LOG;  // strided stages, then 12 contiguous ones
    if (k0 == 0)
      return tt_launch_pass(t, 0, TT_LOG, true, true, in, out, in_stride, out_stride, num_ntts, log_n, bitrev_inputs,
                            inverse, log_ext, coset_idx, stream);
    for (uint32_t q = 0; q < 2; q++) {
      const bool strided = bitrev_inputs ? q == 1 : q == 0;
      const int e = tt_launch_pass(t, strided ? 0 : k0, strided ? k0 : TT_LOG, q == 0, q == 1, in, out, in_stride, out_stride,
                                   num_ntts, log_n, bitrev_inputs, inverse, log_ext, coset_idx, stream);
      if (e) return e;
    }
    return 0;
  }
  const uint64_t n = 1ull << log_n;
  if (l2_chunk_cols == 0) {
    // keep one chunk of columns resident in L2 across the passes
    // (chunking trades HBM traffic for CTAs that each cover fewer columns and rebuild their
    // twiddles more often; on B200 the NTT is integer-bound, so one chunk usually wins)
    const uint64_t budget = (uint64_t)tu.l2_chunk_mb << 20;
    l2_chunk_cols = tu.l2_chunk_mb ? (uint32_t)std::max<uint64_t>(1, budget / (n * 8)) : num_ntts;
  }
  if (np == 1) l2_chunk_cols = num_ntts;
  for (uint32_t c0 = 0; c0 < num_ntts; c0 += l2_chunk_cols) {
    const uint32_t cols = std::min(l2_chunk_cols, num_ntts - c0);
    for (uint32_t q = 0; q < np; q++) {
      const Pass &ps = passes[q];
      PassArgs a;
      const PassShape sh = make_pass(a, t, tu, ps, q, np, in + (uint64_t)c0 * in_stride, out + (uint64_t)c0 * out_stride,
                                     in_stride, out_stride, cols, log_n, bitrev_inputs, inverse, log_ext, coset_idx,
                                     tu.max_cols_per_cta);
      const uint64_t tiles_per_col = sh.tiles_per_col;
      const uint32_t cpc = a.cols_per_cta, gy = sh.groups, threads = sh.threads;
      const size_t smem = sh.smem;
      if (gy > 65535) count_launches((gy - 1) / 65535);
      for (uint32_t y0 = 0; y0 < gy; y0 += 65535) {
        PassArgs b = a;
        const uint32_t ycount = std::min<uint32_t>(65535, gy - y0);
        b.in += (uint64_t)y0 * cpc * b.in_stride;
        b.out += (uint64_t)y0 * cpc * b.out_stride;
        b.num_cols = std::min<uint32_t>(cols - y0 * cpc, ycount * cpc);
        const dim3 grid((uint32_t)tiles_per_col, ycount);
        b.early = launches_early(grid);
        const size_t bytes = b.early ? std::max(smem, EARLY_SMEM) : smem;
        if (tu.radix_bits == 2)
          launch(ntt_pass_kernel<2>, grid, threads, bytes, stream, b);
        else if (tu.radix_bits == 4)
          launch(ntt_pass_kernel<4>, grid, threads, bytes, stream, b);
        else
          launch(ntt_pass_kernel<3>, grid, threads, bytes, stream, b);
      }
      const int e = last_launch_error();
      if (e) return e;
    }
  }
  return 0;
}

static int ntt_check(uint32_t log_n, uint32_t num_ntts, uint64_t in_stride, uint64_t out_stride, uint32_t log_ext,
                     uint32_t coset_idx) {
  (void)num_ntts;
  // ntt.rs:192-200
  if (log_n < 1) return fail("NTT: log_n must be >= 1");
  if (log_n + log_ext > OMEGA_LOG_ORDER) return fail("NTT: log_n + log_extension_degree must be <= 30");
  if (log_n > MAX_LOG_N) return fail("NTT: log_n must be <= 24");
  const uint64_t n = 1ull << log_n;
  if (n > in_stride || n > out_stride) return fail("NTT: n must be <= the strides between arrays");
  if (coset_idx > 0) {
    if (log_ext == 0) return fail("NTT: coset_index > 0 requires log_extension_degree > 0");
    if (coset_idx >= (1u << log_ext)) return fail("NTT: coset_index must be < 2^log_extension_degree");
  }
  return 0;
}

}  // namespace glc

using namespace glc;

extern "C" glc_status glc_batch_ntt_out_of_place(const uint64_t *inputs_matrix, size_t inputs_len,
                                                 uint64_t *outputs_matrix, size_t outputs_len, uint32_t log_n,
                                                 uint32_t num_ntts, uint32_t inputs_offset, uint32_t outputs_offset,
                                                 uint32_t stride_between_input_arrays,
                                                 uint32_t stride_between_output_arrays, bool bitrev_inputs,
                                                 bool inverse, uint32_t log_extension_degree, uint32_t coset_index,
                                                 void *stream) {
  // ntt.rs:308-320
  if (log_n >= 32) return fail("NTT: log_n out of range");
  const uint64_t n = 1ull << log_n;
  if ((uint64_t)inputs_offset + n > stride_between_input_arrays)
    return fail("NTT: inputs_offset + n must be <= stride_between_input_arrays");
  if ((uint64_t)outputs_offset + n > stride_between_output_arrays)
    return fail("NTT: outputs_offset + n must be <= stride_between_output_arrays");
  if (inputs_len < (uint64_t)num_ntts * stride_between_input_arrays)
    return fail("NTT: inputs_matrix shorter than num_ntts * stride_between_input_arrays");
  if (outputs_len < (uint64_t)num_ntts * stride_between_output_arrays)
    return fail("NTT: outputs_matrix shorter than num_ntts * stride_between_output_arrays");
  if (inputs_matrix == outputs_matrix) return fail("NTT: out-of-place call with identical matrices");
  if (inputs_matrix + inputs_offset == outputs_matrix + outputs_offset)
    return fail("NTT: out-of-place call with identical offset pointers");
  int e = ntt_check(log_n, num_ntts, stride_between_input_arrays, stride_between_output_arrays, log_extension_degree,
                    coset_index);
  if (e) return e;
  return ntt_launch(inputs_matrix + inputs_offset, outputs_matrix + outputs_offset, log_n, num_ntts,
                    stride_between_input_arrays, stride_between_output_arrays, bitrev_inputs, inverse,
                    log_extension_degree, coset_index, (cudaStream_t)stream, 0);
}

extern "C" glc_status glc_batch_ntt_in_place(uint64_t *inputs_matrix, size_t inputs_len, uint32_t log_n,
                                             uint32_t num_ntts, uint32_t inputs_offset,
                                             uint32_t stride_between_input_arrays, bool bitrev_inputs, bool inverse,
                                             uint32_t log_extension_degree, uint32_t coset_index, void *stream) {
  // ntt.rs:350-353
  if (log_n >= 32) return fail("NTT: log_n out of range");
  const uint64_t n = 1ull << log_n;
  if ((uint64_t)inputs_offset + n > stride_between_input_arrays)
    return fail("NTT: inputs_offset + n must be <= stride_between_input_arrays");
  if (inputs_len < (uint64_t)num_ntts * stride_between_input_arrays)
    return fail("NTT: inputs_matrix shorter than num_ntts * stride_between_input_arrays");
  int e = ntt_check(log_n, num_ntts, stride_between_input_arrays, stride_between_input_arrays, log_extension_degree,
                    coset_index);
  if (e) return e;
  uint64_t *p = inputs_matrix + inputs_offset;
  return ntt_launch(p, p, log_n, num_ntts, stride_between_input_arrays, stride_between_input_arrays, bitrev_inputs,
                    inverse, log_extension_degree, coset_index, (cudaStream_t)stream, 0);
}

static int bitrev_check(uint32_t rows, uint64_t src_stride, uint64_t dst_stride) {
  // ops_complex.rs:280-283
  if (rows == 0 || (rows & (rows - 1))) return fail("bit_reverse: rows must be a power of two");
  if (src_stride < rows || dst_stride < rows) return fail("bit_reverse: stride must be >= rows");
  return 0;
}

extern "C" glc_status glc_bit_reverse(const uint64_t *src, uint64_t src_stride, uint64_t *dst, uint64_t dst_stride,
                                      uint32_t rows, uint32_t cols, void *stream) {
  int e = bitrev_check(rows, src_stride, dst_stride);
  if (e) return e;
  return bitrev_launch(src, src_stride, dst, dst_stride, 31 - __builtin_clz(rows), cols, (cudaStream_t)stream);
}

extern "C" glc_status glc_bit_reverse_in_place(uint64_t *values, uint64_t stride, uint32_t rows, uint32_t cols,
                                               void *stream) {
  int e = bitrev_check(rows, stride, stride);
  if (e) return e;
  return bitrev_launch(values, stride, values, stride, 31 - __builtin_clz(rows), cols, (cudaStream_t)stream);
}
