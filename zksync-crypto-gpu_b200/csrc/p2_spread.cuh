// One Poseidon2 permutation on 4 or 16 lanes, for launches too small to fill the GPU with one thread
// per permutation.  Included by poseidon2.cu, whose S-box, 96-bit sums and constants it uses.
//
// A thread alone issues about 14 K instructions for a permutation, mostly one after another: 16.8 us
// on B200 however few there are, and a tree's narrow layers wait for one another.  A quad's lane
// holds elements l, 4 + l and 8 + l; of 16 lanes, 12 hold one element each.  In a full round M_E's
// sum over the blocks of four and its M4 take the other lanes' values by shuffles.  In the partial
// rounds every lane keeps its own copy of element 0 and computes its S-box, and the sum of the other
// elements is reduced over the lanes beside it, so that nothing waits for a shuffle after the S-box.
// Bound: the chain of each round's S-box (three products deep), additions and reduction.  Measured
// per permutation when few run: 16.8 us (a thread), 11.4 (4 lanes), 9.5 (16 lanes).  Full, the quads
// reach 0.93 G permutations/s and the 16 lanes 0.4, a thread each 1.67.  A tree of 2^12 leaves of 8
// columns, cap 8: 198 -> 91 us.
#pragma once

namespace glc {

__device__ __forceinline__ uint64_t shfl_xor64(uint64_t x, int mask) {
  return pack(__shfl_xor_sync(0xFFFFFFFFu, lo32(x), mask), __shfl_xor_sync(0xFFFFFFFFu, hi32(x), mask));
}
__device__ __forceinline__ uint64_t shfl64(uint64_t x, int lane, int width) {
  return pack(__shfl_sync(0xFFFFFFFFu, lo32(x), lane, width), __shfl_sync(0xFFFFFFFFu, hi32(x), lane, width));
}

// A permutation spread over G = 4 or 16 lanes: lane l of a quad holds elements l, 4 + l and 8 + l;
// of 16 lanes, lane l < 12 holds element l and the last four hold zeros.
template <int G>
struct Spread {
  static constexpr int E = G == 4 ? 3 : 1;  // elements a lane holds

  // e <- M_E e + rc.  M4's rows seen from a lane: an even lane takes 5, 7, 1, 3 times its own, its
  // neighbour's (lane ^ 1), lane ^ 2's and lane ^ 3's value, an odd one 6, 4, 1, 1 times.
  static __device__ __forceinline__ void external(uint64_t (&e)[E], const uint64_t (&rc)[E]) {
    const bool odd = threadIdx.x & 1;
    const uint32_t c0 = odd ? 6 : 5, c1 = odd ? 4 : 7, c3 = odd ? 1 : 3;
    uint64_t L[E], H[E];
#pragma unroll
    for (int t = 0; t < E; t++) {
      const uint64_t x1 = shfl_xor64(e[t], 1), x2 = shfl_xor64(e[t], 2), x3 = shfl_xor64(e[t], 3);
      L[t] = madw(lo32(e[t]), c0, madw(lo32(x1), c1, madw(lo32(x3), c3, (uint64_t)lo32(x2))));
      H[t] = madw(hi32(e[t]), c0, madw(hi32(x1), c1, madw(hi32(x3), c3, (uint64_t)hi32(x2))));
    }
    if constexpr (G == 4) {
      const uint64_t sl = L[0] + L[1] + L[2], sh = H[0] + H[1] + H[2];
#pragma unroll
      for (int t = 0; t < 3; t++) e[t] = fold(L[t] + sl + lo32(rc[t]), H[t] + sh + hi32(rc[t]));
    } else {
      // the other blocks' values of this place: lanes l + 4 and l + 8 of the 12 (of the last four
      // lanes' own blocks, zeros, nothing is used)
      const uint64_t z = fold(L[0], H[0]);
      const int l = threadIdx.x & 15;
      const uint64_t za = shfl64(z, l < 8 ? l + 4 : l - 8, 16), zb = shfl64(z, l < 4 ? l + 8 : l - 4, 16);
      const uint64_t v = w_red(w_add(w_add(w_add64(z, z), w_from(za)), w_add64(zb, rc[0])));
      e[0] = l < 12 ? v : 0;
    }
  }

  static __device__ __forceinline__ w96 sum_lanes(w96 a) {
#pragma unroll
    for (int mask = 1; mask < G; mask <<= 1)
      a = w_add(a, {__shfl_xor_sync(0xFFFFFFFFu, a.l0, mask), __shfl_xor_sync(0xFFFFFFFFu, a.l1, mask),
                    __shfl_xor_sync(0xFFFFFFFFu, a.h, mask)});
    return a;
  }

  // One partial round from round constant rc: every lane has s0; element i of the others becomes
  // sum + 2^k_i element i, partially reduced every second round as in internal_lazy.
  template <bool REDUCE>
  static __device__ __forceinline__ void internal(uint64_t &s0, w96 (&e)[E], const uint32_t (&k)[E], uint32_t keep,
                                                  uint64_t rc) {
    w96 rest = e[0];
    if constexpr (E == 3) rest = w_add(w_add(rest, e[1]), e[2]);
    rest = sum_lanes(rest);
    const uint64_t x = sbox(s0);
    const w96 sum = w_add(rest, w_from(x));
    s0 = w_red(w_add(sum, w_add(w_shl64(x, 4), w_from(rc))));
#pragma unroll
    for (int t = 0; t < E; t++) {
      e[t] = w_add(sum, w_shl(e[t], k[t]));
      if (REDUCE) e[t] = w_partial(e[t]);
      if (t == 0) e[0] = {e[0].l0 & keep, e[0].l1 & keep, e[0].h & keep};
    }
  }

  // The permutation; every lane of the warp calls it.
  static __device__ __forceinline__ void permutation(uint64_t (&e)[E]) {
    const uint32_t l = threadIdx.x & (G - 1);
    const uint32_t place = l < 12 ? l : 0;
    auto constants = [&](uint64_t (&rc)[E], int r) {
#pragma unroll
      for (int t = 0; t < E; t++) rc[t] = c_rc[r][4 * t + place];
    };
    uint64_t rc[E];
    constants(rc, 0);
    external(e, rc);
#pragma unroll 1
    for (int q = 0; q < 8; q++) {
#pragma unroll
      for (int t = 0; t < E; t++) e[t] = sbox(e[t]);
      if (q == 3 || q == 7) {
#pragma unroll
        for (int t = 0; t < E; t++) rc[t] = 0;
        if (q == 3 && l == 0) rc[0] = c_rc[4][0];
      } else {
        constants(rc, q < 3 ? q + 1 : q + 23);
      }
      external(e, rc);
      if (q == 3) {
        uint32_t k[E];
#pragma unroll
        for (int t = 0; t < E; t++) {
          const uint32_t i = 4 * t + place;  // 4, 14, 11, 8, 0, 5, 2, 9, 13, 6, 3, 12
          k[t] = (uint32_t)((i < 8 ? 0x09020500080B0E04ull >> (8 * i) : 0x0C03060Dull >> (8 * (i - 8))) & 31);
        }
        const uint32_t keep = l == 0 || l >= 12 ? 0 : ~0u;  // lane 0's element 0 is s0
        uint64_t s0 = shfl64(e[0], 0, G);
        w96 w[E];
#pragma unroll
        for (int t = 0; t < E; t++) w[t] = w_from(e[t]);
        w[0] = {w[0].l0 & keep, w[0].l1 & keep, 0};
#pragma unroll 1
        for (int r = 5; r <= 26; r += 2) {
          internal<false>(s0, w, k, keep, c_rc[r][0]);
          internal<true>(s0, w, k, keep, c_rc[r + 1][0]);
        }
        constants(rc, 26);  // s0 has its own
#pragma unroll
        for (int t = 0; t < E; t++) e[t] = w_red(w_add(w[t], w_from(rc[t])));
        if (l == 0) e[0] = s0;
      }
    }
#pragma unroll
    for (int t = 0; t < E; t++) e[t] = canon(e[t]);
  }
};

static constexpr uint32_t SPREAD_THREADS = 256;

// Leaf hashes (as p2_leaves_kernel): G lanes a leaf.  Lane l takes the words of a chunk that are its
// elements, and words l of the capacity and the digest.
template <int G>
__global__ void __launch_bounds__(SPREAD_THREADS) p2_leaves_spread_kernel(const uint64_t *values, uint64_t *results,
                                                                          uint32_t log_rows, uint64_t cols, uint64_t count,
                                                                          bool load_intermediate, bool store_intermediate) {
  const uint64_t gid = ((uint64_t)blockIdx.x * SPREAD_THREADS + threadIdx.x) / G;
  const uint32_t l = threadIdx.x & (G - 1);
  const bool live = gid < count;
  const uint64_t rows = 1ull << log_rows, total = rows * cols, col_stride = rows * count;
  const uint64_t *v = values + (gid << log_rows);
  auto load = [&](uint64_t o) {
    return live && o < total ? __ldcs(v + (o & (rows - 1)) + (o >> log_rows) * col_stride) : 0;
  };
  uint64_t e[Spread<G>::E] = {};
  if constexpr (G == 4) {
    if (load_intermediate && live) e[2] = results[gid + l * count];
    uint64_t n0 = load(l), n1 = load(4 + l);
    for (uint64_t off = 0; off < total; off += 8) {
      e[0] = n0;
      e[1] = n1;
      n0 = load(off + 8 + l);
      n1 = load(off + 12 + l);
      Spread<G>::permutation(e);
    }
    if (live) results[gid + l * count] = canon(store_intermediate ? e[2] : e[0]);
  } else {
    if (load_intermediate && live && l >= 8 && l < 12) e[0] = results[gid + (l - 8) * count];
    uint64_t n0 = l < 8 ? load(l) : 0;
    for (uint64_t off = 0; off < total; off += 8) {
      if (l < 8) {
        e[0] = n0;
        n0 = load(off + 8 + l);
      }
      Spread<G>::permutation(e);
    }
    const uint32_t from = store_intermediate ? 8 : 0;
    if (live && l >= from && l < from + 4) results[gid + (l - from) * count] = canon(e[0]);
  }
}

// Node layers: the CTA owns 2 * SPREAD_THREADS / G consecutive children of layer `in` ([4][2 * count])
// and produces up to `layers` parent layers, down to one node, each stored after the previous one
// (reference tree layout, poseidon2.rs:276-314).  A layer of at most 16 nodes takes 16 lanes a node.
template <int G>
__global__ void __launch_bounds__(SPREAD_THREADS) p2_subtree_spread_kernel(const uint64_t *in, uint64_t *out,
                                                                           uint64_t count, uint32_t layers, bool aligned) {
  constexpr uint32_t NODES = SPREAD_THREADS / G;
  __shared__ uint64_t sh[4][NODES];
  uint64_t layer_count = count, *dst = out;
  uint32_t active = NODES;
  // the next layer: half the nodes, children in sh
  auto advance = [&]() {
    dst += 4 * layer_count;
    layer_count >>= 1;
    active >>= 1;
    layers--;
    __syncthreads();
  };
  if constexpr (G == 4) {
    const uint32_t l = threadIdx.x & 3, n = threadIdx.x >> 2;
    for (bool first = true; layers && active > 16; first = false) {
      const uint64_t node = (uint64_t)blockIdx.x * active + n;
      const bool live = n < active && node < layer_count;
      uint64_t e[3] = {0, 0, 0};
      if (live && first) {
        const uint64_t *src = in + l * 2 * count + 2 * node;
        if (aligned) {
          const ulonglong2 lr = __ldcs(reinterpret_cast<const ulonglong2 *>(src));
          e[0] = lr.x;
          e[1] = lr.y;
        } else {
          e[0] = __ldcs(src);
          e[1] = __ldcs(src + 1);
        }
      } else if (live) {
        e[0] = sh[l][2 * n];
        e[1] = sh[l][2 * n + 1];
      }
      if ((threadIdx.x & ~31u) < 4 * active) Spread<4>::permutation(e);  // whole warps
      __syncthreads();
      if (live) {
        dst[l * layer_count + node] = e[0];
        sh[l][n] = e[0];
      }
      advance();
    }
  }
  const uint32_t l = threadIdx.x & 15, n = threadIdx.x >> 4;
  for (bool first = G == 16; layers; first = false) {
    const uint64_t node = (uint64_t)blockIdx.x * active + n;
    const bool live = n < active && node < layer_count;
    uint64_t e[1] = {0};
    if (live && l < 8)
      e[0] = first ? __ldcs(in + (l & 3) * 2 * count + 2 * node + (l >> 2)) : sh[l & 3][2 * n + (l >> 2)];
    if ((threadIdx.x & ~31u) < 16 * active) Spread<16>::permutation(e);
    __syncthreads();
    if (live && l < 4) {
      dst[l * layer_count + node] = e[0];
      sh[l][n] = e[0];
    }
    advance();
  }
}

}  // namespace glc
