// Exact integer products on the fifth-generation tensor cores (tcgen05, kind::i8): the PTX wrappers
// and the digit representation shared by the kernels that use them.
//
// A linear map over the field with constant coefficients becomes a contraction of bytes.  A
// uint64_t input word is its own string of 8 base-256 digits x_b; with coefficient C the digit
// contributes x_b * (C * 2^(8b) mod p), whose 8 digits are one column of the constant matrix B.  A
// row of input bytes times B (u8 x u8 -> s32) gives 8 sums per output word, its digits before
// carries; carry_digits and reduce_digits turn them into a field element.  The sums are exact: they
// stay below 2^24 (digit_limit).
#pragma once
#include "glc_field.cuh"

namespace glc {
namespace tc {

// A digit sum v may be at most this for v + 2^8 v' to stay below 2^32.
static constexpr uint32_t digit_limit = 0xFFFFFFFFu / 257;

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory descriptor of a K-major operand without swizzle: core matrices of 8 rows x 16
// bytes, consecutive groups of 8 rows 128 bytes apart, consecutive 16-byte K chunks `lbo` apart.
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t lbo) {
  return (uint64_t)(addr >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}
// Instruction descriptor: D s32, A u8, B u8, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc(uint32_t n) { return (2u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, bool accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(desc),
               "r"((uint32_t)accumulate)
               : "memory");
}
// The mbarrier at `bar` completes its phase when the products issued by this thread so far are done.
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Orders this thread's shared-memory writes before the tensor cores' reads of them.
__device__ __forceinline__ void fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 TMEM columns of this thread's lane; the values are there after ld_wait on the same array.
__device__ __forceinline__ void ld32(uint32_t (&v)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void ld_wait(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                 "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
                 "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
               :
               : "memory");
}

// TMEM allocation by one full warp: the address lands in shared memory at `slot`.
template <uint32_t COLUMNS>
__device__ __forceinline__ void tmem_alloc(uint32_t slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(COLUMNS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <uint32_t COLUMNS>
__device__ __forceinline__ void tmem_free(uint32_t addr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "n"(COLUMNS) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Waits for the barrier's current phase: bounded (`polls` of up to 20 us, about a second).  `phase` bit
// 0 is the phase's parity, bit 1 records that a wait gave up, after which later waits poll once.  Every
// thread has a limit of its own, and each whose wait gave up counts itself in *expired; the kernel then
// runs to its end with wrong results, and finish() below waits for what it left in flight.
static constexpr uint32_t WAIT_POLLS = 50000;
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t &phase, unsigned long long *expired,
                                          uint32_t polls = WAIT_POLLS) {
  uint32_t done = 0;
  for (uint32_t tries = 0; tries < polls; tries++) {
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(phase & 1u), "r"(20000u)  // sleeps up to 20 us
                 : "memory");
    if (done || (phase >> 1)) break;
  }
  phase ^= 1u;
  if (!done) {
    phase |= 2u;
    atomicAdd(expired, 1ull);
  }
  fence_after();
}

// The CTA's end: frees its TMEM (by warp 0).  After a wait that gave up, products may still read the
// operand rows and write the TMEM: the threads that issued them (`issuer`, `issuers` of them) then
// commit once more, to the unused barrier `drain`, and everyone waits for that, bounded, first.
template <uint32_t COLUMNS>
__device__ __forceinline__ void finish(uint32_t tmem, uint32_t phase, uint32_t drain, bool issuer, uint32_t issuers,
                                       unsigned long long *expired) {
  fence_before();
  if (__syncthreads_or(phase >> 1)) {
    if (threadIdx.x == 0) mbar_init(drain, issuers);
    fence_smem();
    __syncthreads();
    if (issuer) commit(drain);
    __syncwarp();
    uint32_t last = 0;
    mbar_wait(drain, last, expired);
    fence_before();
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    fence_after();
    tmem_free<COLUMNS>(tmem);
  }
}

// The field element with these 8 digit sums (each at most digit_limit), in [0, 2^64).  Pairs of
// digits first (p = v + 2^8 v' below 2^32), then the four pairs at their 16-bit places carried into
// l0, l1 and h < 2^17, then h folded in: h * 2^64 = h * EPS, whose sum with l carries at most once,
// and then leaves a value below 2^50 to add EPS to.
__device__ __forceinline__ uint64_t reduce_digits(const uint32_t *v) {
  const uint32_t p0 = v[0] + (v[1] << 8), p1 = v[2] + (v[3] << 8), p2 = v[4] + (v[5] << 8), p3 = v[6] + (v[7] << 8);
  uint32_t r0, r1, k;
  asm("{\n\t.reg .u32 l0, l1, h, u;\n\t"
      "add.cc.u32 l0, %3, %4;\n\taddc.cc.u32 l1, %5, %6;\n\taddc.u32 h, %7, 0;\n\t"
      "sub.cc.u32 %0, l0, h;\n\tsubc.u32 u, h, 0;\n\t"
      "add.cc.u32 %1, l1, u;\n\taddc.u32 %2, 0, 0;\n\t}"
      : "=&r"(r0), "=&r"(r1), "=&r"(k)
      : "r"(p0), "r"(p1 << 16), "r"(p2), "r"(__byte_perm(p1, p3, 0x5432)), "r"(p3 >> 16));
  return madw(k, 0xFFFFFFFFu, pack(r0, r1));
}

}  // namespace tc
}  // namespace glc
