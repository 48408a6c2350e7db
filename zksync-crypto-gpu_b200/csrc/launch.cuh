// Kernel launches that may begin before the previous kernel of their stream has ended.
#pragma once
#include <cuda_runtime.h>

namespace glc {

// Small launches carry the programmatic-stream-serialisation attribute: their CTAs may become
// resident, and do what depends on nothing (twiddles from the context's tables), while the previous
// kernel runs out; each then waits (dependency_wait) for that kernel's end and its writes.  A chain of
// small kernels is bound by the gaps between them: the two passes of a 2^16 NTT, a commitment of 2^12
// rows.  Only launches of at most one CTA per SM: waiting CTAs of a larger one would hold SMs that
// other streams' kernels could use.  CTAs that arrive while the kernel before still holds most SMs
// crowd onto the others, hence:
//  * not for the hash kernels (2^15-leaf tree: 170 us becomes 189);
//  * an NTT pass asks for EARLY_SMEM of shared memory, so that an SM takes at most two CTAs, one of
//    them the kernel's before (2^17 x 1 forward: 16.5 us without early launches, 18.8 crowded, 9.4 so);
//  * only NTT passes that are early themselves let the next launch begin (2^17 x 2 forward, whose first
//    has 256 CTAs: 16.5 us without early launches, 22.6 when it did, 14.4 so; 2^13 x 8 inverse on a
//    coset, whose larger pass has short CTAs: 16.6, 12.4, 14.4).
// Measured on B200, us a call back to back: a 2^16 NTT forward and back 28.8 -> 16.6 on the device (with
// other work between the calls about 1.3x).
static constexpr uint64_t EARLY_CTAS = 148;
static constexpr size_t EARLY_SMEM = 77 * 1024;
inline bool launches_early(dim3 grid) { return (uint64_t)grid.x * grid.y * grid.z <= EARLY_CTAS; }

template <typename... Params, typename... Args>
inline void launch(void (*kernel)(Params...), dim3 grid, uint32_t threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = &early;
  c.numAttrs = launches_early(grid) ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, static_cast<Params>(args)...);  // last_launch_error() has its status
}

// Every kernel launched early calls it before it touches memory that other kernels write or read.  It
// also lets the next launch begin.  (In a launch that is not early it waits for nothing.)
__device__ __forceinline__ void dependency_wait() {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace glc
