// Kernel launches that may begin before the previous kernel of their stream has ended.
#pragma once
#include <cuda_runtime.h>

namespace glc {

// Small launches carry the programmatic-stream-serialisation attribute: their CTAs may become
// resident, and do what depends on nothing (twiddles from the context's tables), while the previous
// kernel runs out; each then waits (dependency_wait) for that kernel's end and its writes.  A chain of
// small kernels is bound by the gaps between them: the two passes of a 2^16 NTT, a commitment of 2^12
// rows.  Only launches of at most one CTA per SM: waiting CTAs of a larger one would hold SMs that
// other streams' kernels could use.  Not for the hash kernels: a layer's CTAs that arrive while the
// layer before still holds most SMs crowd onto the others (2^15-leaf tree: 170 us becomes 189).
// Measured on B200: a 2^16 NTT forward and back 28.7 -> 16.7 us.
static constexpr uint64_t EARLY_CTAS = 148;

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
  c.numAttrs = (uint64_t)grid.x * grid.y * grid.z <= EARLY_CTAS ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, static_cast<Params>(args)...);  // last_launch_error() has its status
}

// Every kernel launched this way calls it before it touches memory that other kernels write or read.
// It also lets the next launch begin.
__device__ __forceinline__ void dependency_wait() {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace glc
