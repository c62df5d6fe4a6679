// Launches in a chain: a kernel's blocks are brought up as its predecessor's
// last blocks leave.
//
// A small grid's step is a chain of 3 to 20 us kernels, and between two of them
// lies about a microsecond in which the first one's results are flushed and the
// second one's blocks are started.  launch_chained sets the programmatic stream
// serialisation attribute (inside a captured graph: a programmatic edge), which
// overlaps the two; grid_wait holds the blocks until every earlier grid of the
// stream has completed and its writes are visible.  Only kernels that call
// grid_wait may be launched this way.
//
// Measured, a call before -> after: 128x32 RK222 72.0 -> 68.1 us, 256x64 (20
// steps) 1416 -> 1335, four 512x129 field transforms 47.6 -> 43.2, twelve-member
// ensemble (10 steps) 4700 -> 4225.  An explicit early trigger
// (griddepcontrol.launch_dependents) is not used: waiting blocks then sit on the
// SMs through the whole predecessor and unbalance the next grid (1024x256 RK443
// 435 -> 471 us).  The turbulence and 3D kernels gained nothing and stay as they
// were.
#pragma once

#include <cuda_runtime.h>

#include <initializer_list>
#include <utility>

namespace tb {

// Waits for the preceding grid.  Nothing that an earlier kernel of the stream
// writes is read, and nothing is written, before it; tables of the plan may be.
// The pointers given are hidden from the compiler across the wait: a load
// through a const __restrict__ parameter counts as invariant and could be moved
// above it.
template <class... P>
__device__ __forceinline__ void grid_wait(P&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (void)std::initializer_list<int>{([&] { asm volatile("" : "+l"(p)); }(), 0)...};
}

// Grids of up to three blocks an SM: at 1024x256, whose grids are larger, the
// attribute on every launch cost 0.6 % (435.5 -> 438.2 us, 434.6 with the limit);
// one block an SM loses the gain of the transforms and of the ensemble (47.4 and
// 4432 us).
constexpr long long kChainBlocks = 3 * 148;

template <class... K, class... A>
inline void launch_chained(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = (long long)grid.x * grid.y * grid.z <= kChainBlocks ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);  // a failure is seen by the caller's check_launch
}

}  // namespace tb
