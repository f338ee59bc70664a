// Kernels of one stream launched behind one another without a gap.
//
// Back to back on a stream, a kernel's blocks are set up only after the last block of the kernel before it has ended:
// 2 to 3 us for kernels of a few us.  Launched with programmatic stream serialisation, they are set up while that kernel
// drains, and wait in `after_previous_kernel` until it has ended and its memory is visible.  A kernel launched this way
// calls that first and touches no global memory before it; it then lets the kernel behind it be set up in turn, which is
// therefore never ahead of a kernel before this one.
//
// The two instructions cost a block some 20 ns on its SM (65,536 blocks of block-per-row SpMV: 61 -> 70 us), the gap they
// close is 2 us: only grids of up to kChainBlocks are chained, the others are launched, and run, as usual.
#pragma once
#include <cuda_runtime.h>

namespace swb {

constexpr unsigned kChainBlocks = 12288;

__device__ __forceinline__ void after_previous_kernel() {
  if (gridDim.x > kChainBlocks) return;
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                           Args... args) {
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attribute;
  cfg.numAttrs = grid <= kChainBlocks ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace swb
