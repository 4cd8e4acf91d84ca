// Launching a kernel as a programmatic dependent of the one before it.
//
// The kernels of a cycle are launched as programmatic dependents: a kernel's
// blocks may start once those of the one before have left, before its stores
// are known to be visible. They read what no kernel writes (LDG: connectivity,
// masses, volumes of the undeformed mesh) and wait for the rest. Loads after the
// wait are ordinary ones: a block that started early may not take them through
// the read-only path. Per cycle 30.4 -> 27.2 us at 8^3, 44.5 -> 41.8 at 30^3,
// 710 -> 657 at 100^3, 2,233 -> 2,142 at 150^3. Letting the next kernel in
// earlier, from the first instruction or before the last phase of each block,
// packs its blocks onto the SMs that are free first: 58.7 and 51.1 us at 30^3.
#pragma once

#include <cuda_runtime.h>

namespace lulesh {

__device__ __forceinline__ void wait_for_last_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A programmatic dependent of the kernel before it on the stream (after
// anything else on the stream, an ordinary launch).
template <class... P, class... A>
void launch(void (*kernel)(P...), int grid, int block, cudaStream_t s, const A&... args) {
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.stream = s;
  c.attrs = &early;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, args...);
}

}  // namespace lulesh
