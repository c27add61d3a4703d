// Launches with the programmatic stream-serialization attribute: a kernel may begin while the kernel before it in the
// stream is still running, as far as that kernel has declared (grid_launch_dependents, else its end), and blocks in
// grid_dependency_wait until that kernel has completed and its memory is visible.  Every kernel launched this way calls
// grid_dependency_wait before it touches memory, so results cannot differ; what overlaps is the launch itself and the
// set-up (barriers, TMEM, descriptors).  A kernel of another library before it simply completes first.  Kernels declare
// themselves only after their own wait: at most two neighbours are ever in flight, and a kernel cannot have begun on an
// SM whose read-only cache the kernel before the last one is still filling.
//
// Not for kernels that live on L1 hits (pooling, contractions without tensor cores, operand splitting): beside a
// tensor-core kernel an SM keeps the carve-out for its shared memory, and they would run with what little L1 is left, as
// predecessor or as successor (a 4000 x 4000 x 130 product with its operand splitting 58 -> 74 us).
//
// Measured on replayed ResNet-50 passes (57 launches of 4 to 17 us at 16 images): batch 1 399 -> 363 us, 4 455 -> 408,
// 16 559 -> 514, 64 1016 -> 984, 256 2743 -> 2738; an int8 GEMM of 64 x 64 x 128 4.2 -> 3.5 us, 4096^3 50.2 -> 49.5 us.
// It pays where launches are short and costs nothing where they are long.
#pragma once

#include <cuda_runtime.h>

#include "ptx.cuh"

namespace pmlb {

inline cudaLaunchAttribute dependent_launch_attribute() {
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

// First statement of a kernel without set-up of its own.
__device__ __forceinline__ void dependent_entry() {
  grid_dependency_wait();
  grid_launch_dependents();
}

template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, unsigned block, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr = dependent_launch_attribute();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace pmlb
