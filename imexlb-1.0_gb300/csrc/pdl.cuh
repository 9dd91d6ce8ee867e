// Programmatic dependent launch: a kernel's blocks start, and do what does not
// depend on the previous kernel of the stream (reads of the cell mask and the
// boundary records, of the launch parameters; tables and tensor memory), while
// that one drains; pdl_wait() then holds them until it has completed and its
// writes are visible. A kernel launched without the attribute finds nothing to
// wait for. Small lattices and short chains gain: FP32 256x128 4.38 -> 4.13 us an
// iteration, FP16 1024x512 7.28 -> 6.9 us (both before k_step_pair, whose reads ahead
// of the wait depend on it), FP32 24x16x16 5.47 -> 4.82, 64x32x32 8.22 -> 7.88; on larger
// D3Q27 lattices it is 2 to 0.5% (128x64x64 25.4 -> 25.0, 256x128x128 149.5 -> 148.8). Not used where a large step is bound
// by a pipe: the next step's blocks then settle on the SMs that finish first
// (FP64 512x256 20.8 -> 26.3 us; fixed point 256x128x128 447 -> 445 or 457 us by
// place of the trigger). The trigger comes after the wait: before it, blocks of the
// step after next settle too, ever more unevenly along a chain (FP64 200x100 in
// runs of 64 launches 17.7 us an iteration against 6.3; FP16 512x256 4.54 against
// 4.20).
#pragma once

#include <utility>

#include <cuda_runtime.h>

namespace imx {

#ifdef __CUDACC__
// The next kernel of the stream may start its blocks once every block of this
// one has called this (or ended).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// After pdl_wait(): p without what the compiler knows of it. (A load through a
// `const __restrict__` parameter may take the non-coherent path and be moved
// ahead of the wait.)
template <class P>
__device__ __forceinline__ P* pdl_fresh(P* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

template <class... P, class... A>
cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, unsigned block, unsigned smem, cudaStream_t s,
                             A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, P(std::forward<A>(args))...);
}

template <class... P, class... A>
cudaError_t launch_pdl(void (*kern)(P...), unsigned grid, unsigned block, cudaStream_t s, A&&... args) {
  return launch_dependent(kern, dim3(grid), block, 0u, s, std::forward<A>(args)...);
}
#endif

}  // namespace imx
