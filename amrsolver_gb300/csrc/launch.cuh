// Launches whose setup overlaps the end of the kernel before them (programmatic
// dependent launch): the next kernel is set up while the previous one ends, and
// waits for it in dep_begin.  Every kernel launched by launch_dep calls dep_begin
// first; nothing is read or written before it, so the order of memory accesses
// is that of plain launches.
//
// Why: a stage is a chain of four to seven kernels, and on small boxes each is
// a few microseconds of latency.  With the box record in the launch (see
// BoxTable::one): KEEP4 RHS 16^3 47 -> 30 us, KEEP6 step 45 x 33 x 27 272 -> 216 us,
// KEEP4 step 128^3 3.13 -> 3.07 ms.  No kernel lets its dependents in before its
// blocks exit (griddepcontrol.launch_dependents): blocks of the static marches
// that get in early pile up on the SMs that happen to be free (272 -> 312 us
// and 3.16 ms in these steps).
#pragma once
#include <cuda_runtime.h>

namespace amrs {

// Blocks per SM of a grid-stride launch that has more work than that: divisible by
// 2, 3, 4, 5 and 6, so that every round of resident blocks is full whatever a
// kernel's registers allow (with 8 the third round of a kernel with three resident
// blocks ran with two).  A step, KEEP4 128^3: 2978 us with 8, 2928 with 12, 2922 with
// 24, 2910 with 60; level of 32^3 boxes 3518 and 3439; WENO5 64^3 1754 and 1726.
constexpr int GRID_CTAS = 60;

// Waits until all earlier grids are complete and their writes visible.
__device__ __forceinline__ void dep_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... K, class... A>
cudaError_t launch_dep(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, K(args)...);
}

}  // namespace amrs
