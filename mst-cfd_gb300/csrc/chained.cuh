// Launches that follow one another in a stream: the next kernel's blocks are
// placed while this one still runs and wait for its end themselves, so that
// launch and drain are hidden between the short kernels of a time step: 50 FP64
// RK2 steps of 4,000 cells 3,147 -> 2,490 us, 30 viscous FP32 steps of 97k cells
// 1,289 -> 1,086, 20 FP32 steps of 2M cells 7,114 -> 6,945; in 3D 10 FP32 steps
// of 3,072 / 48,000 cells 493 -> 372 / 732 -> 612, 20 of 1.6M 9,322 -> 9,066.
// Blocks placed early go where the previous kernel has left room, not evenly:
// the launchers leave out the kernels that lose by that.
//
// Every kernel launched with launch_chained calls chain() in every thread that
// goes on, and in at least one thread of every block: a block that ended without
// it could let a later kernel start before an earlier one has ended.  Before
// chain() only tables may be read that no kernel writes.
// Pointers to what kernels write carry no __restrict__, and inline loads of it
// are volatile: neither a read-only load nor one moved above chain() would see
// the previous kernel's result.  Launched the ordinary way, chain() returns at
// once.
#pragma once
#include <cuda_runtime.h>

namespace mst {

// next = false: the last kernel on a caller's stream, whose next launch is not ours
__device__ __forceinline__ void chain(bool next = true) {
  // the previous kernel has ended and its writes are visible
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the next one may be placed
  if (next) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// on = false: launched the ordinary way
template <class... P, class... A>
cudaError_t launch_chained(bool on, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                           cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = on ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace mst
