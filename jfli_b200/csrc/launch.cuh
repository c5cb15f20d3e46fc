// Launches that overlap their start with the end of the kernel before them in the stream
// (programmatic dependent launch). A chain of passes over a small mesh spends more time
// between its kernels than a pass needs to start: with plain launches a 64^3 force took 51 us for
// 37 us of kernels, a 128^3 gradient 7.4 ms for 6.7.
//
// The protocol, for every kernel launched with launch_next:
//   * grid_wait() in every thread before it touches memory: it returns when the grids before this
//     one have finished and their writes are visible. No CTA leaves without it, or the grid
//     after this one could start ahead of the one before. (Reading the twiddle tables, which
//     never change, ahead of it gave 64^3 forces 0.7 us and cost large meshes 0.4%, as the
//     tile's loads then start behind them.)
//   * grid_release() ahead of the last stage: once every CTA of this grid is there (or has exited),
//     CTAs of the next one may take up free places on the SMs. Not earlier: CTAs that wait hold
//     shared memory, and with it L1, that the kernels of other streams, and of this one, could
//     use. Released at the top, where all of a small chain could start at once, three
//     concurrent 128^3 reverse sweeps took 11.0 ms, 10.7 released after the wait, 9.6 released late, 9.5
//     with plain launches; one 128^3 sweep 3.15, 3.15, 3.09 and 3.30 ms; a 96^3 Poisson chain 30, 21, 22
//     and 24 us; 64^3 forces 36.5, 36.5, 36.2 and 43.8. A kernel that is not followed by one of
//     launch_next's has none (its CTAs' exits release).
// Both are no-ops in a plain launch, and a kernel without them is a full dependency on either
// side, as are copies, memsets and events.
#pragma once

#include <cuda_runtime.h>

namespace jfli {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;"); }

// Whether a pass over `cells` cells (of all meshes of a batch) starts before its predecessor has
// ended: below 2^24, where a pass takes 3 to 30 us and the meshes of a step are in L2. Above,
// there is nothing to win, and the CTAs that wait take shared memory and L1 from the ones at
// work. Off -> on, forces: 48^3 36.9 -> 27.9 us, 64^3 43.8 -> 36.2, 96^3 75.5 -> 69.5, 128^3 133.3 -> 126.2,
// 192^3 366 -> 353, 216^3 537 -> 525; ICs, 2LPT and 19 steps: 108^3 2.00 -> 1.80 ms, 144^3 3.19 -> 3.04, 192^3
// 5.72 -> 5.42; reverse sweeps of 10 steps: 64^3 971 -> 749 us, 144^3 4.85 -> 4.67 ms (2LPT, 40 steps at
// 256^3 25.9 -> 26.3 ms, with grid_release at the top). The particle passes are left out at every
// size (launched plainly, no grid_release): with the next pass's CTAs on their SMs their
// gathers lose L1 (256^3 step 345 -> 470 us, 64^3 forces 40 -> 45).
inline bool overlap_starts(long long cells) { return cells < (1ll << 24); }

template <class... Params, class... Args>
inline cudaError_t launch_next(bool overlap, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t s, Args&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = s;
  config.attrs = &attr;
  config.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

}  // namespace jfli
