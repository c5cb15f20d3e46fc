// Launches that overlap their start with the end of the kernel before them in the stream
// (programmatic dependent launch). A chain of passes over a small mesh spends more time
// between its kernels than a pass needs to start: with plain launches a 64^3 force took 51 us for
// 37 us of kernels, a 128^3 gradient 7.4 ms for 6.7.
//
// The protocol, for every kernel launched with launch_next:
//   * grid_release() at the top: once every CTA of this grid has started (or exited), CTAs of
//     the next one may take up free places on the SMs;
//   * grid_wait() in every thread before it touches memory: it returns when the grids before this
//     one have finished and their writes are visible. No CTA leaves without it, or the grid
//     after this one could start ahead of the one before. (Reading the twiddle tables, which
//     never change, ahead of it gave 64^3 forces 0.7 us and cost large meshes 0.4%, as the
//     tile's loads then start behind them.)
// Both are no-ops in a plain launch, and a kernel without them is a full dependency on either
// side, as are copies, memsets and events.
#pragma once

#include <cuda_runtime.h>

namespace jfli {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether a pass over `cells` cells (of all meshes of a batch) starts before its predecessor has
// ended: below 2^24, where a pass takes 3 to 30 us and the meshes of a step are in L2. Above,
// there is nothing to win, and the CTAs that wait take shared memory and L1 from the ones at
// work. Off -> on, forces: 48^3 48.0 -> 37.1 us, 64^3 51.4 -> 40.3, 96^3 74.8 -> 67.2, 128^3 130.6 ->
// 128.4, 216^3 452 -> 437, 256^3 682 -> 687; 2LPT and 10 steps: 128^3 1.73 -> 1.62 ms, 216^3
// 6.48 -> 6.27, 256^3 7.65 -> 7.67; 2LPT, 40 steps at 256^3 25.9 -> 26.3 ms (measured with the z
// and y passes apart at every size; 64^3 forces are 35.8 us with them together). The particle passes
// are left out at every size (launched plainly, no grid_release): with the next pass's CTAs on
// their SMs their gathers lose L1 (256^3 step 345 -> 470 us, 64^3 forces 40 -> 45).
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
