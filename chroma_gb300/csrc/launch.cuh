// Launches of the solvers' iteration kernels with programmatic dependent launch: a kernel may be placed on
// the SMs while its predecessor on the stream still runs, and waits there (pdl_begin) for that
// predecessor's completion and memory.  Its blocks then fill the places that the last wave leaves.
//
// A kernel launched this way calls pdl_begin() before it touches memory, and reads what other kernels
// write with ordinary loads (ldw) or cp.async: the read-only path is for data that no kernel in flight writes (links,
// clover: packed before a host synchronisation).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace gbc {

__device__ __forceinline__ void pdl_begin() {
  // the next kernel may be placed as soon as every block of this one has started
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Which grids are placed early: those of more than about a wave, whose gaps and tails shrink (CGNE of one
// source on 24^3 x 48 29.0 -> 27.4 ms, four uneven lattices 28.9 -> 27.6 ms), and those of a few blocks
// that only combine sums.  Grids of less than a wave are not: placed around their predecessor's
// blocks instead of evenly over the SMs, they end later (FP64 CG on 8^3 x 16 5.4 -> 7.5 ms, symmetric
// BiCGStab on 12 x 12 x 10 x 22 4.4 -> 4.6 ms).
inline bool place_early(long blocks) { return blocks <= 32 || blocks > 152 * 8; }

template <class... P, class... A>
inline void launch_pdl_if(bool early, void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);
}
template <class... P, class... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A&&... args) {
  launch_pdl_if(place_early((long)grid.x * grid.y * grid.z), kernel, grid, block, s, std::forward<A>(args)...);
}

}  // namespace gbc
