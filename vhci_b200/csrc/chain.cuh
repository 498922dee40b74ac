// Launches whose start overlaps the end of the kernel before them in their stream (programmatic
// dependent launch), for the chains of short kernels of a Lanczos step and of the dense eigensolver:
// a kernel that follows another one begins about 2 us after its last block ended; launched this way its
// blocks are placed while the other one drains (12-mode solve of 5,500 launches 139.0 -> 132.2 ms; 100
// states of 60,011 in FP32 storage, 2,100 launches, 66.9 -> 63.8 ms).
//
// launch_chained starts kernel k once every block of the kernel before it in the stream has called
// chain_wait, or ended; k calls chain_wait before it reads or writes anything in global memory, which
// returns when that kernel has ended and its writes are visible.  (It ended after its own chain_wait, so
// all that came before it has ended too.)  A kernel that does not call chain_wait is launched plainly,
// before or after a chained one, as ever.
//
// k's life overlaps that of the kernel before it, so what that kernel writes is not read-only during k:
// k reads it by ordinary loads, never by __ldg or ld.global.nc (which a compiler may also move to before
// the wait) nor through const __restrict__ pointers (whose loads it may turn into such).  The matrix and
// other tables are complete before the kernel before k begins, and stay with the read-only loads.
#pragma once

#include <cuda_runtime.h>

namespace vhci {

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
inline void launch_chained(void (*k)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, static_cast<P>(a)...);
}

}  // namespace vhci
