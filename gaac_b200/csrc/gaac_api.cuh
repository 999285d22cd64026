// Helpers shared by the C-ABI entry points.
#pragma once
#include <cuda_runtime.h>
#include <utility>
#include <stdint.h>
#include "../../include/gaac_b200.h"

namespace gaac {
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int launch_status() { return cudaGetLastError() == cudaSuccess ? GAAC_OK : GAAC_E_LAUNCH; }

// ---- programmatic dependent launch.  A kernel launched with launch_overlapped may become resident while the kernel before it in the stream is still
// running, once every block of that one has executed griddep_launch() or exited; it begins with griddep_wait(), which returns when that
// kernel has completed and its writes are visible, and touches no memory before (but see exponent_hist_kernel behind clear_kernel).  Behind an ordinary kernel, and with the switch off, all of
// this does nothing.  It takes a launch's latency (1-2 us) off chains of short kernels.
inline int g_launch_overlap = 1;      // see gaac_set_launch_overlap
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::); }
// shared_bytes: dynamic shared memory;  carveout: per cent of an SM's memory that shared memory should have, the rest being L1 (0: as the driver has it).
template <class... Params, class... Args>
int launch_overlapped_with(int shared_bytes, int carveout, void (*kernel)(Params...), dim3 grid, unsigned threads, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = shared_bytes; cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = g_launch_overlap;
  at[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout; at[1].val.sharedMemCarveout = (unsigned)carveout;
  cfg.attrs = at; cfg.numAttrs = carveout > 0 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) != cudaSuccess) { cudaGetLastError(); return GAAC_E_LAUNCH; }
  return launch_status();
}
template <class... Params, class... Args>
int launch_overlapped(void (*kernel)(Params...), dim3 grid, unsigned threads, cudaStream_t stream, Args&&... args) {
  return launch_overlapped_with(0, 0, kernel, grid, threads, stream, std::forward<Args>(args)...);
}
}  // namespace gaac
