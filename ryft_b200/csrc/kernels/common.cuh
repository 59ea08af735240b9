// Shared launch helpers for the kernel translation units.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstdlib>
#include <stdint.h>

namespace b2x {
extern std::atomic<int64_t> g_launch_count;
inline void count_launch(int n = 1) { g_launch_count.fetch_add(n, std::memory_order_relaxed); }
// Programmatic dependent launch.  A kernel launched through `launch_overlapped` may start while the kernel before it on the
// stream is still running, once every CTA of that one has called `pdl_trigger` or left; it sets itself up (barriers, TMEM)
// and must call `pdl_wait`, in every thread that touches global memory, before it reads or writes any: the wait ends when all
// earlier kernels of the stream have finished and their results are visible.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... P, typename... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
#endif
constexpr int kNumSms = 148;  // B200: 2 dies x 74 SMs
// B2X_VM_STATIC=0 makes every fused-elementwise program run through the interpreter, also those that have a build-time
// specialised form (for measuring what the specialisation is worth, and for testing the interpreter on the same programs).
inline bool vm_static_enabled() {
  const char* e = getenv("B2X_VM_STATIC");
  return !(e && e[0] == '0');
}
}  // namespace b2x
