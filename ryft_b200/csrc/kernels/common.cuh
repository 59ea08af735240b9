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
// What such a kernel reads may have been written while it was already running.  The read-only path (__ldg, ld.global.nc,
// const __restrict__) promises data that does not change during the kernel, and is closed to it.  Open are `ld_global` below
// and __ldcs / __ldcg, whose volatile asm stays behind the wait, plain accesses through pointers that carry no such promise,
// and TMA.  k_gemm_simt keeps the read-only path and is launched in its turn instead: coherent loads cost it 5 to 12 % (1023 x
// 777 x 1001 bf16 65.2 -> 69.4 us, 1 x 4096 x 4096 f32 72 -> 79), the later start 2 us (65.2 -> 67.7, 72 -> 74; 17 x 33 x 5 6.0 -> 8.3).
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Coherent loads of 1 to 16 bytes.
__device__ __forceinline__ uint32_t ld_global(const uint8_t* p) {
  uint32_t v;
  asm volatile("ld.global.u8 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ uint32_t ld_global(const uint16_t* p) {
  uint16_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ uint32_t ld_global(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ uint2 ld_global(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ uint4 ld_global(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ float ld_global(const float* p) { return __uint_as_float(ld_global((const uint32_t*)p)); }
__device__ __forceinline__ float4 ld_global(const float4* p) {
  const uint4 v = ld_global((const uint4*)p);
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
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
