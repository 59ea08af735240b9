// Row softmax of a dense f32 matrix: out[r][:] = exp(x[r][:] - max) / sum, stored as f32, bf16 or f16.
//
// The planner recognises the chain reduce max -> subtract -> exponential -> reduce add -> divide over the last dimension
// (crates/ryft-mlir/src/dialects/stable_hlo/operations/functional.rs:188-219 and the elementwise builders) and replaces
// its four passes over memory with this one: a row is read once, kept in registers between the maximum, the exponentials
// and the quotient, and written once.  The operations are the chain's own (expf, IEEE division, f32 sums; the terms of a sum
// are added in another order, with an error against 64 bits that is no larger at any width), so infinities
// and NaN go the same way: a NaN or +inf score, or a row of -inf only, makes the row NaN.
//
// HBM-bound: 4 bytes read and the result's bytes written per element.  A row belongs to a warp up to 1024 elements (two
// shuffle reductions, no barrier) and to a CTA of 256 or 512 threads above; E elements per thread cover the row exactly
// once, so E is the smallest power of two that does.  [8192, 4096] f32: 424 us in four passes, two of them interpreted
// (805 MB); 43.6 us in one (6.15 TB/s). [1387, 151]: 38.9 us in four launches, 4.1 in one.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../../../include/b2x_kernels.h"
#include "common.cuh"
#include "vm.cuh"

namespace b2x {

__device__ __forceinline__ float sm_max(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// The sum of N values from v[AT] on, added in pairs.
template <int AT, int N, int E>
__device__ __forceinline__ float sm_tree_sum(const float (&v)[E]) {
  if constexpr (N == 1) return v[AT];
  else return sm_tree_sum<AT, N / 2>(v) + sm_tree_sum<AT + N / 2, N / 2>(v);
}

// T threads per row (32: eight rows per CTA), E elements per thread in pieces of V adjacent ones, OUT: B2xElem of the result.
template <int T, int E, int V, int OUT>
__global__ void __launch_bounds__(T == 32 ? 256 : T) k_softmax_rows(const float* x, char* out, int64_t rows, int n) {
  __shared__ float smem[2][T / 32];
  constexpr int ROWS = T == 32 ? 8 : 1;
  constexpr int P = E / V;                              // pieces per thread
  pdl_trigger();
  pdl_wait();
  const int tid = T == 32 ? (threadIdx.x & 31) : threadIdx.x;
  // a row's threads leave together: with T == 32 they are one warp, otherwise the whole CTA
  for (int64_t row = (int64_t)blockIdx.x * ROWS + (T == 32 ? threadIdx.x >> 5 : 0); row < rows; row += (int64_t)gridDim.x * ROWS) {
    const float* src = x + row * n;
    float v[E];
#pragma unroll
    for (int i = 0; i < P; i++) {
      const int c = (i * T + tid) * V;
      if constexpr (V == 4) {
        // streaming: a row is read once, by this CTA only
        const float4 f = c < n ? __ldcs((const float4*)(src + c)) : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
        v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
      } else {
        v[i] = c < n ? __ldcs(src + c) : -CUDART_INF_F;
      }
    }
    float m = v[0];
#pragma unroll
    for (int i = 1; i < E; i++) m = sm_max(m, v[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = sm_max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if constexpr (T > 32) {
      if ((tid & 31) == 0) smem[0][tid >> 5] = m;
      __syncthreads();
      m = smem[0][0];
#pragma unroll
      for (int w = 1; w < T / 32; w++) m = sm_max(m, smem[0][w]);
    }
    // a piece's four values are added in pairs, and pieces go to two partial sums in turn (single values to eight): at most six
    // additions in a row instead of E
    constexpr int PARTS = V == 4 ? 2 : 8;
    float part[PARTS];
#pragma unroll
    for (int i = 0; i < PARTS; i++) part[i] = 0.f;
#pragma unroll
    for (int i = 0; i < P; i++) {
      if ((i * T + tid) * V < n) {
        float piece[V];
#pragma unroll
        for (int j = 0; j < V; j++) piece[j] = v[i * V + j] = expf(v[i * V + j] - m);
        part[i % PARTS] += sm_tree_sum<0, V>(piece);
      }
    }
    float s = sm_tree_sum<0, PARTS>(part);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if constexpr (T > 32) {
      // smem[1] is read again only behind the next row's first barrier
      if ((tid & 31) == 0) smem[1][tid >> 5] = s;
      __syncthreads();
      s = sm_tree_sum<0, T / 32>(smem[1]);
    }
    constexpr int ES = OUT == EL_F32 ? 4 : 2;
    char* dst = out + row * n * ES;
#pragma unroll
    for (int i = 0; i < P; i++) {
      const int c = (i * T + tid) * V;
      if (c < n) {
        uint32_t q[V];
#pragma unroll
        for (int j = 0; j < V; j++) q[j] = vm_encode(f2u(__fdiv_rn(v[i * V + j], s)), OUT);
        if constexpr (ES == 4) vm_st_bytes<V * 4>(dst + c * 4, q);
        else if constexpr (V == 1) vm_st_bytes<2>(dst + c * 2, q);
        else {
          const uint32_t w[2] = {q[0] | (q[1] << 16), q[2] | (q[3] << 16)};
          vm_st_bytes<8>(dst + c * 2, w);
        }
      }
    }
  }
}

template <int T, int E, int V>
static int launch_rows(const float* x, char* out, uint8_t elem, int64_t rows, int n, cudaStream_t stream) {
  constexpr int ROWS = T == 32 ? 8 : 1;
  int64_t grid = (rows + ROWS - 1) / ROWS;
  if (grid > (int64_t)kNumSms * 512) grid = (int64_t)kNumSms * 512;
  const unsigned block = T == 32 ? 256 : T;
  cudaError_t e;
  if (elem == EL_F32) e = launch_overlapped(k_softmax_rows<T, E, V, EL_F32>, dim3((unsigned)grid), dim3(block), 0, stream, x, out, rows, n);
  else if (elem == EL_BF16) e = launch_overlapped(k_softmax_rows<T, E, V, EL_BF16>, dim3((unsigned)grid), dim3(block), 0, stream, x, out, rows, n);
  else if (elem == EL_F16) e = launch_overlapped(k_softmax_rows<T, E, V, EL_F16>, dim3((unsigned)grid), dim3(block), 0, stream, x, out, rows, n);
  else return (int)cudaErrorInvalidValue;
  if (e != cudaSuccess) return (int)e;
  count_launch();
  return (int)cudaGetLastError();
}

template <int V>
static int launch_width(const float* x, char* out, uint8_t elem, int64_t rows, int n, cudaStream_t stream) {
  if (n <= 32 * 4) return launch_rows<32, 4, V>(x, out, elem, rows, n, stream);
  if (n <= 32 * 8) return launch_rows<32, 8, V>(x, out, elem, rows, n, stream);
  if (n <= 32 * 16) return launch_rows<32, 16, V>(x, out, elem, rows, n, stream);
  if (n <= 32 * 32) return launch_rows<32, 32, V>(x, out, elem, rows, n, stream);
  if (n <= 256 * 8) return launch_rows<256, 8, V>(x, out, elem, rows, n, stream);
  if (n <= 256 * 16) return launch_rows<256, 16, V>(x, out, elem, rows, n, stream);
  if (n <= 512 * 16) return launch_rows<512, 16, V>(x, out, elem, rows, n, stream);
  return launch_rows<512, 32, V>(x, out, elem, rows, n, stream);
}

}  // namespace b2x

extern "C" int b2x_launch_softmax(const void* x, void* out, uint8_t out_elem, int64_t rows, int64_t n, b2x_stream_t stream) {
  using namespace b2x;
  if (rows <= 0 || n <= 0) return 0;
  if (n > B2X_SOFTMAX_MAX_ROW) return (int)cudaErrorInvalidValue;
  const bool wide = n % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)out & 15) == 0;
  return wide ? launch_width<4>((const float*)x, (char*)out, out_elem, rows, (int)n, (cudaStream_t)stream)
              : launch_width<1>((const float*)x, (char*)out, out_elem, rows, (int)n, (cudaStream_t)stream);
}
