// CUDA-core strided batched GEMM with the fused-elementwise epilogue.
//
// This is the general path of stablehlo.dot_general: any element type the executor supports (f32/bf16/f16 with f32
// accumulation, 8/16/32-bit integers with 32-bit accumulation), any strides, any sizes (down to the 2x3x2 example
// in the reference's README).  Large aligned bf16/f16/f32 problems go to the tcgen05 kernel instead.
//
// 256 threads compute a BM x 64 tile (BM = 128 with 8 x 4 results per thread, or 64 with 4 x 4) over 16-deep k-slabs in
// two shared-memory buffers; the next slab's operands travel from global memory into registers while the current one is
// multiplied.  f32 products go two at a time through fma.rn.f32x2, each rounded as a scalar fma would round it.  A
// problem with fewer tiles than the chip has room for is cut along K: the CTAs of a cluster take one piece each, and
// then each sums and finishes its share of the tile out of the others' shared memory, always in the same order.
// The finished tile passes through shared memory, so that the epilogue program runs (and stores) along rows, from one
// copy of its code; a program that only stores the accumulator is recognised on the host and is a plain store.
// Bound: FMA issue for large problems; below ~10^7 products the chain of latencies of one slab after the other.
//   1023 x 777 x 1001 bf16           162 us -> 68 us
//   1500 x 1999 x 2047 f16           817 us -> 361 us
//   17 x 33 x 5 f32                   31 us -> 8.2 us (before: sixteen inlined interpreted stores per thread)
//   8 x 2048 x 9 f32                 229 us -> 16.4 us (before: one CTA walked all of K)
#include <cooperative_groups.h>

#include "../../../include/b2x_kernels.h"
#include "common.cuh"
#include "vm.cuh"

namespace b2x {

struct GemmK {
  const char* a; const char* b;
  int elem, es;
  int64_t batch, M, N, K;
  int64_t sab, sam, sak, sbb, sbn, sbk;
  int64_t k_piece;         // k range of one CTA of a cluster (a multiple of 16)
  int32_t tiles_n, CL;
  char* plain_out;         // dense row-major result of a program that only stores the accumulator
  int32_t plain_elem;
};

enum SimtKind { SIMT_F32 = 0, SIMT_HALF = 1, SIMT_INT = 2 };

template <int KIND>
__device__ __forceinline__ uint32_t simt_load(const char* p, int es) {
  if constexpr (KIND == SIMT_F32) return __ldg((const uint32_t*)p);
  else if constexpr (KIND == SIMT_HALF) return __ldg((const uint16_t*)p);
  else {
    if (es == 4) return __ldg((const uint32_t*)p);
    if (es == 2) return __ldg((const uint16_t*)p);
    return __ldg((const uint8_t*)p);
  }
}
template <int KIND>
__device__ __forceinline__ uint32_t simt_decode(uint32_t raw, int elem) {
  if constexpr (KIND == SIMT_F32) return raw;
  else if constexpr (KIND == SIMT_HALF) return elem == EL_BF16 ? raw << 16 : f2u(__half2float(__ushort_as_half((unsigned short)raw)));
  else return vm_decode(raw, (uint8_t)elem);
}

// One operand's share of a slab: ROWS x 16 elements, ROWS * 16 / 256 per thread.  Threads run along k where k is
// contiguous in memory and along the rows otherwise.
template <int KIND, int ROWS>
struct SimtSide {
  static constexpr int E = ROWS * 16 / 256;
  const char* p;           // element 0 of this thread at k = 0 of the piece
  int64_t step, slab;      // bytes between a thread's elements, and from one slab to the next
  int row0, k0, drow, dk;  // element e: row row0 + e * drow, k k0 + e * dk of the slab
  __device__ __forceinline__ void begin(const char* base, int64_t srow, int64_t sk, int64_t row_at, int64_t k_at, int es) {
    if (sk == 1) { k0 = threadIdx.x & 15; row0 = threadIdx.x >> 4; dk = 0; drow = 16; }
    else { row0 = threadIdx.x % ROWS; k0 = threadIdx.x / ROWS; drow = 0; dk = 256 / ROWS; }
    p = base + ((row_at + row0) * srow + (k_at + k0) * sk) * es;
    step = (drow * srow + dk * sk) * es;
    slab = 16 * sk * es;
  }
  __device__ __forceinline__ void load(uint32_t (&raw)[E], int64_t rows_left, int64_t k_left, int es) {
#pragma unroll
    for (int e = 0; e < E; e++) raw[e] = (row0 + e * drow < rows_left && k0 + e * dk < k_left) ? simt_load<KIND>(p + e * step, es) : 0u;
    p += slab;
  }
  __device__ __forceinline__ void store(uint32_t* sm, const uint32_t (&raw)[E], int elem) const {
#pragma unroll
    for (int e = 0; e < E; e++) sm[(k0 + e * dk) * (ROWS + 4) + row0 + e * drow] = simt_decode<KIND>(raw[e], elem);
  }
};

__device__ __forceinline__ uint64_t simt_pair(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}

// V: 0 the program only stores the accumulator; 1 / 4 elements per run of the epilogue program.
template <int KIND, int BM, int V>
__global__ void __launch_bounds__(256) k_gemm_simt(const __grid_constant__ GemmK G, const __grid_constant__ B2xVmProgram P) {
  namespace cg = cooperative_groups;
  constexpr int BN = 64, TM = BM / 16, TN = 4;
  constexpr int A_WORDS = 16 * (BM + 4), B_WORDS = 16 * (BN + 4);
  constexpr int RING = 2 * (A_WORDS + B_WORDS), TILE = BM * BN;
  __shared__ __align__(16) uint32_t sm[RING > TILE ? RING : TILE];
  pdl_trigger();     // nothing to wait for: the operands come through the read-only path, so this kernel is launched in its turn
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int rank = G.CL > 1 ? (int)(blockIdx.x % (unsigned)G.CL) : 0;
  const unsigned tile = blockIdx.x / (unsigned)G.CL;
  const int64_t m0 = (int64_t)(tile / (unsigned)G.tiles_n) * BM, n0 = (int64_t)(tile % (unsigned)G.tiles_n) * BN;
  const int64_t kb = rank * G.k_piece, ke = min(G.K, kb + G.k_piece);
  for (int64_t bi = blockIdx.z; bi < G.batch; bi += gridDim.z) {
    uint64_t c[TM][TN / 2];          // pairs of f32 sums, or of 32-bit integer sums
#pragma unroll
    for (int i = 0; i < TM; i++) { c[i][0] = 0; c[i][1] = 0; }
    SimtSide<KIND, BM> A;
    SimtSide<KIND, BN> B;
    A.begin(G.a + bi * G.sab * G.es, G.sam, G.sak, m0, kb, G.es);
    B.begin(G.b + bi * G.sbb * G.es, G.sbn, G.sbk, n0, kb, G.es);
    uint32_t ra[SimtSide<KIND, BM>::E], rb[SimtSide<KIND, BN>::E];
    if (kb < ke) {
      A.load(ra, G.M - m0, ke - kb, G.es);
      B.load(rb, G.N - n0, ke - kb, G.es);
    }
    int buf = 0;
    for (int64_t k = kb; k < ke; k += 16) {
      uint32_t* sa = sm + buf * (A_WORDS + B_WORDS);
      uint32_t* sb = sa + A_WORDS;
      A.store(sa, ra, G.elem);
      B.store(sb, rb, G.elem);
      __syncthreads();               // also: everybody is done with the buffer that the next slab overwrites
      if (k + 16 < ke) {
        A.load(ra, G.M - m0, ke - k - 16, G.es);
        B.load(rb, G.N - n0, ke - k - 16, G.es);
      }
#pragma unroll
      for (int kk = 0; kk < 16; kk++) {
        uint32_t av[TM], bv[TN];
#pragma unroll
        for (int i = 0; i < TM; i += 4) *(uint4*)(av + i) = *(const uint4*)(sa + kk * (BM + 4) + (i / 4) * 64 + ty * 4);
        *(uint4*)bv = *(const uint4*)(sb + kk * (BN + 4) + tx * 4);
#pragma unroll
        for (int i = 0; i < TM; i++) {
          if constexpr (KIND == SIMT_INT) {
#pragma unroll
            for (int j = 0; j < 2; j++) {
              const uint32_t lo = (uint32_t)c[i][j] + av[i] * bv[2 * j], hi = (uint32_t)(c[i][j] >> 32) + av[i] * bv[2 * j + 1];
              c[i][j] = simt_pair(lo, hi);
            }
          } else {
            const uint64_t aa = simt_pair(av[i], av[i]);
#pragma unroll
            for (int j = 0; j < 2; j++)
              asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[i][j]) : "l"(aa), "l"(simt_pair(bv[2 * j], bv[2 * j + 1])));
          }
        }
      }
      buf ^= 1;
    }
    // the tile, row-major in shared memory; row of result i: 64 * (i / 4) + 4 * ty + i % 4
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; i++)
      *(uint4*)(sm + ((i / 4) * 64 + ty * 4 + (i & 3)) * BN + tx * 4) =
          make_uint4((uint32_t)c[i][0], (uint32_t)(c[i][0] >> 32), (uint32_t)c[i][1], (uint32_t)(c[i][1] >> 32));
    if (G.CL > 1) cg::this_cluster().sync(); else __syncthreads();
    constexpr int W = V == 0 ? 1 : V;
    const int share = TILE / G.CL;   // elements that this CTA finishes: whole rows of the tile
    for (int i = rank * share + (int)threadIdx.x * W; i < (rank + 1) * share; i += 256 * W) {
      const int64_t m = m0 + i / BN, n = n0 + i % BN;
      uint32_t v[W];
      if (G.CL > 1) {
#pragma unroll
        for (int j = 0; j < W; j++) v[j] = 0;
        for (int r = 0; r < G.CL; r++) {
          const uint32_t* o = cg::this_cluster().map_shared_rank(sm, r) + i;
#pragma unroll
          for (int j = 0; j < W; j++) v[j] = KIND == SIMT_INT ? v[j] + o[j] : f2u(u2f(v[j]) + u2f(o[j]));
        }
      } else {
#pragma unroll
        for (int j = 0; j < W; j++) v[j] = sm[i + j];
      }
      if (m < G.M && n < G.N) {
        const int64_t at = (bi * G.M + m) * G.N + n;
        if constexpr (V == 0) {
          const uint32_t e = vm_encode(v[0], (uint8_t)G.plain_elem);
          const int es = vm_elem_size((uint8_t)G.plain_elem);
          if (es == 4) ((uint32_t*)G.plain_out)[at] = e; else if (es == 2) ((uint16_t*)G.plain_out)[at] = (uint16_t)e; else ((uint8_t*)G.plain_out)[at] = (uint8_t)e;
        } else {
          uint32_t acc[V];
          vm_run<V>(P, (uint64_t)at, v, acc);
        }
      }
    }
    // the tile has been read, by the other CTAs of the cluster as well
    if (G.CL > 1) cg::this_cluster().sync(); else __syncthreads();
  }
}

// Whether the program is `load acc0; store T0` into the dense row-major result.
static bool simt_plain_store(const B2xVmProgram& P, const GemmK& G) {
  const B2xVmInstr* c = P.code;
  if (P.n_instr != 2 || P.n_tensors != 1 || c[0].op != VM_LOAD || c[0].src_kind != VM_SRC_ACC0 || c[0].rnd != VM_RN_NONE || c[1].op != VM_STORE ||
      c[1].src_kind != VM_SRC_TENSOR || c[1].src_idx != 0 || c[1].rnd != VM_RN_NONE || vm_elem_size(P.tensors[0].elem) > 4) return false;
  int64_t total = 1;
  for (int d = P.n_dims - 1; d >= 0; d--) {
    if (P.tensors[0].stride[d] != total && P.dim[d] != 1) return false;
    total *= P.dim[d];
  }
  return total == G.batch * G.M * G.N;
}

template <int KIND>
static int launch_simt(GemmK G, const B2xVmProgram& P, int vec, cudaStream_t stream) {
  // The 128-row tile does twice the work per byte of shared memory; it is taken when its tiles cover two thirds of the SMs.
  const int64_t tiles_n = (G.N + 63) / 64;
  const bool large = (G.M + 127) / 128 * tiles_n * G.batch >= kNumSms * 2 / 3;
  const int64_t tiles = (large ? (G.M + 127) / 128 : (G.M + 63) / 64) * tiles_n;
  // K is cut while that adds CTAs that fit (two per SM) and leaves each at least four slabs
  int CL = 1;
  while (CL < 8 && tiles * G.batch * CL < 2 * kNumSms && G.K >= (int64_t)CL * 2 * 64) CL *= 2;
  G.CL = CL;
  G.k_piece = (((G.K + CL - 1) / CL + 15) / 16) * 16;
  G.tiles_n = (int)tiles_n;
  if (tiles * CL > 0x7fffffff || tiles_n > 0x7fffffff) return (int)cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles * CL), 1, (unsigned)(G.batch > 1024 ? 1024 : G.batch));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)CL; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = CL > 1 ? 1 : 0;
  const int V = simt_plain_store(P, G) ? 0 : ((vec >= 4 && G.N % 4 == 0) ? 4 : 1);
  if (V == 0) { G.plain_out = (char*)P.tensors[0].ptr; G.plain_elem = P.tensors[0].elem; }
  cudaError_t e;
#define B2X_SIMT(BM_) (V == 0 ? cudaLaunchKernelEx(&cfg, k_gemm_simt<KIND, BM_, 0>, G, P) : V == 4 ? cudaLaunchKernelEx(&cfg, k_gemm_simt<KIND, BM_, 4>, G, P) \
                                                                                        : cudaLaunchKernelEx(&cfg, k_gemm_simt<KIND, BM_, 1>, G, P))
  if (large) e = B2X_SIMT(128); else e = B2X_SIMT(64);
#undef B2X_SIMT
  if (e != cudaSuccess) return (int)e;
  count_launch();
  return (int)cudaGetLastError();
}

}  // namespace b2x

extern "C" int b2x_launch_gemm_simt(const B2xGemmArgs* a, const B2xVmProgram* epilogue, int vec, b2x_stream_t stream_) {
  using namespace b2x;
  cudaStream_t stream = (cudaStream_t)stream_;
  if (a->batch <= 0 || a->M <= 0 || a->N <= 0) return 0;
  GemmK G{};
  G.a = (const char*)a->a; G.b = (const char*)a->b;
  G.elem = a->elem;
  switch (a->elem) {
    case EL_F32: case EL_S32: case EL_U32: G.es = 4; break;
    case EL_BF16: case EL_F16: case EL_S16: case EL_U16: G.es = 2; break;
    case EL_S8: case EL_U8: case EL_PRED: G.es = 1; break;
    default: return (int)cudaErrorInvalidValue;
  }
  const bool is_int = !(a->elem == EL_F32 || a->elem == EL_BF16 || a->elem == EL_F16);
  G.batch = a->batch; G.M = a->M; G.N = a->N; G.K = a->K;
  G.sab = a->a_batch_stride; G.sam = a->a_row_stride; G.sak = a->a_k_stride;
  G.sbb = a->b_batch_stride; G.sbn = a->b_row_stride; G.sbk = a->b_k_stride;
  if ((a->M + 63) / 64 > 65535) return (int)cudaErrorInvalidValue;
  if (is_int) return launch_simt<SIMT_INT>(G, *epilogue, vec, stream);
  return a->elem == EL_F32 ? launch_simt<SIMT_F32>(G, *epilogue, vec, stream) : launch_simt<SIMT_HALF>(G, *epilogue, vec, stream);
}
