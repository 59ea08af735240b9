// Entry points of the tcgen05 GEMM (kernel: gemm_tc.cuh) and the f32 hi/lo split used by the 3xTF32 scheme.
#include "gemm_tc.cuh"

#include <atomic>
#include <map>
#include <mutex>

namespace b2x {

static __device__ int32_t g_sched[kSchedSlots * 2];

// Scheduler pair for launches on `stream` of the current device.  Launches on one stream run in order, and a pair is
// back at zero when its launch retires, so every stream can keep one pair for good; launches that may overlap (different
// streams) never share a tile counter.  Only the address of the array is taken here; device code reads and resets it.
// Returns nullptr when more than kSchedSlots different streams have launched GEMMs on this device.
int32_t* sched_slot(cudaStream_t stream) {
  static std::mutex mu;
  static int32_t* base[64] = {};
  static std::map<cudaStream_t, int> slot_of[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!base[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_sched) != cudaSuccess) return nullptr;
    base[dev] = (int32_t*)p;
  }
  auto it = slot_of[dev].find(stream);
  if (it == slot_of[dev].end()) {
    if ((int)slot_of[dev].size() >= kSchedSlots) return nullptr;
    it = slot_of[dev].emplace(stream, (int)slot_of[dev].size()).first;
  }
  return base[dev] + 2 * it->second;
}

// ---- f32 -> hi/lo TF32 split for the 3xTF32 scheme ------------------------------------------------------------------
// out rows are K-major: sel 0 -> [hi | hi | lo] and sel 1 -> [hi | lo | hi] with 3K elements, sel 2 -> [hi | lo] with 2 ld
// elements, each half padded with zeros from K to ld.  One launch splits both operands, in tiles of 32 x 128.  A source that
// is contiguous along k is read along k, 16 bytes per lane where its rows allow; any other source is read along the rows and
// turned through shared memory.  Either way 16 values per thread are in flight before the first is needed, and the halves
// leave as 16-byte pieces of rows.  HBM-bound: 4 bytes in, 8 out per element (sel 2).  2 x [2048, 4096] contracted over the
// first dimension: 64 us with 32 x 32 tiles and 4 bytes per access; the whole product 389 -> 364 us.
// Elements of one half of a paired row: whole k-blocks, so that none straddles the two halves.
static int64_t paired_ld(int64_t K) { return (K + 31) / 32 * 32; }
struct SplitSide {
  const float* src; float* dst;
  int64_t rows, K, ld, pitch, sb, sr, sk;   // ld: elements of a half, pitch: of an output row
  int64_t tiles_r, tiles_k, n_tiles;
  int sel, wide;                            // wide: rows of the source can be read, rows of the result written, 16 bytes at a time
};
__device__ __forceinline__ float2 split_value(float x, bool& nonfinite) {
  const float hi = __uint_as_float(__float_as_uint(x) & 0xffffe000u);
  const float lo = __uint_as_float(__float_as_uint(x - hi) & 0xffffe000u);
  // an infinite value is its high half alone, and so is a NaN, made quiet: its set bits may all lie in the part cut off
  const bool special = (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u;
  nonfinite |= special;
  return special ? make_float2(x + x, 0.f) : make_float2(hi, lo);
}
__device__ __forceinline__ void split_write(const SplitSide& S, float* o, int64_t k, const float (&x)[4], bool& nonfinite) {
  float2 v[4];
#pragma unroll
  for (int j = 0; j < 4; j++) v[j] = split_value(x[j], nonfinite);
  if (S.wide) {
    const float4 hi = make_float4(v[0].x, v[1].x, v[2].x, v[3].x), lo = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
    *(float4*)(o + k) = hi;
    *(float4*)(o + S.ld + k) = S.sel == 0 ? hi : lo;
    if (S.sel != 2) *(float4*)(o + 2 * S.ld + k) = S.sel == 0 ? lo : hi;
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (k + j < S.ld) {
        o[k + j] = v[j].x;
        o[S.ld + k + j] = S.sel == 0 ? v[j].x : v[j].y;
        if (S.sel != 2) o[2 * S.ld + k + j] = S.sel == 0 ? v[j].y : v[j].x;
      }
  }
}
__global__ void __launch_bounds__(256, 4) k_split_f32(const __grid_constant__ SplitSide A, const __grid_constant__ SplitSide B, uint32_t* nonfinite) {
  __shared__ float tile[32][129];
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t total = A.n_tiles + B.n_tiles;
  bool bad = false;
  for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
    const bool second = t >= A.n_tiles;
    const SplitSide& S = second ? B : A;
    int64_t u = second ? t - A.n_tiles : t;
    const int64_t tk = u % S.tiles_k; u /= S.tiles_k;
    const int64_t tr = u % S.tiles_r;
    const int64_t b = u / S.tiles_r;
    const float* src = S.src + b * S.sb;
    float* dst = S.dst + b * S.rows * S.pitch;
    if (S.sk == 1) {
      // 32 rows x 128 k: a warp per row, four rows each
      const int64_t r0 = tr * 32 + warp, k = tk * 128 + lane * 4;
      float x[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int64_t r = r0 + i * 8;
        const float* p = src + r * S.sr + k;
#pragma unroll
        for (int j = 0; j < 4; j++) x[i][j] = 0.f;
        if (r < S.rows) {
          if (S.wide && k + 3 < S.K) {
            const float4 f = ld_global((const float4*)p);
            x[i][0] = f.x; x[i][1] = f.y; x[i][2] = f.z; x[i][3] = f.w;
          } else {
#pragma unroll
            for (int j = 0; j < 4; j++) if (k + j < S.K) x[i][j] = ld_global(p + j);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int64_t r = r0 + i * 8;
        if (r < S.rows && k < S.ld) split_write(S, dst + r * S.pitch, k, x[i], bad);
      }
    } else {
      // 128 rows x 32 k: read along the rows, four k lines per warp; written along k, eight lanes to a row's 128 bytes
      const int64_t r0 = tr * 128, k0 = tk * 32;
      float x[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int64_t k = k0 + warp * 4 + i, r = r0 + j * 32 + lane;
          x[i][j] = (r < S.rows && k < S.K) ? ld_global(src + r * S.sr + k * S.sk) : 0.0f;
        }
      __syncthreads();        // the previous tile has been written out
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) tile[warp * 4 + i][j * 32 + lane] = x[i][j];
      __syncthreads();
      const int kk = (lane & 7) * 4;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int rr = i * 32 + warp * 4 + (lane >> 3);
        const float y[4] = {tile[kk][rr], tile[kk + 1][rr], tile[kk + 2][rr], tile[kk + 3][rr]};
        if (r0 + rr < S.rows && k0 + kk < S.ld) split_write(S, dst + (r0 + rr) * S.pitch, k0 + kk, y, bad);
      }
    }
  }
  bad = __syncthreads_or(bad);
  if (nonfinite && threadIdx.x == 0) nonfinite[blockIdx.x] = bad ? 1u : 0u;
}

constexpr int kSplitCtas = kNumSms * 8;
// `nonfinite`: kSplitCtas words, or null; *n_nonfinite (may be null): how many of them are written.
static int launch_split(const B2xGemmArgs* a, float* a_split, float* b_split, bool paired, uint32_t* nonfinite, int32_t* n_nonfinite, cudaStream_t stream) {
  if (a->elem != EL_F32) return (int)cudaErrorInvalidValue;
  auto side = [&](const void* src, float* dst, int64_t rows, int64_t sb, int64_t sr, int64_t sk, int sel) {
    SplitSide s{};
    s.src = (const float*)src; s.dst = dst; s.rows = rows; s.K = a->K; s.sb = sb; s.sr = sr; s.sk = sk; s.sel = sel;
    s.ld = paired ? paired_ld(a->K) : a->K; s.pitch = paired ? 2 * s.ld : 3 * a->K;
    const int tr = sk == 1 ? 32 : 128, tk = sk == 1 ? 128 : 32;
    s.tiles_r = (rows + tr - 1) / tr; s.tiles_k = (s.ld + tk - 1) / tk; s.n_tiles = a->batch * s.tiles_r * s.tiles_k;
    s.wide = (uintptr_t)dst % 16 == 0 && s.ld % 4 == 0 && s.pitch % 4 == 0 && (sk != 1 || ((uintptr_t)src % 16 == 0 && sr % 4 == 0 && (a->batch == 1 || sb % 4 == 0)));
    return s;
  };
  const SplitSide A = side(a->a, a_split, a->M, a->a_batch_stride, a->a_row_stride, a->a_k_stride, paired ? 2 : 0);
  const SplitSide B = side(a->b, b_split, a->N, a->b_batch_stride, a->b_row_stride, a->b_k_stride, paired ? 2 : 1);
  int64_t grid = A.n_tiles + B.n_tiles;
  if (grid > kSplitCtas) grid = kSplitCtas;
  if (n_nonfinite) *n_nonfinite = (int32_t)grid;
  if (grid < 1) return 0;
  const cudaError_t e = launch_overlapped(k_split_f32, dim3((unsigned)grid), dim3(256), 0, stream, A, B, nonfinite);
  if (e != cudaSuccess) return (int)e;
  count_launch(1);
  return (int)cudaGetLastError();
}
}  // namespace b2x

extern "C" int b2x_launch_split_f32(const B2xGemmArgs* a, float* a_split, float* b_split, b2x_stream_t stream) {
  return b2x::launch_split(a, a_split, b_split, false, nullptr, nullptr, (cudaStream_t)stream);
}

namespace b2x {
// Everything the launcher decides from the problem's shape and the epilogue program, before any device work.
struct TcRoute {
  bool tf32 = false, a_mn = false, b_mn = false;
  int es = 2, BK = 64, CHUNK = 64, BN = 256;
  int64_t a_ld = 0, b_ld = 0;
  int static_id = 0;        // build-time specialised epilogue that will run (0: the interpreter)
  TcParams p{};
};

// paired: the operands are rows of [hi | lo] (TcParams::paired), K counts one half
static int tc_route(const B2xGemmArgs* a, const B2xVmProgram* epilogue, bool paired, TcRoute* r) {
  if (a->batch <= 0 || a->M <= 0 || a->N <= 0 || a->K <= 0) return (int)cudaErrorInvalidValue;
  r->tf32 = a->elem == EL_F32;
  if (!r->tf32 && a->elem != EL_BF16 && a->elem != EL_F16) return (int)cudaErrorInvalidValue;
  const int es = r->es = r->tf32 ? 4 : 2;
  const int BK = r->BK = 128 / es;
  r->CHUNK = 128 / es;
  const int64_t al = 16 / es;
  r->a_mn = !(a->a_k_stride == 1) && a->a_row_stride == 1;
  r->b_mn = !(a->b_k_stride == 1) && a->b_row_stride == 1;
  if (!r->a_mn && a->a_k_stride != 1) return (int)cudaErrorInvalidValue;
  if (!r->b_mn && a->b_k_stride != 1) return (int)cudaErrorInvalidValue;
  r->a_ld = r->a_mn ? a->a_k_stride : a->a_row_stride;
  r->b_ld = r->b_mn ? a->b_k_stride : a->b_row_stride;
  if (r->a_ld % al || r->b_ld % al || (a->batch > 1 && (a->a_batch_stride % al || a->b_batch_stride % al))) return (int)cudaErrorInvalidValue;
  if (a->N % 8) return (int)cudaErrorInvalidValue;
  // widest tile that the result allows; a problem with fewer tiles than half the SMs takes narrower ones, so that
  // more SMs share the operand traffic (each CTA streams its own A and B tiles)
  int BN = a->N >= 256 ? 256 : (a->N >= 128 ? 128 : 64);
  {
    const int64_t m_tiles = (a->M + TC_BM - 1) / TC_BM;
    while (BN > 64 && m_tiles * ((a->N + BN - 1) / BN) * a->batch < kNumSms / 2) BN /= 2;
  }
  r->BN = BN;
  TcParams& p = r->p;
  p.batch = a->batch; p.M = a->M; p.N = a->N; p.K = a->K;
  p.a_mn_major = r->a_mn; p.b_mn_major = r->b_mn;
  p.num_m_tiles = (int)((a->M + TC_BM - 1) / TC_BM);
  p.num_n_tiles = (int)((a->N + BN - 1) / BN);
  p.num_tiles = (int64_t)p.num_m_tiles * p.num_n_tiles * a->batch;
  if (p.num_tiles >= (1ll << 31)) return (int)cudaErrorInvalidValue;
  p.k_blocks = (int)((a->K + BK - 1) / BK);
  p.transposed = a->K <= 8192 ? 1 : 0;
  p.paired = paired ? 1 : 0;
  p.lo_off = paired ? (int32_t)paired_ld(a->K) : 0;
  p.epi_groups = p.k_blocks * (paired ? 3 : 1) <= 8 ? 1 : 2;
  // Tall (256 x 256) tiles: long-K 16-bit problems whose tall tiles still fill the last round of the 148 SMs.  Their
  // epilogue is not overlapped, so K must be long enough to make it small; B2X_GEMM_TALL=0 / 1 switches them off / forces
  // them wherever the kernel can run them.
  p.tall = 0;
  // short K: three stages, the fourth holds the second set of staging tiles of the bulk-store epilogue (gemm_tc.cuh)
  p.short_k = (BN == 256 && !r->tf32 && p.k_blocks <= 3) ? 1 : 0;
  { static const int sk = [] { const char* e = getenv("B2X_GEMM_SHORT_K"); return e ? atoi(e) : -1; }(); if (sk == 0) p.short_k = 0; }
  int64_t bm = TC_BM;
  if (!r->tf32 && BN == 256 && a->M >= 2 * TC_BM) {
    static const int mode = [] { const char* e = getenv("B2X_GEMM_TALL"); return e ? atoi(e) : -1; }();
    // how full the rounds of the 148 SMs are with either tile height; tall tiles were measured 20-25 % faster per FLOP
    // (MLP step, K = 4096 ... 16384), so they are taken unless their last round wastes more than that
    const int64_t tall_tiles = ((a->M + 2 * TC_BM - 1) / (2 * TC_BM)) * p.num_n_tiles * a->batch;
    auto fill = [](int64_t tiles) { const int64_t rounds = (tiles + kNumSms - 1) / kNumSms; return (double)tiles / (double)(rounds * kNumSms); };
    const bool pays = fill(tall_tiles) * 1.2 > fill(p.num_tiles);
    if (mode == 1 || (mode != 0 && p.k_blocks >= 32 && pays)) {
      p.tall = 1;
      p.epi_groups = 2;
      p.transposed = 1;   // the epilogue of a tall tile is not hidden behind the next tile, so the form with fewer store cycles wins at every K
      bm = 2 * TC_BM;
      p.num_m_tiles = (int)((a->M + bm - 1) / bm);
      p.num_tiles = (int64_t)p.num_m_tiles * p.num_n_tiles * a->batch;
    }
  }
  {
    // A slab of a group ~ 32 MiB (a quarter of the 126 MB L2)
    const int64_t slab_per_m_tile = bm * a->K * es * (paired ? 2 : 1);
    int64_t gm = (32ll << 20) / (slab_per_m_tile > 0 ? slab_per_m_tile : 1);
    if (gm < 4) gm = 4;
    if (gm > 64) gm = 64;
    if (gm > p.num_m_tiles) gm = p.num_m_tiles;
    p.group_m = (int)gm;
  }
  p.idesc = sm100::make_idesc(r->tf32 ? 2u : (a->elem == EL_BF16 ? 1u : 0u), r->a_mn, r->b_mn, TC_BM, (uint32_t)BN);
  const int id = vm_static_enabled() ? vm_static_lookup(vm_signature_hash(*epilogue)) : 0;
  r->static_id = (id && (r->tf32 ? tc_static_has_tf32(id, BN) : tc_static_has(id, BN))) ? id : 0;
  return 0;
}
}  // namespace b2x

namespace b2x {
// The product that the tensor cores make of an f32 problem once its operands lie in scratch as rows of [hi | lo]: K stays.
static B2xGemmArgs paired_problem(const B2xGemmArgs& a) {
  B2xGemmArgs g = a;
  g.a_k_stride = g.b_k_stride = 1;
  g.a_row_stride = g.b_row_stride = 2 * paired_ld(a.K);
  g.a_batch_stride = a.M * g.a_row_stride;
  g.b_batch_stride = a.N * g.b_row_stride;
  return g;
}

static int report_route(const B2xGemmArgs& a, const B2xVmProgram* epilogue, bool paired, int32_t out[12]) {
  TcRoute r;
  int rc = tc_route(&a, epilogue, paired, &r);
  if (rc) return rc;
  out[0] = r.BN; out[1] = r.static_id; out[2] = r.p.epi_groups;
  out[3] = (r.static_id && r.p.transposed && tc_static_stores(r.static_id) >= 2) ? 1 : 0;
  out[4] = r.p.group_m; out[5] = r.p.num_m_tiles; out[6] = r.p.num_n_tiles; out[7] = r.p.k_blocks;
  out[8] = r.static_id ? tc_static_stores(r.static_id) : 0;
  out[9] = (int32_t)(r.p.num_tiles < kNumSms ? r.p.num_tiles : kNumSms);
  out[10] = r.p.tall ? 2 * TC_BM : TC_BM;
  out[11] = r.p.paired;
  return 0;
}
}  // namespace b2x

extern "C" int b2x_gemm_tc_route(const B2xGemmArgs* a, const B2xVmProgram* epilogue, int32_t out[12]) {
  return b2x::report_route(*a, epilogue, false, out);
}

extern "C" int b2x_gemm_f32_route(const B2xGemmArgs* a, const B2xVmProgram* epilogue, int32_t out[12]) {
  if (a->elem != EL_F32) return (int)cudaErrorInvalidValue;
  return b2x::report_route(b2x::paired_problem(*a), epilogue, true, out);
}

namespace b2x {
// nonfinite, n_nonfinite: see launch_split; for paired operands only
static int launch_gemm_tc(const B2xGemmArgs* a, const B2xVmProgram* epilogue, bool paired, const uint32_t* nonfinite, int32_t n_nonfinite, int32_t* status,
                          cudaStream_t stream) {
  TcRoute r;
  int rc = tc_route(a, epilogue, paired, &r);
  if (rc) return rc;
  if (((uintptr_t)a->a & 15) || ((uintptr_t)a->b & 15)) return (int)cudaErrorInvalidValue;
  const bool tf32 = r.tf32, a_mn = r.a_mn, b_mn = r.b_mn;
  const int es = r.es, BK = r.BK, CHUNK = r.CHUNK, BN = r.BN;
  const int64_t a_ld = r.a_ld, b_ld = r.b_ld;
  CUtensorMapDataType dt = tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : (a->elem == EL_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
  CUtensorMap tmA, tmB;
  bool ok;
  TcParams p = r.p;
  p.nonfinite = nonfinite;
  p.n_nonfinite = n_nonfinite;
  p.split_a = paired ? (const float*)a->a : nullptr;
  p.split_b = paired ? (const float*)a->b : nullptr;
  // B2X_GEMM_LOADS=3d keeps one load per 128-byte-wide sub-tile of an MN-major operand (for comparison)
  static const bool folded = [] { const char* e = getenv("B2X_GEMM_LOADS"); return !(e && e[0] == '3'); }();
  p.a_mn_4d = p.b_mn_4d = 0;
  const uint64_t k_extent = paired ? 2 * (uint64_t)paired_ld(a->K) : (uint64_t)a->K;
  const uint32_t bm = p.tall ? 2 * TC_BM : TC_BM;   // rows of A per stage
  if (!a_mn) ok = encode_3d(&tmA, dt, es, a->a, k_extent, (uint64_t)a->M, (uint64_t)a->batch, (uint64_t)a_ld, (uint64_t)a->a_batch_stride, BK, bm);
  else {
    ok = folded && encode_mn_major_4d(&tmA, dt, es, a->a, (uint64_t)a->M, (uint64_t)a->K, (uint64_t)a->batch, (uint64_t)a_ld, (uint64_t)a->a_batch_stride, CHUNK, BK, bm);
    if (ok) p.a_mn_4d = 1;
    else ok = encode_3d(&tmA, dt, es, a->a, (uint64_t)a->M, (uint64_t)a->K, (uint64_t)a->batch, (uint64_t)a_ld, (uint64_t)a->a_batch_stride, CHUNK, BK);
  }
  if (!ok) return (int)cudaErrorInvalidValue;
  if (!b_mn) ok = encode_3d(&tmB, dt, es, a->b, k_extent, (uint64_t)a->N, (uint64_t)a->batch, (uint64_t)b_ld, (uint64_t)a->b_batch_stride, BK, BN);
  else {
    ok = folded && encode_mn_major_4d(&tmB, dt, es, a->b, (uint64_t)a->N, (uint64_t)a->K, (uint64_t)a->batch, (uint64_t)b_ld, (uint64_t)a->b_batch_stride, CHUNK, BK, BN);
    if (ok) p.b_mn_4d = 1;
    else ok = encode_3d(&tmB, dt, es, a->b, (uint64_t)a->N, (uint64_t)a->K, (uint64_t)a->batch, (uint64_t)b_ld, (uint64_t)a->b_batch_stride, CHUNK, BK);
  }
  if (!ok) return (int)cudaErrorInvalidValue;
  if (tf32) {
    if (r.static_id) {
      rc = launch_tc_static_tf32(r.static_id, BN, tmA, tmB, p, *epilogue, status, stream);
      if (rc >= 0) return rc;
    }
    if (BN == 256) return launch_tc<256, 4, true, 0>(tmA, tmB, p, *epilogue, status, stream);
    if (BN == 128) return launch_tc<128, 6, true, 0>(tmA, tmB, p, *epilogue, status, stream);
    return launch_tc<64, 8, true, 0>(tmA, tmB, p, *epilogue, status, stream);
  }
  if (r.static_id) {
    rc = launch_tc_static(r.static_id, BN, tmA, tmB, p, *epilogue, status, stream);
    if (rc >= 0) return rc;
  }
  if (BN == 256) return launch_tc<256, 4, false, 0>(tmA, tmB, p, *epilogue, status, stream);
  if (BN == 128) return launch_tc<128, 6, false, 0>(tmA, tmB, p, *epilogue, status, stream);
  return launch_tc<64, 8, false, 0>(tmA, tmB, p, *epilogue, status, stream);
}
}  // namespace b2x

extern "C" int b2x_launch_gemm_tc(const B2xGemmArgs* a, const B2xVmProgram* epilogue, int32_t* status, b2x_stream_t stream) {
  return b2x::launch_gemm_tc(a, epilogue, false, nullptr, 0, status, (cudaStream_t)stream);
}

extern "C" int64_t b2x_gemm_f32_scratch_bytes(int64_t batch, int64_t M, int64_t N, int64_t K) {
  const int64_t pitch = 2 * b2x::paired_ld(K) * 4;
  return (batch * M * pitch + 1023) / 1024 * 1024 + batch * N * pitch + b2x::kSplitCtas * 4;   // pitch: whole 256 bytes
}

extern "C" int b2x_launch_gemm_f32(const B2xGemmArgs* a, const B2xVmProgram* epilogue, void* scratch, int32_t* status, b2x_stream_t stream_) {
  using namespace b2x;
  cudaStream_t stream = (cudaStream_t)stream_;
  if (a->elem != EL_F32 || !scratch || paired_ld(a->K) > (1ll << 29)) return (int)cudaErrorInvalidValue;
  B2xGemmArgs g = paired_problem(*a);
  char* b_split = (char*)scratch + (a->batch * g.a_batch_stride * 4 + 1023) / 1024 * 1024;
  g.a = scratch; g.b = b_split;
  uint32_t* nonfinite = (uint32_t*)(b_split + a->batch * g.b_batch_stride * 4);
  int32_t n_nonfinite = 0;
  int rc = launch_split(a, (float*)scratch, (float*)b_split, true, nonfinite, &n_nonfinite, stream);
  if (rc) return rc;
  return launch_gemm_tc(&g, epilogue, true, nonfinite, n_nonfinite, status, stream);
}
