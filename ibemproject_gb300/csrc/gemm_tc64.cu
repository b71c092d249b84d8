// FP64 trailing updates of the dense factorisation on the tensor cores:  C -= A * B with FP64
// storage on sm_103a's BF16 tcgen05 pipe (Ozaki's error-free splitting).
//
// Why: GB300's FP64 pipe does 2 multiply-adds per clock and SM (0.60 T/s measured), so a SIMT
// FP64 update is bound by it whatever its tiling; the BF16 tensor pipe does 3,200 times as
// many, and 28 BF16 products carry one FP64 product.
//
// Scheme.  Row i of A is written as 2^ea_i times fixed-point numbers of 55 bits and a sign (the
// largest one between 2^54 and 2^55), column j of B likewise, and each number as seven signed
// 8-bit digits (|d| <= 128, exact in BF16).  The digit products of equal weight, g = p + q, are
// summed in one FP32 accumulator of TMEM: over a chunk of 192 columns |sum| <= (g + 1) 192 128^2
// = (g + 1) 3 2^20, which FP32 holds exactly for g <= 4.  g = 5 and 6 (weights 2^-40 and below of
// the leading one) lose the units of a few additions past 2^24, for data whose digits are all
// of one sign and near the largest: below 0.1 k 2^-53 of what the bound below counts in.
// (Chunks of 256 columns let g = 4 past 2^24 too; the additions truncate, and such data came
// out off by 7 k 2^-53.)  After every chunk the accumulators are added to two 64-bit integers
// per entry (g <= 3 and g >= 4, exact), which are converted to FP64 once at the end.
//
// Accuracy is to the largest entry of a row and column, not to each entry.  In units where the
// largest products are 2^108 to 2^110, the products left out (g >= 7) are worth at most 6.03
// 2^54 a term and the rounding of the two operands 2 2^54: an entry of the product is off by at
// most 4.1 k 2^-53 max|a_i.| max|b_.j|, typically far less than the rounding of an FP64 sum of k
// products (tests/test_gemm64_product.py).  Entries that are small beside their row keep fewer
// than 53 bits: the solve gives the digits that this costs back by a step of refinement
// (solver.cu).  A row or column that holds an infinity or NaN gives NaN in its whole row or
// column of C.
//
// Measured (random normal entries): 3600^3 28 TFLOP/s, 8192 x 8192 x 2048 31 TFLOP/s (the FP64
// pipe gives 1.2), rms error 7e-18 and 9e-18 of sum |a||b| where FP64 multiply-adds give 5e-17.
//
// Kernels: k_split64 makes the digit planes (one pass for the exponents, one for the digits,
// the second from L2), K-major as the MMA reads them; k_umma_f64 is one CTA per 128 x 64
// tile: a TMA producer warp (two 86 KB stages of 32 columns x 7 digit planes of A and B), an
// MMA warp (56 tcgen05.mma of 128 x 64 x 16 per stage into seven accumulators of 64 TMEM
// columns), eight epilogue warps.  The tile is as wide as seven accumulators allow (448 of
// 512 TMEM columns).  The accumulators are read back once per 192 columns, about an eighth of
// the chunk's MMA time, so they are not double-buffered.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "prof.h"
#include "solver.h"
#include "umma.cuh"

namespace ibem {
namespace {

constexpr int NS = 7;                               // digits of an operand, accumulators
constexpr int BM = 128, BN = 64, BK = 32, STAGES = 2;
constexpr int CHUNK = 6;                            // K blocks between two readings of the accumulators (192 columns)
constexpr int A_PLANE = BM * BK * 2, B_PLANE = BN * BK * 2;   // 8 and 4 KB
constexpr int STAGE_BYTES = NS * (A_PLANE + B_PLANE);         // 86,016
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
constexpr int EPI_WARPS = 8, THREADS = 32 * (EPI_WARPS + 2);
constexpr int TMEM_COLS = 512;
constexpr int GROUP_M = 16;                         // tile order: groups of 16 row tiles, columns inner
constexpr int64_t kMaxK = 2048;                     // columns per call of the kernel (bounds the digit planes)
constexpr uint32_t kIdesc = umma_idesc(BN);

// ---------------------------------------------------------------- digits
// Exponent field of a row's scale: at least 32, so that the scale 2^(E - 1041) is a normal
// number; entries below 2^-1046 then round to zero.
__device__ __forceinline__ int scale_field(int maxhi) { return max(maxhi >> 20, 32); }
__device__ __forceinline__ double scale_of(int maxhi) {
  if ((maxhi >> 20) == 0x7ff) return __longlong_as_double(0x7ff8000000000000LL);
  return __longlong_as_double((long long)(scale_field(maxhi) - 1041 + 1023) << 52);
}
// the seven digits of x, most significant first, each as the bits of a BF16 integer
__device__ __forceinline__ void digits7(double x, int field, uint32_t (&d)[NS]) {
  const long long bits = __double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7ff);
  long long f = (bits & 0xfffffffffffffLL) | 0x10000000000000LL;
  const int s = ex - field + 2;                     // at most 2: |f| < 2^55
  if (ex == 0 || ex == 0x7ff || s < -54) f = 0;     // (non-finite: the scale is NaN)
  else if (s >= 0) f <<= s;
  else f = (f + (1LL << (-s - 1))) >> -s;
  if (bits < 0) f = -f;
  f += 0x808080808080LL;                            // bytes 0..5 become digit + 128
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    // byte b in the mantissa of 2^23: subtracting 2^23 + 128 leaves the integer b - 128; the
    // top digit (f >> 48, in [-128, 128]) is shifted by 256 the same way
    const uint32_t b = i == 0 ? (uint32_t)((int)(f >> 48) + 256) : (uint32_t)(f >> (8 * (6 - i))) & 0xffu;
    const float v = __uint_as_float(0x4b000000u | b) - (i == 0 ? 8388608.0f + 256.0f : 8388608.0f + 128.0f);
    d[i] = __float_as_uint(v) >> 16;
  }
}
__device__ __forceinline__ void put8(const double (&v)[8], int field, __nv_bfloat16* out, int64_t plane) {
  uint32_t w[NS][4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    uint32_t d0[NS], d1[NS];
    digits7(v[2 * t], field, d0);
    digits7(v[2 * t + 1], field, d1);
#pragma unroll
    for (int i = 0; i < NS; ++i) w[i][t] = d0[i] | (d1[i] << 16);
  }
#pragma unroll
  for (int i = 0; i < NS; ++i)
    *reinterpret_cast<uint4*>(out + i * plane) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// Digit planes of A (m x k, first mb blocks: 32 rows each) and B (k x n, the other blocks: 32
// columns each).  Planes are [digit][row or column][kp], rows padded with zeros to mp and np.
// 256 threads.  A: lane = row, so loads are coalesced down the columns; B: a warp takes four
// columns, a lane 8 consecutive entries of one.
__global__ void __launch_bounds__(256) k_split64(int m, int n, int k, int kp, int mp, int np,
                                                 const double* __restrict__ A, int64_t lda,
                                                 const double* __restrict__ B, int64_t ldb,
                                                 __nv_bfloat16* __restrict__ pa, __nv_bfloat16* __restrict__ pb,
                                                 double* __restrict__ sa, double* __restrict__ sb, int mb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int)blockIdx.x < mb) {
    __shared__ int smax[8][32];
    const int row = blockIdx.x * 32 + lane;
    const bool in = row < m;
    const double* a = A + row;
    int mx = 0;
    if (in) {
#pragma unroll 8
      for (int c = warp; c < k; c += 8) mx = max(mx, __double2hiint(a[c * lda]) & 0x7fffffff);
    }
    smax[warp][lane] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) mx = max(mx, smax[w][lane]);
    if (warp == 0) sa[row] = scale_of(mx);
    const int field = scale_field(mx);
    const int64_t plane = (int64_t)mp * kp;
    for (int c0 = 8 * warp; c0 < kp; c0 += 64) {
      double v[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = in && c0 + t < k ? a[(c0 + t) * lda] : 0.0;
      put8(v, field, pa + (int64_t)row * kp + c0, plane);
    }
  } else {
    const int64_t plane = (int64_t)np * kp;
    for (int q = 0; q < 4; ++q) {
      const int col = ((int)blockIdx.x - mb) * 32 + 4 * warp + q;
      const bool in = col < n;
      const double* b = B + (int64_t)col * ldb;
      int mx = 0;
      if (in) {
#pragma unroll 8
        for (int r = lane; r < k; r += 32) mx = max(mx, __double2hiint(b[r]) & 0x7fffffff);
      }
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0) sb[col] = scale_of(mx);
      const int field = scale_field(mx);
      for (int r0 = 8 * lane; r0 < kp; r0 += 256) {
        double v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] = in && r0 + t < k ? b[r0 + t] : 0.0;
        put8(v, field, pb + (int64_t)col * kp + r0, plane);
      }
    }
  }
}

// ---------------------------------------------------------------- the GEMM kernel
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

__global__ void __launch_bounds__(THREADS, 1)
    k_umma_f64(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tB, double* __restrict__ C,
               int64_t ldc, int m, int n, int kblocks, const double* __restrict__ sa, const double* __restrict__ sb,
               int* err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + STAGES * STAGE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 3);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
  const uint32_t ready = smem_u32(bars + 2 * STAGES), drained = smem_u32(bars + 2 * STAGES + 1),
                 settled = smem_u32(bars + 2 * STAGES + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tm, tn;
  {
    const int tiles_m = (m + BM - 1) / BM, tiles_n = (n + BN - 1) / BN;
    const int b = blockIdx.x, per_group = GROUP_M * tiles_n;
    const int first = (b / per_group) * GROUP_M, gsz = min(GROUP_M, tiles_m - first);
    tm = first + (b % per_group) % gsz;
    tn = (b % per_group) / gsz;
  }
  const int m0 = tm * BM, n0 = tn * BN;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(ready, 1);
    mbar_init(drained, EPI_WARPS);
    mbar_init(settled, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int chunks = (kblocks + CHUNK - 1) / CHUNK;

  if (warp == EPI_WARPS) {
    if (lane == 0) {
      // ---- TMA producer
      int issued[STAGES] = {};
      for (int kb = 0; kb < kblocks; ++kb) {
        const int s = kb % STAGES;
        if (kb >= STAGES && !mbar_wait(empty0 + 8 * s, (uint32_t)((kb / STAGES - 1) & 1), err)) break;
        unsigned char* st = base + s * STAGE_BYTES;
        const uint32_t fb = full0 + 8 * s;
        mbar_expect_tx(fb, STAGE_BYTES);
        tma_load_3d(smem_u32(st), &tA, fb, kb * BK, m0, 0);
        tma_load_3d(smem_u32(st + NS * A_PLANE), &tB, fb, kb * BK, n0, 0);
        ++issued[s];
      }
      // copies still in flight (only on an early exit) are waited for, bounded
      for (int s = 0; s < STAGES; ++s)
        if (issued[s]) mbar_settle(full0 + 8 * s, (uint32_t)((issued[s] - 1) & 1));
    }
  } else if (warp == EPI_WARPS + 1) {
    if (lane == 0) {
      // ---- MMA issuer
      for (int kb = 0; kb < kblocks; ++kb) {
        const int s = kb % STAGES, ch = kb / CHUNK;
        if (kb % CHUNK == 0 && ch > 0 && !mbar_wait(drained, (uint32_t)((ch - 1) & 1), err)) break;
        if (!mbar_wait(full0 + 8 * s, (uint32_t)((kb / STAGES) & 1), err)) break;
        tc_fence_after();
        const uint32_t a0 = smem_u32(base + s * STAGE_BYTES), b0 = a0 + NS * A_PLANE;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
#pragma unroll
          for (int g = 0; g < NS; ++g)
#pragma unroll
            for (int p = 0; p <= g; ++p)
              umma(tmem + g * BN, umma_desc(a0 + p * A_PLANE + kk * 32), umma_desc(b0 + (g - p) * B_PLANE + kk * 32), kIdesc,
                   (uint32_t)((kb % CHUNK) | kk | p));
        umma_commit(empty0 + 8 * s);
        if (kb % CHUNK == CHUNK - 1 || kb == kblocks - 1) umma_commit(ready);
      }
      umma_commit(settled);   // no MMA may be in flight when the TMEM is freed, also after an early exit
      mbar_settle(settled, 0);
    }
  } else {
    // ---- epilogue: warp w reads the TMEM lanes (rows) of its quarter w % 4, columns of half w / 4
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t t0 = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(half * (BN / 2));
    long long hi[BN / 2], lo[BN / 2];
#pragma unroll
    for (int j = 0; j < BN / 2; ++j) hi[j] = lo[j] = 0;
    bool ok = true;
    for (int ch = 0; ch < chunks; ++ch) {
      ok = __all_sync(0xffffffffu, mbar_wait(ready, (uint32_t)(ch & 1), err));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int j0 = 0; j0 < BN / 2; j0 += 4) {
        uint32_t r[NS][4];
#pragma unroll
        for (int g = 0; g < NS; ++g) tmem_ld4(t0 + g * BN + j0, r[g]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          int v[NS];
#pragma unroll
          for (int g = 0; g < NS; ++g) v[g] = __float2int_rn(__uint_as_float(r[g][j]));
          hi[j0 + j] += (long long)v[0] * (1 << 24) + (long long)v[1] * (1 << 16) + (long long)v[2] * (1 << 8) + v[3];
          lo[j0 + j] += (long long)v[4] * (1 << 16) + (long long)v[5] * (1 << 8) + v[6];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(drained);
    }
    const int row = m0 + 32 * quarter + lane;
    if (ok && row < m) {
      const double fa = sa[row];
      double* c = C + row;
#pragma unroll
      for (int j0 = 0; j0 < BN / 2; j0 += 8) {
        double cv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = n0 + half * (BN / 2) + j0 + j;
          cv[j] = col < n ? c[(int64_t)col * ldc] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = n0 + half * (BN / 2) + j0 + j;
          // 2^-24 and the 2^36 in each scale undo the digits' weights
          const double v = fma((double)lo[j0 + j], 0x1p-24, (double)hi[j0 + j]);
          if (col < n) c[(int64_t)col * ldc] = fma(-(v * fa), sb[col], cv[j]);
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------- host side
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;
bool g_attr_set[64] = {};
std::mutex g_attr_mu;

ibem_status encode_planes(CUtensorMap* map, const __nv_bfloat16* ptr, int64_t rows, int64_t kp, uint32_t box_rows) {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  if (!g_encode) return fail(IBEM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  const cuuint64_t dims[3] = {(cuuint64_t)kp, (cuuint64_t)rows, NS};
  const cuuint64_t strides[2] = {(cuuint64_t)kp * sizeof(__nv_bfloat16), (cuuint64_t)(kp * rows) * sizeof(__nv_bfloat16)};
  const cuuint32_t box[3] = {BK, box_rows, NS};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(ptr), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(IBEM_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return IBEM_OK;
}

constexpr int64_t pad_to(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

}  // namespace

// planes of mp + np rows and the scales; a 256-byte boundary before each part
size_t gemm_tc64_workspace_bytes(int64_t max_m, int64_t max_n) {
  const int64_t rows = pad_to(max_m, BM) + pad_to(max_n, BN);
  return (size_t)rows * (kMaxK * NS * sizeof(__nv_bfloat16) + sizeof(double)) + 4 * 256;
}

ibem_status gemm_sub_f64_tc(int64_t m, int64_t n, int64_t k, const double* A, int64_t lda, const double* B,
                            int64_t ldb, double* C, int64_t ldc, void* ws, size_t ws_bytes, int* err,
                            cudaStream_t st) {
  if (m <= 0 || n <= 0 || k <= 0) return IBEM_OK;
  if (m > (1 << 30) || n > (1 << 30)) return fail(IBEM_ERR_ARG, "gemm_tc64: dimension too large");
  int dev = 0;
  IBEM_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(g_attr_mu);
    if (dev >= 64 || !g_attr_set[dev]) {
      IBEM_CUDA(cudaFuncSetAttribute((const void*)k_umma_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
      if (dev < 64) g_attr_set[dev] = true;
    }
  }
  const int64_t mp = pad_to(m, BM), np = pad_to(n, BN);
  for (int64_t k0 = 0; k0 < k; k0 += kMaxK) {
    const int64_t kc = std::min<int64_t>(kMaxK, k - k0), kp = pad_to(kc, BK);
    unsigned char* w = static_cast<unsigned char*>(ws);
    auto take = [&](size_t bytes) {
      unsigned char* q = w;
      w += (bytes + 255) / 256 * 256;
      return q;
    };
    __nv_bfloat16* pa = reinterpret_cast<__nv_bfloat16*>(take((size_t)NS * mp * kp * sizeof(__nv_bfloat16)));
    __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(take((size_t)NS * np * kp * sizeof(__nv_bfloat16)));
    double* sa = reinterpret_cast<double*>(take(mp * sizeof(double)));
    double* sb = reinterpret_cast<double*>(take(np * sizeof(double)));
    if ((size_t)(w - static_cast<unsigned char*>(ws)) > ws_bytes) return fail(IBEM_ERR_ARG, "gemm_tc64: workspace too small");
    const int mb = (int)(mp / 32), nb = (int)(np / 32);
    {
      ProfScope ps(PROF_GEMM_SPLIT, st);
      ::ibem::count_launch(), k_split64<<<mb + nb, 256, 0, st>>>((int)m, (int)n, (int)kc, (int)kp, (int)mp, (int)np,
                                                                 A + k0 * lda, lda, B + k0, ldb, pa, pb, sa, sb, mb);
      IBEM_LAUNCH_CHECK("gemm_tc64 split");
    }
    alignas(64) CUtensorMap ta, tb;
    ibem_status s;
    if ((s = encode_planes(&ta, pa, mp, kp, BM))) return s;
    if ((s = encode_planes(&tb, pb, np, kp, BN))) return s;
    const unsigned grid = (unsigned)((mp / BM) * (np / BN));
    ProfScope ps(PROF_GEMM_TC, st, 2.0 * m * n * kc);
    ::ibem::count_launch(), k_umma_f64<<<grid, THREADS, SMEM_BYTES, st>>>(ta, tb, C, ldc, (int)m, (int)n, (int)(kp / BK), sa,
                                                                         sb, err);
    IBEM_LAUNCH_CHECK("gemm_tc64");
  }
  return IBEM_OK;
}

}  // namespace ibem
