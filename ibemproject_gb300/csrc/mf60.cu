// Matrix-free products of the layout-60 sphere systems (eigenstrain orders 0, 1 and 2): the
// pair blocks that ibem_e3d_pair_blocks(layout 60) assembles (integratorElastic3D.cpp:
// 341-682: ...EquivalentInclusion, ...FirstOrderInclusion, ...SecondOrderInclusion) are
// applied inside the product (mf60_contract.cuh: in the frame of the pair's offset, where a
// block has 520 entries instead of 3,600), so a batch of quadratic realisations is solved
// without storing its matrices.
//
// Scaled system As = Dr A Dc with Dr = a_s^order / mu0 (rows of target s), Dc = a_h^-order
// (columns of source h): in coordinates x' = (c_s - c_h) / a_h and with the moduli divided by
// mu0 a block is the unit-sphere block times (a_s / a_h)^(row order).  The kernels scale a
// source's powers of 1/r by a_h^-(row order) and the sums by a_s^(row order) once.
//
// One thread per target particle, 64 consecutive targets of one realisation per CTA, source
// slices over gridDim.y (and their pieces over gridDim.z), partial sums added atomically to the
// target's own block times its coefficients (k_self_apply60, which also clears the sums).  A
// target whose centre lies inside a source (overlapping spheres) takes that pair from the
// generated dense block (FP64: k_mf60_inside).
//
// Bound by the FP32 (FP64) multiply-adds.  FP32: one kernel for all 60 rows, which rotates a
// source's coefficients once.  FP64: the rows of orders 0 and 1 in one kernel and those of order
// 2 in another, because 60 sums and 60 rotated coefficients do not fit 255 registers; the
// rotation of the coefficients is repeated.  Measured, 12 realisations of 50 to 300 spheres
// (437,000 pairs): FP32 product 1.13 -> 0.09 ms, FP64 product 45.2 -> 3.5 ms, against the
// generated blocks in 18 and 7 kernels.
#include <cuda_runtime.h>

#include <type_traits>

#include "gen_sphere60.cuh"
#include "gen_sphere60_f32.cuh"
#include "mf.h"
#include "fp64_math.cuh"
#include "mf60_contract.cuh"
#include "prof.h"

namespace ibem {
namespace {

constexpr int kNu = 60;
constexpr int kT = kMf60Targets;   // targets per CTA
constexpr int kChunk = 16;         // sources staged per chunk

// acc[r] += v * xs[c]
template <class T>
struct RowSink {
  T* acc;
  const T* xs;
  __device__ __forceinline__ void operator()(int r, int c, T v) const { acc[r] += v * xs[c]; }
};

// Offset of a target (centre p) from a source (centre c, ia = 1 / radius) in units of the source's
// radius.  True: outside the source.  The FP64 product decides this for a pair in three kernels,
// which have to agree on a centre within a rounding of the surface: hence rounded operations,
// which the compiler does not fuse into multiply-adds of its own choice.
__device__ __forceinline__ bool offset60(const double* p, const double* c, double ia, double (&x)[3], double& r2) {
#pragma unroll
  for (int d = 0; d < 3; ++d) x[d] = __dmul_rn(__dsub_rn(p[d], c[d]), ia);
  r2 = __dadd_rn(__dadd_rn(__dmul_rn(x[0], x[0]), __dmul_rn(x[1], x[1])), __dmul_rn(x[2], x[2]));
  return r2 > 1.0;
}

// A pair whose target centre lies inside the source, from the generated blocks (dense): rare
// (overlapping spheres), so out of line and straight into y.  as, ia: radius of the target,
// 1 / radius of the source; xs: the source's coefficients.
__device__ __noinline__ void pair_inside(float x0, float x1, float x2, float as, float ia, const SphMatF& mc,
                                         const float* xs, float* y) {
  float acc[kNu];
  for (int r = 0; r < kNu; ++r) acc[r] = 0.f;
  RowSink<float> sk{acc, xs};
#define IBEM_B(NM) sph_block60f##NM(x0, x1, x2, 1.0f, mc, sk)
  IBEM_B(m_c0_r0); IBEM_B(m_c1_r0); IBEM_B(m_c2_r0); IBEM_B(m_c0_r1); IBEM_B(m_c1_r1); IBEM_B(m_c0_r2);
  IBEM_B(_c2g0_r1); IBEM_B(_c2g1_r1); IBEM_B(_c2g2_r1); IBEM_B(_c2g3_r1); IBEM_B(_c2g4_r1); IBEM_B(_c2g5_r1);
  IBEM_B(_c1g0_r2); IBEM_B(_c1g1_r2); IBEM_B(_c1g2_r2);
  IBEM_B(_c2g0_r2); IBEM_B(_c2g1_r2); IBEM_B(_c2g2_r2); IBEM_B(_c2g3_r2); IBEM_B(_c2g4_r2); IBEM_B(_c2g5_r2);
#undef IBEM_B
  for (int r = 0; r < kNu; ++r) atomicAdd(y + r, acc[r] * (r < 6 ? 1.f : r < 24 ? as * ia : as * ia * as * ia));
}
// the nine FP64 sub-blocks (column order, row order) of the unit sphere
template <class Sink>
__device__ __forceinline__ void blocks60(int which, double x0, double x1, double x2, const SphMat& mc, Sink& sk) {
  switch (which) {
#define IBEM_B(I, NM) case I: sph_block60_##NM(x0, x1, x2, 1.0, mc, sk); break
    IBEM_B(0, c2_r2); IBEM_B(1, c2_r1); IBEM_B(2, c1_r2); IBEM_B(3, c2_r0); IBEM_B(4, c0_r2);
    IBEM_B(5, c1_r1); IBEM_B(6, c1_r0); IBEM_B(7, c0_r1); IBEM_B(8, c0_r0);
#undef IBEM_B
  }
}
__device__ __noinline__ void pair_inside(double x0, double x1, double x2, double as, double ia, const SphMat& mc,
                                         const double* xs, double* y) {
  double acc[kNu];
  for (int r = 0; r < kNu; ++r) acc[r] = 0.0;
  RowSink<double> sk{acc, xs};
  // the sub-blocks compare |x|^2 with 1 themselves, by operations of their own: a centre within a few
  // roundings of the surface is moved 2^-50 of its distance inwards, so that all of them see it inside
  if (x0 * x0 + x1 * x1 + x2 * x2 > 1.0 - 0x1p-48) x0 -= 0x1p-50 * x0, x1 -= 0x1p-50 * x1, x2 -= 0x1p-50 * x2;
  for (int i = 0; i < 9; ++i) blocks60(i, x0, x1, x2, mc, sk);
  for (int r = 0; r < kNu; ++r) atomicAdd(y + r, acc[r] * (r < 6 ? 1.0 : r < 24 ? as * ia : as * ia * as * ia));
}

// Own block of a realisation's particles (unit sphere at x = 0 plus C0, moduli / mu0; the same
// for all of them in the scaled system): S[seg][column][row].  One CTA per realisation, the
// nine sub-blocks by one thread of a warp each.
__global__ void __launch_bounds__(288) k_self60(const SphMat* __restrict__ mats, double* __restrict__ S,
                                                float* __restrict__ Sf) {
  __shared__ double M[kNu * kNu];
  for (int i = threadIdx.x; i < kNu * kNu; i += blockDim.x) M[i] = 0.0;
  __syncthreads();
  const SphMat mc = mats[blockIdx.x];
  struct Put {
    double* M;
    __device__ void operator()(int r, int c, double v) const { M[c * kNu + r] += v; }
  } put{M};
  if (threadIdx.x % 32 == 0) blocks60(threadIdx.x / 32, 0.0, 0.0, 0.0, mc, put);
  __syncthreads();
  if (threadIdx.x == 0) sph_self60(mc, put);
  __syncthreads();
  for (int i = threadIdx.x; i < kNu * kNu; i += blockDim.x) {
    S[(int64_t)blockIdx.x * kNu * kNu + i] = M[i];
    Sf[(int64_t)blockIdx.x * kNu * kNu + i] = (float)M[i];
  }
}

// Row of M x with a realisation's 60 x 60 block stored by columns: a warp's rows are neighbours.
__device__ __forceinline__ float block60_row(const float* __restrict__ m, const float* __restrict__ x) {
  const float4* x4 = reinterpret_cast<const float4*>(x);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < kNu / 4; ++c) {
    const float4 v = x4[c];
    s = fmaf(m[(4 * c) * kNu], v.x, s);
    s = fmaf(m[(4 * c + 1) * kNu], v.y, s);
    s = fmaf(m[(4 * c + 2) * kNu], v.z, s);
    s = fmaf(m[(4 * c + 3) * kNu], v.w, s);
  }
  return s;
}

// y = own block times the particle's coefficients, or 0 for a realisation masked out.  The FP32
// form reads an FP32 copy of the blocks: converting their entries took the FP64 pipe 13 of
// 17 us for 2,100 particles.
template <class T>
__global__ void __launch_bounds__(240) k_self_apply60(int64_t n, const int* __restrict__ seg_of,
                                                      const int* __restrict__ mask, int mask_on,
                                                      const T* __restrict__ S, const T* __restrict__ x,
                                                      T* __restrict__ y) {
  chain_wait();
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t p = t / kNu;
  const int seg = seg_of[p];
  T s = T(0);
  if (!mask || mask[seg] == mask_on) {
    const T* m = S + (int64_t)seg * kNu * kNu + t % kNu;
    const T* v = x + p * kNu;
    if constexpr (sizeof(T) == 4) {
      s = block60_row(m, v);
    } else {
#pragma unroll 10
      for (int c = 0; c < kNu; ++c) s += m[c * kNu] * v[c];
    }
  }
  y[t] = s;
}

__global__ void __launch_bounds__(kT)
    k_mf60_f32(const MfTile* __restrict__ tiles, const int* __restrict__ seg_begin, const int* __restrict__ mask,
               int mask_on, const float4* __restrict__ gh, const float4* __restrict__ gl,
               const SphMatF* __restrict__ mats, const float* __restrict__ x, float* __restrict__ y) {
  chain_wait();
  __shared__ float4 sgh[kChunk], sgl[kChunk];
  __shared__ __align__(16) float sx[kChunk * kNu];
  const MfTile t = tiles[blockIdx.x];
  if (mask && mask[t.seg] != mask_on) return;
  const int hb0 = seg_begin[t.seg], he0 = seg_begin[t.seg + 1];
  const int ns = gridDim.y * gridDim.z, per = (he0 - hb0 + ns - 1) / ns;
  const int hb = hb0 + (blockIdx.y * gridDim.z + blockIdx.z) * per, he = min(he0, hb + per);
  if (hb >= he) return;
  const int s = t.s0 + threadIdx.x;
  const bool act = threadIdx.x < t.ns;
  const float kmu = mats[t.seg].kmu, klam = mats[t.seg].klam, nu = 0.5f * mats[t.seg].tn2;
  const float4 ph = act ? gh[s] : make_float4(0.f, 0.f, 0.f, 1.f);
  const float4 pl = act ? gl[s] : make_float4(0.f, 0.f, 0.f, 1.f);
  float acc[kNu];
#pragma unroll
  for (int r = 0; r < kNu; ++r) acc[r] = 0.f;
  for (int h0 = hb; h0 < he; h0 += kChunk) {
    const int nh = min(kChunk, he - h0);
    __syncthreads();
    for (int i = threadIdx.x; i < nh; i += kT) {
      sgh[i] = gh[h0 + i];
      sgl[i] = gl[h0 + i];
    }
    for (int i = threadIdx.x; i < nh * kNu; i += kT) sx[i] = x[(int64_t)kNu * h0 + i] * mf60_weight(i % kNu);
    __syncthreads();
    if (!act) continue;
#pragma unroll 1
    for (int hh = 0; hh < nh; ++hh) {
      const float4 qh = sgh[hh], ql = sgl[hh];
      const float ia = ql.w;
      const float x0 = ((ph.x - qh.x) + (pl.x - ql.x)) * ia;
      const float x1 = ((ph.y - qh.y) + (pl.y - ql.y)) * ia;
      const float x2 = ((ph.z - qh.z) + (pl.z - ql.z)) * ia;
      const float r2 = x0 * x0 + x1 * x1 + x2 * x2;
      if (!(r2 > 1.f)) {
        if (h0 + hh != s) pair_inside(x0, x1, x2, ph.w, ia, mats[t.seg], x + (int64_t)kNu * (h0 + hh), y + (int64_t)kNu * s);
        continue;
      }
      const float ir = rsqrtf(r2);
      Mf60Frame<float> f;
      mf60_frame(x0 * ir, x1 * ir, x2 * ir, f);
      float A0[6], A1[6][3], A2[6][6];
      mf60_source(f, sx + kNu * hh, A0, A1, A2);
      mf60_rows<0>(f, A0, A1, A2, ir, 1.f, nu, acc);
      mf60_rows<1>(f, A0, A1, A2, ir, ia, nu, acc + 6);
      mf60_rows<2>(f, A0, A1, A2, ir, ia * ia, nu, acc + 24);
    }
  }
  if (!act) return;
  mf60_map<0>(kmu, klam, acc);
  mf60_map<1>(kmu, klam, acc + 6);
  mf60_map<2>(kmu, klam, acc + 24);
  float* o = y + (int64_t)kNu * s;
#pragma unroll
  for (int r = 0; r < kNu; ++r) atomicAdd(o + r, acc[r] * (r < 6 ? 1.f : r < 24 ? ph.w : ph.w * ph.w));
}

// The pairs of the FP64 product whose target centre lies inside the source sphere (overlapping
// spheres; usually none), by the generated block: a few operations a pair to look for them.  In the
// product's own loop the call cost its kernel 87 registers.
__global__ void __launch_bounds__(kT)
    k_mf60_inside(const MfTile* __restrict__ tiles, const int* __restrict__ seg_begin, const int* __restrict__ mask,
                  int mask_on, const double* __restrict__ cen, const double* __restrict__ rad,
                  const SphMat* __restrict__ mats, const double* __restrict__ x, double* __restrict__ y) {
  const MfTile t = tiles[blockIdx.x];
  if (mask && mask[t.seg] != mask_on) return;
  const int hb0 = seg_begin[t.seg], he0 = seg_begin[t.seg + 1];
  const int ns = gridDim.y * gridDim.z, per = (he0 - hb0 + ns - 1) / ns;
  const int hb = hb0 + (blockIdx.y * gridDim.z + blockIdx.z) * per, he = min(he0, hb + per);
  if (threadIdx.x >= t.ns) return;
  const int s = t.s0 + threadIdx.x;
  const double p[3] = {cen[3 * (int64_t)s], cen[3 * (int64_t)s + 1], cen[3 * (int64_t)s + 2]};
#pragma unroll 4
  for (int h = hb; h < he; ++h) {
    const double ia = 1.0 / rad[h];
    double u[3], r2;
    if (!offset60(p, cen + 3 * (int64_t)h, ia, u, r2) && h != s)
      pair_inside(u[0], u[1], u[2], rad[s], ia, mats[t.seg], x + (int64_t)kNu * h, y + (int64_t)kNu * s);
  }
}

// FP64 product, bound by the FP64 pipe: HI false, the rows of orders 0 and 1, and true, of order 2.
// One kernel for all 60 rows spills; one per order turned each source's coefficients into the
// frame of the offset three times (12 realisations of U[50, 300]: 4.3 ms a product, now 3.5).
template <bool HI>
__global__ void __launch_bounds__(kT)
    k_mf60_f64(const MfTile* __restrict__ tiles, const int* __restrict__ seg_begin, const int* __restrict__ mask,
               int mask_on, const double* __restrict__ cen, const double* __restrict__ rad,
               const SphMat* __restrict__ mats, const double* __restrict__ x, double* __restrict__ y) {
  constexpr int NR = HI ? 36 : 24;
  __shared__ double sc[kChunk * 4];
  __shared__ __align__(16) double sx[kChunk * kNu];
  const MfTile t = tiles[blockIdx.x];
  if (mask && mask[t.seg] != mask_on) return;
  const int hb0 = seg_begin[t.seg], he0 = seg_begin[t.seg + 1];
  const int ns = gridDim.y * gridDim.z, per = (he0 - hb0 + ns - 1) / ns;
  const int hb = hb0 + (blockIdx.y * gridDim.z + blockIdx.z) * per, he = min(he0, hb + per);
  if (hb >= he) return;
  const int s = t.s0 + threadIdx.x;
  const bool act = threadIdx.x < t.ns;
  const double kmu = mats[t.seg].kmu, klam = mats[t.seg].klam, nu = 0.5 * mats[t.seg].tn2;
  double p[3] = {0.0, 0.0, 0.0}, as = 1.0;
  if (act) {
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d] = cen[3 * (int64_t)s + d];
    as = rad[s];
  }
  double acc[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0;
  for (int h0 = hb; h0 < he; h0 += kChunk) {
    const int nh = min(kChunk, he - h0);
    __syncthreads();
    for (int i = threadIdx.x; i < nh; i += kT) {
      sc[4 * i] = cen[3 * (int64_t)(h0 + i)];
      sc[4 * i + 1] = cen[3 * (int64_t)(h0 + i) + 1];
      sc[4 * i + 2] = cen[3 * (int64_t)(h0 + i) + 2];
      sc[4 * i + 3] = 1.0 / rad[h0 + i];
    }
    for (int i = threadIdx.x; i < nh * kNu; i += kT) sx[i] = x[(int64_t)kNu * h0 + i] * (double)mf60_weight(i % kNu);
    __syncthreads();
    if (!act) continue;
#pragma unroll 1
    for (int hh = 0; hh < nh; ++hh) {
      const double ia = sc[4 * hh + 3];
      double u[3], r2;
      if (!offset60(p, sc + 4 * hh, ia, u, r2)) continue;   // k_mf60_inside
      const double ir = rsqrt_h3(r2);
      Mf60Frame<double> f;
      mf60_frame(u[0] * ir, u[1] * ir, u[2] * ir, f);
      double A0[6], A1[6][3], A2[6][6];
      mf60_source(f, sx + kNu * hh, A0, A1, A2);
      if constexpr (HI) {
        mf60_rows<2>(f, A0, A1, A2, ir, ia * ia, nu, acc);
      } else {
        mf60_rows<0>(f, A0, A1, A2, ir, 1.0, nu, acc);
        mf60_rows<1>(f, A0, A1, A2, ir, ia, nu, acc + 6);
      }
    }
  }
  if (!act) return;
  if constexpr (HI) {
    mf60_map<2>(kmu, klam, acc);
  } else {
    mf60_map<0>(kmu, klam, acc);
    mf60_map<1>(kmu, klam, acc + 6);
  }
  double* o = y + (int64_t)kNu * s + (HI ? 24 : 0);
#pragma unroll
  for (int r = 0; r < NR; ++r) atomicAdd(o + r, acc[r] * (HI ? as * as : r < 6 ? 1.0 : as));
}

// The own block of a realisation's particles inverted by Gauss-Jordan elimination in place, with
// partial pivoting, in FP64; one CTA per realisation.  P is stored by columns, as its product
// reads it.  Bound by the FP64 pipe (3,600 multiply-adds a step at 2 per clock) and three
// barriers and a pivot search a step: 154 us; on the augmented matrix with 64 threads and a
// serial search 711 us.
constexpr int kBjThreads = 512;
__global__ void __launch_bounds__(kBjThreads) k_block_jacobi60(const double* __restrict__ S, float* __restrict__ P) {
  __shared__ double M[kNu][kNu + 1];
  __shared__ double f[kNu], ipiv;
  __shared__ int piv[kNu], from[kNu];
  const int p = blockIdx.x;
  const int t = threadIdx.x;
  for (int i = t; i < kNu * kNu; i += kBjThreads) M[i % kNu][i / kNu] = S[(int64_t)p * kNu * kNu + i];
  __syncthreads();
  for (int k = 0; k < kNu; ++k) {
    if (t < 32) {   // the first of the largest entries of column k
      double v = t >= k ? fabs(M[t][k]) : -1.0;
      int r = t;
      if (t + 32 < kNu && t + 32 >= k && fabs(M[t + 32][k]) > v) {
        v = fabs(M[t + 32][k]);
        r = t + 32;
      }
      for (int o = 16; o; o >>= 1) {
        const double vo = __shfl_xor_sync(0xffffffffu, v, o);
        const int ro = __shfl_xor_sync(0xffffffffu, r, o);
        if (vo > v || (vo == v && ro < r)) {
          v = vo;
          r = ro;
        }
      }
      if (t == 0) {
        r = r >= k ? r : k;   // no number in the column
        const double d = M[r][k];
        piv[k] = r;
        ipiv = d != 0.0 ? 1.0 / d : 0.0;
      }
    } else if (t >= 64 && t < 64 + kNu) {
      f[t - 64] = M[t - 64][k];
    }
    __syncthreads();
    const int pr = piv[k];
    if (t < kNu) {   // swap rows k and pr, scale row k
      const double a = M[k][t], b = M[pr][t];
      M[pr][t] = a;
      M[k][t] = t == k ? ipiv : b * ipiv;
    }
    __syncthreads();
    for (int i = t; i < kNu * kNu; i += kBjThreads) {
      const int r = i / kNu, c = i % kNu;
      if (r != k) M[r][c] = (c == k ? 0.0 : M[r][c]) - f[r == pr ? k : r] * M[k][c];
    }
    __syncthreads();
  }
  if (t == 0) {   // the row swaps, undone on the columns of the inverse
    for (int c = 0; c < kNu; ++c) from[c] = c;
    for (int k = kNu - 1; k >= 0; --k) {
      const int c = from[k];
      from[k] = from[piv[k]];
      from[piv[k]] = c;
    }
  }
  __syncthreads();
  float* o = P + (int64_t)kNu * kNu * p;
  for (int i = t; i < kNu * kNu; i += kBjThreads) o[i] = (float)M[i % kNu][from[i / kNu]];
}

// z = P v with the realisation's block (Pseg[seg], 60 x 60 by columns); kdev: v is column
// *kdev of a basis with column stride vstride (Arnoldi steps).  With the block by rows a warp's
// loads touched 32 lines each: 13.0 -> 4.3 us for 2,100 particles.
__global__ void __launch_bounds__(240) k_precond_apply60(int num, const int* __restrict__ seg_of,
                                                         const float* __restrict__ Pseg, const float* __restrict__ v,
                                                         float* __restrict__ z, const int* __restrict__ kdev,
                                                         int64_t vstride) {
  chain_wait();
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)num * kNu) return;
  if (kdev) v += (int64_t)(*kdev) * vstride;
  const int64_t p = t / kNu;
  z[t] = block60_row(Pseg + (int64_t)seg_of[p] * kNu * kNu + t % kNu, v + p * kNu);
}

}  // namespace

ibem_status mf60_self(const MfBatch& b, cudaStream_t st) {
  ::ibem::count_launch(), k_self60<<<b.nseg, 288, 0, st>>>(b.mats, b.self60, b.self60f);
  IBEM_LAUNCH_CHECK("mf60 own blocks");
  return IBEM_OK;
}

ibem_status mf60_apply_f32(const MfBatch& b, const float* x, float* y, cudaStream_t st, const int* mask,
                           int mask_on) {
  launch_chained(k_self_apply60<float>, (unsigned)((b.N + 239) / 240), 240, st, b.N, b.seg_of, mask, mask_on,
                 b.self60f, x, y);
  launch_chained(k_mf60_f32, dim3(b.ntiles_s[0], b.split.slices, b.split.pieces), kT, st, b.tiles_s[0], b.seg_begin, mask,
                 mask_on, b.gh, b.gl, b.matf, x, y);
  IBEM_LAUNCH_CHECK("mf60 apply f32");
  return IBEM_OK;
}

ibem_status mf60_apply_f64(const MfBatch& b, const double* x, double* y, cudaStream_t st, const int* mask,
                           int mask_on) {
  const dim3 grid(b.ntiles_s[0], b.split_wide.slices, b.split_wide.pieces);
  ::ibem::count_launch(), k_self_apply60<double><<<(unsigned)((b.N + 239) / 240), 240, 0, st>>>(b.N, b.seg_of, mask, mask_on,
                                                                                                b.self60, x, y);
#define IBEM_MF60_F64(HI)                                                                                         \
  ::ibem::count_launch(), k_mf60_f64<HI><<<grid, kT, 0, st>>>(b.tiles_s[0], b.seg_begin, mask, mask_on, b.cen, b.rad, \
                                                              b.mats, x, y)
  IBEM_MF60_F64(true);
  IBEM_MF60_F64(false);
  ::ibem::count_launch(), k_mf60_inside<<<grid, kT, 0, st>>>(b.tiles_s[0], b.seg_begin, mask, mask_on, b.cen, b.rad, b.mats,
                                                             x, y);
#undef IBEM_MF60_F64
  IBEM_LAUNCH_CHECK("mf60 apply f64");
  return IBEM_OK;
}

ibem_status mf60_block_jacobi(const MfBatch& b, float* Pseg, cudaStream_t st) {
  ::ibem::count_launch(), k_block_jacobi60<<<b.nseg, kBjThreads, 0, st>>>(b.self60, Pseg);
  IBEM_LAUNCH_CHECK("mf60 block jacobi");
  return IBEM_OK;
}

ibem_status mf60_precond_apply(const MfBatch& b, const float* Pseg, const float* v, float* z, const int* kdev,
                               int64_t vstride, cudaStream_t st) {
  const int64_t n = (int64_t)b.num * kNu;
  launch_chained(k_precond_apply60, (unsigned)((n + 239) / 240), 240, st, b.num, b.seg_of, Pseg, v, z, kdev, vstride);
  IBEM_LAUNCH_CHECK("mf60 preconditioner");
  return IBEM_OK;
}

}  // namespace ibem
