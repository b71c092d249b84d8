// Matrix-free solves of the layout-24 sphere systems, one realisation or a batch of them.
//
// The pair blocks that ibem_e3d_pair_blocks stores (integratorElastic3D.cpp:341-567,
// orders 0 and 1) are never formed: their products with the coefficients are evaluated
// as the contracted strain and its gradient (mf_contract.cuh):
//   k_mf_apply_f32  As x in FP32 on the scaled system (mf.h), the GMRES operator;
//   k_mf_apply_f64  As x in FP64, the refinement residual Dr b - As xs; for the residual
//                   that decides convergence it takes only the source chunks near each
//                   warp's targets and k_mf_apply_df the far ones (both visit particles in
//                   the Morton order of their centres, so warps and chunks are compact).
// One thread per target particle s, 128 consecutive targets of one realisation per CTA;
// the CTA's source particles h (a slice of the realisation, or a piece of one) are staged
// through shared memory in chunks with their coefficients, and every thread sums the
// pair products in registers.  Slices add their partial sums atomically.
//
// Solver: iterative refinement x += Dc d; each correction d solves As d = Dr r with a
// restarted FP32 GMRES right-preconditioned by a block-sparse P (block-Jacobi, Neumann or
// learned); the residual that drives the next correction is a double-float product
// (k_mf_apply_df, ~48 bits) and the one that decides convergence the split product.  All
// realisations of a batch run in lock step (per-realisation Arnoldi: segmented dot
// products, Hessenberg updates and Givens rotations on the device, one thread per
// realisation), stopping each realisation on its own residual estimate.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <map>
#include <mutex>
#include <thread>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "gen_sphere24.cuh"
#include "mf.h"
#include "dfnum.cuh"
#include "mf_contract.cuh"
#include "prof.h"
#include "solver.h"

namespace ibem {
namespace {

constexpr int kMfThreads = 128;
constexpr int kMfChunk = 32;
constexpr double kMfFarRadii = 4.0;   // near / far split of the deciding residual
constexpr int kMfSplitMin = 1280;     // smallest realisation (particles) that uses the split
constexpr int kMfSkipMin = 5000;      // from here the far pass skips near sources (256-thread CTAs)

// sink of a generated block: acc[r] += v * x[c] (r, c compile-time constants after inlining)
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
template <class T>
struct MvSink {
  T (&acc)[kMfNu];
  const T* __restrict__ xs;
  __device__ __forceinline__ void operator()(int r, int c, T v) const { acc[r] = fma_t(v, xs[c], acc[r]); }
};

// Source records (mf_contract.cuh) of a chunk: the coefficients are staged with a zero behind each
// source's 24, the records summed from them, TT threads over the entries.
__device__ const MfRecTab g_rec_tab = mf_rec_tab();
template <class T>
struct MfStage {
  __align__(16) T rec[kMfChunk * kRecLen];
  T raw[kMfChunk * (kMfNu + 1)];
  unsigned tab[kRecLen];
  __device__ __forceinline__ void init() {
    for (int i = threadIdx.x; i < kRecLen; i += blockDim.x) tab[i] = g_rec_tab.v[i];
  }
  template <class F>
  __device__ __forceinline__ void load(int nh, F value) {   // value(source of the chunk, coefficient)
    for (int i = threadIdx.x; i < nh * (kMfNu + 1); i += blockDim.x) {
      const int h = i / (kMfNu + 1), c = i % (kMfNu + 1);
      raw[i] = c < kMfNu ? value(h, c) : T(0);
    }
  }
  __device__ __forceinline__ void build(int nh) {
    for (int i = threadIdx.x; i < nh * kRecLen; i += blockDim.x)
      rec[i] = mf_rec_entry(tab[i % kRecLen], raw + (kMfNu + 1) * (i / kRecLen));
  }
};

// One work item of the FP32 product: the TT targets of a tile against source slice `slice`
// of `nslice` of its realisation (TT = blockDim.x, the tile shape the autotuner picks).
template <int TT>
__device__ __forceinline__ void mf_f32_item(const MfTile t, int slice, int nslice, const int* __restrict__ seg_begin,
                                            const int* __restrict__ mask, int mask_on,
                                            const float4* __restrict__ gh, const float4* __restrict__ gl,
                                            const SphMatF* __restrict__ mats, const float* __restrict__ x,
                                            float* __restrict__ y, float4* sgh, float4* sgl, MfStage<float>& sx) {
  if (mask && mask[t.seg] != mask_on) return;  // realisation left out of this product
  const int hb0 = seg_begin[t.seg], he0 = seg_begin[t.seg + 1];
  const int per = (he0 - hb0 + nslice - 1) / nslice;
  const int hb = hb0 + slice * per, he = min(he0, hb + per);
  if (hb >= he) return;
  const int s = t.s0 + threadIdx.x;
  const bool act = threadIdx.x < t.ns;
  const SphMatF mc = mats[t.seg];
  const float4 ph = act ? gh[s] : make_float4(0.f, 0.f, 0.f, 1.f);
  const float4 pl = act ? gl[s] : make_float4(0.f, 0.f, 0.f, 1.f);
  float acc[kMfNu];
#pragma unroll
  for (int r = 0; r < kMfNu; ++r) acc[r] = 0.f;
  for (int h0 = hb; h0 < he; h0 += kMfChunk) {
    const int nh = min(kMfChunk, he - h0);
    __syncthreads();
    for (int i = threadIdx.x; i < nh; i += TT) {
      sgh[i] = gh[h0 + i];
      sgl[i] = gl[h0 + i];
    }
    sx.load(nh, [&](int h, int c) { return x[(int64_t)kMfNu * (h0 + h) + c]; });
    __syncthreads();
    sx.build(nh);
    __syncthreads();
    if (!act) continue;
#pragma unroll 1
    for (int hh = 0; hh < nh; ++hh) {
      const float4 qh = sgh[hh], ql = sgl[hh];
      const float ia = ql.w;
      // offset from the source centre in units of its radius (hi/lo parts keep ~48 bits)
      const float x0 = ((ph.x - qh.x) + (pl.x - ql.x)) * ia;
      const float x1 = ((ph.y - qh.y) + (pl.y - ql.y)) * ia;
      const float x2 = ((ph.z - qh.z) + (pl.z - ql.z)) * ia;
      sph_pair_raw24<float>(x0, x1, x2, 2.f - mc.tn2, sx.rec + kRecLen * hh, ph.w * ia, acc);
    }
  }
  if (!act) return;
  float yv[kMfNu];
  sph_pair_map24<float>(acc, mc.kmu, mc.klam, yv);
  if (s >= hb && s < he) {  // the slice holding the target adds its self term (C0 / mu0)
    MvSink<float> sk{yv, x + (int64_t)kMfNu * s};
    sph_self24f(mc, sk);
  }
  float* o = y + (int64_t)kMfNu * s;
#pragma unroll
  for (int r = 0; r < kMfNu; ++r) atomicAdd(o + r, yv[r]);
}

// one CTA per (tile, slice): grid (ntiles, nslice)
template <int TT>
__global__ void __launch_bounds__(TT)
    k_mf_apply_f32(const MfTile* __restrict__ tiles, const int* __restrict__ seg_begin,
                   const int* __restrict__ mask, int mask_on,
                   const float4* __restrict__ gh, const float4* __restrict__ gl,
                   const SphMatF* __restrict__ mats, const float* __restrict__ x, float* __restrict__ y) {
  chain_wait();
  __shared__ float4 sgh[kMfChunk], sgl[kMfChunk];
  __shared__ MfStage<float> sx;
  sx.init();
  mf_f32_item<TT>(tiles[blockIdx.x], blockIdx.y * gridDim.z + blockIdx.z, gridDim.y * gridDim.z,
                  seg_begin, mask, mask_on, gh, gl, mats, x, y, sgh, sgl, sx);
}

// persistent form: as many CTAs as fit on the GPU at once walk a work list of (tile,
// slice) pairs sorted by decreasing cost (sources x targets), CTA c taking items c,
// c + gridDim.x, ... (the longest first, so that the realisations of a ragged batch finish
// together)
template <int TT>
__global__ void __launch_bounds__(TT)
    k_mf_apply_f32_persist(const MfTile* __restrict__ tiles, const int2* __restrict__ work, int nwork, int nslice,
                           const int* __restrict__ seg_begin, const int* __restrict__ mask, int mask_on,
                           const float4* __restrict__ gh, const float4* __restrict__ gl,
                           const SphMatF* __restrict__ mats, const float* __restrict__ x, float* __restrict__ y) {
  chain_wait();
  __shared__ float4 sgh[kMfChunk], sgl[kMfChunk];
  __shared__ MfStage<float> sx;
  sx.init();
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const int2 it = work[w];
    mf_f32_item<TT>(tiles[it.x], it.y, nslice, seg_begin, mask, mask_on, gh, gl, mats, x, y, sgh, sgl, sx);
  }
}

// FP64 product of the scaled system (the refinement residual): the same evaluation as the
// FP32 kernel in double precision, offsets from FP64 centres.
// Split products (the deciding residual): particles are visited in the Morton order of
// their centres within each realisation (perm: position -> particle), so the 32 targets of a
// warp form a compact cluster.  mode 0: every pair; 1: only the sources near the warp's
// targets (within kMfFarRadii of their radius of the targets' bounding box), and the self
// term; 2 and 3: only the far sources, no self term.  The test is per (warp, source) and
// warp-uniform.  The double-float pair code is longer than the instruction cache: warps of
// an SM that run it at different places each fetch their own instructions, and issue fell
// to half when the far pass let every warp skip its own near sources.  So the far pass
// keeps them together: mode 2 (two 128-thread CTAs per SM) evaluates every source of the
// chunk, a warp's near ones against zero coefficients, so every CTA does the same work;
// mode 3 (one 256-thread CTA per SM) skips them, the barrier at each chunk realigning the
// warps of the SM.
__device__ __forceinline__ void warp_box(bool act, double x, double y, double z, double* lo, double* hi) {
  double v[3] = {x, y, z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double a = act ? v[d] : 1e300, b = act ? v[d] : -1e300;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
      b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    lo[d] = a;
    hi[d] = b;
  }
}

// whether a source sphere (c, r) lies beyond kMfFarRadii of its radius from the box of the
// warp's targets: the same for every lane; rounded operations without contraction, so that
// the FP64 and double-float kernels of a split product classify every pair the same way
__device__ __forceinline__ bool source_is_far(const double* wlo, const double* whi, double cx, double cy, double cz,
                                              double r) {
  const double c[3] = {cx, cy, cz};
  double d2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double g = fmax(0.0, fmax(__dadd_rn(wlo[d], -c[d]), __dadd_rn(c[d], -whi[d])));
    d2 = __dadd_rn(d2, __dmul_rn(g, g));
  }
  const double lim = __dmul_rn(kMfFarRadii, r);
  return d2 > __dmul_rn(lim, lim);
}
// The sources of one CTA (piece blockIdx.z of slice blockIdx.y), in chunks of kMfChunk: chunk j
// starts at first + j * step and ends at end at the latest.  The full product (mode 0) takes
// a contiguous range of the realisation; the split ones deal the chunks
// out to the CTAs in turn.  In Morton order the near sources of a tile sit in a few neighbouring chunks:
// this way every CTA gets about the average share of them.
struct MfSlice {
  int first, step, end;
  __device__ __forceinline__ bool holds(int p) const {
    return p >= first && p < end && (p - first) % step < kMfChunk;
  }
};
__device__ __forceinline__ MfSlice mf_slice(int hb0, int he0, int mode) {
  const int k = blockIdx.y * gridDim.z + blockIdx.z, ns = gridDim.y * gridDim.z;
  if (mode) return {hb0 + kMfChunk * k, kMfChunk * ns, he0};
  const int per = (he0 - hb0 + ns - 1) / ns;
  const int hb = hb0 + k * per;
  return {hb, kMfChunk, min(he0, hb + per)};
}

// Sources of the chunk at h0 (nh of them) that this warp evaluates, as a bit mask (bit i:
// source h0 + i); the same for every lane.  Lane i classifies source i.  Evaluating the
// selected sources in turn keeps the warps of a CTA at the same place in the long
// straight-line pair code (instruction fetches shared), which skipping inside the loop
// would not.
__device__ __forceinline__ unsigned chunk_mask(int mode, bool warp_on, const double* wlo, const double* whi, int h0,
                                               int nh, const int* __restrict__ perm, const double* __restrict__ cen,
                                               const double* __restrict__ rad) {
  const int lane = threadIdx.x & 31;
  bool take = lane < nh;
  if (mode && take) {
    const int h = perm[h0 + lane];
    take = source_is_far(wlo, whi, cen[3 * (int64_t)h], cen[3 * (int64_t)h + 1], cen[3 * (int64_t)h + 2], rad[h]) ==
           (mode >= 2);
  }
  const unsigned m = __ballot_sync(0xffffffffu, take);
  return warp_on ? m : 0u;
}

__global__ void __launch_bounds__(kMfThreads)
    k_mf_apply_f64(const MfTile* __restrict__ tiles, const int* __restrict__ seg_begin,
                   const int* __restrict__ mask, int mask_on,
                   const double* __restrict__ cen, const double* __restrict__ rad,
                   const SphMat* __restrict__ mats, const double* __restrict__ x, double* __restrict__ y,
                   const int* __restrict__ perm, int mode) {
  __shared__ double sc[kMfChunk * 4];
  __shared__ MfStage<double> sx;
  sx.init();
  const MfTile t = tiles[blockIdx.x];
  if (mask && mask[t.seg] != mask_on) return;  // realisation left out of this product
  const MfSlice sl = mf_slice(seg_begin[t.seg], seg_begin[t.seg + 1], mode);
  if (sl.first >= sl.end) return;
  const int pos = t.s0 + threadIdx.x;
  const bool act = threadIdx.x < t.ns;
  const int s = act ? perm[pos] : 0;
  const SphMat mc = mats[t.seg];   // moduli divided by mu0 (scaled system)
  double p0 = 0, p1 = 0, p2 = 0, as = 1;
  if (act) {
    p0 = cen[3 * (int64_t)s];
    p1 = cen[3 * (int64_t)s + 1];
    p2 = cen[3 * (int64_t)s + 2];
    as = rad[s];
  }
  double wlo[3], whi[3];
  warp_box(act, p0, p1, p2, wlo, whi);
  double acc[kMfNu];
#pragma unroll
  for (int r = 0; r < kMfNu; ++r) acc[r] = 0.0;
  const bool warp_on = __any_sync(0xffffffffu, act);
  for (int h0 = sl.first; h0 < sl.end; h0 += sl.step) {
    const int nh = min(kMfChunk, sl.end - h0);
    // mode 1: the sources near the warp's targets; 2: the far ones; 0: all
    unsigned m = chunk_mask(mode, warp_on, wlo, whi, h0, nh, perm, cen, rad);
    if (!__syncthreads_or(m != 0u)) continue;   // no warp of the CTA needs this chunk
    for (int i = threadIdx.x; i < nh; i += blockDim.x) {
      const int h = perm[h0 + i];
      sc[4 * i] = cen[3 * (int64_t)h];
      sc[4 * i + 1] = cen[3 * (int64_t)h + 1];
      sc[4 * i + 2] = cen[3 * (int64_t)h + 2];
      sc[4 * i + 3] = 1.0 / rad[h];
    }
    sx.load(nh, [&](int h, int c) { return x[(int64_t)kMfNu * perm[h0 + h] + c]; });
    __syncthreads();
    sx.build(nh);
    __syncthreads();
    if (!act) continue;
#pragma unroll 1
    for (; m; m &= m - 1u) {
      const int hh = __ffs(m) - 1;
      const double ia = sc[4 * hh + 3];
      const double x0 = (p0 - sc[4 * hh]) * ia, x1 = (p1 - sc[4 * hh + 1]) * ia, x2 = (p2 - sc[4 * hh + 2]) * ia;
      sph_pair_raw24<double>(x0, x1, x2, 2.0 - mc.tn2, sx.rec + kRecLen * hh, as * ia, acc);
    }
  }
  if (!act) return;
  double yv[kMfNu];
  sph_pair_map24<double>(acc, mc.kmu, mc.klam, yv);
  if (sl.holds(pos) && mode < 2) {
    MvSink<double> sk{yv, x + (int64_t)kMfNu * s};
    sph_self24(mc, sk);
  }
  double* o = y + (int64_t)kMfNu * s;
#pragma unroll
  for (int r = 0; r < kMfNu; ++r) atomicAdd(o + r, yv[r]);
}

// The scaled product in double-float arithmetic (~48 bits): the residual that drives a
// refinement step (the final residual, which decides convergence, is the FP64 kernel's).
// Centres, inverse radii and coefficients are staged as double-float pairs.
struct DfSink {
  DF (&acc)[kMfNu];
  const double* __restrict__ xs;
  __device__ __forceinline__ void operator()(int r, int c, double v) const { acc[r] += DF(v) * DF(xs[c]); }
};

template <int TT>
__global__ void __launch_bounds__(TT)
    k_mf_apply_df(const MfTile* __restrict__ tiles, const int* __restrict__ seg_begin,
                   const int* __restrict__ mask, int mask_on,
                  const double* __restrict__ cen, const double* __restrict__ rad,
                  const SphMat* __restrict__ mats, const double* __restrict__ x, double* __restrict__ y,
                  const int* __restrict__ perm, int mode) {
  __shared__ DF sc[kMfChunk * 4];
  __shared__ MfStage<DF> sx;
  __shared__ __align__(16) DF szero[kRecLen];   // the record of a skipped source in mode 2
  sx.init();
  for (int i = threadIdx.x; i < kRecLen; i += TT) szero[i] = DF();
  const MfTile t = tiles[blockIdx.x];
  if (mask && mask[t.seg] != mask_on) return;  // realisation left out of this product
  const MfSlice sl = mf_slice(seg_begin[t.seg], seg_begin[t.seg + 1], mode);
  if (sl.first >= sl.end) return;
  const int pos = t.s0 + threadIdx.x;
  const bool act = threadIdx.x < t.ns;
  const int s = act ? perm[pos] : 0;
  const SphMat mc = mats[t.seg];   // moduli divided by mu0 (scaled system)
  DF p0, p1, p2, as(1.0);
  double q0 = 0, q1 = 0, q2 = 0;
  if (act) {
    q0 = cen[3 * (int64_t)s];
    q1 = cen[3 * (int64_t)s + 1];
    q2 = cen[3 * (int64_t)s + 2];
    p0 = DF(q0);
    p1 = DF(q1);
    p2 = DF(q2);
    as = DF(rad[s]);
  }
  double wlo[3], whi[3];
  warp_box(act, q0, q1, q2, wlo, whi);
  const DF tf(2.0 - mc.tn2);
  DF acc[kMfNu];
  const bool warp_on = __any_sync(0xffffffffu, act);
  for (int h0 = sl.first; h0 < sl.end; h0 += sl.step) {
    const int nh = min(kMfChunk, sl.end - h0);
    unsigned m = chunk_mask(mode, warp_on, wlo, whi, h0, nh, perm, cen, rad);
    if (!__syncthreads_or(m != 0u)) continue;   // no warp of the CTA needs this chunk
    for (int i = threadIdx.x; i < nh; i += blockDim.x) {
      const int h = perm[h0 + i];
      sc[4 * i] = DF(cen[3 * (int64_t)h]);
      sc[4 * i + 1] = DF(cen[3 * (int64_t)h + 1]);
      sc[4 * i + 2] = DF(cen[3 * (int64_t)h + 2]);
      sc[4 * i + 3] = DF(1.0 / rad[h]);
    }
    sx.load(nh, [&](int h, int c) { return DF(x[(int64_t)kMfNu * perm[h0 + h] + c]); });
    __syncthreads();
    sx.build(nh);
    __syncthreads();
    if (!act) continue;
    const unsigned all = nh >= 32 ? 0xffffffffu : (1u << nh) - 1u;
#pragma unroll 1
    for (unsigned k = mode == 2 ? all : m; k; k &= k - 1u) {
      const int hh = __ffs(k) - 1;
      const DF* xs = (m >> hh) & 1u ? sx.rec + kRecLen * hh : szero;
      const DF ia = sc[4 * hh + 3];
      const DF x0 = (p0 - sc[4 * hh]) * ia, x1 = (p1 - sc[4 * hh + 1]) * ia, x2 = (p2 - sc[4 * hh + 2]) * ia;
      sph_pair_raw24<DF>(x0, x1, x2, tf, xs, as * ia, acc);
    }
  }
  if (!act) return;
  DF yv[kMfNu];
  sph_pair_map24<DF>(acc, DF(mc.kmu), DF(mc.klam), yv);
  if (sl.holds(pos) && mode < 2) {
    DfSink sk{yv, x + (int64_t)kMfNu * s};
    sph_self24(mc, sk);
  }
  double* o = y + (int64_t)kMfNu * s;
#pragma unroll
  for (int r = 0; r < kMfNu; ++r) atomicAdd(o + r, df_value(yv[r]));
}

// Geometry in the FP32 layout, scalings, segment of every particle.
__global__ void k_mf_prep(int nu, int num, const double* __restrict__ cen, const double* __restrict__ rad,
                          const int* __restrict__ seg_of, const SphMat* __restrict__ mats, float4* __restrict__ gh,
                          float4* __restrict__ gl, double* __restrict__ dr, double* __restrict__ dc) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= num) return;
  float hi[3], lo[3];
  for (int k = 0; k < 3; ++k) {
    const double c = cen[3 * (int64_t)p + k];
    hi[k] = (float)c;
    lo[k] = (float)(c - (double)hi[k]);
  }
  const double a = rad[p];
  gh[p] = make_float4(hi[0], hi[1], hi[2], (float)a);
  gl[p] = make_float4(lo[0], lo[1], lo[2], (float)(1.0 / a));
  const double imu = 1.0 / mats[seg_of[p]].mu0;
  // rows / columns of eigenstrain order o (0: 6, 1: 18, 2: 36 unknowns): a^o / mu0, a^-o
  for (int r = 0; r < nu; ++r) {
    const int o = r < 6 ? 0 : (r < 24 ? 1 : 2);
    const double ao = o == 0 ? 1.0 : (o == 1 ? a : a * a);
    dr[(int64_t)nu * p + r] = ao * imu;
    dc[(int64_t)nu * p + r] = 1.0 / ao;
  }
}

// Scaled diagonal block (FP64, x = 0, unit sphere, moduli / mu0) inverted by Gauss-Jordan
// with partial pivoting; one CTA per realisation: in the scaled system a sphere's own block
// depends on the materials only, so every sphere of a realisation shares it (k_bcast_blocks
// copies it to each).  One CTA's latency bounds it: 64 clocks per dependent-free FP64
// multiply-add and warp.  24 threads form a column each by the pair contraction (~750
// operations; one thread generating the block, ~6,000, and 32 threads eliminating: 133 us),
// four warps eliminate: 56 us.
constexpr int kBjThreads24 = 128;
__global__ void __launch_bounds__(kBjThreads24) k_block_jacobi(const SphMat* __restrict__ mats, float* __restrict__ P) {
  __shared__ double M[kMfNu][2 * kMfNu + 1];
  const int p = blockIdx.x;   // realisation
  const int t = threadIdx.x;
  SphMat mc = mats[p];
  const double sc = 1.0 / mc.mu0;
  mc.kmu *= sc;
  mc.klam *= sc;
  mc.lam0 *= sc;
  mc.mu0 = 1.0;
  if (t < kMfNu) {
    double e[kMfNu], y[kMfNu] = {};
#pragma unroll
    for (int r = 0; r < kMfNu; ++r) {
      e[r] = r == t ? 1.0 : 0.0;
      M[r][kMfNu + t] = e[r];
    }
    sph_pair_apply24<double>(0.0, 0.0, 0.0, 1.0, mc.kmu, mc.klam, mc.tn1, mc.tn2, e, 1.0, y);
#pragma unroll
    for (int r = 0; r < kMfNu; ++r) M[r][t] = y[r];
  }
  __syncthreads();
  if (t == 0) {
    struct Put {
      double (*M)[2 * kMfNu + 1];
      __device__ void operator()(int r, int c, double v) const { M[r][c] += v; }
    } put{M};
    sph_self24(mc, put);
  }
  __syncthreads();
  __shared__ int piv;
  __shared__ double f[kMfNu];
  for (int k = 0; k < kMfNu; ++k) {
    if (t < 32) {   // the first of the largest entries
      double v = t >= k && t < kMfNu ? fabs(M[t][k]) : -1.0;
      int r = t;
      for (int o = 16; o; o >>= 1) {
        const double vo = __shfl_xor_sync(0xffffffffu, v, o);
        const int ro = __shfl_xor_sync(0xffffffffu, r, o);
        if (vo > v || (vo == v && ro < r)) {
          v = vo;
          r = ro;
        }
      }
      if (t == 0) piv = min(r, kMfNu - 1);
    }
    __syncthreads();
    const int pr = piv;
    if (pr != k)
      for (int c = t; c < 2 * kMfNu; c += kBjThreads24) {
        const double v = M[k][c];
        M[k][c] = M[pr][c];
        M[pr][c] = v;
      }
    __syncthreads();
    const double d = M[k][k];
    const double id = d != 0.0 ? 1.0 / d : 0.0;
    __syncthreads();
    for (int c = t; c < 2 * kMfNu; c += kBjThreads24) M[k][c] *= id;
    if (t < kMfNu) f[t] = M[t][k];  // column k of the other rows (row k is being scaled, unused)
    __syncthreads();
    for (int i = t; i < kMfNu * 2 * kMfNu; i += kBjThreads24) {
      const int r = i / (2 * kMfNu), c = i % (2 * kMfNu);
      if (r != k) M[r][c] -= f[r] * M[k][c];
    }
    __syncthreads();
  }
  float* o = P + (int64_t)kMfNu * kMfNu * p;
  for (int i = t; i < kMfNu * kMfNu; i += kBjThreads24) o[i] = (float)M[i / kMfNu][kMfNu + i % kMfNu];
}

// P[p] = Pseg[seg_of[p]] (24 x 24 blocks, float4 copies)
__global__ void k_bcast_blocks(int num, const int* __restrict__ seg_of, const float* __restrict__ Pseg,
                               float* __restrict__ P) {
  constexpr int kQ = kMfNu * kMfNu / 4;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)num * kQ) return;
  const int64_t p = t / kQ;
  const int q = (int)(t % kQ);
  reinterpret_cast<float4*>(P)[t] = reinterpret_cast<const float4*>(Pseg)[(int64_t)seg_of[p] * kQ + q];
}

// Control of the Arnoldi steps of a cycle, on the device: the kernels of a step read the step's
// index and return at once when the cycle has stopped, so that steps can be launched ahead of
// the host's knowing how many there will be.
struct StepCtl {
  int k;         // steps taken
  int stop;      // the cycle is over
  int nactive, arrived;   // of the update's CTAs
};
// what the host reads, in pinned memory
struct HostCtl {
  volatile int steps;   // steps finished (taken or skipped)
  volatile int stop;
};

// z = P v for the block-sparse preconditioner: z_p = D_p v_p + sum_slot Q_(p,slot) v_nbr
// (24 x 24 row-major blocks).  zero: cleared (the step's product adds to it).  ctl (Arnoldi
// steps): v is column ctl->k of a basis with column stride vstride; nothing to do once ctl->stop.
//
// Bound by reading Q once (37 KB a particle).  144 threads take a particle, each the same four
// columns of the same row of all 17 blocks, so that a block is read in one piece and a thread
// has 16 independent loads.  With a row per thread (and four lanes to a row) every cache line was
// asked for by eight loads: 45 -> 25 us for 4,200 particles (154 MB).
constexpr int kPreQ = kMfNu * kMfNu / 4;         // float4 of a block, threads of a particle
constexpr int kPrePart = 2;                      // particles of a CTA
constexpr int kPreThreads = kPreQ * kPrePart;
__global__ void __launch_bounds__(kPreThreads) k_precond_apply(int num, const float* __restrict__ D,
                                                               const float* __restrict__ Q, const int* __restrict__ nbr,
                                                               const float* __restrict__ v, float* __restrict__ z,
                                                               float* __restrict__ zero, const StepCtl* __restrict__ ctl,
                                                               int64_t vstride) {
  chain_wait();
  __shared__ float red[kPreThreads];
  if (ctl) {
    if (ctl->stop) return;
    v += (int64_t)ctl->k * vstride;
  }
  const int64_t p = (int64_t)blockIdx.x * kPrePart + threadIdx.x / kPreQ;
  const int e = threadIdx.x % kPreQ, c = e % (kMfNu / 4);
  const float4* v4 = reinterpret_cast<const float4*>(v) + c;
  auto dot = [](const float4& a, const float4& b, float s) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s))));
  };
  float s = 0.f;
  if (p < num) {
    s = dot(reinterpret_cast<const float4*>(D)[p * kPreQ + e], v4[p * (kMfNu / 4)], 0.f);
    if (Q) {
      const float4* q = reinterpret_cast<const float4*>(Q) + p * kKnn * kPreQ + e;
      const int* nb = nbr + p * kKnn;
#pragma unroll
      for (int k = 0; k < kKnn; ++k) {
        const int j = nb[k];
        if (j >= 0) s = dot(q[k * kPreQ], v4[(int64_t)j * (kMfNu / 4)], s);
      }
    }
  }
  red[threadIdx.x] = s;
  __syncthreads();
  const int64_t row = (int64_t)blockIdx.x * kPrePart * kMfNu + threadIdx.x;
  if (threadIdx.x >= kPrePart * kMfNu || row >= (int64_t)num * kMfNu) return;
  const float* r = red + threadIdx.x * (kMfNu / 4);
  z[row] = ((r[0] + r[1]) + (r[2] + r[3])) + (r[4] + r[5]);
  if (zero) zero[row] = 0.f;
}

// out[seg * ldo + j] += sum over the segment's rows of V_j[row] * w[row], j < nv (Arnoldi steps:
// j <= ctl->k).  grid (nseg, splits, column groups); a CTA of 256 threads holds up to 8 rows per
// thread in registers and takes kDotCols columns, whose sums it reduces together (one column at
// a time, with a CTA reduction each, took 1.5 us a column).
constexpr int kDotRows = 8, kDotThreads = 256, kDotCols = 8;
template <class TV>
__global__ void __launch_bounds__(kDotThreads)
    k_seg_dots(int nu, const int* __restrict__ seg_begin, int nv, const TV* __restrict__ V, int64_t ldv,
               const TV* __restrict__ w, double* __restrict__ out, int ldo, const StepCtl* __restrict__ ctl = nullptr) {
  chain_wait();
  if (ctl) {
    if (ctl->stop) return;
    nv = ctl->k + 1;
  }
  const int j0 = blockIdx.z * kDotCols;
  if (j0 >= nv) return;
  const int nj = min(kDotCols, nv - j0);
  const int seg = blockIdx.x;
  const int64_t r0 = (int64_t)nu * seg_begin[seg], r1 = (int64_t)nu * seg_begin[seg + 1];
  const int64_t base = r0 + (int64_t)blockIdx.y * kDotThreads * kDotRows;
  if (base >= r1) return;
  TV wr[kDotRows];
#pragma unroll
  for (int i = 0; i < kDotRows; ++i) {
    const int64_t r = base + threadIdx.x + (int64_t)i * kDotThreads;
    wr[i] = r < r1 ? w[r] : TV(0);
  }
  __shared__ double red[kDotThreads / 32][kDotCols];
#pragma unroll 2
  for (int j = 0; j < nj; ++j) {
    const TV* vj = V + (int64_t)(j0 + j) * ldv;
    double s = 0;
#pragma unroll
    for (int i = 0; i < kDotRows; ++i) {
      const int64_t r = base + threadIdx.x + (int64_t)i * kDotThreads;
      if (r < r1) s += (double)vj[r] * (double)wr[i];
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][j] = s;
  }
  __syncthreads();
  if (threadIdx.x < nj) {
    double tot = 0;
    for (int k = 0; k < kDotThreads / 32; ++k) tot += red[k][threadIdx.x];
    atomicAdd(out + (int64_t)seg * ldo + j0 + threadIdx.x, tot);
  }
}

// w[row] -= sum_j h[seg(row) * ldh + j] V_j[row], j <= ctl->k; with n2, n2[seg] += w[row]^2
__global__ void __launch_bounds__(256) k_seg_sub(int nu, int64_t N, const int* __restrict__ seg_of,
                                                 const float* __restrict__ V, int64_t ldv, const double* __restrict__ h,
                                                 int ldh, float* __restrict__ w, double* __restrict__ n2,
                                                 const StepCtl* __restrict__ ctl) {
  chain_wait();
  if (ctl->stop) return;
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int nv = ctl->k + 1;
  const bool in = r < N;
  const int seg = in ? seg_of[r / nu] : -1;
  float s = 0.f;
  if (in) {
    const double* hs = h + (int64_t)seg * ldh;
    s = w[r];
#pragma unroll 4
    for (int j = 0; j < nv; ++j) s -= (float)hs[j] * V[(int64_t)j * ldv + r];
    w[r] = s;
  }
  if (!n2) return;
  // a warp's rows belong to one realisation, but for its borders
  double q = (double)s * (double)s;
  if (__all_sync(0xffffffffu, seg == __shfl_sync(0xffffffffu, seg, 0))) {
    for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if ((threadIdx.x & 31) == 0 && in) atomicAdd(n2 + seg, q);
  } else if (in) {
    atomicAdd(n2 + seg, q);
  }
}

// y[row] (+)= scale[seg(row)] * x[row] (FP32 <- FP64 / FP32); with ctl (after the step's update,
// which has counted it), y is column ctl->k of a basis with column stride ystride
template <class TX, class TY>
__global__ void k_seg_scale(int nu, int64_t N, const int* __restrict__ seg_of, const double* __restrict__ scale,
                            const TX* __restrict__ x, TY* __restrict__ y, int add,
                            const StepCtl* __restrict__ ctl = nullptr, int64_t ystride = 0) {
  chain_wait();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= N) return;
  if (ctl) {
    if (ctl->stop) return;
    y += (int64_t)ctl->k * ystride;
  }
  const double v = scale[seg_of[r / nu]] * (double)x[r];
  y[r] = add ? (TY)((double)y[r] + v) : (TY)v;
}

// Per-realisation Arnoldi bookkeeping after step k (one thread per realisation):
// H(:,k) = d1 + d2 (two Gram-Schmidt passes), H(k+1,k) = sqrt(n2), previous Givens
// rotations, the new one, g; inv = 1 / H(k+1,k) for normalising the new basis vector.
struct Krylov {
  double* H;      // nseg x (m+1) x m, row-major per realisation
  double* g;      // nseg x (m+1)
  double* cs;     // nseg x m
  double* sn;
  double* beta;   // nseg
  double* inv;    // nseg
  int* kc;        // nseg: Arnoldi columns accepted in this cycle
  int* active;    // nseg: 1 while the cycle continues for the realisation
  double* d1;     // nseg x (m+1) dot products, pass 1
  double* d2;     // pass 2
  double* n2;     // nseg
  double* yv;     // nseg x m
  double* thr;    // nseg: |g| target of the current GMRES solve (inner_tol * first beta)
  double* est;    // nseg: latest Arnoldi estimate of the GMRES residual norm
  int* nsteps;    // nseg: Arnoldi steps taken while active (reported)
  int* nactive;   // 1
};

// The last CTA then counts the step: ctl->k += 1, and stop once k == m or no realisation is
// active; `host` (pinned) is told.  d1, d2 and n2 are left zero for the next step.
__global__ void k_arnoldi_update(int nseg, int m, Krylov K, StepCtl* __restrict__ ctl, HostCtl* __restrict__ host) {
  chain_wait();
  if (ctl->stop) {
    if (host && blockIdx.x == 0 && threadIdx.x == 0) host->steps = host->steps + 1;
    return;
  }
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = ctl->k;
  int still = 0;
  if (s < nseg) {
    double* d1 = K.d1 + (int64_t)s * (m + 1);
    double* d2 = K.d2 + (int64_t)s * (m + 1);
    if (K.active[s]) {
      double* H = K.H + (int64_t)s * (m + 1) * m;
      double* g = K.g + (int64_t)s * (m + 1);
      double* cs = K.cs + (int64_t)s * m;
      double* sn = K.sn + (int64_t)s * m;
      // ||w|| after the two Gram-Schmidt passes
      const double hn = sqrt(fmax(K.n2[s], 0.0));
      double a = d1[0] + d2[0];
      for (int i = 0; i < k; ++i) {   // column k through the previous Givens rotations
        const double b = d1[i + 1] + d2[i + 1];
        H[i * m + k] = cs[i] * a + sn[i] * b;
        a = -sn[i] * a + cs[i] * b;
      }
      const double den = hypot(a, hn);
      cs[k] = den > 0 ? a / den : 1.0;
      sn[k] = den > 0 ? hn / den : 0.0;
      H[k * m + k] = den;
      H[(k + 1) * m + k] = 0.0;
      const double gk = g[k], gn = -sn[k] * gk;
      g[k + 1] = gn;
      g[k] = cs[k] * gk;
      K.kc[s] = k + 1;
      K.nsteps[s] += 1;
      K.est[s] = fabs(gn);
      still = !(fabs(gn) <= K.thr[s] || hn == 0.0 || k + 1 == m);
      K.inv[s] = still ? 1.0 / hn : 0.0;
      if (!still) K.active[s] = 0;
    } else {
      K.inv[s] = 0.0;
    }
    for (int i = 0; i <= k; ++i) d1[i] = d2[i] = 0.0;
    K.n2[s] = 0.0;
  }
  const int n = __syncthreads_count(still);
  if (threadIdx.x != 0) return;
  if (n) atomicAdd(&ctl->nactive, n);
  __threadfence();
  if (atomicAdd(&ctl->arrived, 1) + 1 < (int)gridDim.x) return;
  __threadfence();
  const int na = *reinterpret_cast<volatile int*>(&ctl->nactive);
  ctl->nactive = 0;
  ctl->arrived = 0;
  ctl->k = k + 1;
  ctl->stop = !(k + 1 < m && na > 0);
  if (host) {
    if (ctl->stop) host->stop = 1;
    __threadfence_system();
    host->steps = host->steps + 1;
  }
}

// y = H(0:kc, 0:kc)^-1 g(0:kc) per realisation (zeros beyond kc)
__global__ void k_hess_solve(int nseg, int m, Krylov K) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  const double* H = K.H + (int64_t)s * (m + 1) * m;
  const double* g = K.g + (int64_t)s * (m + 1);
  double* y = K.yv + (int64_t)s * m;
  const int kc = K.kc[s];
  for (int i = m - 1; i >= kc; --i) y[i] = 0.0;
  for (int i = kc - 1; i >= 0; --i) {
    double t = g[i];
    for (int j = i + 1; j < kc; ++j) t -= H[i * m + j] * y[j];
    y[i] = H[i * m + i] != 0.0 ? t / H[i * m + i] : 0.0;
  }
}

// start of a GMRES cycle: beta = sqrt(n2), g = (beta, 0, ...); on the first cycle of a
// solve thr = inner_tol[s] * beta; active while beta > thr and the realisation is not done
__global__ void k_cycle_start(int nseg, int m, Krylov K, const int* __restrict__ done, int first,
                              const double* __restrict__ inner_tol) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  const double b = sqrt(fmax(K.n2[s], 0.0));
  K.beta[s] = b;
  K.n2[s] = 0.0;
  if (first) K.thr[s] = inner_tol[s] * b;
  K.est[s] = b;
  double* g = K.g + (int64_t)s * (m + 1);
  for (int i = 0; i <= m; ++i) g[i] = 0.0;
  g[0] = b;
  const int a = (b > K.thr[s] && b > 0.0 && !done[s]) ? 1 : 0;
  K.active[s] = a;
  K.kc[s] = 0;
  K.inv[s] = a ? 1.0 / b : 0.0;
  if (a) atomicAdd(K.nactive, 1);
}

// x[row] = sum_j y[seg][j] V_j[row], j < ctl->k
__global__ void k_seg_combine(int nu, int64_t N, const int* __restrict__ seg_of, const float* __restrict__ V,
                              int64_t ldv, const double* __restrict__ y, int ldy, float* __restrict__ x,
                              const StepCtl* __restrict__ ctl) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= N) return;
  const int nv = ctl->k;
  const double* ys = y + (int64_t)seg_of[r / nu] * ldy;
  double s = 0;
  for (int j = 0; j < nv; ++j) s += ys[j] * (double)V[(int64_t)j * ldv + r];
  x[r] = (float)s;
}

template <class T>
__global__ void k_fill(T* p, int64_t n, T v) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}
__global__ void k_mul(int64_t n, const double* __restrict__ a, const double* __restrict__ x, double* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = a[i] * x[i];
}
__global__ void k_div_to_f32(int64_t n, const double* __restrict__ x, const double* __restrict__ d, float* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = (float)(x[i] / d[i]);
}
__global__ void k_f32_div(int64_t n, const float* __restrict__ x, const double* __restrict__ d, double* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = (double)x[i] / d[i];
}
// out = a - b (FP64)
__global__ void k_sub64(int64_t n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] - b[i];
}
// out = a - b (FP64) on the rows of realisations with done == 0
__global__ void k_sub64_masked(int nu, int64_t n, const int* __restrict__ seg_of, const int* __restrict__ done,
                               const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && !done[seg_of[i / nu]]) out[i] = a[i] - b[i];
}
// y = x / d (FP64)
__global__ void k_div64(int64_t n, const double* __restrict__ x, const double* __restrict__ d, double* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = x[i] / d[i];
}
__global__ void k_to_f32(int64_t n, const double* __restrict__ x, float* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = (float)x[i];
}
// y += x (FP32)
__global__ void k_add_f32(int64_t n, const float* __restrict__ x, float* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] += x[i];
}
// xs += d (FP64 += FP32)
__global__ void k_acc_f32(int64_t n, const float* __restrict__ d, double* __restrict__ xs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) xs[i] += (double)d[i];
}
// out = a - b (FP32)
__global__ void k_sub_f32(int64_t n, const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] - b[i];
}
// mean order-0 eigenstrain weighted by volume: out[seg*6 + r] += V_p E_p[r]
// Volume integral of each particle's eigenstrain polynomial, summed per realisation.  Over a
// sphere of radius a the linear terms average to zero and x_k x_l averages to a^2/5 delta_kl,
// so the order-2 coefficients E_ijkk (diagonal (k, k) slots: 0, 3, 5 of the six p <= q of
// layout 60; 0, 4, 8 of the nine (p, q) of layout 78) add a^2/5 each.
__global__ void k_vol_eigen(int num, int nu, const int* __restrict__ seg_of, const double* __restrict__ rad,
                            const double* __restrict__ axes, const double* __restrict__ x, double* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= num) return;
  const double a = rad[p];
  // particle volume (an ellipsoid's linear eigenstrain averages to its uniform part)
  const double vp = 4.0 / 3.0 * 3.141592653589793 *
                    (axes ? axes[3 * (int64_t)p] * axes[3 * (int64_t)p + 1] * axes[3 * (int64_t)p + 2] : a * a * a);
  const double q = a * a / 5.0;
  const double* e = x + (int64_t)nu * p;
  for (int r = 0; r < 6; ++r) {
    double v = e[r];
    if (nu == 60) v += q * (e[24 + 6 * r] + e[24 + 6 * r + 3] + e[24 + 6 * r + 5]);
    if (nu == 78) v += q * (e[24 + 9 * r] + e[24 + 9 * r + 4] + e[24 + 9 * r + 8]);
    atomicAdd(out + 6 * seg_of[p] + r, vp * v);
  }
}

inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// Source slices of a product hold at least 32 sources.  Where that leaves too few CTAs, a slice
// is cut into up to kMfPieces pieces (gridDim.z): a thread takes its sources one after the other
// (64 clocks per FP64 multiply-add and warp), so in a small realisation the slice is the
// product's latency: 64 spheres with one and with four pieces a slice (32 and 8 sources), FP64
// product 570 us and 156 us, FP32 product 25 and 13 us.
static int slice_cap(int max_seg) { return std::max(1, (max_seg + 31) / 32); }

static MfSplit mf_split(int ctas, int max_seg) {
  const int cap = slice_cap(max_seg);
  const int pieces = std::max(1, std::min(kMfPieces, (ctas + cap - 1) / cap));
  return {std::max(1, std::min(cap, (ctas + pieces - 1) / pieces)), pieces};
}

// ------------------------------------------------------------------ batch set-up
ibem_status mf_batch_init(MfBatch& b, const ibem_e3d_batch& in, cudaStream_t st, int layout) {
  if (layout != 24 && layout != 60) return fail(IBEM_ERR_ARG, "mf: layout 24 or 60");
  b.nu = layout;
  if (in.nseg <= 0 || !in.seg_begin || !in.centers_dev || !in.radius_dev || !in.mats)
    return fail(IBEM_ERR_ARG, "mf: bad batch");
  b.st = st;
  b.nseg = in.nseg;
  b.seg_begin_h.assign(in.seg_begin, in.seg_begin + in.nseg + 1);
  b.mats_h.assign(in.mats, in.mats + in.nseg);
  if (b.seg_begin_h[0] != 0) return fail(IBEM_ERR_ARG, "mf: seg_begin[0] must be 0");
  b.max_seg = 0;
  for (int s = 0; s < in.nseg; ++s) {
    const int n = b.seg_begin_h[s + 1] - b.seg_begin_h[s];
    if (n < 1) return fail(IBEM_ERR_ARG, "mf: every realisation needs at least one particle");
    b.max_seg = std::max(b.max_seg, n);
  }
  b.num = b.seg_begin_h[in.nseg];
  b.N = (int64_t)b.nu * b.num;
  b.cen = in.centers_dev;
  b.rad = in.radius_dev;
  b.axes = in.axes_dev;
  std::vector<int> seg_of(b.num);
  std::vector<MfTile> tiles;
  for (int s = 0; s < in.nseg; ++s) {
    for (int p = b.seg_begin_h[s]; p < b.seg_begin_h[s + 1]; ++p) seg_of[p] = s;
    for (int p = b.seg_begin_h[s]; p < b.seg_begin_h[s + 1]; p += kMfThreads)
      tiles.push_back({s, p, std::min(kMfThreads, b.seg_begin_h[s + 1] - p), 0});
  }
  b.ntiles = (int)tiles.size();
  std::vector<MfTile> tiles_s[3];
  for (int k = 0; k < 3; ++k) {
    const int tt = 64 << k;
    for (int s = 0; s < in.nseg; ++s)
      for (int p = b.seg_begin_h[s]; p < b.seg_begin_h[s + 1]; p += tt)
        tiles_s[k].push_back({s, p, std::min(tt, b.seg_begin_h[s + 1] - p), 0});
    b.ntiles_s[k] = (int)tiles_s[k].size();
  }
  // slices of the source range: about 4 CTAs per SM in total, at least 32 sources per slice
  int dev = 0, nsm = 0;
  IBEM_CUDA(cudaGetDevice(&dev));
  IBEM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int want = std::max(1, nsm) * 4;
  b.split = b.split_wide = mf_split((want + b.ntiles - 1) / b.ntiles, b.max_seg);
  std::vector<SphMat> md(in.nseg), ms(in.nseg);
  std::vector<SphMatF> mf(in.nseg);
  for (int s = 0; s < in.nseg; ++s) {
    const ibem_material& m = in.mats[s];
    md[s] = sph_mat_init(m.E0, m.nu0, m.E1, m.nu1);
    mf[s] = sph_matf_init(md[s]);
    ms[s] = md[s];  // scaled: moduli / mu0
    const double k = 1.0 / md[s].mu0;
    ms[s].kmu *= k;
    ms[s].klam *= k;
    ms[s].lam0 *= k;
    ms[s].twomu0 *= k;
    ms[s].mu0 = 1.0;
  }
  IBEM_CUDA(alloc_async((void**)&b.seg_begin, sizeof(int) * (in.nseg + 1), st));
  IBEM_CUDA(alloc_async((void**)&b.seg_of, sizeof(int) * b.num, st));
  IBEM_CUDA(alloc_async((void**)&b.gh, sizeof(float4) * b.num, st));
  IBEM_CUDA(alloc_async((void**)&b.gl, sizeof(float4) * b.num, st));
  IBEM_CUDA(alloc_async((void**)&b.matd, sizeof(SphMat) * in.nseg, st));
  IBEM_CUDA(alloc_async((void**)&b.matf, sizeof(SphMatF) * in.nseg, st));
  IBEM_CUDA(alloc_async((void**)&b.mats, sizeof(SphMat) * in.nseg, st));
  IBEM_CUDA(alloc_async((void**)&b.dr, sizeof(double) * b.N, st));
  IBEM_CUDA(alloc_async((void**)&b.dc, sizeof(double) * b.N, st));
  IBEM_CUDA(alloc_async((void**)&b.tiles, sizeof(MfTile) * b.ntiles, st));
  for (int k = 0; k < 3; ++k) IBEM_CUDA(alloc_async((void**)&b.tiles_s[k], sizeof(MfTile) * b.ntiles_s[k], st));
  // Morton order of the centres within each realisation (10 bits per axis of its bounding box)
  std::vector<int> perm(b.num);
  {
    std::vector<double> ch(3 * (size_t)b.num);
    IBEM_CUDA(cudaMemcpyAsync(ch.data(), in.centers_dev, sizeof(double) * ch.size(), cudaMemcpyDeviceToHost, st));
    IBEM_CUDA(cudaStreamSynchronize(st));
    auto spread = [](uint32_t v) {
      v &= 0x3ffu;
      v = (v | (v << 16)) & 0x030000ffu;
      v = (v | (v << 8)) & 0x0300f00fu;
      v = (v | (v << 4)) & 0x030c30c3u;
      v = (v | (v << 2)) & 0x09249249u;
      return v;
    };
    std::vector<std::pair<uint32_t, int>> key;
    for (int s = 0; s < in.nseg; ++s) {
      const int p0 = b.seg_begin_h[s], p1 = b.seg_begin_h[s + 1];
      double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
      for (int p = p0; p < p1; ++p)
        for (int d = 0; d < 3; ++d) {
          lo[d] = std::min(lo[d], ch[3 * (size_t)p + d]);
          hi[d] = std::max(hi[d], ch[3 * (size_t)p + d]);
        }
      key.clear();
      for (int p = p0; p < p1; ++p) {
        uint32_t q[3];
        for (int d = 0; d < 3; ++d) {
          const double w = hi[d] > lo[d] ? (ch[3 * (size_t)p + d] - lo[d]) / (hi[d] - lo[d]) : 0.0;
          q[d] = (uint32_t)std::min(1023.0, std::max(0.0, std::floor(w * 1024.0)));
        }
        key.push_back({spread(q[0]) | (spread(q[1]) << 1) | (spread(q[2]) << 2), p});
      }
      std::sort(key.begin(), key.end());
      for (int i = 0; i < p1 - p0; ++i) perm[p0 + i] = key[i].second;
    }
  }
  IBEM_CUDA(alloc_async((void**)&b.perm, sizeof(int) * b.num, st));
  IBEM_CUDA(cudaMemcpyAsync(b.perm, perm.data(), sizeof(int) * b.num, cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaMemcpyAsync(b.seg_begin, b.seg_begin_h.data(), sizeof(int) * (in.nseg + 1), cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaMemcpyAsync(b.seg_of, seg_of.data(), sizeof(int) * b.num, cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaMemcpyAsync(b.matd, md.data(), sizeof(SphMat) * in.nseg, cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaMemcpyAsync(b.matf, mf.data(), sizeof(SphMatF) * in.nseg, cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaMemcpyAsync(b.mats, ms.data(), sizeof(SphMat) * in.nseg, cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaMemcpyAsync(b.tiles, tiles.data(), sizeof(MfTile) * b.ntiles, cudaMemcpyHostToDevice, st));
  for (int k = 0; k < 3; ++k)
    IBEM_CUDA(cudaMemcpyAsync(b.tiles_s[k], tiles_s[k].data(), sizeof(MfTile) * b.ntiles_s[k], cudaMemcpyHostToDevice,
                              st));
  b.tshape = 1;   // 128 targets per CTA until the autotuner says otherwise
  ::ibem::count_launch(), k_mf_prep<<<nblk(b.num), 256, 0, st>>>(b.nu, b.num, b.cen, b.rad, b.seg_of, b.matd, b.gh, b.gl,
                                                                 b.dr, b.dc);
  IBEM_LAUNCH_CHECK("mf prep");
  if (b.nu == 60) {
    IBEM_CUDA(alloc_async((void**)&b.self60, sizeof(double) * 3600 * in.nseg, st));
    IBEM_CUDA(alloc_async((void**)&b.self60f, sizeof(float) * 3600 * in.nseg, st));
    if (ibem_status q = mf60_self(b, st)) return q;
  }
  // the host vectors above must outlive the copies
  IBEM_CUDA(cudaStreamSynchronize(st));
  return IBEM_OK;
}

void mf_batch_free(MfBatch& b) {
  const cudaStream_t st = b.st;
  free_async(b.seg_begin, st);
  free_async(b.seg_of, st);
  free_async(b.gh, st);
  free_async(b.gl, st);
  free_async(b.matd, st);
  free_async(b.matf, st);
  free_async(b.mats, st);
  free_async(b.self60, st);
  free_async(b.self60f, st);
  free_async(b.dr, st);
  free_async(b.dc, st);
  free_async(b.tiles, st);
  for (int k = 0; k < 3; ++k) free_async(b.tiles_s[k], st);
  free_async(b.work, st);
  free_async(b.perm, st);
  b = MfBatch();
}

ibem_status mf_set_f32_shape(MfBatch& b, int tshape, MfSplit split, int persist, cudaStream_t st) {
  const int hsplit = split.slices;
  b.tshape = tshape;
  b.split = split;
  b.persist = persist;
  if (!persist) return IBEM_OK;
  // work list: every (tile, slice) with sources, by decreasing targets x sources
  std::vector<MfTile> tiles(b.ntiles_s[tshape]);
  {
    // tiles of this shape, rebuilt on the host from the segment table (as at batch init)
    const int tt = 64 << tshape;
    int n = 0;
    for (int s = 0; s < b.nseg; ++s)
      for (int p = b.seg_begin_h[s]; p < b.seg_begin_h[s + 1]; p += tt)
        tiles[n++] = {s, p, std::min(tt, b.seg_begin_h[s + 1] - p), 0};
  }
  std::vector<std::pair<int64_t, int2>> items;
  for (int t = 0; t < (int)tiles.size(); ++t) {
    const int hb0 = b.seg_begin_h[tiles[t].seg], he0 = b.seg_begin_h[tiles[t].seg + 1];
    const int per = (he0 - hb0 + hsplit - 1) / hsplit;
    for (int j = 0; j < hsplit; ++j) {
      const int len = std::min(he0, hb0 + (j + 1) * per) - (hb0 + j * per);
      if (len > 0) items.push_back({(int64_t)len * tiles[t].ns, make_int2(t, j)});
    }
  }
  std::stable_sort(items.begin(), items.end(), [](const auto& a, const auto& c) { return a.first > c.first; });
  std::vector<int2> w(items.size());
  for (size_t i = 0; i < items.size(); ++i) w[i] = items[i].second;
  free_async(b.work, st);
  b.work = nullptr;
  b.nwork = (int)w.size();
  IBEM_CUDA(alloc_async((void**)&b.work, sizeof(int2) * std::max<size_t>(1, w.size()), st));
  IBEM_CUDA(cudaMemcpyAsync(b.work, w.data(), sizeof(int2) * w.size(), cudaMemcpyHostToDevice, st));
  IBEM_CUDA(cudaStreamSynchronize(st));   // w must outlive the copy
  int dev = 0, sms = 0, per_sm = 0;
  IBEM_CUDA(cudaGetDevice(&dev));
  IBEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int tt = 64 << tshape;
  cudaError_t e = tshape == 0   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mf_apply_f32_persist<64>, tt, 0)
                  : tshape == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mf_apply_f32_persist<128>, tt, 0)
                                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mf_apply_f32_persist<256>, tt, 0);
  if (e != cudaSuccess) return cuda_fail(e, "mf persistent occupancy");
  b.persist_ctas = std::max(1, std::min(b.nwork, std::max(1, per_sm) * sms));
  return IBEM_OK;
}

// ------------------------------------------------------------------ autotuner
// The products' launch shape is (target tiles) x (source slices); the slice count trades
// parallelism and tail effects against the atomic adds of the partial sums.  For the FP32
// product (the GMRES operator, launched once per Arnoldi step) the tuner also picks the
// tile shape (64, 128 or 256 targets per CTA) and the launch form: one CTA per (tile,
// slice), or persistent CTAs (as many as fit on the GPU) over a list of (tile, slice) items
// sorted by decreasing cost.  For a shape class (log2 buckets of the tile count and of the
// largest realisation, and the number of SMs) every candidate is run once to warm up and
// once timed with CUDA events (inputs of zeros: the same work as any input); the fastest is
// kept for the process.  The double-float / FP64 kernels (~255 registers) keep 128-target
// tiles and get their own slice count.
namespace {
struct TuneKey {
  int tiles_b, seg_b, sms;
  bool operator<(const TuneKey& o) const {
    return tiles_b != o.tiles_b ? tiles_b < o.tiles_b : seg_b != o.seg_b ? seg_b < o.seg_b : sms < o.sms;
  }
};
struct TuneVal {
  MfSplit split, split_wide;
  int tshape, persist;
};
std::mutex g_tune_mu;
std::map<TuneKey, TuneVal> g_tune;

int log2_bucket(int v) {
  int b = 0;
  while ((1 << b) < v) ++b;
  return b;
}
// splits of the source range that give 1, 2, 4 and 8 CTAs per SM in total
std::vector<MfSplit> split_candidates(int ntiles, int max_seg, int sms) {
  std::vector<MfSplit> cand;
  for (int per_sm : {1, 2, 4, 8}) {
    const MfSplit h = mf_split((sms * per_sm + ntiles - 1) / ntiles, max_seg);
    if (std::find(cand.begin(), cand.end(), h) == cand.end()) cand.push_back(h);
  }
  return cand;
}
}  // namespace

ibem_status mf_tune(MfBatch& b, cudaStream_t st) {
  int dev = 0, sms = 0;
  IBEM_CUDA(cudaGetDevice(&dev));
  IBEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const TuneKey key{log2_bucket(b.ntiles), log2_bucket(b.max_seg), sms * 100 + b.nu};
  const int cap = slice_cap(b.max_seg);
  // IBEM_MF_F32_SHAPE="shape,persistent,slices[,pieces]" fixes the FP32 product's launch (tests and
  // measurements of every shape); the wide products keep the batch's initial split
  if (const char* f = b.nu == 24 ? std::getenv("IBEM_MF_F32_SHAPE") : nullptr) {
    int ts = 1, pers = 0, h = 1, pc = 1;
    if (std::sscanf(f, "%d,%d,%d,%d", &ts, &pers, &h, &pc) >= 3 && ts >= 0 && ts < 3 && (pers == 0 || pers == 1) && h >= 1 &&
        pc >= 1 && pc <= (pers ? 1 : kMfPieces))
      return mf_set_f32_shape(b, ts, {std::min(h, cap), pc}, pers, st);
    return fail(IBEM_ERR_ARG, "IBEM_MF_F32_SHAPE: expected shape (0-2),persistent (0/1),slices (>= 1)[,pieces (1-4, persistent 1)]");
  }
  {
    bool hit = false;
    TuneVal v{};
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      auto it = g_tune.find(key);
      if (it != g_tune.end()) {
        hit = true;
        v = it->second;
      }
    }
    if (hit) {
      b.split_wide = {std::min(v.split_wide.slices, cap), v.split_wide.pieces};
      return mf_set_f32_shape(b, v.tshape, {std::min(v.split.slices, cap), v.split.pieces}, v.persist, st);
    }
  }
  float* xf = nullptr;
  float* yf = nullptr;
  double* xd = nullptr;
  double* yd = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  ibem_status s = IBEM_OK;
  {
    cudaError_t e = alloc_async((void**)&xf, sizeof(float) * b.N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&yf, sizeof(float) * b.N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&xd, sizeof(double) * b.N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&yd, sizeof(double) * b.N, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(xf, 0, sizeof(float) * b.N, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(xd, 0, sizeof(double) * b.N, st);
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e != cudaSuccess) s = cuda_fail(e, "mf tune");
  }
  // runs the product twice (warm-up, then timed) and returns the timed milliseconds
  auto time_it = [&](bool wide, float& ms) -> ibem_status {
    for (int rep = 0; rep < 2; ++rep) {
      cudaEventRecord(e0, st);
      ibem_status r = wide ? mf_apply_df(b, xd, yd, st) : mf_apply_f32(b, xf, yf, st);
      cudaEventRecord(e1, st);
      if (r) return r;
    }
    const cudaError_t e = cudaEventSynchronize(e1);
    if (e != cudaSuccess) return cuda_fail(e, "mf tune");
    cudaEventElapsedTime(&ms, e0, e1);
    return IBEM_OK;
  };
  TuneVal best{b.split, b.split_wide, b.tshape, 0};
  float best_ms = 1e30f;
  for (int ts = 0; ts < 3 && !s; ++ts)
    for (MfSplit h : split_candidates(b.ntiles_s[ts], b.max_seg, sms)) {
      if (b.nu == 60 && ts != 0) break;   // the layout-60 products have 64-target tiles only
      for (int pers = 0; pers < (b.nu == 60 ? 1 : 2) && !s; ++pers) {
        if (pers && h.pieces > 1) continue;   // the work list is of whole slices
        if ((s = mf_set_f32_shape(b, ts, h, pers, st))) break;
        float ms = 0.f;
        if ((s = time_it(false, ms))) break;
        if (ms < best_ms) {
          best_ms = ms;
          best.tshape = ts;
          best.split = h;
          best.persist = pers;
        }
      }
      if (s) break;
    }
  best_ms = 1e30f;
  for (MfSplit h : split_candidates(b.nu == 60 ? b.ntiles_s[0] : b.ntiles, b.max_seg, sms)) {
    if (s) break;
    b.split_wide = h;
    float ms = 0.f;
    if ((s = time_it(true, ms))) break;
    if (ms < best_ms) {
      best_ms = ms;
      best.split_wide = h;
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  free_async(xf, st);
  free_async(yf, st);
  free_async(xd, st);
  free_async(yd, st);
  if (s) return s;
  b.split_wide = best.split_wide;
  if ((s = mf_set_f32_shape(b, best.tshape, best.split, best.persist, st))) return s;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune[key] = best;
  return IBEM_OK;
}

template <int TT>
void launch_f32(const MfBatch& b, const float* x, float* y, cudaStream_t st, const int* mask, int mask_on) {
  const MfTile* tiles = b.tiles_s[TT == 64 ? 0 : (TT == 128 ? 1 : 2)];
  if (b.persist)
    launch_chained(k_mf_apply_f32_persist<TT>, b.persist_ctas, TT, st, tiles, b.work, b.nwork, b.split.slices, b.seg_begin,
                   mask, mask_on, b.gh, b.gl, b.matf, x, y);
  else
    launch_chained(k_mf_apply_f32<TT>, dim3(b.ntiles_s[TT == 64 ? 0 : (TT == 128 ? 1 : 2)], b.split.slices, b.split.pieces),
                   TT, st, tiles, b.seg_begin, mask, mask_on, b.gh, b.gl, b.matf, x, y);
}

ibem_status mf_apply_f32(const MfBatch& b, const float* x, float* y, cudaStream_t st, const int* mask, int mask_on,
                         bool clear) {
  ProfScope ps(PROF_MF_F32, st, 0.0);
  if (b.nu == 60) return mf60_apply_f32(b, x, y, st, mask, mask_on);
  if (clear) IBEM_CUDA(cudaMemsetAsync(y, 0, sizeof(float) * b.N, st));
  if (b.tshape == 0) launch_f32<64>(b, x, y, st, mask, mask_on);
  else if (b.tshape == 2) launch_f32<256>(b, x, y, st, mask, mask_on);
  else launch_f32<128>(b, x, y, st, mask, mask_on);
  IBEM_LAUNCH_CHECK("mf apply f32");
  return IBEM_OK;
}

ibem_status mf_apply_f64(const MfBatch& b, const double* x, double* y, cudaStream_t st, const int* mask, int mask_on) {
  ProfScope ps(PROF_MF_F64, st, 0.0);
  if (b.nu == 60) return mf60_apply_f64(b, x, y, st, mask, mask_on);
  IBEM_CUDA(cudaMemsetAsync(y, 0, sizeof(double) * b.N, st));
  // near sources in FP64, far sources (beyond kMfFarRadii of their radius from the box of
  // the warp's targets) in double-float: their contributions are at most kMfFarRadii^-3 of a
  // touching one, so the double-float rounding (~2^-44 per operation, times 4^-3) is ~1e-15
  // of the largest term, the level of the FP64 rounding of the near pairs (measured: split
  // against all pairs in FP64 6.6e-16 relative, 5.2e-16 with 8 radii, 1.7e-14 for
  // double-float everywhere).  In realisations below kMfSplitMin particles most (warp,
  // source) pairs are near, and one FP64 launch over every pair is faster than the two passes:
  // 900 spheres 0.73 and 0.90 ms, 1,280 1.55 and 1.16 ms, 20,000 395 and 94 ms.  Skipping near
  // sources in the far pass against evaluating them with zero coefficients: 2,000 spheres 1.76 and
  // 1.69 ms, 5,000 7.3 and 8.1 ms
  const bool split = b.max_seg >= kMfSplitMin;
  ::ibem::count_launch(), k_mf_apply_f64<<<dim3(b.ntiles, b.split_wide.slices, b.split_wide.pieces), kMfThreads, 0, st>>>(
      b.tiles, b.seg_begin, mask, mask_on, b.cen, b.rad, b.mats, x, y, b.perm, split ? 1 : 0);
  if (split && b.max_seg < kMfSkipMin)
    ::ibem::count_launch(), k_mf_apply_df<kMfThreads><<<dim3(b.ntiles, b.split_wide.slices, b.split_wide.pieces), kMfThreads, 0, st>>>(
        b.tiles, b.seg_begin, mask, mask_on, b.cen, b.rad, b.mats, x, y, b.perm, 2);
  else if (split)   // the same number of warps per SM, one CTA of 256 targets (tiles_s[2])
    ::ibem::count_launch(),
        k_mf_apply_df<2 * kMfThreads><<<dim3(b.ntiles_s[2], std::min((b.max_seg + 31) / 32, 2 * b.split_wide.slices)),
                                         2 * kMfThreads, 0, st>>>(b.tiles_s[2], b.seg_begin, mask, mask_on, b.cen,
                                                                  b.rad, b.mats, x, y, b.perm, 3);
  IBEM_LAUNCH_CHECK("mf apply f64");
  return IBEM_OK;
}

ibem_status mf_apply_f64_all(const MfBatch& b, const double* x, double* y, cudaStream_t st) {
  ProfScope ps(PROF_MF_F64, st, 0.0);
  if (b.nu == 60) return mf60_apply_f64(b, x, y, st, nullptr, 1);
  IBEM_CUDA(cudaMemsetAsync(y, 0, sizeof(double) * b.N, st));
  ::ibem::count_launch(), k_mf_apply_f64<<<dim3(b.ntiles, b.split_wide.slices, b.split_wide.pieces), kMfThreads, 0, st>>>(
      b.tiles, b.seg_begin, nullptr, 1, b.cen, b.rad, b.mats, x, y, b.perm, 0);
  IBEM_LAUNCH_CHECK("mf apply f64 (all pairs)");
  return IBEM_OK;
}

ibem_status mf_apply_df(const MfBatch& b, const double* x, double* y, cudaStream_t st, const int* mask, int mask_on) {
  ProfScope ps(PROF_MF_DF, st, 0.0);
  if (b.nu == 60) return mf60_apply_f64(b, x, y, st, mask, mask_on);   // no double-float form of layout 60
  IBEM_CUDA(cudaMemsetAsync(y, 0, sizeof(double) * b.N, st));
  ::ibem::count_launch(), k_mf_apply_df<kMfThreads><<<dim3(b.ntiles, b.split_wide.slices, b.split_wide.pieces), kMfThreads, 0, st>>>(
      b.tiles, b.seg_begin, mask, mask_on, b.cen, b.rad, b.mats, x, y, b.perm, 0);
  IBEM_LAUNCH_CHECK("mf apply df");
  return IBEM_OK;
}

ibem_status mf_block_jacobi(const MfBatch& b, float* P, cudaStream_t st) {
  float* Pseg = nullptr;
  IBEM_CUDA(alloc_async((void**)&Pseg, sizeof(float) * kMfNu * kMfNu * (size_t)b.nseg, st));
  ::ibem::count_launch(), k_block_jacobi<<<b.nseg, kBjThreads24, 0, st>>>(b.matd, Pseg);
  ::ibem::count_launch(), k_bcast_blocks<<<nblk((int64_t)b.num * kMfNu * kMfNu / 4), 256, 0, st>>>(b.num, b.seg_of, Pseg, P);
  free_async(Pseg, st);
  IBEM_LAUNCH_CHECK("block jacobi");
  return IBEM_OK;
}


// ------------------------------------------------------------------ solver
namespace {

// A HostCtl in pinned memory for the life of one solve.  The slots are a page per process,
// allocated on first use; a solve that finds none free (or is told not to) runs step by step.
struct HostSlot {
  static constexpr int kSlots = 64;
  HostCtl* ctl = nullptr;
  explicit HostSlot(bool wanted) {
    if (!wanted) return;
    std::lock_guard<std::mutex> l(mu());
    Slots& p = slots();
    if (!p.mem && !p.tried) {
      p.tried = true;
      void* m = nullptr;
      CaptureSafe safe;
      if (cudaHostAlloc(&m, kSlots * kStride, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess)
        p.mem = static_cast<char*>(m);
      else
        cudaGetLastError();
    }
    for (int i = 0; p.mem && i < kSlots; ++i)
      if (!p.used[i]) {
        p.used[i] = true;
        ctl = reinterpret_cast<HostCtl*>(p.mem + i * kStride);
        break;
      }
  }
  ~HostSlot() {
    if (!ctl) return;
    std::lock_guard<std::mutex> l(mu());
    slots().used[(reinterpret_cast<char*>(ctl) - slots().mem) / kStride] = false;
  }
  HostSlot(const HostSlot&) = delete;
  HostSlot& operator=(const HostSlot&) = delete;

 private:
  static constexpr size_t kStride = 64;   // a cache line each
  struct Slots {
    char* mem = nullptr;
    bool tried = false, used[kSlots] = {};
  };
  static std::mutex& mu() {
    static std::mutex m;
    return m;
  }
  static Slots& slots() {
    static Slots s;
    return s;
  }
};

struct MfSolver {
  const MfBatch& b;
  cudaStream_t st;
  int m;
  int64_t N;
  float* V = nullptr;    // (m+1) x N Krylov basis
  float* z = nullptr;    // N
  float* w = nullptr;    // N   new Arnoldi vector before normalisation (and scratch)
  float* d = nullptr;    // N   correction of the current refinement step
  float* rin = nullptr;  // N   right-hand side of the current GMRES solve
  float* r32 = nullptr;  // N   residual of a restarted cycle
  int* done = nullptr;   // nseg
  double* tolv = nullptr;  // nseg: residual reduction asked of this GMRES solve
  StepCtl* ctl = nullptr;  // control of the cycle's steps
  HostSlot host;           // the host's view of it (none: the host reads ctl after every step)
  Krylov K{};
  void* kmem = nullptr;
  int splits = 1;
  MfSolver(const MfBatch& bb, cudaStream_t s, int mm, bool ahead) : b(bb), st(s), m(mm), N(bb.N), host(ahead) {
    splits = (int)((b.nu * (int64_t)b.max_seg + kDotThreads * kDotRows - 1) / (kDotThreads * kDotRows));
  }
  ~MfSolver() {
    if (host.ctl) cudaStreamSynchronize(st);   // after an error steps may still report to the slot
    free_async(V, st);
    free_async(z, st);
    free_async(w, st);
    free_async(d, st);
    free_async(rin, st);
    free_async(r32, st);
    free_async(done, st);
    free_async(tolv, st);
    free_async(kmem, st);
  }
  ibem_status alloc() {
    IBEM_CUDA(alloc_async((void**)&V, sizeof(float) * N * (m + 1), st));
    IBEM_CUDA(alloc_async((void**)&z, sizeof(float) * N, st));
    IBEM_CUDA(alloc_async((void**)&w, sizeof(float) * N, st));
    IBEM_CUDA(alloc_async((void**)&d, sizeof(float) * N, st));
    IBEM_CUDA(alloc_async((void**)&rin, sizeof(float) * N, st));
    IBEM_CUDA(alloc_async((void**)&r32, sizeof(float) * N, st));
    IBEM_CUDA(alloc_async((void**)&done, sizeof(int) * b.nseg, st));
    IBEM_CUDA(alloc_async((void**)&tolv, sizeof(double) * b.nseg, st));
    const size_t S = b.nseg;
    const size_t nd = S * ((size_t)(m + 1) * m + (m + 1) + 2 * (size_t)m + 5 + 2 * (size_t)(m + 1) + m);
    const size_t ni = 3 * S + 1 + 4;
    IBEM_CUDA(alloc_async((void**)&kmem, nd * sizeof(double) + sizeof(int) * ni, st));
    double* p = (double*)kmem;
    K.H = p; p += S * (m + 1) * m;
    K.g = p; p += S * (m + 1);
    K.cs = p; p += S * m;
    K.sn = p; p += S * m;
    K.beta = p; p += S;
    K.inv = p; p += S;
    K.n2 = p; p += S;
    K.thr = p; p += S;
    K.est = p; p += S;
    K.d1 = p; p += S * (m + 1);
    K.d2 = p; p += S * (m + 1);
    K.yv = p; p += S * m;
    int* ip = (int*)p;
    K.kc = ip; ip += S;
    K.active = ip; ip += S;
    K.nsteps = ip; ip += S;
    K.nactive = ip; ip += 1;
    ctl = reinterpret_cast<StepCtl*>(ip);
    IBEM_CUDA(cudaMemsetAsync(kmem, 0, nd * sizeof(double) + sizeof(int) * ni, st));
    return IBEM_OK;
  }
  template <class T>
  ibem_status seg_norm2(const T* v, double* n2, cudaStream_t s) {
    IBEM_CUDA(cudaMemsetAsync(n2, 0, sizeof(double) * b.nseg, s));
    ::ibem::count_launch(), k_seg_dots<T><<<dim3(b.nseg, splits), kDotThreads, 0, s>>>(b.nu, b.seg_begin, 1, v, 0, v, n2, 1);
    IBEM_LAUNCH_CHECK("seg norm");
    return IBEM_OK;
  }
  template <class T>
  ibem_status seg_norm2(const T* v, double* n2) { return seg_norm2(v, n2, st); }
  int read_int(const int* p, ibem_status& s) {
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, p, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "gmres: read active count");
    return h;
  }
  // z = P v (layout 24: the block-sparse preconditioner; layout 60: the realisation's
  // block-Jacobi block, P.D holding one 60 x 60 block per realisation)
  ibem_status precond(const MfPrecond& P, const float* v, float* z, float* zero, const StepCtl* c, int64_t vstride) {
    if (b.nu == 60) return mf60_precond_apply(b, P.D, v, z, c ? &c->k : nullptr, vstride, st);
    launch_chained(k_precond_apply, nblk(b.num, kPrePart), kPreThreads, st, b.num, P.D, P.Q, P.nbr, v, z, zero, c, vstride);
    IBEM_LAUNCH_CHECK("preconditioner");
    return IBEM_OK;
  }
  // The next Arnoldi step: w = As P v_k, two Gram-Schmidt passes against v_0..v_k, the
  // per-realisation Hessenberg update, v_(k+1) = w / ||w||, k = ctl->k read by the kernels.
  ibem_status arnoldi_step(const MfPrecond& P) {
    const int S = b.nseg;
    const dim3 dots(S, splits, (m + kDotCols - 1) / kDotCols);
    ibem_status r = precond(P, V, z, w, ctl, N);
    if (r) return r;
    r = mf_apply_f32(b, z, w, st, K.active, 1, false);   // converged realisations sit out
    if (r) return r;
    ProfScope pg(PROF_GMRES_OTHER, st);
    launch_chained(k_seg_dots<float>, dots, kDotThreads, st, b.nu, b.seg_begin, 0, V, N, w, K.d1, m + 1, ctl);
    launch_chained(k_seg_sub, nblk(N), 256, st, b.nu, N, b.seg_of, V, N, K.d1, m + 1, w, nullptr, ctl);
    launch_chained(k_seg_dots<float>, dots, kDotThreads, st, b.nu, b.seg_begin, 0, V, N, w, K.d2, m + 1, ctl);
    launch_chained(k_seg_sub, nblk(N), 256, st, b.nu, N, b.seg_of, V, N, K.d2, m + 1, w, K.n2, ctl);
    launch_chained(k_arnoldi_update, nblk(S, 128), 128, st, S, m, K, ctl, host.ctl);
    launch_chained(k_seg_scale<float, float>, nblk(N), 256, st, b.nu, N, b.seg_of, K.inv, w, V, 0, ctl, N);
    IBEM_LAUNCH_CHECK("arnoldi step");
    return IBEM_OK;
  }
  // The steps of a cycle, each launched while the one before is still running: the update kernel
  // reports through pinned memory, so the stream never runs dry between steps, and the kernels of
  // steps past the end return at once.  A while node of a CUDA graph around one captured step
  // cost its capture and instantiation on every solve, and its kernels could not be set up early
  // (chain_wait): solve of 64 particles 1.90 ms, 1.55 ms with this form.
  ibem_status run_steps(const MfPrecond& P) {
    constexpr int kAhead = 1;
    ibem_status s = IBEM_OK;
    if (!host.ctl) {   // step by step
      do {
        if ((s = arnoldi_step(P))) return s;
      } while (!read_int(&ctl->stop, s) && !s);
      return s;
    }
    host.ctl->steps = 0;
    host.ctl->stop = 0;
    for (int launched = 0; launched < m; ++launched) {
      long long spins = 0;
      while (launched - __atomic_load_n(const_cast<int*>(&host.ctl->steps), __ATOMIC_ACQUIRE) > kAhead) {
        // the flag can only stay behind when the stream failed; look at it now and then
        if (++spins % 65536 == 0) {
          const cudaError_t e = cudaStreamQuery(st);
          if (e != cudaSuccess && e != cudaErrorNotReady) return cuda_fail(e, "gmres: Arnoldi steps");
          if (e == cudaSuccess && launched - host.ctl->steps > kAhead) return fail(IBEM_ERR_CUDA, "gmres: lost an Arnoldi step");
        }
      }
      if (host.ctl->stop) break;
      if ((s = arnoldi_step(P))) return s;
    }
    return s;
  }
  // FP32 GMRES(m) with restarts on As d = rin, right-preconditioned by P; d overwritten.
  // Realisations flagged in `done` take no step.  Stops each realisation once
  // ||rin - As d|| <= inner_tol ||rin|| (Arnoldi estimate).
  ibem_status gmres(const MfPrecond& P, int max_cycles) {
    const int S = b.nseg;
    ibem_status s = IBEM_OK;
    IBEM_CUDA(cudaMemsetAsync(d, 0, sizeof(float) * N, st));
    for (int cyc = 0; cyc < max_cycles && !s; ++cyc) {
      const float* r = rin;
      if (cyc > 0) {  // residual of the restarted cycle, rin - As d
        if ((s = mf_apply_f32(b, d, w, st, done, 0))) break;
        ::ibem::count_launch(), k_sub_f32<<<nblk(N), 256, 0, st>>>(N, rin, w, r32);
        r = r32;
      }
      if ((s = seg_norm2(r, K.n2))) break;
      IBEM_CUDA(cudaMemsetAsync(K.nactive, 0, sizeof(int) + sizeof(StepCtl), st));   // and ctl behind it
      ::ibem::count_launch(), k_cycle_start<<<nblk(S, 128), 128, 0, st>>>(S, m, K, done, cyc == 0, tolv);
      ::ibem::count_launch(), k_seg_scale<float, float><<<nblk(N), 256, 0, st>>>(b.nu, N, b.seg_of, K.inv, r, V, 0);
      IBEM_LAUNCH_CHECK("gmres cycle start");
      const int na = read_int(K.nactive, s);
      if (s || na == 0) break;
      if ((s = run_steps(P))) break;
      // d += P V y
      ::ibem::count_launch(), k_hess_solve<<<nblk(S, 128), 128, 0, st>>>(S, m, K);
      ::ibem::count_launch(), k_seg_combine<<<nblk(N), 256, 0, st>>>(b.nu, N, b.seg_of, V, N, K.yv, m, w, ctl);
      if ((s = precond(P, w, z, nullptr, nullptr, 0))) break;
      ::ibem::count_launch(), k_add_f32<<<nblk(N), 256, 0, st>>>(N, z, d);
      IBEM_LAUNCH_CHECK("gmres update");
    }
    return s;
  }
};

}  // namespace

ibem_status mf_solve(const MfBatch& b, const double* bvec, double* x, const MfPrecond& P, const ibem_mf_options& o,
                     ibem_mf_report* rep, cudaStream_t st) {
  const int S = b.nseg;
  const int64_t N = b.N;
  MfSolver g(b, st, o.restart, o.stepwise == 0);
  ibem_status s = g.alloc();
  double *xs = nullptr, *rs = nullptr, *y = nullptr, *bs = nullptr, *bn2 = nullptr;
  if (!s) {
    cudaError_t e = alloc_async((void**)&xs, sizeof(double) * N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&rs, sizeof(double) * N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&y, sizeof(double) * N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&bs, sizeof(double) * N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&bn2, sizeof(double) * 2 * S, st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf solve workspace");
  }
  std::vector<double> hb(S), hr(S), htol(S);
  std::vector<int> hdone(S, 0), outer_of(S, 0);
  if (!s) {
    cudaMemsetAsync(xs, 0, sizeof(double) * N, st);
    ::ibem::count_launch(), k_mul<<<nblk(N), 256, 0, st>>>(N, b.dr, bvec, bs);  // bs = Dr b
    cudaMemcpyAsync(rs, bs, sizeof(double) * N, cudaMemcpyDeviceToDevice, st);  // rs = bs (x = 0)
    s = g.seg_norm2(rs, bn2);
    if (!s) {
      cudaMemcpyAsync(hb.data(), bn2, sizeof(double) * S, cudaMemcpyDeviceToHost, st);
      const cudaError_t e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) s = cuda_fail(e, "mf solve: rhs norms");
    }
  }
  // rs holds the residual of the current iterate; `exact` says whether it came from the
  // FP64 product (or x = 0).  A double-float residual drives the next correction; once it
  // shows every realisation within tol, the FP64 residual of the same iterate decides.
  bool exact = true;
  auto read_rel = [&]() -> ibem_status {
    ibem_status r = g.seg_norm2(rs, bn2 + S);
    if (r) return r;
    cudaMemcpyAsync(hr.data(), bn2 + S, sizeof(double) * S, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "mf solve: residual norms");
    return IBEM_OK;
  };
  auto fp64_residual = [&]() -> ibem_status {
    ibem_status r = mf_apply_f64(b, xs, y, st);   // As xs in FP64
    if (r) return r;
    ::ibem::count_launch(), k_sub64<<<nblk(N), 256, 0, st>>>(N, bs, y, rs);   // rs = bs - As xs
    IBEM_LAUNCH_CHECK("mf residual");
    exact = true;
    return read_rel();
  };
  int outer = 0;
  hr = hb;
  while (!s) {
    bool all = true;
    for (int i = 0; i < S; ++i) all = all && (hb[i] > 0 ? std::sqrt(hr[i] / hb[i]) : 0.0) <= o.tol;
    if (!exact && (all || outer >= o.max_outer)) {
      if ((s = fp64_residual())) break;
      all = true;
      for (int i = 0; i < S; ++i) all = all && (hb[i] > 0 ? std::sqrt(hr[i] / hb[i]) : 0.0) <= o.tol;
    }
    for (int i = 0; i < S; ++i) {
      const double rel = hb[i] > 0 ? std::sqrt(hr[i] / hb[i]) : 0.0;
      rep[i].rel_residual = rel;
      hdone[i] = rel <= o.tol ? 1 : 0;
    }
    if (all || outer >= o.max_outer) break;
    for (int i = 0; i < S; ++i)
      if (!hdone[i]) outer_of[i] = outer + 1;
    cudaMemcpyAsync(g.done, hdone.data(), sizeof(int) * S, cudaMemcpyHostToDevice, st);
    // reduction asked of each realisation's GMRES: inner_tol, or deeper when that is what
    // brings the next residual within tol (never below the ~1e-6 the FP32 products allow)
    for (int i = 0; i < S; ++i)
      htol[i] = std::max(1e-6, std::min(o.inner_tol, rep[i].rel_residual > 0 ? 0.1 * o.tol / rep[i].rel_residual : o.inner_tol));
    cudaMemcpyAsync(g.tolv, htol.data(), sizeof(double) * S, cudaMemcpyHostToDevice, st);
    // FP32 correction of the scaled system, then the double-float residual of the new iterate
    ::ibem::count_launch(), k_to_f32<<<nblk(N), 256, 0, st>>>(N, rs, g.rin);
    if ((s = g.gmres(P, o.max_cycles))) break;
    ::ibem::count_launch(), k_acc_f32<<<nblk(N), 256, 0, st>>>(N, g.d, xs);
    ++outer;
    // expected residual of every realisation still running: its previous residual times the
    // reduction its GMRES reached (Arnoldi estimate over the first beta), but no better than
    // the FP32 products allow (~1e-6 of the correction).  When all are expected to meet tol,
    // go straight to the deciding FP64 residual; otherwise a double-float one.
    std::vector<double> est(S), thr(S);
    cudaMemcpyAsync(est.data(), g.K.est, sizeof(double) * S, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(thr.data(), g.K.thr, sizeof(double) * S, cudaMemcpyDeviceToHost, st);
    {
      const cudaError_t e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) { s = cuda_fail(e, "mf solve: GMRES estimates"); break; }
    }
    bool expect = true;
    for (int i = 0; i < S; ++i) {
      if (hdone[i]) continue;
      const double beta0 = thr[i] > 0 ? thr[i] / htol[i] : 0.0;
      const double red = beta0 > 0 ? std::max(est[i] / beta0, 1e-6) : 1.0;
      expect = expect && rep[i].rel_residual * red <= 0.5 * o.tol;
    }
    if (expect) {
      if ((s = fp64_residual())) break;
      continue;
    }
    if ((s = mf_apply_df(b, xs, y, st, g.done, 0))) break;   // done realisations keep their residual
    ::ibem::count_launch(), k_sub64_masked<<<nblk(N), 256, 0, st>>>(b.nu, N, b.seg_of, g.done, bs, y, rs);
    IBEM_LAUNCH_CHECK("mf refinement");
    exact = false;
    if ((s = read_rel())) break;
  }
  if (!s) {
    ::ibem::count_launch(), k_mul<<<nblk(N), 256, 0, st>>>(N, b.dc, xs, x);
    std::vector<int> steps(S);
    cudaMemcpyAsync(steps.data(), g.K.nsteps, sizeof(int) * S, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf solve: finish");
    for (int i = 0; i < S; ++i) {
      rep[i].outer = outer_of[i];
      rep[i].inner = steps[i];
    }
    for (int i = 0; i < S && !s; ++i)
      if (!(rep[i].rel_residual <= o.tol)) s = fail(IBEM_ERR_NOCONV, "mf solve: a realisation missed the tolerance");
  }
  free_async(xs, st);
  free_async(rs, st);
  free_async(y, st);
  free_async(bs, st);
  free_async(bn2, st);
  return s;
}

}  // namespace ibem

// ------------------------------------------------------------------ C ABI
using namespace ibem;

extern "C" ibem_status ibem_e3d_mf_matvec(const ibem_e3d_batch* batch, int precision, const double* x_dev,
                                          double* y_dev, void* stream) {
  return ibem_e3d_mf_matvec_layout(batch, 24, precision, x_dev, y_dev, stream);
}

extern "C" ibem_status ibem_e3d_mf_matvec_layout(const ibem_e3d_batch* batch, int layout, int precision,
                                                 const double* x_dev, double* y_dev, void* stream) {
  if (batch && batch->axes_dev) return fail(IBEM_ERR_ARG, "matrix-free products and the learned preconditioner take spheres; solve ellipsoid batches with ibem_e3d_batch_dense_solve");
  if (!batch || !x_dev || !y_dev || (precision != 32 && precision != 48 && precision != 64 && precision != 65))
    return fail(IBEM_ERR_ARG, "mf_matvec: bad arguments");
  if (layout != 24 && layout != 60) return fail(IBEM_ERR_ARG, "mf_matvec: layout 24 or 60");
  cudaStream_t st = as_stream(stream);
  MfBatch b;
  ibem_status s = mf_batch_init(b, *batch, st, layout);
  if (!s) {
    if (precision != 32) {
      double *xs = nullptr, *ys = nullptr;
      cudaError_t e = alloc_async((void**)&xs, sizeof(double) * b.N, st);
      if (e == cudaSuccess) e = alloc_async((void**)&ys, sizeof(double) * b.N, st);
      if (e != cudaSuccess) s = cuda_fail(e, "mf_matvec workspace");
      if (!s) {
        ::ibem::count_launch(), k_div64<<<nblk(b.N), 256, 0, st>>>(b.N, x_dev, b.dc, xs);  // xs = x / Dc
        s = precision == 64 ? mf_apply_f64(b, xs, ys, st)
                            : precision == 65 ? mf_apply_f64_all(b, xs, ys, st) : mf_apply_df(b, xs, ys, st);
        if (!s) ::ibem::count_launch(), k_div64<<<nblk(b.N), 256, 0, st>>>(b.N, ys, b.dr, y_dev);  // y = ys / Dr
      }
      if (!s) {
        const cudaError_t e2 = cudaStreamSynchronize(st);
        if (e2 != cudaSuccess) s = cuda_fail(e2, "mf_matvec");
      }
      free_async(xs, st);
      free_async(ys, st);
    } else {
      float *xf = nullptr, *yf = nullptr;
      s = mf_tune(b, st);   // the tile shape the solver's GMRES uses
      cudaError_t e = s ? cudaSuccess : alloc_async((void**)&xf, sizeof(float) * b.N, st);
      if (e == cudaSuccess && !s) e = alloc_async((void**)&yf, sizeof(float) * b.N, st);
      if (e != cudaSuccess) s = cuda_fail(e, "mf_matvec workspace");
      if (!s) {
        ::ibem::count_launch(), k_div_to_f32<<<nblk(b.N), 256, 0, st>>>(b.N, x_dev, b.dc, xf);  // xs = x / Dc
        s = mf_apply_f32(b, xf, yf, st);
        if (!s) ::ibem::count_launch(), k_f32_div<<<nblk(b.N), 256, 0, st>>>(b.N, yf, b.dr, y_dev);  // y = ys / Dr
      }
      if (!s) {
        const cudaError_t e2 = cudaStreamSynchronize(st);
        if (e2 != cudaSuccess) s = cuda_fail(e2, "mf_matvec");
      }
      free_async(xf, st);
      free_async(yf, st);
    }
  }
  if (!s) {
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf_matvec");
  }
  mf_batch_free(b);
  return s;
}

extern "C" ibem_status ibem_e3d_mf_solve(const ibem_e3d_batch* batch, const double* b_dev, double* x_dev,
                                         ibem_precond pc, const float* gnn_params_dev, const ibem_mf_options* opt,
                                         ibem_mf_report* reports, void* stream) {
  return ibem_e3d_mf_solve_layout(batch, 24, b_dev, x_dev, pc, gnn_params_dev, opt, reports, stream);
}

extern "C" ibem_status ibem_e3d_mf_solve_layout(const ibem_e3d_batch* batch, int layout, const double* b_dev,
                                                double* x_dev, ibem_precond pc, const float* gnn_params_dev,
                                                const ibem_mf_options* opt, ibem_mf_report* reports, void* stream) {
  if (layout != 24 && layout != 60) return fail(IBEM_ERR_ARG, "mf_solve: layout 24 or 60");
  if (layout == 60 && pc != IBEM_PRECOND_BLOCK_JACOBI)
    return fail(IBEM_ERR_ARG, "mf_solve: layout 60 takes the block-Jacobi preconditioner");
  if (batch && batch->axes_dev) return fail(IBEM_ERR_ARG, "matrix-free products and the learned preconditioner take spheres; solve ellipsoid batches with ibem_e3d_batch_dense_solve");
  if (!batch || !b_dev || !x_dev || !reports) return fail(IBEM_ERR_ARG, "mf_solve: bad arguments");
  if (pc != IBEM_PRECOND_BLOCK_JACOBI && pc != IBEM_PRECOND_LEARNED && pc != IBEM_PRECOND_NEUMANN)
    return fail(IBEM_ERR_ARG, "mf_solve: preconditioner");
  if (pc == IBEM_PRECOND_LEARNED && !gnn_params_dev) return fail(IBEM_ERR_ARG, "mf_solve: learned form needs parameters");
  ibem_mf_options o{};
  if (opt) o = *opt;
  if (o.restart <= 0) o.restart = 50;
  if (o.max_cycles <= 0) o.max_cycles = 20;
  if (o.max_outer <= 0) o.max_outer = 8;
  if (o.tol <= 0) o.tol = 1e-10;
  if (o.inner_tol <= 0) o.inner_tol = 1e-5;
  if (o.restart > 200) return fail(IBEM_ERR_ARG, "mf_solve: restart > 200");
  cudaStream_t st = as_stream(stream);
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  for (auto& e : ev) IBEM_CUDA(cudaEventCreate(&e));
  IBEM_CUDA(cudaEventRecord(ev[0], st));
  MfBatch b;
  ibem_status s = mf_batch_init(b, *batch, st, layout);
  if (!s) s = mf_tune(b, st);
  MfPrecond P;
  if (!s) {
    // layout 24: one 24 x 24 block per particle (the learned and Neumann forms change them);
    // layout 60: one 60 x 60 block per realisation
    const size_t nblocks = layout == 60 ? (size_t)b.nseg : (size_t)b.num;
    const cudaError_t e = alloc_async((void**)&P.D, sizeof(float) * layout * layout * nblocks, st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf_solve: preconditioner blocks");
  }
  {
    ProfScope pp(PROF_PRECOND, st);
    if (!s) s = layout == 60 ? mf60_block_jacobi(b, P.D, st) : mf_block_jacobi(b, P.D, st);
    if (!s && pc != IBEM_PRECOND_BLOCK_JACOBI)
      s = mf_neighbour_precond(b, pc == IBEM_PRECOND_LEARNED ? gnn_params_dev : nullptr, P, st);
  }
  cudaEventRecord(ev[1], st);
  for (int i = 0; i < batch->nseg; ++i) reports[i] = ibem_mf_report{};
  if (!s) s = mf_solve(b, b_dev, x_dev, P, o, reports, st);
  cudaEventRecord(ev[2], st);
  float t_set = 0.f, t_sol = 0.f;
  if (cudaEventSynchronize(ev[2]) == cudaSuccess) {
    cudaEventElapsedTime(&t_set, ev[0], ev[1]);
    cudaEventElapsedTime(&t_sol, ev[1], ev[2]);
  }
  for (auto& e : ev) cudaEventDestroy(e);
  for (int i = 0; i < batch->nseg; ++i) {
    reports[i].t_setup_ms = t_set;
    reports[i].t_solve_ms = t_sol;
  }
  free_async(P.D, st);
  free_async(P.Q, st);
  free_async(P.nbr, st);
  mf_batch_free(b);
  return s;
}

extern "C" ibem_status ibem_e3d_batch_farfield_rhs_layout(const ibem_e3d_batch* batch, int layout,
                                                          const double* sig_inf, double* b_dev, void* stream) {
  const int nu = ibem_layout_size(layout);
  if (!batch || !batch->seg_begin || !batch->mats || !sig_inf || !b_dev || nu < 0)
    return fail(IBEM_ERR_ARG, "batch_farfield_rhs: bad arguments");
  for (int s = 0; s < batch->nseg; ++s) {
    const int p0 = batch->seg_begin[s], n = batch->seg_begin[s + 1] - p0;
    const ibem_status r = ibem_e3d_farfield_rhs(n, &batch->mats[s], layout, sig_inf, b_dev + (int64_t)nu * p0, stream);
    if (r) return r;
  }
  return IBEM_OK;
}

extern "C" ibem_status ibem_e3d_batch_farfield_rhs(const ibem_e3d_batch* batch, const double* sig_inf, double* b_dev,
                                                   void* stream) {
  return ibem_e3d_batch_farfield_rhs_layout(batch, 24, sig_inf, b_dev, stream);
}

extern "C" ibem_status ibem_e3d_batch_dense_solve(const ibem_e3d_batch* batch, int layout, ibem_solver_form form,
                                                  const double* b_dev, double* x_dev, double tol,
                                                  ibem_solve_report* reports, void* stream) {
  const int nu = ibem_layout_size(layout);
  if (!batch || !batch->seg_begin || !batch->mats || !batch->centers_dev || !batch->radius_dev || !b_dev || !x_dev ||
      nu < 0 || batch->nseg < 0 || batch->seg_begin[0] != 0)
    return fail(IBEM_ERR_ARG, "batch_dense_solve: bad arguments");
  int64_t nmax = 0;
  for (int s = 0; s < batch->nseg; ++s) {
    const int n = batch->seg_begin[s + 1] - batch->seg_begin[s];
    if (n < 0) return fail(IBEM_ERR_ARG, "batch_dense_solve: seg_begin must not decrease");
    nmax = std::max<int64_t>(nmax, (int64_t)nu * n);
  }
  if (form != IBEM_SOLVE_FP64 && form != IBEM_SOLVE_MIXED_IR && form != IBEM_SOLVE_GMRES_BJ)
    return fail(IBEM_ERR_ARG, "batch_dense_solve: unknown solver form");
  if (batch->axes_dev && (layout != 24 || !batch->quats_dev))
    return fail(IBEM_ERR_ARG, "batch_dense_solve: ellipsoids take layout 24 and need quaternions");
  cudaStream_t st = as_stream(stream);
  // Workers: each owns a stream, the largest realisation's N x N matrix and (block-Jacobi
  // form) its FP32 copy, and takes the next unsolved realisation until none is left.  The
  // block-Jacobi form runs several workers at once, so that one realisation's
  // latency-bound steps (host-driven GMRES, small kernels) overlap another's products; the
  // factorising forms run one worker (their panel kernel needs every SM to itself).  As many
  // workers as fit in a quarter of the free device memory (what the library keeps unused is
  // free to it), at most kDenseWorkers.
  constexpr int kDenseWorkers = 4;
  const size_t per_worker = sizeof(double) * nmax * nmax +
                            (form == IBEM_SOLVE_GMRES_BJ ? sizeof(float) * ((nmax + 3) / 4 * 4) * nmax : 0);
  int nwork = 1;
  if (form == IBEM_SOLVE_GMRES_BJ && per_worker > 0) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess)
      nwork = (int)std::max<size_t>(1, std::min<size_t>({(size_t)kDenseWorkers, (size_t)batch->nseg,
                                                         (free_b + pool_kept()) / 4 / per_worker}));
  }
  // b_dev is written on the caller's stream: let it land before the workers read it
  cudaError_t e0 = cudaStreamSynchronize(st);
  if (e0 != cudaSuccess) return cuda_fail(e0, "batch_dense_solve");
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int> next{0};
  std::atomic<bool> failed{false};
  std::mutex err_mu;
  ibem_status first = IBEM_OK;
  std::string first_msg;
  auto worker = [&](bool own_stream) {
    cudaSetDevice(dev);
    cudaStream_t ws = st;
    ibem_status s = IBEM_OK;
    if (own_stream) {
      const cudaError_t e = cudaStreamCreateWithFlags(&ws, cudaStreamNonBlocking);
      if (e != cudaSuccess) s = cuda_fail(e, "batch_dense_solve: stream");
    }
    double* A = nullptr;
    float* W = nullptr;
    if (!s && nmax) {
      cudaError_t e = alloc_async((void**)&A, sizeof(double) * nmax * nmax, ws);
      if (e == cudaSuccess && form == IBEM_SOLVE_GMRES_BJ)
        e = alloc_async((void**)&W, sizeof(float) * ((nmax + 3) / 4 * 4) * nmax, ws);
      if (e != cudaSuccess) s = cuda_fail(e, "batch_dense_solve: matrix");
    }
    while (!s && !failed.load()) {
      const int i = next.fetch_add(1);
      if (i >= batch->nseg) break;
      const int p0 = batch->seg_begin[i], n = batch->seg_begin[i + 1] - p0;
      const int64_t N = (int64_t)nu * n, off = (int64_t)nu * p0;
      ibem_solve_report rep{};
      if (n) {
        s = batch->axes_dev
                ? ibem_e3d_ell_pair_blocks(batch->centers_dev + 3 * (int64_t)p0, batch->axes_dev + 3 * (int64_t)p0,
                                           batch->quats_dev + 4 * (int64_t)p0, n, &batch->mats[i], A, N, 0, 0, ws)
                : ibem_e3d_pair_blocks(batch->centers_dev + 3 * (int64_t)p0, batch->radius_dev + p0, n,
                                       &batch->mats[i], layout, A, N, 0, 0, ws);
        if (!s) s = solve_dense(form, N, A, N, b_dev + off, x_dev + off, tol, &rep, ws, nu, W);
      }
      if (reports) reports[i] = rep;
    }
    free_async(A, ws);
    free_async(W, ws);
    cudaStreamSynchronize(ws);
    if (own_stream && ws) cudaStreamDestroy(ws);
    if (s) {
      failed.store(true);
      std::lock_guard<std::mutex> l(err_mu);
      if (!first) first = s, first_msg = ibem_last_error();
    }
  };
  if (nwork == 1) {
    worker(false);
  } else {
    std::vector<std::thread> pool;
    for (int t = 0; t < nwork; ++t) pool.emplace_back(worker, true);
    for (auto& t : pool) t.join();
  }
  return first ? fail(first, first_msg) : IBEM_OK;
}

extern "C" ibem_status ibem_e3d_effective_modulus(const ibem_e3d_batch* batch, const double* x_dev,
                                                  const double* volume, const double* sig_inf, double* mean_strain,
                                                  double* e_eff, void* stream) {
  return ibem_e3d_effective_modulus_layout(batch, 24, x_dev, volume, sig_inf, mean_strain, e_eff, stream);
}

extern "C" ibem_status ibem_e3d_effective_modulus_layout(const ibem_e3d_batch* batch, int layout, const double* x_dev,
                                                         const double* volume, const double* sig_inf,
                                                         double* mean_strain, double* e_eff, void* stream) {
  const int nu = ibem_layout_size(layout);
  if (!batch || !x_dev || !volume || !sig_inf || !e_eff || nu < 0)
    return fail(IBEM_ERR_ARG, "effective_modulus: bad arguments");
  if (batch->axes_dev && layout != 24) return fail(IBEM_ERR_ARG, "effective_modulus: ellipsoids take layout 24");
  cudaStream_t st = as_stream(stream);
  MfBatch b;
  ibem_status s = mf_batch_init(b, *batch, st);
  double* acc = nullptr;
  const int S = batch->nseg;
  std::vector<double> h(6 * (size_t)S);
  if (!s) {
    cudaError_t e = alloc_async((void**)&acc, sizeof(double) * 6 * S, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(acc, 0, sizeof(double) * 6 * S, st);
    if (e != cudaSuccess) s = cuda_fail(e, "effective_modulus");
  }
  if (!s) {
    ::ibem::count_launch(), k_vol_eigen<<<nblk(b.num), 256, 0, st>>>(b.num, nu, b.seg_of, b.rad, b.axes, x_dev, acc);
    cudaMemcpyAsync(h.data(), acc, sizeof(double) * 6 * S, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "effective_modulus");
  }
  if (!s) {
    for (int i = 0; i < S; ++i) {
      const ibem_material& m = batch->mats[i];
      const double tr = sig_inf[0] + sig_inf[3] + sig_inf[5];
      double eps[6];
      for (int r = 0; r < 6; ++r) {
        const bool diag = (r == 0 || r == 3 || r == 5);
        eps[r] = ((1 + m.nu0) * sig_inf[r] - (diag ? m.nu0 * tr : 0.0)) / m.E0 + h[6 * i + r] / volume[i];
      }
      if (mean_strain)
        for (int r = 0; r < 6; ++r) mean_strain[6 * i + r] = eps[r];
      e_eff[i] = eps[5] != 0 ? sig_inf[5] / eps[5] : 0.0;
    }
  }
  free_async(acc, st);
  mf_batch_free(b);
  return s;
}

// Host buffers in, host buffers out, copied straight between the caller's (pageable) arrays
// and the device: on a Grace host the GPU reads and writes pageable memory at full link speed
// (12.6 MB of stresses: 0.08 ms, the same as from pinned memory), and a pinned staging copy
// would cost a host memcpy (0.74 ms for the same stresses).  The points, needed only by the
// stress sums, go on a second stream ahead of the solve.  Output arrays whose pages are not
// yet mapped (a fresh allocation) would be faulted in by the device copy at a far lower rate:
// a helper thread writes one byte of every page while the device solves.
extern "C" ibem_status ibem_e3d_run_host_mf(const ibem_material* mat, int num, const double* centers,
                                            const double* radius, int nump, const double* points,
                                            const double* sig_inf, ibem_precond pc, const float* gnn_params,
                                            const ibem_mf_options* opt, double* X, double* stress,
                                            ibem_mf_report* report) {
  if (!mat || num <= 0 || !centers || !radius || nump < 0 || (nump > 0 && !points) || !sig_inf || !X ||
      (nump > 0 && !stress) || !report)
    return fail(IBEM_ERR_ARG, "run_host_mf: bad arguments");
  if (pc == IBEM_PRECOND_LEARNED && !gnn_params) return fail(IBEM_ERR_ARG, "run_host_mf: learned form needs parameters");
  const int64_t N = (int64_t)kMfNu * num;
  const int64_t np = gnn_param_count();
  const size_t pts_bytes = sizeof(double) * 3 * (size_t)nump, str_bytes = sizeof(double) * 6 * (size_t)nump;
  double *cen = nullptr, *rad = nullptr, *pts = nullptr, *b = nullptr, *x = nullptr, *S = nullptr;
  float* prm = nullptr;
  cudaStream_t st = nullptr, st2 = nullptr;
  cudaEvent_t ev = nullptr;
  ibem_status s = IBEM_OK;
  {
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st2, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = alloc_async((void**)&cen, sizeof(double) * 3 * num, st);
    if (e == cudaSuccess) e = alloc_async((void**)&rad, sizeof(double) * num, st);
    if (e == cudaSuccess) e = alloc_async((void**)&pts, sizeof(double) * 3 * std::max(nump, 1), st);
    if (e == cudaSuccess) e = alloc_async((void**)&b, sizeof(double) * N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&x, sizeof(double) * N, st);
    if (e == cudaSuccess) e = alloc_async((void**)&S, sizeof(double) * 6 * std::max(nump, 1), st);
    if (e == cudaSuccess && gnn_params) e = alloc_async((void**)&prm, sizeof(float) * np, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(cen, centers, sizeof(double) * 3 * num, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(rad, radius, sizeof(double) * num, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && gnn_params) e = cudaMemcpyAsync(prm, gnn_params, sizeof(float) * np, cudaMemcpyHostToDevice, st);
    // pts is allocated on st: st2 waits for that before it copies into it
    if (e == cudaSuccess) e = cudaEventRecord(ev, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st2, ev, 0);
    if (e == cudaSuccess && nump > 0) e = cudaMemcpyAsync(pts, points, pts_bytes, cudaMemcpyHostToDevice, st2);
    if (e == cudaSuccess) e = cudaEventRecord(ev, st2);
    if (e != cudaSuccess) s = cuda_fail(e, "run_host_mf: set-up");
  }
  std::thread toucher;
  if (!s)
    toucher = std::thread([=]() {
      const size_t step = 4096;   // no larger than any page size
      auto touch = [step](double* p, size_t bytes) {
        for (size_t o = 0; o < bytes; o += step) reinterpret_cast<volatile char*>(p)[o] = 0;
      };
      touch(X, sizeof(double) * (size_t)N);
      if (nump > 0) touch(stress, str_bytes);
    });
  const int seg[2] = {0, num};
  const ibem_e3d_batch bt{1, seg, cen, rad, mat};
  if (!s) s = ibem_e3d_farfield_rhs(num, mat, kMfNu, sig_inf, b, st);
  if (!s) s = ibem_e3d_mf_solve(&bt, b, x, pc, prm, opt, report, st);
  if (!s && nump > 0) {
    const cudaError_t e = cudaStreamWaitEvent(st, ev, 0);
    if (e != cudaSuccess) s = cuda_fail(e, "run_host_mf: points");
  }
  if (!s && nump > 0)
    s = ibem_e3d_field_form(IBEM_SOLVE_MIXED_IR, pts, nump, cen, rad, num, mat, kMfNu, x, nullptr, 0, nullptr, 0,
                            nullptr, nullptr, sig_inf, S, st);
  if (toucher.joinable()) toucher.join();
  if (!s) {
    cudaError_t e = cudaMemcpyAsync(X, x, sizeof(double) * N, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && nump > 0) e = cudaMemcpyAsync(stress, S, str_bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "run_host_mf: results");
  }
  if (st2) cudaStreamSynchronize(st2);
  if (st) cudaStreamSynchronize(st);
  free_async(cen, st);
  free_async(rad, st);
  free_async(pts, st);
  free_async(b, st);
  free_async(x, st);
  free_async(S, st);
  free_async(prm, st);
  if (ev) cudaEventDestroy(ev);
  if (st2) cudaStreamDestroy(st2);
  if (st) cudaStreamDestroy(st);
  return s;
}

extern "C" ibem_status ibem_e3d_mf_tuning(const ibem_e3d_batch* batch, int* slices_fp32, int* slices_wide,
                                          void* stream) {
  if (batch && batch->axes_dev) return fail(IBEM_ERR_ARG, "matrix-free products and the learned preconditioner take spheres; solve ellipsoid batches with ibem_e3d_batch_dense_solve");
  if (!batch || !slices_fp32 || !slices_wide) return fail(IBEM_ERR_ARG, "mf_tuning: bad arguments");
  cudaStream_t st = as_stream(stream);
  MfBatch b;
  ibem_status s = mf_batch_init(b, *batch, st);
  if (!s) s = mf_tune(b, st);
  if (!s) {
    *slices_fp32 = b.split.slices;
    *slices_wide = b.split_wide.slices;
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf_tuning");
  }
  mf_batch_free(b);
  return s;
}

extern "C" ibem_status ibem_e3d_mf_pieces(const ibem_e3d_batch* batch, int* pieces_fp32, int* pieces_wide,
                                         void* stream) {
  if (batch && batch->axes_dev) return fail(IBEM_ERR_ARG, "matrix-free products and the learned preconditioner take spheres; solve ellipsoid batches with ibem_e3d_batch_dense_solve");
  if (!batch || !pieces_fp32 || !pieces_wide) return fail(IBEM_ERR_ARG, "mf_pieces: bad arguments");
  cudaStream_t st = as_stream(stream);
  MfBatch b;
  ibem_status s = mf_batch_init(b, *batch, st);
  if (!s) s = mf_tune(b, st);
  if (!s) {
    *pieces_fp32 = b.split.pieces;
    *pieces_wide = b.split_wide.pieces;
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf_pieces");
  }
  mf_batch_free(b);
  return s;
}

extern "C" ibem_status ibem_e3d_mf_tile_shape(const ibem_e3d_batch* batch, int* targets_per_cta, int* persistent,
                                              int* slices, void* stream) {
  if (batch && batch->axes_dev) return fail(IBEM_ERR_ARG, "matrix-free products and the learned preconditioner take spheres; solve ellipsoid batches with ibem_e3d_batch_dense_solve");
  if (!batch || !targets_per_cta || !persistent || !slices) return fail(IBEM_ERR_ARG, "mf_tile_shape: bad arguments");
  cudaStream_t st = as_stream(stream);
  MfBatch b;
  ibem_status s = mf_batch_init(b, *batch, st);
  if (!s) s = mf_tune(b, st);
  if (!s) {
    *targets_per_cta = 64 << b.tshape;
    *persistent = b.persist;
    *slices = b.split.slices;
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "mf_tile_shape");
  }
  mf_batch_free(b);
  return s;
}
