// Boundary-element kernels of the 3D elastic iBEM path (FP64).
//
//  bem_hg        classical Q4 BEM H and G with 8x8 Gauss-Legendre quadrature, the singular
//                element split into two degenerate triangles, and the rigid-body diagonal
//                (BEMBuilderElastic3D.cpp:1169-1509, BEMElasticHelper3D.cpp:29-321).
//                One thread per (collocation node, element), a warp per singular pair; the
//                element's 12 traction columns are summed per node in a fixed order (the
//                reference accumulates them under `omp critical`, :1432-1454).
//  bem_to_incl   stress and its 1st/2nd gradient at particle centres from unit boundary
//                displacements/tractions (addFluxEquivalent{,FirstOrder,SecondOrder}BEM,
//                :1511-1867), from moments of the derivatives of R over each element.
//  bem_post      boundary part of the stress at sample points (post_stress_BEM,
//                postProcessorElastic3D.cpp:224-365), contracted with U and T at every
//                Gauss point: a per-call quadrature table (point, normal, weight x Jacobian,
//                interpolated U and T per Gauss point) staged through shared memory, one
//                thread per sample point.
#include <algorithm>
#include <cuda_runtime.h>

#include "bem_contract.cuh"
#include "bem_moments.cuh"
#include "ibem_internal.h"
#include "prof.h"

namespace {

__constant__ double kGP[8] = {0.960289856497536,  -0.960289856497536, 0.796666477413627,
                              -0.796666477413627, 0.525532409916329,  -0.525532409916329,
                              0.183434642495650,  -0.183434642495650};
__constant__ double kGW[8] = {0.101228536290376, 0.101228536290376, 0.222381034453374,
                              0.222381034453374, 0.313706645877887, 0.313706645877887,
                              0.362683783378362, 0.362683783378362};

struct Elem {
  double c[12];  // 4 corners x 3
};

// Corner coordinates of element e; false (nothing read) if a node number is outside
// 1..NN, so a bad connectivity table can never address outside the node array.
__device__ __forceinline__ bool load_elem(const double* __restrict__ nodes, int NN, const int* __restrict__ conn,
                                          int e, Elem& el, int* sc) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sc[j] = conn[4 * e + j];
    if (sc[j] < 1 || sc[j] > NN) return false;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) el.c[3 * j + k] = nodes[3 * (sc[j] - 1) + k];
  return true;
}

// Serendip_func, Normal_Jac, Cartesian (BEMElasticHelper3D.cpp:199-280)
__device__ __forceinline__ void q4_point(const double* c, double xi, double et, double* N,
                                         double* gc, double* nv, double& jac) {
  N[0] = 0.25 * (1 - xi) * (1 - et);
  N[1] = 0.25 * (1 + xi) * (1 - et);
  N[2] = 0.25 * (1 + xi) * (1 + et);
  N[3] = 0.25 * (1 - xi) * (1 + et);
  const double dxi[4] = {-0.25 * (1 - et), 0.25 * (1 - et), 0.25 * (1 + et), -0.25 * (1 + et)};
  const double det[4] = {-0.25 * (1 - xi), -0.25 * (1 + xi), 0.25 * (1 + xi), 0.25 * (1 - xi)};
  double vx[3], ve[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    vx[i] = dxi[0] * c[i] + dxi[1] * c[3 + i] + dxi[2] * c[6 + i] + dxi[3] * c[9 + i];
    ve[i] = det[0] * c[i] + det[1] * c[3 + i] + det[2] * c[6 + i] + det[3] * c[9 + i];
    gc[i] = N[0] * c[i] + N[1] * c[3 + i] + N[2] * c[6 + i] + N[3] * c[9 + i];
  }
  nv[0] = vx[1] * ve[2] - ve[1] * vx[2];
  nv[1] = vx[2] * ve[0] - vx[0] * ve[2];
  nv[2] = vx[0] * ve[1] - vx[1] * ve[0];
  jac = sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
  nv[0] /= jac;
  nv[1] /= jac;
  nv[2] /= jac;
}

// Trans_Tri + Triangle_Coord (BEMElasticHelper3D.cpp:29-191): Gauss point (xb, eb) of the
// square mapped onto triangle `ntr` of the split at corner l_pi; jb its Jacobian.
__device__ __forceinline__ void tri_map(int ntr, int l_pi, double xb, double eb, double& xi,
                                        double& et, double& jb) {
  // corner/mid-side indices of the two triangles for each singular corner
  const int tab[2][4][3] = {{{1, 2, 0}, {2, 3, 1}, {0, 1, 2}, {0, 1, 3}},
                            {{2, 3, 0}, {3, 0, 1}, {3, 0, 2}, {1, 2, 3}}};
  const double xs[4] = {-1, 1, 1, -1};
  const double es[4] = {-1, -1, 1, 1};
  double cx[3], ce[3];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    cx[n] = xs[tab[ntr][l_pi][n]];
    ce[n] = es[tab[ntr][l_pi][n]];
  }
  const double Nb[3] = {0.25 * (1 + xb) * (1 - eb), 0.25 * (1 + xb) * (1 + eb), 0.5 * (1 - xb)};
  const double dNx[3] = {0.25 * (1 - eb), 0.25 * (1 + eb), -0.5};
  const double dNe[3] = {-0.25 * (1 + xb), 0.25 * (1 + xb), 0.0};
  xi = Nb[0] * cx[0] + Nb[1] * cx[1] + Nb[2] * cx[2];
  et = Nb[0] * ce[0] + Nb[1] * ce[1] + Nb[2] * ce[2];
  const double J00 = dNx[0] * cx[0] + dNx[1] * cx[1] + dNx[2] * cx[2];
  const double J01 = dNx[0] * ce[0] + dNx[1] * ce[1] + dNx[2] * ce[2];
  const double J10 = dNe[0] * cx[0] + dNe[1] * cx[1] + dNe[2] * cx[2];
  const double J11 = dNe[0] * ce[0] + dNe[1] * ce[1] + dNe[2] * ce[2];
  jb = J00 * J11 - J01 * J10;
}

struct KelvinC {
  double cu, c1, ct, c3;  // UK: c/(r) (c1 + r_i r_j);  TK: c2 / r^2, c3 = 1 - 2 nu
};

// Integ3 for one (collocation node, element): dU, dT (3 x 12), BEMBuilderElastic3D.cpp:1169-1353
// The traction part of this element is written to TG, laid out like G (column 12e + 3a + j,
// row 3i + ii; zero for the singular corner); node_gather then sums the columns of the
// elements that share a node in a fixed order, so H is the same bit for bit on every run.

// UK / TK (BEMElasticHelper3D.cpp:269-321) at offset x from the collocation node, without the
// quadrature weight: U symmetric (xx xy xz yy yz zz), T row-major 3 x 3
__device__ __forceinline__ void kelvin_ut(double x0, double x1, double x2, const double* nv, const KelvinC& kc,
                                          double (&U)[6], double (&T)[9]) {
  const double ir = ibem::rsqrt_h3(x0 * x0 + x1 * x1 + x2 * x2);
  const double dr[3] = {x0 * ir, x1 * ir, x2 * ir};
  const double conr = kc.cu * ir, c0 = conr * kc.c1;
  const double cth = nv[0] * dr[0] + nv[1] * dr[1] + nv[2] * dr[2];
  const double cr = kc.ct * (ir * ir), c3 = cr * kc.c3, ct3 = -3.0 * cr * cth;
  int q = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j, ++q) {
      const double dd = dr[i] * dr[j];
      U[q] = i == j ? conr * dd + c0 : conr * dd;
      if (i == j) T[3 * i + i] = ct3 * dd - c3 * cth;
      else {
        const double as = c3 * (nv[j] * dr[i] - nv[i] * dr[j]);
        T[3 * i + j] = ct3 * dd + as;
        T[3 * j + i] = ct3 * dd - as;
      }
    }
}

// Pairs whose node is not a corner of the element: one thread per node, 128 nodes per CTA and
// one element, whose 64 Gauss points (position, normal, shape functions x weight x Jacobian:
// the part that does not depend on the node, with its square root and divisions) are formed
// once per CTA in shared memory.  U is symmetric, so 15 sums of four shape functions are kept
// instead of 72 entries formed one by one.  Bound by the FP64 pipe, about 135 operations per
// (node, Gauss point); 600 elements, 602 nodes: 18.7 -> 5.1 ms, the singular pairs included.
__global__ void __launch_bounds__(128) bem_hg_kernel(const double* __restrict__ nodes, int NN,
                                                     const int* __restrict__ conn, KelvinC kc,
                                                     double* __restrict__ TG, int64_t ldt,
                                                     double* __restrict__ G, int64_t ldg) {
  __shared__ double sg[64][10];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int e = blockIdx.y;
  Elem el;
  int sc[4];
  if (!load_elem(nodes, NN, conn, e, el, sc)) return;   // the same for the whole CTA
  if (threadIdx.x < 64) {
    const int mq = threadIdx.x / 8, kq = threadIdx.x % 8;
    double N[4], gc[3], nv[3], jac;
    q4_point(el.c, kGP[mq], kGP[kq], N, gc, nv, jac);
    const double wj = kGW[mq] * kGW[kq] * jac;
    double* g = sg[threadIdx.x];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      g[d] = gc[d];
      g[3 + d] = nv[d];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) g[6 + a] = N[a] * wj;
  }
  __syncthreads();
  if (i >= NN) return;
#pragma unroll
  for (int n = 0; n < 4; ++n)
    if (sc[n] == i + 1) return;   // bem_hg_singular
  const double p0 = nodes[3 * i], p1 = nodes[3 * i + 1], p2 = nodes[3 * i + 2];
  double aU[6][4], aT[9][4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int q = 0; q < 6; ++q) aU[q][n] = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) aT[q][n] = 0.0;
  }
#pragma unroll 1
  for (int q = 0; q < 64; ++q) {
    const double* g = sg[q];
    double U[6], T[9];
    kelvin_ut(g[0] - p0, g[1] - p1, g[2] - p2, g + 3, kc, U, T);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const double w = g[6 + n];
#pragma unroll
      for (int t = 0; t < 6; ++t) aU[t][n] += w * U[t];
#pragma unroll
      for (int t = 0; t < 9; ++t) aT[t][n] += w * T[t];
    }
  }
  const int sym[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
  for (int ii = 0; ii < 3; ++ii)
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      G[(12 * (int64_t)e + k) * ldg + 3 * i + ii] = aU[sym[3 * ii + k % 3]][k / 3];
      TG[(12 * (int64_t)e + k) * ldt + 3 * i + ii] = aT[3 * ii + k % 3][k / 3];
    }
}

// Pairs whose node is a corner of the element: a warp per (element, corner), two triangles of 64
// Gauss points, four points per lane, the 60 sums added over the warp by a butterfly (the same
// order on every run).  An element that names a node twice keeps the last of its corners, as
// the first form of this loop did.
__global__ void __launch_bounds__(128) bem_hg_singular(const double* __restrict__ nodes, int NN,
                                                       const int* __restrict__ conn, int NE, KelvinC kc,
                                                       double* __restrict__ TG, int64_t ldt,
                                                       double* __restrict__ G, int64_t ldg) {
  const int id = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (id >= 4 * NE) return;
  const int e = id / 4, l_pi = id % 4;
  Elem el;
  int sc[4];
  if (!load_elem(nodes, NN, conn, e, el, sc)) return;
  for (int n = l_pi + 1; n < 4; ++n)
    if (sc[n] == sc[l_pi]) return;
  const int i = sc[l_pi] - 1;
  double aU[6][4], aT[9][4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int q = 0; q < 6; ++q) aU[q][n] = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) aT[q][n] = 0.0;
  }
  for (int g = lane; g < 128; g += 32) {
    const int mq = (g & 63) / 8, kq = g % 8;
    double xi, et, jb;
    tri_map(g / 64, l_pi, kGP[mq], kGP[kq], xi, et, jb);
    double N[4], gc[3], nv[3], jac;
    q4_point(el.c, xi, et, N, gc, nv, jac);
    const double wj = jac * jb * (kGW[mq] * kGW[kq]);
    double U[6], T[9];
    kelvin_ut(gc[0] - el.c[3 * l_pi], gc[1] - el.c[3 * l_pi + 1], gc[2] - el.c[3 * l_pi + 2], nv, kc, U, T);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const double w = N[n] * wj;
#pragma unroll
      for (int t = 0; t < 6; ++t) aU[t][n] += w * U[t];
      if (n != l_pi) {
#pragma unroll
        for (int t = 0; t < 9; ++t) aT[t][n] += w * T[t];
      }
    }
  }
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int t = 0; t < 6; ++t) aU[t][n] += __shfl_xor_sync(0xffffffffu, aU[t][n], off);
#pragma unroll
      for (int t = 0; t < 9; ++t) aT[t][n] += __shfl_xor_sync(0xffffffffu, aT[t][n], off);
    }
  }
  if (lane != 0) return;
  const int sym[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
  for (int ii = 0; ii < 3; ++ii)
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      G[(12 * (int64_t)e + k) * ldg + 3 * i + ii] = aU[sym[3 * ii + k % 3]][k / 3];
      TG[(12 * (int64_t)e + k) * ldt + 3 * i + ii] = k / 3 != l_pi ? aT[3 * ii + k % 3][k / 3] : 0.0;
    }
}

// ---- node incidence: the (element, corner) slots of every node, in increasing order ----
// inc_start[c] .. inc_start[c + 1] - 1 index inc_slot, whose entries are 4e + a for the
// corners a of elements e at node c.  Built with integer atomics, then each node's list is
// sorted, so the order (and every sum over it) does not depend on scheduling.
__global__ void k_inc_count(const int* __restrict__ conn, int NE, int NN, int* __restrict__ cnt) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= 4 * NE) return;
  const int c = conn[id] - 1;
  if (c >= 0 && c < NN) atomicAdd(cnt + c, 1);
}

// exclusive prefix sum of n counts into start[0..n] (one block, sequential chunks)
__global__ void k_inc_scan(const int* __restrict__ cnt, int n, int* __restrict__ start) {
  __shared__ int sh[1024];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int i = base + threadIdx.x;
    const int v = i < n ? cnt[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
      const int t = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
      __syncthreads();
      sh[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < n) start[i] = carry + sh[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += sh[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) start[n] = carry;
}

__global__ void k_inc_fill(const int* __restrict__ conn, int NE, int NN, const int* __restrict__ start,
                           int* __restrict__ cursor, int* __restrict__ slot) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= 4 * NE) return;
  const int c = conn[id] - 1;
  if (c < 0 || c >= NN) return;
  slot[start[c] + atomicAdd(cursor + c, 1)] = id;
}

__global__ void k_inc_sort(int NN, const int* __restrict__ start, int* __restrict__ slot) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= NN) return;
  for (int i = start[c] + 1; i < start[c + 1]; ++i) {
    const int v = slot[i];
    int j = i - 1;
    while (j >= start[c] && slot[j] > v) { slot[j + 1] = slot[j]; --j; }
    slot[j + 1] = v;
  }
}

// H[(3c + d) ldh + r] (+)= sum over node c's slots 4e + a, in order, of S[(12e + 3a + d) lds + r]
// for rows r < nrows; the element columns of S are laid out like G.
__global__ void __launch_bounds__(256) k_node_gather(int64_t nrows, int NN, const int* __restrict__ start,
                                                     const int* __restrict__ slot, const double* __restrict__ S,
                                                     int64_t lds, double* __restrict__ H, int64_t ldh, int accumulate) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= nrows) return;
  for (int c = blockIdx.y; c < NN; c += gridDim.y) {
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
    for (int q = start[c]; q < start[c + 1]; ++q) {
      const int64_t col = 3 * (int64_t)slot[q];   // 12e + 3a
      acc0 += S[col * lds + r];
      acc1 += S[(col + 1) * lds + r];
      acc2 += S[(col + 2) * lds + r];
    }
    double* h = H + 3 * (int64_t)c * ldh + r;
    if (accumulate) {
      h[0] += acc0;
      h[ldh] += acc1;
      h[2 * ldh] += acc2;
    } else {
      h[0] = acc0;
      h[ldh] = acc1;
      h[2 * ldh] = acc2;
    }
  }
}

// Rigid-body diagonal (:1478-1501): H(r, 3i+l) = -sum_c H(r, c) over columns c with c%3 == l.
__global__ void bem_diag_kernel(int NN, double* __restrict__ H, int64_t ldh) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= 3 * NN) return;
  double s0 = 0, s1 = 0, s2 = 0;
  for (int c = 0; c < NN; ++c) {
    s0 += H[(3 * (int64_t)c) * ldh + r];
    s1 += H[(3 * (int64_t)c + 1) * ldh + r];
    s2 += H[(3 * (int64_t)c + 2) * ldh + r];
  }
  const int64_t i = r / 3;
  H[(3 * i) * ldh + r] = -s0;
  H[(3 * i + 1) * ldh + r] = -s1;
  H[(3 * i + 2) * ldh + r] = -s2;
}

// ---- boundary -> inclusion rows ----
// One CTA per element and group of particles, two particles at a time:
//  1. a thread per (particle, Gauss point): the derivatives of R of orders 3 .. 4 + MAXO;
//  2. their moments over the element (bem_moments.cuh), a thread per (derivative, column);
//  3. the rows of orders 0 .. MAXO from the moments, a thread per (row, dof, corner).
// Rows of the layout: order 0 -> t; order 1 -> 6 + 3t + w; order 2 -> 24 + 9t + 3w + z (layout
// 78, both orders of w and z) or 24 + 6t + pairidx(w <= z) (layout 60).
// The displacement part (the H rows) is written per element into UG, laid out like G;
// node_gather sums it per node in a fixed element order (no atomics on matrix entries).
// Bound by the FP64 pipe: about 2,200 operations per (particle, Gauss point) for all three
// orders (derivatives 700, moments 950, rows 500), 1,100 without order 2, where forming the
// stress kernels of one derivative tuple at a time took 15,000.  64 particles, 600 elements, 78
// unknowns: 106 -> 9.2 ms; 21 particles, 294 elements, 24 unknowns: 12.0 -> 0.76 ms.
constexpr int kInclK = 2;           // particles at a time
constexpr int kInclGroup = 8;       // particles per CTA
template <int MAXO>
struct InclShape {
  static constexpr int nd = MAXO == 2 ? 74 : 46;             // derivatives of orders 3 .. 4 + MAXO
  static constexpr int mid = MAXO == 2 ? 36 : 15;            // of orders 4 .. 3 + MAXO
  static constexpr int top = MAXO == 2 ? 28 : 21;            // of order 4 + MAXO
  static constexpr int tasks = 10 + 4 * mid + 3 * top;       // moments: (derivative, column)
  static constexpr int rows = MAXO == 2 ? 60 : 24;
  static constexpr size_t smem = sizeof(double) * (kInclK * nd * 65 + kInclK * nd * 16 + 64 * 16 + 64 * 3);
};
struct InclMom {
  const double* m;   // [derivative][column * 4 + corner], offset to the corner
  __device__ __forceinline__ double operator()(int c, int i) const { return m[16 * i + 4 * c]; }
};

template <int MAXO>
__global__ void __launch_bounds__(128) bem_incl_kernel(const double* __restrict__ nodes, int NN,
                                                       const int* __restrict__ conn, const double* __restrict__ cen,
                                                       int num, BemMat bm, int nu, double* __restrict__ UG, int64_t ldu,
                                                       double* __restrict__ G, int64_t ldg) {
  using S = InclShape<MAXO>;
  extern __shared__ __align__(16) double incl_smem[];
  double* sd = incl_smem;                          // [particle][derivative][65]: value at the Gauss points
  double* sm = sd + kInclK * S::nd * 65;           // [particle][derivative][16]: moments
  double* sw = sm + kInclK * S::nd * 16;           // [Gauss point][16]: N_j w J {1, n}
  double* sp = sw + 64 * 16;                       // [Gauss point][3]
  const int e = blockIdx.x;
  Elem el;
  int sc[4];
  if (!load_elem(nodes, NN, conn, e, el, sc)) return;   // the same for the whole CTA
  if (threadIdx.x < 64) {
    const int mq = threadIdx.x / 8, kq = threadIdx.x % 8;
    double N[4], gc[3], nv[3], jac;
    q4_point(el.c, kGP[mq], kGP[kq], N, gc, nv, jac);
    const double wj = kGW[mq] * kGW[kq] * jac;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double w = N[j] * wj;
      sw[16 * threadIdx.x + j] = w;
#pragma unroll
      for (int m = 0; m < 3; ++m) sw[16 * threadIdx.x + 4 + 4 * m + j] = w * nv[m];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) sp[3 * threadIdx.x + d] = gc[d];
  }
  __syncthreads();
  const int kb = blockIdx.y * kInclGroup, ke = min(num, kb + kInclGroup);
  for (int k0 = kb; k0 < ke; k0 += kInclK) {
    const int nk = min(kInclK, ke - k0);
    {
      const int kk = threadIdx.x / 64, g = threadIdx.x % 64;
      if (kk < nk) {
        const double* c = cen + 3 * (int64_t)(k0 + kk);
        const double x0 = sp[3 * g] - c[0], x1 = sp[3 * g + 1] - c[1], x2 = sp[3 * g + 2] - c[2];
        double* d = sd + kk * S::nd * 65 + g;
        ibem::bmo_derivatives<4 + MAXO>(x0, x1, x2, ibem::rsqrt_h3(x0 * x0 + x1 * x1 + x2 * x2),
                                        [&](int i, double v) { d[65 * i] = v; });
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nk * S::tasks; t += 128) {
      const int kk = t / S::tasks, i = t % S::tasks;
      int a, c;   // column 0 for orders 3 .. 3 + MAXO, the normal's for 4 .. 4 + MAXO
      if (i < 10) {
        a = i;
        c = 0;
      } else if (i < 10 + 4 * S::mid) {
        a = 10 + (i - 10) % S::mid;
        c = (i - 10) / S::mid;
      } else {
        a = 10 + S::mid + (i - 10 - 4 * S::mid) % S::top;
        c = 1 + (i - 10 - 4 * S::mid) / S::top;
      }
      const double* d = sd + (kk * S::nd + a) * 65;
      const double* w = sw + 4 * c;
      double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0;
#pragma unroll 8
      for (int g = 0; g < 64; ++g) {
        const double v = d[g];
        const double2 w01 = *reinterpret_cast<const double2*>(w + 16 * g), w23 = *reinterpret_cast<const double2*>(w + 16 * g + 2);
        m0 += v * w01.x;
        m1 += v * w01.y;
        m2 += v * w23.x;
        m3 += v * w23.y;
      }
      double* o = sm + (kk * S::nd + a) * 16 + 4 * c;
      o[0] = m0;
      o[1] = m1;
      o[2] = m2;
      o[3] = m3;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nk * S::rows * 12; t += 128) {
      const int r = t % S::rows, col = (t / S::rows) % 12, kk = t / (S::rows * 12), n = col % 3;
      int o, tt, w = 0, z = 0, row = r;
      if (r < 6) {
        o = 0;
        tt = r;
      } else if (r < 24) {
        o = 1;
        tt = (r - 6) / 3;
        w = (r - 6) % 3;
      } else {
        o = 2;
        tt = (r - 24) / 6;
        const int q = (r - 24) % 6;
        w = q < 3 ? 0 : (q < 5 ? 1 : 2);
        z = q < 3 ? q : (q < 5 ? q - 2 : 2);
        if (nu == 78) row = 24 + 9 * tt + 3 * w + z;
      }
      const int k = tt < 3 ? 0 : (tt < 5 ? 1 : 2), l = tt < 3 ? tt : (tt < 5 ? tt - 2 : 2);
      const ibem::BmoEntries<InclMom> en{InclMom{sm + kk * S::nd * 16 + col / 3}, bm.kA, bm.kB, bm.lam0, bm.mu0, bm.dlam,
                                         bm.dmu};
      const int cnt = o == 0 ? 0 : ibem::bmo_e(w) + (o == 2 ? ibem::bmo_e(z) : 0);
      double st, su;
      en.entry(k, l, o, cnt, n, st, su);
      const double fac = o == 2 ? 0.5 : 1.0;
      const int64_t at = (int64_t)nu * (k0 + kk), c = 12 * (int64_t)e + col;
      UG[c * ldu + at + row] = -fac * su;   // summed per node by node_gather
      G[c * ldg + at + row] = fac * st;
      if (nu == 78 && o == 2 && w != z) {
        const int64_t mirror = at + 24 + 9 * tt + 3 * z + w;
        UG[c * ldu + mirror] = -fac * su;
        G[c * ldg + mirror] = fac * st;
      }
    }
    __syncthreads();   // sd and sm are refilled
  }
}

// ---- boundary part of the stress at sample points ----
// Everything at a Gauss point that does not depend on the sample point -- its position, unit
// normal, weight x Jacobian, and U and T interpolated there -- is one record of the
// quadrature table, formed once per call (one thread per (element, Gauss point)); the
// per-point kernel then only evaluates the Kelvin stress kernels and contracts them.
constexpr int kPostQ = 64;        // 8 x 8 Gauss points per element
constexpr int kPostRec = 13;      // x y z, nx ny nz, w*J, u(3), t(3)
constexpr int kPostStage = 128;   // Gauss points per slice are a multiple of this

__global__ void bem_post_table(const double* __restrict__ nodes, int NN, const int* __restrict__ conn, int NE,
                               const double* __restrict__ U, const double* __restrict__ T,
                               double* __restrict__ tab) {
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (id >= (int64_t)NE * kPostQ) return;
  const int e = (int)(id / kPostQ), q = (int)(id % kPostQ), mq = q / 8, kq = q % 8;
  double c[12], u[12], t[12];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    int node = conn[4 * e + a] - 1;
    if (node < 0 || node >= NN) node = 0;  // out-of-range connectivity: never index outside
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      c[3 * a + d] = nodes[3 * node + d];
      u[3 * a + d] = U[3 * node + d];
    }
  }
#pragma unroll
  for (int k = 0; k < 12; ++k) t[k] = T[12 * (int64_t)e + k];
  double N[4], gc[3], nv[3], jac;
  q4_point(c, kGP[mq], kGP[kq], N, gc, nv, jac);
  double* r = tab + id * kPostRec;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r[d] = gc[d];
    r[3 + d] = nv[d];
    r[7 + d] = N[0] * u[d] + N[1] * u[3 + d] + N[2] * u[6 + d] + N[3] * u[9 + d];
    r[10 + d] = N[0] * t[d] + N[1] * t[3 + d] + N[2] * t[6 + d] + N[3] * t[9 + d];
  }
  r[6] = kGW[mq] * kGW[kq] * jac;
}

// Gauss points [q_begin, q_end) of slice blockIdx.y of gridDim.y (a multiple of kPostStage)
__device__ __forceinline__ void post_slice(int64_t nq, int64_t& qb, int64_t& qe) {
  const int64_t per = ((nq + gridDim.y - 1) / gridDim.y + kPostStage - 1) / kPostStage * kPostStage;
  qb = min(nq, (int64_t)blockIdx.y * per);
  qe = min(nq, qb + per);
}

// the sums' records of the Gauss points (one thread each)
__global__ void k_post_rec(const double* __restrict__ tab, int64_t nq, BemPostCoef cf, BemPostRec* __restrict__ out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < nq) out[q] = bem_post_rec(tab + q * kPostRec, cf);
}

// FP64 sums: one thread per sample point, the records of 64 Gauss points at a time in shared
// memory.  Bound by the FP64 pipe: 59 operations per (point, Gauss point).  600 elements, 32^3
// points: 238 -> 144 ms.
constexpr int kPostStageRec = 64;
__global__ void __launch_bounds__(128) bem_post_kernel(const double* __restrict__ pts, int nump,
                                                       const BemPostRec* __restrict__ rec, int64_t nq, BemPostCoef cf,
                                                       double* __restrict__ part) {
  static_assert(sizeof(BemPostRec) == 12 * sizeof(double2), "BemPostRec is copied as 12 double2");
  __shared__ __align__(16) BemPostRec sq[kPostStageRec];
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = s < nump;
  double P0 = 0, P1 = 0, P2 = 0;
  if (act) { P0 = pts[3 * (int64_t)s]; P1 = pts[3 * (int64_t)s + 1]; P2 = pts[3 * (int64_t)s + 2]; }
  double acc[6] = {0, 0, 0, 0, 0, 0};
  int64_t qb, qe;
  post_slice(nq, qb, qe);   // slice boundaries are multiples of kPostStage, hence of kPostStageRec
  for (int64_t q0 = qb; q0 < qe; q0 += kPostStageRec) {
    const int nqs = (int)min((int64_t)kPostStageRec, qe - q0);
    __syncthreads();
    {
      const double2* src = reinterpret_cast<const double2*>(rec + q0);
      double2* dst = reinterpret_cast<double2*>(sq);
      for (int i = threadIdx.x; i < nqs * 12; i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    if (!act) continue;
#pragma unroll 2
    for (int qq = 0; qq < nqs; ++qq) bem_post_add(P0, P1, P2, sq[qq], cf, acc);
  }
  if (act)
#pragma unroll
    for (int t = 0; t < 6; ++t) part[6 * ((int64_t)blockIdx.y * nump + s) + t] = bem_post_value(acc, t);
}

// stress = sum of the slices' partial sums, in slice order (the same result on every run)
__global__ void k_post_reduce(int nump, int nslice, const double* __restrict__ part, double* __restrict__ stress) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= 6 * (int64_t)nump) return;
  double v = 0.0;
  for (int k = 0; k < nslice; ++k) v += part[(int64_t)k * 6 * nump + i];
  stress[i] = v;
}

// double-float records of the Gauss points (one thread each)
__global__ void k_post_df_table(const double* __restrict__ tab, int64_t nq, BemPostCoef cf,
                                ibem::BemPostDF* __restrict__ out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < nq) out[q] = ibem::bem_post_df_record(tab + q * kPostRec, cf);
}

// the mixed form's boundary sums: double-float contraction (bem_contract.cuh), the records
// staged in shared memory 64 at a time, compensated sums per component
constexpr int kPostStageDF = 64;
__global__ void __launch_bounds__(128) bem_post_kernel_df(const double* __restrict__ pts, int nump,
                                                          const ibem::BemPostDF* __restrict__ tab, int64_t nq,
                                                          ibem::BemPostCoefDF cf, double* __restrict__ part) {
  static_assert(sizeof(ibem::BemPostDF) == 11 * sizeof(float4), "BemPostDF is copied as 11 float4");
  __shared__ __align__(16) ibem::BemPostDF sq[kPostStageDF];
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = s < nump;
  ibem::dfloat p[3] = {};
  if (act)
    for (int k = 0; k < 3; ++k) p[k] = ibem::df_make(pts[3 * (int64_t)s + k]);
  ibem::dacc acc[6] = {};
  int64_t qb, qe;
  post_slice(nq, qb, qe);   // slice boundaries are multiples of kPostStage, hence of kPostStageDF
  for (int64_t q0 = qb; q0 < qe; q0 += kPostStageDF) {
    const int nqs = (int)min((int64_t)kPostStageDF, qe - q0);
    __syncthreads();
    {
      const float4* src = reinterpret_cast<const float4*>(tab + q0);
      float4* dst = reinterpret_cast<float4*>(sq);
      for (int i = threadIdx.x; i < nqs * 11; i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    if (!act) continue;
#pragma unroll 1
    for (int qq = 0; qq < nqs; ++qq) ibem::bem_post_contracted_df(p, sq[qq], cf, acc);
  }
  if (act)
#pragma unroll
    for (int t = 0; t < 6; ++t) part[6 * ((int64_t)blockIdx.y * nump + s) + t] = (double)acc[t].s + (double)acc[t].c;
}

}  // namespace

namespace ibem {

// Node incidence lists of the mesh (see k_inc_*), in stream-ordered memory freed by the caller
// with cudaFreeAsync: *start (NN + 1 ints) then the slots (4 NE ints) in one allocation.
static ibem_status node_incidence(const int* conn, int NN, int NE, int** start, int** slot, cudaStream_t st) {
  int* buf = nullptr;
  const size_t n = (size_t)(NN + 1) + 2 * (size_t)NN + 4 * (size_t)NE;
  IBEM_CUDA(pool_alloc((void**)&buf, sizeof(int) * n, st));
  int* s0 = buf;
  int* cnt = s0 + NN + 1;
  int* cur = cnt + NN;
  int* sl = cur + NN;
  IBEM_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * 2 * (size_t)NN, st));
  const unsigned g4 = (unsigned)((4 * (int64_t)NE + 255) / 256);
  if (NE > 0) ::ibem::count_launch(), k_inc_count<<<g4, 256, 0, st>>>(conn, NE, NN, cnt);
  ::ibem::count_launch(), k_inc_scan<<<1, 1024, 0, st>>>(cnt, NN, s0);
  if (NE > 0) ::ibem::count_launch(), k_inc_fill<<<g4, 256, 0, st>>>(conn, NE, NN, s0, cur, sl);
  ::ibem::count_launch(), k_inc_sort<<<(NN + 255) / 256, 256, 0, st>>>(NN, s0, sl);
  IBEM_LAUNCH_CHECK("node incidence");
  *start = s0;
  *slot = sl;
  return IBEM_OK;
}

static dim3 gather_grid(int64_t nrows, int NN) {
  return dim3((unsigned)((nrows + 255) / 256), (unsigned)std::min(NN, 65535));
}

ibem_status bem_hg(const double* nodes, int NN, const int* conn, int NE, const ibem_material& m,
                   double* H, int64_t ldh, int64_t hrow0, int64_t hcol0, double* G, int64_t ldg,
                   int64_t grow0, int64_t gcol0, cudaStream_t st) {
  double* Hb = H + hcol0 * ldh + hrow0;
  double* Gb = G + gcol0 * ldg + grow0;
  if (NN <= 0) return IBEM_OK;
  const int64_t ldt = 3 * (int64_t)NN;
  double* TG = nullptr;
  const size_t tg_bytes = sizeof(double) * ldt * 12 * (size_t)(NE > 0 ? NE : 1);
  IBEM_CUDA(pool_alloc((void**)&TG, tg_bytes, st));
  IBEM_CUDA(cudaMemsetAsync(TG, 0, tg_bytes, st));   // an element with bad connectivity adds nothing
  int *start = nullptr, *slot = nullptr;
  ibem_status s = node_incidence(conn, NN, NE, &start, &slot, st);
  if (s) { pool_free(TG, st); return s; }
  const double mu = m.E0 / (2 * (1 + m.nu0));
  KelvinC kc;
  kc.cu = 1.0 / (16 * IBEM_PI * mu * (1 - m.nu0));
  kc.c1 = 3 - 4 * m.nu0;
  kc.ct = 1.0 / (8 * IBEM_PI * (1 - m.nu0));
  kc.c3 = 1 - 2 * m.nu0;
  dim3 grid((NN + 127) / 128, NE);
  if (NE > 0) {
    ::ibem::count_launch(), bem_hg_kernel<<<grid, 128, 0, st>>>(nodes, NN, conn, kc, TG, ldt, Gb, ldg);
    ::ibem::count_launch(), bem_hg_singular<<<(unsigned)NE, 128, 0, st>>>(nodes, NN, conn, NE, kc, TG, ldt, Gb, ldg);
  }
  ::ibem::count_launch(), k_node_gather<<<gather_grid(ldt, NN), 256, 0, st>>>(ldt, NN, start, slot, TG, ldt, Hb, ldh, 0);
  ::ibem::count_launch(), bem_diag_kernel<<<(3 * NN + 127) / 128, 128, 0, st>>>(NN, Hb, ldh);
  pool_free(start, st);
  pool_free(TG, st);
  IBEM_LAUNCH_CHECK("bem_hg");
  return IBEM_OK;
}

ibem_status bem_to_incl(const double* nodes, int NN, const int* conn, int NE, const double* cen,
                        int num, const ibem_material& m, int layout, double* H, int64_t ldh,
                        int64_t hcol0, double* G, int64_t ldg, int64_t gcol0, int64_t row0,
                        cudaStream_t st) {
  BemMat bm = bem_mat_init(m.E0, m.nu0, m.E1, m.nu1);
  double* Hb = H + hcol0 * ldh + row0;
  double* Gb = G + gcol0 * ldg + row0;
  if (NN <= 0 || NE <= 0 || num <= 0) return IBEM_OK;
  const int64_t rows = (int64_t)layout * num;
  double* UG = nullptr;
  const size_t ug_bytes = sizeof(double) * rows * 12 * (size_t)NE;
  IBEM_CUDA(pool_alloc((void**)&UG, ug_bytes, st));
  IBEM_CUDA(cudaMemsetAsync(UG, 0, ug_bytes, st));   // an element with bad connectivity adds nothing
  int *start = nullptr, *slot = nullptr;
  ibem_status s = node_incidence(conn, NN, NE, &start, &slot, st);
  if (s) { pool_free(UG, st); return s; }
  const dim3 grid((unsigned)NE, (unsigned)((num + kInclGroup - 1) / kInclGroup));
  cudaError_t ce = cudaSuccess;
  if (layout == 24) {
    ce = cudaFuncSetAttribute((const void*)bem_incl_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)InclShape<1>::smem);
    ::ibem::count_launch(), bem_incl_kernel<1><<<grid, 128, InclShape<1>::smem, st>>>(nodes, NN, conn, cen, num, bm, layout, UG,
                                                                                     rows, Gb, ldg);
  } else {
    ce = cudaFuncSetAttribute((const void*)bem_incl_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)InclShape<2>::smem);
    ::ibem::count_launch(), bem_incl_kernel<2><<<grid, 128, InclShape<2>::smem, st>>>(nodes, NN, conn, cen, num, bm, layout, UG,
                                                                                     rows, Gb, ldg);
  }
  ::ibem::count_launch(), k_node_gather<<<gather_grid(rows, NN), 256, 0, st>>>(rows, NN, start, slot, UG, rows, Hb, ldh, 1);
  pool_free(start, st);
  pool_free(UG, st);
  if (ce != cudaSuccess) return cuda_fail(ce, "bem_to_incl");
  IBEM_LAUNCH_CHECK("bem_to_incl");
  return IBEM_OK;
}

ibem_status bem_post(const double* pts, int nump, const double* nodes, int NN, const int* conn,
                     int NE, const ibem_material& m, const double* U, const double* T,
                     double* stress, cudaStream_t st, bool mixed) {
  BemMat bm = bem_mat_init(m.E0, m.nu0, m.E1, m.nu1);
  const BemPostCoef cf = bem_post_coef(bm);
  ProfScope ps(PROF_BEM, st);
  const int64_t nq = (int64_t)NE * kPostQ;
  double* tab = nullptr;
  // source slices of the Gauss points: about 8 CTAs per SM in total, at least one staged
  // chunk each (few sample points would otherwise leave most SMs idle)
  int dev = 0, nsm = 0;
  IBEM_CUDA(cudaGetDevice(&dev));
  IBEM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int gx = (nump + 127) / 128;
  const int64_t chunks = (nq + kPostStage - 1) / kPostStage;
  const int nslice = (int)std::max<int64_t>(1, std::min<int64_t>((8 * (int64_t)nsm + gx - 1) / gx, chunks));
  const size_t tab_bytes = (sizeof(double) * kPostRec * (nq > 0 ? nq : 1) + 255) / 256 * 256;
  const size_t df_bytes = ((mixed ? sizeof(BemPostDF) : sizeof(BemPostRec)) * (nq > 0 ? nq : 1) + 255) / 256 * 256;
  const size_t part_bytes = sizeof(double) * 6 * (size_t)nslice * (size_t)nump;
  IBEM_CUDA(pool_alloc((void**)&tab, tab_bytes + df_bytes + part_bytes, st));
  void* recs = reinterpret_cast<char*>(tab) + tab_bytes;   // the form's records of the Gauss points
  double* part = reinterpret_cast<double*>(reinterpret_cast<char*>(tab) + tab_bytes + df_bytes);
  const unsigned gq = (unsigned)((nq + 127) / 128);
  const dim3 grid((unsigned)gx, (unsigned)nslice);
  if (nq > 0)
    ::ibem::count_launch(), bem_post_table<<<gq, 128, 0, st>>>(nodes, NN, conn, NE, U, T, tab);
  if (mixed) {
    BemPostDF* tdf = static_cast<BemPostDF*>(recs);
    if (nq > 0) ::ibem::count_launch(), k_post_df_table<<<gq, 128, 0, st>>>(tab, nq, cf, tdf);
    ::ibem::count_launch(), bem_post_kernel_df<<<grid, 128, 0, st>>>(pts, nump, tdf, nq, bem_post_coef_df(cf), part);
  } else {
    BemPostRec* trec = static_cast<BemPostRec*>(recs);
    if (nq > 0) ::ibem::count_launch(), k_post_rec<<<gq, 128, 0, st>>>(tab, nq, cf, trec);
    ::ibem::count_launch(), bem_post_kernel<<<grid, 128, 0, st>>>(pts, nump, trec, nq, cf, part);
  }
  ::ibem::count_launch(), k_post_reduce<<<(unsigned)((6 * (int64_t)nump + 255) / 256), 256, 0, st>>>(nump, nslice,
                                                                                                   part, stress);
  pool_free(tab, st);
  IBEM_LAUNCH_CHECK("bem_post");
  return IBEM_OK;
}

}  // namespace ibem
