// Dense pairwise matrices of the dual-interpolation BEM (DIBEM): for every
// pair of collocation points i != j with R = |x_j - x_i|,
//   F_ij = phi(R)                      radial basis function
//   D_ij = u*(x_i, x_j)                fundamental solution
// restating `_dibem_FD_kernel!` (src/Laplace/DIBEM_GPU.jl:194-208, Laplace:
// D = -log(R)/(2 pi k)) and `_elast_dibem_FD_kernel!`
// (src/Elasticity/Assembly_GPU.jl:258-280, Kelvin: D holds the 2x2 block
// U(r) of `_kelvin2d_UT`).  phi: `_dibem_phi` (DIBEM_GPU.jl:116-139), kinds
// 1-7 the polyharmonic splines R, R^2 log(R+e), R^3, R^4 log(R+e), R^5,
// R^6 log(R+e), R^7, kind 10 the fundamental solution.  Entries with
// i == j or R^2 <= eps^2 stay zero.  Outputs column-major (Julia layout).
#include <cfloat>
#include <cmath>

#include "bem_abi_internal.h"
#include "bem_device.cuh"
#include "fast64.cuh"

namespace bem {
namespace {

// FP64 through the short functions (fast64.cuh), FP32 through the platform's
__device__ __forceinline__ double fd_log(double x) { return f64::log(x); }
__device__ __forceinline__ float fd_log(float x) { return logf(x); }
__device__ __forceinline__ double fd_sqrt(double x) { return f64::sqrt(x); }
__device__ __forceinline__ float fd_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double fd_rcp(double x) { return f64::rcp(x); }
__device__ __forceinline__ float fd_rcp(float x) { return 1.f / x; }

template <typename T>
__device__ __forceinline__ T dibem_phi(int kind, T R, T kcond, T epsa) {
  const T R2 = R * R;
  switch (kind) {
    case 1: return R;
    case 2: return R2 * fd_log(R + epsa);
    case 3: return R2 * R;
    case 4: return (R2 * R2) * fd_log(R + epsa);
    case 5: return R2 * R2 * R;
    case 6: return (R2 * R2 * R2) * fd_log(R + epsa);
    case 7: return R2 * R2 * R2 * R;
    default: return -fd_log(R) / (T(2) * T(3.14159265358979323846) * kcond);
  }
}

// F (nt x nt) and D: Laplace (DOF 1) nt x nt, Kelvin (DOF 2) 2nt x 2nt with
// node-major blocks u11 u12; u12 u22.  Every entry depends on R or on products
// of two components of x_j - x_i, so both matrices are symmetric to the bit:
// a CTA forms the TB x TB tile (I, J), I >= J, once, stores it, and stores its
// transpose as tile (J, I) through shared memory.  A warp stores 32
// consecutive rows of a column whatever the leading dimension (a thread with
// 16 bytes of each column, as before, stored element by element when it was
// odd: 8193 points in FP32 145 us, now 108; the write alone takes 80, the rest
// is issue, 82 instructions for an entry and its mirror).  FP64 is bound by its
// arithmetic, which this halves (4095 points: Laplace 2.55 -> 0.63 ms, Kelvin
// 1.84 -> 0.66, with the short logarithm and square root).  One kernel per phi
// and a path without bounds for inner tiles took the FP32 one from 125 to 108.
// Tile rows r and nb - 1 - r share blockIdx.y.
template <typename T>
struct FdArgs {
  int nt, nb;
  const double *px, *py;
  T prm0, prm1, epsa, eps2;
  T *F, *D;
  int64_t ldf, ldd;
};

// one tile and its transpose; EDGE: it may reach beyond the last point or
// hold the diagonal
template <typename T, int DOF, int TB, int KIND, bool EDGE>
__device__ __forceinline__ void dibem_fd_tile(const FdArgs<T>& a, int I, int J, T (*tr)[TB][TB + 1], const T* sx,
                                              const T* sy, T xi, T yi) {
  constexpr int NV = DOF == 1 ? 2 : 4, STEP = 256 / TB;
  const int t = threadIdx.x, row = t & (TB - 1), c0 = t / TB;
  const T pi = T(3.14159265358979323846);
  // Laplace: -log(R) / (2 pi k) with the constant's reciprocal formed once;
  // Kelvin: prm0 = mu, prm1 = nu
  const T coef = DOF == 1 ? T(1) / (T(2) * pi * a.prm0) : T(1) / (T(2) * (T(4) * pi * (T(1) - a.prm1)) * a.prm0);
  auto put = [&](T* f, T* d, const T (&v)[NV]) {
    *f = v[0];
    if constexpr (DOF == 1) {
      *d = v[1];
    } else {
      d[0] = v[1];
      d[1] = v[2];
      d[a.ldd] = v[2];
      d[a.ldd + 1] = v[3];
    }
  };
  {
    const int i = I * TB + row;
    T* f = a.F + i + (size_t)(J * TB + c0) * a.ldf;
    T* d = a.D + (size_t)DOF * i + (size_t)(J * TB + c0) * DOF * a.ldd;
#pragma unroll 4
    for (int c = c0; c < TB; c += STEP, f += STEP * a.ldf, d += STEP * DOF * a.ldd) {
      const int j = J * TB + c;
      T v[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] = T(0);
      const T rx = sx[c] - xi, ry = sy[c] - yi;
      const T R2 = rx * rx + ry * ry;
      if ((!EDGE || i != j) && R2 > a.eps2) {
        const T R = fd_sqrt(R2);
        v[0] = dibem_phi<T>(KIND, R, DOF == 1 ? a.prm0 : T(1), a.epsa);
        if constexpr (DOF == 1) {
          v[1] = -fd_log(R) * coef;
        } else {
          // U of the 2-D Kelvin solution (`_kelvin2d_UT`, Elasticity/Fundamental.jl)
          const T invR = fd_rcp(R);
          const T dr1 = rx * invR, dr2 = ry * invR;
          const T prod2 = (T(3) - T(4) * a.prm1) * (-fd_log(R));
          v[1] = (prod2 + dr1 * dr1) * coef;
          v[2] = (dr1 * dr2) * coef;
          v[3] = (prod2 + dr2 * dr2) * coef;
        }
      }
      if (!EDGE || (i < a.nt && j < a.nt)) put(f, d, v);
#pragma unroll
      for (int q = 0; q < NV; ++q) tr[q][c][row] = v[q];
    }
  }
  if (EDGE && I == J) return;
  __syncthreads();
  {
    const int j = J * TB + row;
    T* f = a.F + j + (size_t)(I * TB + c0) * a.ldf;
    T* d = a.D + (size_t)DOF * j + (size_t)(I * TB + c0) * DOF * a.ldd;
#pragma unroll 4
    for (int c = c0; c < TB; c += STEP, f += STEP * a.ldf, d += STEP * DOF * a.ldd) {
      T v[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] = tr[q][row][c];
      if (!EDGE || (I * TB + c < a.nt && j < a.nt)) put(f, d, v);
    }
  }
}

template <typename T, int DOF, int TB, int KIND>
__global__ void __launch_bounds__(256) dibem_fd_kernel(const __grid_constant__ FdArgs<T> a) {
  __shared__ T tr[DOF == 1 ? 2 : 4][TB][TB + 1];
  __shared__ T sx[TB], sy[TB];
  const int y = blockIdx.y, x = blockIdx.x;
  const int I = x <= y ? y : a.nb - 1 - y, J = x <= y ? x : x - y - 1;
  if (x > y && I <= y) return;  // the middle row of an odd count pairs with itself
  const int t = threadIdx.x, i = min(I * TB + (t & (TB - 1)), a.nt - 1);
  if (t < TB) {
    const int j = min(J * TB + t, a.nt - 1);
    sx[t] = (T)a.px[j];
    sy[t] = (T)a.py[j];
  }
  const T xi = (T)a.px[i], yi = (T)a.py[i];
  __syncthreads();
  if (I == J || (I + 1) * TB > a.nt)
    dibem_fd_tile<T, DOF, TB, KIND, true>(a, I, J, tr, sx, sy, xi, yi);
  else
    dibem_fd_tile<T, DOF, TB, KIND, false>(a, I, J, tr, sx, sy, xi, yi);
}

template <typename T, int DOF, int TB>
void launch_fd(int nt, const double* px, const double* py, double prm0, double prm1, int kind, double epsa, T eps,
               T* F, int64_t ldf, T* D, int64_t ldd, cudaStream_t st) {
  const int nb = (nt + TB - 1) / TB;
  const FdArgs<T> a{nt, nb, px, py, (T)prm0, (T)prm1, (T)epsa, eps * eps, F, D, ldf, ldd};
  void (*const k[8])(FdArgs<T>) = {dibem_fd_kernel<T, DOF, TB, 1>, dibem_fd_kernel<T, DOF, TB, 2>,
                                   dibem_fd_kernel<T, DOF, TB, 3>, dibem_fd_kernel<T, DOF, TB, 4>,
                                   dibem_fd_kernel<T, DOF, TB, 5>, dibem_fd_kernel<T, DOF, TB, 6>,
                                   dibem_fd_kernel<T, DOF, TB, 7>, dibem_fd_kernel<T, DOF, TB, 10>};
  k[kind == 10 ? 7 : kind - 1]<<<dim3(nb + 1, (nb + 1) / 2), 256, 0, st>>>(a);
}

template <typename T>
__device__ __forceinline__ T dibem_phi_int(int kind, T R, T kcond, T epsa) {
  const T R2 = R * R;
  switch (kind) {
    case 1: return (R2 * R) / T(3);
    case 2: { const T R4 = R2 * R2; return (T(4) * R4 * log(R + epsa) - R4) / T(16); }
    case 3: return (R2 * R2 * R) / T(5);
    case 4: { const T R6 = R2 * R2 * R2; return R6 * log(R + epsa) / T(6) - R6 / T(36); }
    case 5: return (R2 * R2 * R2 * R) / T(7);
    case 6: { const T R8 = (R2 * R2) * (R2 * R2); return R8 * log(R + epsa) / T(8) - R8 / T(64); }
    case 7: { const T R4 = R2 * R2; return (R4 * R4 * R) / T(9); }
    default: return -(T(2) * R2 * log(R) - R2) / (T(8) * T(3.14159265358979323846) * kcond);
  }
}

// phi_int(R) / R^2 in FP64, times phi_int_divisor: the powers of R
// cancel before they are formed, so a pair needs no quotient (an FP64 quotient
// is five and a half multiply-adds of GB300's small FP64 pipe)
__device__ __forceinline__ double phi_int_over_r2(int kind, double R2, double lgR2, double epsa) {
  if (kind == 10) return 1.0 - lgR2;
  const double R = f64::sqrt(R2);
  switch (kind) {
    case 1: return R;
    case 2: return R2 * (4.0 * f64::log(R + epsa) - 1.0);
    case 3: return R2 * R;
    case 4: return (R2 * R2) * (6.0 * f64::log(R + epsa) - 1.0);
    case 5: return (R2 * R2) * R;
    case 6: return (R2 * R2 * R2) * (8.0 * f64::log(R + epsa) - 1.0);
    default: return (R2 * R2 * R2) * R;
  }
}
// (sums are divided by it once: a factor 1 / 3 would round every sum one way)
__device__ __forceinline__ double phi_int_divisor(int kind, double kcond) {
  switch (kind) {
    case 1: return 3.0;
    case 2: return 16.0;
    case 3: return 5.0;
    case 4: return 36.0;
    case 5: return 7.0;
    case 6: return 64.0;
    case 7: return 9.0;
    default: return 8.0 * kPi * kcond;
  }
}

// An element's box in FP32, rounded outwards, and its near limit widened by
// more than the rounding of coordinates and distances: a point that the FP32
// test calls far is far for the exact FP64 test too.  (The FP64 box test took
// a third of the far kernel, the exact test for every pair half of the near
// kernel.)
struct Box32 {
  float lox, loy, hix, hiy, lim;
};
__device__ __forceinline__ Box32 box32(const double* x, const double* y, int nn, double L, double nf) {
  double lx = INFINITY, ly = INFINITY, hx = -INFINITY, hy = -INFINITY;
  for (int q = 0; q < nn; ++q) {
    lx = fmin(lx, x[q]);
    ly = fmin(ly, y[q]);
    hx = fmax(hx, x[q]);
    hy = fmax(hy, y[q]);
  }
  Box32 b{__double2float_rd(lx), __double2float_rd(ly), __double2float_ru(hx), __double2float_ru(hy), 0.f};
  const float m = fmaxf(fmaxf(fabsf(b.lox), fabsf(b.hix)), fmaxf(fabsf(b.loy), fabsf(b.hiy)));
  b.lim = nf > 1e20 ? INFINITY : __double2float_ru(nf * L * (1.0 + 1e-5)) + 1e-6f * m;
  return b;
}
// (px, py): the point rounded to FP32, pm = 1e-6 times its largest coordinate
__device__ __forceinline__ bool surely_far(const Box32& b, float px, float py, float pm) {
  const float dx = fmaxf(fmaxf(b.lox - px, px - b.hix), 0.f), dy = fmaxf(fmaxf(b.loy - py, py - b.hiy), 0.f);
  const float lim = b.lim + pm;
  return dx * dx + dy * dy > lim * lim;
}

// Far boundary sums IF, ID of the DIBEM domain integrals (restating
// `_dibem_IFID_kernel!`, DIBEM_GPU.jl:234-270): for every collocation point
// i and boundary node j with R > 1e-10, unless the pair (i, element of j) is
// near or i lies on that element (`_near_skip_mask`, the same exact FP64 test
// as the assembly),
//   IF_i += phi_int(R) w_j (r . n_j) / R^2,  ID_i += rad(R) w_j (r . n_j) / R^2,
// rad(R) = -(2 R^2 log R - R^2) / (8 pi k) (`_dibem_rad_id2d`, :173-177),
// w_j = Jacobian_j * elem_weight_k.  With rad(R) / R^2 = (1 - log R^2) / (8 pi k)
// and phi_int(R) / R^2 by phi_int_over_r2 a pair is 27 FP64 operations for an
// odd spline (it was 90; 4098 x 4098 pairs 2.48 -> 1.02 ms, FP64 issue bound).
// Grid: x over 128-point row blocks, y over 32-element chunks staged in
// shared memory; partial sums are added atomically.
constexpr int IF_EC = 32;
struct IfidRule {
  double ew[BEM_MAXNN];
};

template <typename T>
__global__ void __launch_bounds__(128) dibem_ifid_kernel(GeomDev g, IfidRule rw, int rbf, T kcond, T epsa,
                                                        double nf, T* __restrict__ IF, T* __restrict__ ID) {
  __shared__ double sx[IF_EC * BEM_MAXNN], sy[IF_EC * BEM_MAXNN];
  __shared__ T snx[IF_EC * BEM_MAXNN], sny[IF_EC * BEM_MAXNN], sw[IF_EC * BEM_MAXNN];
  __shared__ Box32 sbox[IF_EC];
  __shared__ double belen[IF_EC];
  const int nn = g.nn;
  const int e0 = blockIdx.y * IF_EC;
  const int nel = min(IF_EC, g.ne - e0);
  for (int idx = threadIdx.x; idx < nel * nn; idx += blockDim.x) {
    const int j = e0 * nn + idx;
    sx[idx] = g.px[j];
    sy[idx] = g.py[j];
    sw[idx] = (T)(g.jac[j] * rw.ew[idx % nn]);
    snx[idx] = (T)g.nx[j] * (sizeof(T) == 8 ? sw[idx] : T(1));  // FP64: times the weight
    sny[idx] = (T)g.ny[j] * (sizeof(T) == 8 ? sw[idx] : T(1));
  }
  __syncthreads();
  for (int el = threadIdx.x; el < nel; el += blockDim.x) {
    belen[el] = g.elen[e0 + el];
    sbox[el] = box32(sx + el * nn, sy + el * nn, nn, belen[el], nf);
  }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nt) return;
  const V2 pf{g.px[i], g.py[i]};
  const T pxi = (T)pf.x, pyi = (T)pf.y;
  const float fx = (float)pf.x, fy = (float)pf.y, fm = 1e-6f * fmaxf(fabsf(fx), fabsf(fy));
  T aF = T(0), aD = T(0);
  const T radc = T(1) / (T(8) * T(3.14159265358979323846) * kcond);
  for (int el = 0; el < nel; ++el) {
    const int e = e0 + el;
    if (i >= e * nn && i < (e + 1) * nn) continue;  // source on the element
    if (!surely_far(sbox[el], fx, fy, fm)) {
      V2 xg[BEM_MAXNN];
      for (int q = 0; q < nn; ++q) xg[q] = V2{sx[el * nn + q], sy[el * nn + q]};
      if (near_element(pf, xg, nn, belen[el], nf)) continue;
    }
    for (int q = 0; q < nn; ++q) {
      const int s = el * nn + q;
      const T rx = (T)sx[s] - pxi, ry = (T)sy[s] - pyi;
      const T R2 = rx * rx + ry * ry;
      if constexpr (sizeof(T) == 4) {
        // FP32: the products in the reference's order (quotients are cheap
        // here, and the sums keep their rounding)
        const T R = sqrt(R2);
        if (R > T(1e-10)) {
          const T wJn = sw[s] * (rx * snx[s] + ry * sny[s]) / R2;
          aF += dibem_phi_int<T>(rbf, R, kcond, epsa) * wJn;
          aD += -(T(2) * R2 * log(R) - R2) * radc * wJn;
        }
      } else if (R2 > T(1e-20)) {
        const T rn = rx * snx[s] + ry * sny[s];
        const T lg = f64::log(R2);
        aF += phi_int_over_r2(rbf, R2, lg, epsa) * rn;
        aD += (T(1) - lg) * rn;
      }
    }
  }
  if constexpr (sizeof(T) == 8) {
    aF = f64::div(aF, phi_int_divisor(rbf, kcond));
    aD *= radc;
  }
  atomicAdd(IF + i, aF);
  atomicAdd(ID + i, aD);
}

// Near-pair correction of IF and ID (`_dibem_correct_near_cpu!`,
// src/Laplace/DIBEM_GPU.jl:272-300): for every element near point i (the
// assembly's exact test) or holding it, the npg-point Gauss rule on the
// element's field interpolant (`_rim_build_elements`,
// src/Core/DIBEM_common.jl:112-171: rule points y_q, normals tan2normal of
// the tangent aligned with the element's first nodal normal, w_q J_q),
//   IF_i += phi_int(R) w_q J_q (r . n_q) / R^2,  ID_i += rad(R) w_q J_q (r . n_q) / R^2
// with r = y_q - x_i, points closer than 1e-14 skipped.  FP64.  A CTA takes
// 128 points and 16 elements: its pairs are found first (nearly all CTAs have
// none and leave), then the elements' rule points are built in shared memory
// and 16 lanes take a pair's rule (a thread per point went through its
// elements alone: 13 of a warp's 32 lanes had work at best; 1.39 ms at 4098
// nodes, now 0.14).
constexpr int NR_EC = 16, NR_PT = 128;
__global__ void __launch_bounds__(NR_PT) dibem_near_kernel(const __grid_constant__ GeomDev g,
                                                          const __grid_constant__ Rules R, int rbf, double kcond,
                                                          double epsa, double nf, double* __restrict__ IF,
                                                          double* __restrict__ ID) {
  __shared__ double sx[NR_EC * BEM_MAXNN], sy[NR_EC * BEM_MAXNN];
  __shared__ double qy[NR_EC * BEM_MAXNPG][4];  // y.x, y.y, n.x w J, n.y w J
  __shared__ Box32 sbox[NR_EC];
  __shared__ double belen[NR_EC];
  __shared__ unsigned short s_pair[NR_PT * NR_EC];  // point * 16 + element
  __shared__ int s_count;
  const int nn = g.nn, npg = R.npg, t = threadIdx.x;
  const int e0 = blockIdx.y * NR_EC;
  const int nel = min(NR_EC, g.ne - e0);
  for (int idx = t; idx < nel * nn; idx += NR_PT) {
    sx[idx] = g.px[e0 * nn + idx];
    sy[idx] = g.py[e0 * nn + idx];
  }
  if (t == 0) s_count = 0;
  __syncthreads();
  if (t < nel) {
    belen[t] = g.elen[e0 + t];
    sbox[t] = box32(sx + t * nn, sy + t * nn, nn, belen[t], nf);
  }
  __syncthreads();
  const int i = blockIdx.x * NR_PT + t;
  if (i < g.nt) {
    const V2 pf{g.px[i], g.py[i]};
    const float fx = (float)pf.x, fy = (float)pf.y, fm = 1e-6f * fmaxf(fabsf(fx), fabsf(fy));
    for (int el = 0; el < nel; ++el) {
      const int e = e0 + el;
      bool near = i >= e * nn && i < (e + 1) * nn;
      if (!near && !surely_far(sbox[el], fx, fy, fm)) {
        V2 xg[BEM_MAXNN];
        for (int k = 0; k < nn; ++k) xg[k] = V2{sx[el * nn + k], sy[el * nn + k]};
        near = near_element(pf, xg, nn, belen[el], nf);
      }
      if (near) s_pair[atomicAdd(&s_count, 1)] = (unsigned short)(t * NR_EC + el);
    }
  }
  __syncthreads();
  const int count = s_count;
  if (count == 0) return;
  for (int v = t; v < nel * npg; v += NR_PT) {
    const int el = v / npg, q = v - el * npg;
    double L[BEM_MAXNN], dL[BEM_MAXNN];
    shapefun(R.leg_x, R.leg_bw, R.leg_D, nn, R.qsi[q], L, dL);
    double px = 0, py = 0, dx = 0, dy = 0;
    for (int k = 0; k < nn; ++k) {
      px += L[k] * sx[el * nn + k];
      py += L[k] * sy[el * nn + k];
      dx += dL[k] * sx[el * nn + k];
      dy += dL[k] * sy[el * nn + k];
    }
    const int j0 = (e0 + el) * nn;
    const bool bad = sqrt(dx * dx + dy * dy) < 1e-16;
    const double flip = dy * g.nx[j0] - dx * g.ny[j0] < 0 ? -R.w[q] : R.w[q];
    qy[v][0] = px;
    qy[v][1] = py;
    qy[v][2] = bad ? 0.0 : flip * dy;
    qy[v][3] = bad ? 0.0 : -(flip * dx);
  }
  __syncthreads();
  const double dF = phi_int_divisor(rbf, kcond), cD = 1.0 / (8.0 * kPi * kcond);
  const int lg = t & 15;
  for (int p0 = 0; p0 < count; p0 += NR_PT / 16) {
    const int p = p0 + (t >> 4);
    double aF = 0.0, aD = 0.0;
    int ip = 0;
    if (p < count) {
      const int pr = s_pair[p], el = pr & (NR_EC - 1);
      ip = blockIdx.x * NR_PT + pr / NR_EC;
      const double x = g.px[ip], y = g.py[ip];
      for (int q = lg; q < npg; q += 16) {
        const double* Y = qy[el * npg + q];
        const double rx = Y[0] - x, ry = Y[1] - y;
        const double R2 = rx * rx + ry * ry;
        if (R2 < 1e-28) continue;
        const double rn = rx * Y[2] + ry * Y[3], l = f64::log(R2);
        aF += phi_int_over_r2(rbf, R2, l, epsa) * rn;
        aD += (1.0 - l) * rn;
      }
    }
    for (int o = 8; o > 0; o >>= 1) {
      aF += __shfl_xor_sync(0xffffffffu, aF, o);
      aD += __shfl_xor_sync(0xffffffffu, aD, o);
    }
    if (p < count && lg == 0) {
      atomicAdd(IF + ip, f64::div(aF, dF));
      atomicAdd(ID + ip, aD * cD);
    }
  }
}

}  // namespace
}  // namespace bem

using namespace bem;

extern "C" int bem_dibem_ifid2d(bem_ctx* c, const bem_geom2d* geom, double k, int rbf, double epsa,
                                double near_factor, int dtype, int mem, void* IF, void* ID) {
  if (!c || !geom || !IF || !ID) return BEM_ERR_INVALID;
  if (!((rbf >= 1 && rbf <= 7) || rbf == 10)) return BEM_ERR_INVALID;
  if (dtype != BEM_F32 && dtype != BEM_F64) return BEM_ERR_INVALID;
  if (mem != BEM_MEM_HOST && mem != BEM_MEM_DEVICE) return BEM_ERR_INVALID;
  if (!(k > 0) || !(near_factor >= 0)) return BEM_ERR_INVALID;
  int rc = bem_check_geom(geom, 2, near_factor);
  if (rc) return rc;
  CallScope cs(c);
  cudaSetDevice(c->device);
  GeomDev gd;
  Rules R;
  rc = bem_stage_geom(c, geom, 2, mem, gd, R);
  if (rc) return rc;
  IfidRule rw{};
  for (int q = 0; q < BEM_MAXNN; ++q) rw.ew[q] = R.ew[q];
  const size_t esz = dtype == BEM_F32 ? 4 : 8;
  const size_t nt = (size_t)gd.nt;
  void *dF = IF, *dD = ID;
  if (mem == BEM_MEM_HOST) {
    void* o = c->get(bem_ctx::SLOT_OUT2, 2 * esz * nt);
    if (!o) return BEM_ERR_NOMEM;
    dF = o;
    dD = (char*)o + esz * nt;
  }
  cudaMemsetAsync(dF, 0, esz * nt, c->stream);
  cudaMemsetAsync(dD, 0, esz * nt, c->stream);
  dim3 grid((unsigned)((nt + 127) / 128), (unsigned)((gd.ne + IF_EC - 1) / IF_EC));
  if (dtype == BEM_F64)
    dibem_ifid_kernel<double><<<grid, 128, 0, c->stream>>>(gd, rw, rbf, k, epsa, near_factor, (double*)dF,
                                                            (double*)dD);
  else
    dibem_ifid_kernel<float><<<grid, 128, 0, c->stream>>>(gd, rw, rbf, (float)k, (float)epsa, near_factor,
                                                           (float*)dF, (float*)dD);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->cuda_fail(e, "dibem_ifid_kernel");
  if (mem == BEM_MEM_HOST) {
    cudaMemcpyAsync(IF, dF, esz * nt, cudaMemcpyDeviceToHost, c->stream);
    cudaMemcpyAsync(ID, dD, esz * nt, cudaMemcpyDeviceToHost, c->stream);
  }
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->cuda_fail(e, "dibem_ifid");
  return BEM_OK;
}

extern "C" int bem_dibem_fd2d(bem_ctx* c, int nt, const double* px, const double* py, int kind, double prm0,
                              double prm1, int rbf, double epsa, int dtype, int mem, void* F, int64_t ldf,
                              void* D, int64_t ldd) {
  if (!c || nt <= 0 || !px || !py || !F || !D) return BEM_ERR_INVALID;
  if (kind != 0 && kind != 1) return BEM_ERR_INVALID;
  if (!((rbf >= 1 && rbf <= 7) || rbf == 10)) return BEM_ERR_INVALID;
  if (dtype != BEM_F32 && dtype != BEM_F64) return BEM_ERR_INVALID;
  if (mem != BEM_MEM_HOST && mem != BEM_MEM_DEVICE) return BEM_ERR_INVALID;
  const int dof = kind == 0 ? 1 : 2;
  if (ldf < nt || ldd < (int64_t)dof * nt) return BEM_ERR_INVALID;
  if (kind == 0 && !(prm0 > 0)) return BEM_ERR_INVALID;
  if (kind == 1 && (!(prm0 > 0) || !(prm1 < 0.5) || !(prm1 > -1.0))) return BEM_ERR_INVALID;
  CallScope cs(c);
  cudaSetDevice(c->device);
  const size_t esz = dtype == BEM_F32 ? 4 : 8;
  const size_t n = (size_t)nt;
  const double *dx = px, *dy = py;
  void *dF = F, *dD = D;
  int64_t lf = ldf, lD = ldd;
  if (mem == BEM_MEM_HOST) {
    double* g = (double*)c->get(bem_ctx::SLOT_GEOM, sizeof(double) * 2 * n);
    lf = (int64_t)((n + 3) / 4 * 4);
    lD = (int64_t)((dof * n + 3) / 4 * 4);
    void* o0 = c->get(bem_ctx::SLOT_OUT0, esz * (size_t)lf * n);
    void* o1 = c->get(bem_ctx::SLOT_OUT1, esz * (size_t)lD * dof * n);
    if (!g || !o0 || !o1) return BEM_ERR_NOMEM;
    cudaMemcpyAsync(g, px, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(g + n, py, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream);
    dx = g;
    dy = g + n;
    dF = o0;
    dD = o1;
  }
  // tiles of 64 only where four bytes a value keep two of them in 33 KB
  if (kind == 0) {
    if (dtype == BEM_F64)
      launch_fd<double, 1, 32>(nt, dx, dy, prm0, 0, rbf, epsa, DBL_EPSILON, (double*)dF, lf, (double*)dD, lD, c->stream);
    else
      launch_fd<float, 1, 64>(nt, dx, dy, prm0, 0, rbf, epsa, FLT_EPSILON, (float*)dF, lf, (float*)dD, lD, c->stream);
  } else {
    if (dtype == BEM_F64)
      launch_fd<double, 2, 32>(nt, dx, dy, prm0, prm1, rbf, epsa, DBL_EPSILON, (double*)dF, lf, (double*)dD, lD, c->stream);
    else
      launch_fd<float, 2, 32>(nt, dx, dy, prm0, prm1, rbf, epsa, FLT_EPSILON, (float*)dF, lf, (float*)dD, lD, c->stream);
  }
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->cuda_fail(e, "dibem kernel");
  if (mem == BEM_MEM_HOST) {
    cudaMemcpy2DAsync(F, esz * ldf, dF, esz * lf, esz * n, n, cudaMemcpyDeviceToHost, c->stream);
    cudaMemcpy2DAsync(D, esz * ldd, dD, esz * lD, esz * dof * n, dof * n, cudaMemcpyDeviceToHost, c->stream);
  }
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->cuda_fail(e, "dibem");
  return BEM_OK;
}

extern "C" int bem_dibem_ifid_near2d(bem_ctx* c, const bem_geom2d* geom, double k, int rbf, double epsa,
                                     double near_factor, int npg, int mem, double* IF, double* ID) {
  if (!c || !geom || !IF || !ID) return BEM_ERR_INVALID;
  if (!((rbf >= 1 && rbf <= 7) || rbf == 10)) return BEM_ERR_INVALID;
  if (mem != BEM_MEM_HOST && mem != BEM_MEM_DEVICE) return BEM_ERR_INVALID;
  if (!(k > 0) || !(near_factor >= 0)) return BEM_ERR_INVALID;
  int rc = bem_check_geom(geom, npg, near_factor);
  if (rc) return rc;
  CallScope cs(c);
  cudaSetDevice(c->device);
  GeomDev gd;
  Rules R;
  rc = bem_stage_geom(c, geom, npg, mem, gd, R);
  if (rc) return rc;
  const size_t nt = (size_t)gd.nt;
  double *dF = IF, *dD = ID;
  if (mem == BEM_MEM_HOST) {
    double* o = (double*)c->get(bem_ctx::SLOT_OUT2, 2 * sizeof(double) * nt);
    if (!o) return BEM_ERR_NOMEM;
    dF = o;
    dD = o + nt;
    cudaMemcpyAsync(dF, IF, sizeof(double) * nt, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(dD, ID, sizeof(double) * nt, cudaMemcpyHostToDevice, c->stream);
  }
  dim3 grid((unsigned)((nt + 127) / 128), (unsigned)((gd.ne + NR_EC - 1) / NR_EC));
  dibem_near_kernel<<<grid, 128, 0, c->stream>>>(gd, R, rbf, k, epsa, near_factor, dF, dD);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->cuda_fail(e, "dibem_near_kernel");
  if (mem == BEM_MEM_HOST) {
    cudaMemcpyAsync(IF, dF, sizeof(double) * nt, cudaMemcpyDeviceToHost, c->stream);
    cudaMemcpyAsync(ID, dD, sizeof(double) * nt, cudaMemcpyDeviceToHost, c->stream);
  }
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->cuda_fail(e, "dibem_ifid_near");
  return BEM_OK;
}
