// Adjoint gradient of a boundary-flux misfit with respect to the boundary
// node coordinates (2-D Laplace), through assembly and solve.
//
// The reference has no adjoint of its dense path; this follows the standard
// adjoint-state method on the collocation equations F = H T - G q = 0
// (H, G from `H_G_full_direct`, src/Core/Assembly_full.jl:61-175, with the
// row-sum diagonal :384-390) and the column swap of `applyBC`
// (src/Core/Boundary_conditions.jl:20-75):
//   J = 1/2 sum_{i: BC_i = 0} (q_i - q*_i)^2,   A u = b  <=>  F(u, X) = 0,
//   A^T lambda = dJ/du,   dJ/dX = -lambda^T dF/dX  (T, q held fixed).
// With the diagonal H_ii = -sum_{j != i} H_ij folded in,
//   dJ/dX = sum_{i, j != i} a_ij dH_ij/dX + sum_{i, j} c_ij dG_ij/dX,
//   a_ij = -lambda_i (T_j - T_i),   c_ij = lambda_i q_j.
// Geometry model: elements without CAD nodes, i.e. x(xi) is the Lagrange
// interpolant of the element's p+1 collocation nodes; node normals and
// Jacobians come from that interpolant, so the node coordinates are the only
// geometric parameters.  Boundary data (BC, BV) and the target are held
// fixed.  H and G are never stored: the backward kernels recompute what they
// need.
//   far pairs      analytic derivatives of the nodal lumping (a6), chained
//                  through the node normal and Jacobian to the element nodes
//   near pairs     (same exact near test as the assembly) differences of
//                  the element integral w.r.t. the source and the element's
//                  node coordinates, step 1e-5 element lengths, central
//                  unless a branch switch of the near-field map lies inside
//                  the step (then the smooth one-sided difference)
//   on-element     central differences of the on-element integral w.r.t.
//                  the element's node coordinates (the source moves with its
//                  node)
#include <cmath>
#include <cstring>

#include "bem_abi_internal.h"
#include "bem_lu.h"
#include "near_coop.cuh"
#include "warp_sum.cuh"

int bem_solve_mixed_dev(bem_ctx* c, int N, const double* A64, int64_t lda, const double* b, double tol,
                        int max_iter, int x3, double* x, bem_solve_stats* stats, double* hx = nullptr);

namespace bem {
namespace {

constexpr double kTwoPi = 6.283185307179586476925286766559;

struct AdjArgs {
  GeomDev g;
  Rules R;
  double k, near_factor;
  const double *lam, *T, *q;
  double* gX;      // 2n: dJ/dx, dJ/dy per node (node-major)
  double* gn;      // 2n: dJ/dn per node
  double* gJ;      // n : dJ/dJacobian per node
  const float4* rows;    // records and candidate pairs of the assembly
  const ElemRec* elems;
  const int2* cand;
  const int* ncand;
  int ccap;
  int2* pairs;     // near pairs (i, e)
  int* count;      // [0] near pair count, [1] overflow flag, [2] tasks claimed
  int cap;
  double* S;       // values of the near integrals, neval per pair
};

// derivative contributions of one far pair (source i, node j) -- nodal
// lumping G = -log(R^2)/(4 pi k) J w, H = (r.n)/(2 pi R^2) J w, r = x_j - x_i
__device__ __forceinline__ void far_pair_grad(const AdjArgs& a, int i, int j, double w, double& gxi,
                                              double& gyi, double* node5) {
  const GeomDev& g = a.g;
  const double rx = g.px[j] - g.px[i], ry = g.py[j] - g.py[i];
  const double R2 = rx * rx + ry * ry;
  const double nxj = g.nx[j], nyj = g.ny[j], Jj = g.jac[j];
  const double c = Jj * w;
  const double G = -log(R2) / (2 * kTwoPi * a.k) * c;
  const double rn = rx * nxj + ry * nyj;
  const double H = rn / (kTwoPi * R2) * c;
  const double aH = -a.lam[i] * (a.T[j] - a.T[i]);
  const double aG = a.lam[i] * a.q[j];
  // dG/dr = -r c / (2 pi k R2);  dH/dr = c/(2 pi) (n / R2 - 2 (r.n) r / R2^2)
  const double fG = -c / (kTwoPi * a.k * R2);
  const double fH = c / kTwoPi;
  const double grx = aG * fG * rx + aH * fH * (nxj / R2 - 2 * rn * rx / (R2 * R2));
  const double gry = aG * fG * ry + aH * fH * (nyj / R2 - 2 * rn * ry / (R2 * R2));
  gxi -= grx;
  gyi -= gry;
  node5[0] += grx;
  node5[1] += gry;
  node5[2] += aH * fH * rx / R2;  // dH/dn
  node5[3] += aH * fH * ry / R2;
  node5[4] += (aH * H + aG * G) / Jj;  // d/dJ
}

// Analytic derivatives of the far pairs (those that the assembly's box test
// calls far).  A lane takes one node and walks the CTA's rows, so the five
// sums per node stay in registers; the two sums per row meet across the lanes
// eight rows at a time (warp_sum8: 9 adds for 8 sums; with rows on the lanes
// and five shuffle trees per node the sums were half of the kernel).  With
//   m = lambda_i / R2,  d = -m (T_j - T_i),  g = -(q_j / k) m - 2 d (r.n) / R2
// the pair adds J w / 2 pi times  r g + n d  to x_j (minus that to x_i),
// r d to the normal, and to the Jacobian (d (r.n) - lambda_i q_j log R2 / 2 k)
// / J: 40 FP64 operations and a box test in FP32.
constexpr int AF_ROWS = 64;
__global__ void __launch_bounds__(128) adj_far_kernel(const __grid_constant__ AdjArgs a) {
  __shared__ float4 s_row[AF_ROWS];
  __shared__ double s_x[AF_ROWS], s_y[AF_ROWS], s_l[AF_ROWS], s_T[AF_ROWS];
  const GeomDev& g = a.g;
  const int i0 = blockIdx.y * AF_ROWS, nr = min(AF_ROWS, g.n - i0);
  for (int r = threadIdx.x; r < AF_ROWS; r += blockDim.x) {
    const int i = min(i0 + r, g.n - 1);
    s_row[r] = a.rows[i];
    s_x[r] = g.px[i];
    s_y[r] = g.py[i];
    s_l[r] = a.lam[i];
    s_T[r] = a.T[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = j < g.n;
  const int jc = valid ? j : g.n - 1, e = jc / g.nn;
  const ElemRec E = a.elems[e];
  const double xj = g.px[jc], yj = g.py[jc], nx = g.nx[jc], ny = g.ny[jc], J = g.jac[jc];
  const double Tj = a.T[jc], qk = a.q[jc] / a.k;
  const double c = J * a.R.ew[jc - e * g.nn] / kTwoPi;
  double sx = 0.0, sy = 0.0, tx = 0.0, ty = 0.0, sd = 0.0, sl = 0.0;
  for (int r0 = 0; r0 < nr; r0 += 8) {
    double vx[8], vy[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int r = r0 + q;
      vx[q] = vy[q] = 0.0;
      const float4 rec = s_row[r];
      if (r < nr && valid && box_far(rec.x, rec.y, rec.z, rec.w, E)) {
        const double rx = xj - s_x[r], ry = yj - s_y[r], lam = s_l[r];
        const double R2 = fma(rx, rx, ry * ry), rn = fma(rx, nx, ry * ny);
        const double inv = f64::rcp(R2), m = lam * inv;
        const double d = m * (s_T[r] - Tj);
        const double gm = fma(-2.0 * d, rn * inv, -(qk * m));
        const double gx = fma(rx, gm, nx * d), gy = fma(ry, gm, ny * d);
        sx += gx;
        sy += gy;
        tx = fma(d, rx, tx);
        ty = fma(d, ry, ty);
        sd = fma(d, rn, sd);
        sl = fma(lam, f64::log(R2), sl);
        vx[q] = -c * gx;
        vy[q] = -c * gy;
      }
    }
    const double wx = warp_sum8(vx, lane), wy = warp_sum8(vy, lane);
    const int r = r0 + (lane >> 2);
    if ((lane & 3) < 2 && r < nr) atomicAdd(a.gX + 2 * (i0 + r) + (lane & 3), (lane & 3) ? wy : wx);
  }
  if (valid) {
    atomicAdd(a.gX + 2 * j, c * sx);
    atomicAdd(a.gX + 2 * j + 1, c * sy);
    atomicAdd(a.gn + 2 * j, c * tx);
    atomicAdd(a.gn + 2 * j + 1, c * ty);
    atomicAdd(a.gJ + j, c / J * (sd - 0.5 * qk * sl));
  }
}

// The assembly's candidate pairs by the exact near test: near pairs are
// listed for the difference kernels, the others get their far derivatives.
__global__ void __launch_bounds__(128) adj_pairs_kernel(const __grid_constant__ AdjArgs a) {
  const GeomDev& g = a.g;
  const int nn = g.nn, count = min(*a.ncand, a.ccap);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
    const int2 pr = a.cand[t];
    const int i = pr.x, e = pr.y;
    V2 nodes[BEM_MAXNN];
    for (int kk = 0; kk < nn; ++kk) nodes[kk] = V2{g.px[e * nn + kk], g.py[e * nn + kk]};
    if (near_element(V2{g.px[i], g.py[i]}, nodes, nn, g.elen[e], a.near_factor)) {
      const int slot = atomicAdd(a.count, 1);
      if (slot < a.cap) a.pairs[slot] = pr;
      else a.count[1] = 1;
      continue;
    }
    double gxi = 0.0, gyi = 0.0;
    for (int kk = 0; kk < nn; ++kk) {
      double node5[5] = {0, 0, 0, 0, 0};
      const int j = e * nn + kk;
      far_pair_grad(a, i, j, a.R.ew[kk], gxi, gyi, node5);
      atomicAdd(a.gX + 2 * j, node5[0]);
      atomicAdd(a.gX + 2 * j + 1, node5[1]);
      atomicAdd(a.gn + 2 * j, node5[2]);
      atomicAdd(a.gn + 2 * j + 1, node5[3]);
      atomicAdd(a.gJ + j, node5[4]);
    }
    atomicAdd(a.gX + 2 * i, gxi);
    atomicAdd(a.gX + 2 * i + 1, gyi);
  }
}

// Derivative from S(-h), S(0), S(+h).  The near-field maps switch branch at
// thresholds of the pole position (the reference's tanp3c rules), so the
// discrete integral can jump by its quadrature error inside a step: when the
// one-sided slopes disagree beyond smooth curvature, the jump lies on the
// steeper side and the other side's slope is the derivative.
__device__ __forceinline__ double fd_slope(double sm, double s0, double sp, double h) {
  const double f = (sp - s0) / h, b = (s0 - sm) / h;
  const double d = fabs(f - b);
  if (d <= 1e-3 * fmax(fabs(f), fabs(b)) || d * h <= 1e-13 * fabs(s0)) return 0.5 * (f + b);
  return fabs(f) < fabs(b) ? f : b;
}

// S = sum_k a_k h_k + c_k g_k over the element's nodes for source pf
__device__ double near_value(const AdjArgs& a, int i, int e, const V2* nodes, V2 pf) {
  const GeomDev& g = a.g;
  const int nn = g.nn;
  V2 geo[BEM_MAXGEO];
  double h[BEM_MAXNN], gg[BEM_MAXNN];
  Physics ph{};
  ph.kind = 0;
  ph.k = a.k;
  const V2 nref{g.nx[e * nn], g.ny[e * nn]};
  integrate_near<1>(a.R, ph, nodes, geo, pf, g.elen[e], nref, h, gg);
  double s = 0.0;
  for (int kk = 0; kk < nn; ++kk) {
    const int j = e * nn + kk;
    s += -a.lam[i] * (a.T[j] - a.T[i]) * h[kk] + a.lam[i] * a.q[j] * gg[kk];
  }
  return s;
}

// The near integrals of a pair are wanted at its nodes and source as they
// are (value 0) and with each coordinate c moved by +h (value 2 c + 1) and -h
// (2 c + 2), h = 1e-5 element lengths: c = 0, 1 the source, then the nodes.
__device__ __forceinline__ int near_values(int nn) { return 1 + 2 * (2 + 2 * nn); }

template <int NN>
__device__ __forceinline__ void perturb(int ev, double h, V2& pf, V2* nodes) {
  const int c = (ev - 1) >> 1;
  const double d = ev == 0 ? 0.0 : ((ev & 1) ? h : -h);
  if (ev > 0 && c == 0) pf.x += d;
  if (ev > 0 && c == 1) pf.y += d;
#pragma unroll
  for (int k = 0; k < NN; ++k) {
    if (ev > 0 && c == 2 + 2 * k) nodes[k].x += d;
    if (ev > 0 && c == 3 + 2 * k) nodes[k].y += d;
  }
}

// one value by one thread: the near-field maps other than tanp3c, and the
// pairs that take none of its regular branches
__device__ __noinline__ void near_value_general(const AdjArgs& a, int i, int e, int ev, double* out) {
  const GeomDev& g = a.g;
  V2 nodes[BEM_MAXNN];
  for (int k = 0; k < g.nn; ++k) nodes[k] = V2{g.px[e * g.nn + k], g.py[e * g.nn + k]};
  V2 pf{g.px[i], g.py[i]};
  if (ev > 0) {
    const int c = (ev - 1) >> 1;
    const double d = (ev & 1) ? 1e-5 * g.elen[e] : -1e-5 * g.elen[e];
    if (c == 0) pf.x += d;
    else if (c == 1) pf.y += d;
    else if (c & 1) nodes[(c - 2) >> 1].y += d;
    else nodes[(c - 2) >> 1].x += d;
  }
  *out = near_value(a, i, e, nodes, pf);
}

__global__ void __launch_bounds__(64) adj_near_general_kernel(const __grid_constant__ AdjArgs a) {
  const int ne = near_values(a.g.nn), cnt = min(a.count[0], a.cap);
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (int64_t)cnt * ne;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int2 pr = a.pairs[t / ne];
    near_value_general(a, pr.x, pr.y, (int)(t % ne), a.S + t);
  }
}

// The values by warps, 16 at a time (near_coop.cuh).  One thread per pair
// went through its 17 integrals (quadratic elements) one after another: at
// 1023 nodes 2730 threads, four per scheduler, 4.7 ms; now 46 000 values fill
// the GPU and share their lanes: 0.48 ms.
template <int NN>
__global__ void __launch_bounds__(128) adj_near_kernel(const __grid_constant__ AdjArgs a) {
  using namespace coop;
  __shared__ Slot s_slots[4][PAIRS];
  __shared__ double s_q[BEM_MAXNPG], s_w[BEM_MAXNPG];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const GeomDev& g = a.g;
  const Rules& R = a.R;
  const int nev = near_values(NN);
  const int64_t count = (int64_t)min(a.count[0], a.cap) * nev;
  if (blockIdx.x >= NEAR_CTAS && count <= NEAR_MANY * PAIRS) return;
  for (int q = threadIdx.x; q < R.npg; q += blockDim.x) {
    s_q[q] = R.qsi[q];
    s_w[q] = R.w[q];
  }
  __syncthreads();
  Physics ph{};
  ph.k = a.k;
  const Consts kc = make_consts<1>(ph);
  Slot* slots = s_slots[warp];
  // one task per warp of the first CTAs, the others claimed, as the pairs of
  // an assembly (near_kernel): other gradients of a batch may hold any SMs
  auto claim = [&] {
    int t = 0;
    if (lane == 0) t = atomicAdd(a.count + 2, 1);
    return (int64_t)(4 * NEAR_CTAS + __shfl_sync(FULL, t, 0)) * PAIRS;
  };
  for (int64_t base = blockIdx.x < NEAR_CTAS ? (int64_t)(warp * NEAR_CTAS + (int)blockIdx.x) * PAIRS : claim();
       base < count; base = claim()) {
    const int np = (int)min((int64_t)PAIRS, count - base);
    if (lane < np) {
      const int64_t t = base + lane;
      const int2 pr = a.pairs[t / nev];
      const int i = pr.x, e = pr.y;
      Slot& s = slots[lane];
      V2 nodes[NN];
#pragma unroll
      for (int k = 0; k < NN; ++k) nodes[k] = V2{g.px[e * NN + k], g.py[e * NN + k]};
      V2 pf{g.px[i], g.py[i]};
      perturb<NN>((int)(t % nev), 1e-5 * g.elen[e], pf, nodes);
      s.kind = K_TANGENT;
#pragma unroll
      for (int k = 0; k < NN; ++k) {
        s.cx[k] = nodes[k].x;
        s.cy[k] = nodes[k].y;
      }
      s.sx = pf.x;
      s.sy = pf.y;
      s.nrx = g.nx[e * NN];
      s.nry = g.ny[e * NN];
      complex_pole_1d(R, nodes, NN, pf, s.z0, s.e0);
    }
    __syncwarp();
    map_constants(R, slots, np, lane);
    constexpr int G = 8;
    const int lg = lane & (G - 1);
    for (int p0 = 0; p0 < np; p0 += 32 / G) {
      const int p = p0 + lane / G;
      const bool valid = p < np;
      const Slot& s = slots[valid ? p : 0];
      const int kind = valid ? s.kind : K_NONE;
      double h[NN], gg[NN];
      integrate_group<1, NN, true>(s, kind == K_TANGENT || kind == K_REALPOLE, R.npg, s_q, s_w, R, NN, kc, lg, G, h,
                                   gg);
      // S = sum_k a_k h_k + c_k g_k, this lane's nodes; then over the lanes
      double S = 0.0;
      const int64_t t = base + p;
      int2 pr = make_int2(0, 0);
      if (valid) {
        pr = a.pairs[t / nev];
        const double lam = a.lam[pr.x], Ti = a.T[pr.x];
#pragma unroll
        for (int k = 0; k < NN; ++k) {
          const int j = pr.y * NN + k;
          S += -lam * (a.T[j] - Ti) * h[k] + lam * a.q[j] * gg[k];
        }
      }
      for (int o = G >> 1; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
      if (valid && lg == 0) {
        if (kind == K_GENERAL) near_value_general(a, pr.x, pr.y, (int)(t % nev), a.S + t);
        else a.S[t] = S;
      }
    }
    __syncwarp();
  }
}

// slopes of the near integrals from their values
__global__ void __launch_bounds__(128) adj_near_slope_kernel(const __grid_constant__ AdjArgs a) {
  const int nn = a.g.nn, nev = near_values(nn), nc = 2 + 2 * nn;
  const int64_t count = (int64_t)min(a.count[0], a.cap) * nc;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = t / nc;
    const int c = (int)(t - p * nc);
    const int2 pr = a.pairs[p];
    const double* S = a.S + p * nev;
    const double h = 1e-5 * a.g.elen[pr.y];
    const int at = c < 2 ? 2 * pr.x + c : 2 * (pr.y * nn + ((c - 2) >> 1)) + (c & 1);
    atomicAdd(a.gX + at, fd_slope(S[2 * c + 2], S[0], S[2 * c + 1], h));
  }
}

// On-element integrals, node coordinates perturbed (the source is one of
// them): four lanes per value with the rule's sample weights (singular_table),
// 1 + 4 NN values per node, their differences within the CTA.  The rule run
// step by step by one thread per node, 13 times over, took 2.5 ms at 1023
// quadratic nodes, now 0.06.
template <int NN>
__global__ void __launch_bounds__(128) adj_singular_kernel(const __grid_constant__ AdjArgs a,
                                                           const __grid_constant__ SingularTable<NN> tab) {
  constexpr int NB = 8, NEV = 1 + 4 * NN;  // nodes per CTA, values per node
  __shared__ double s_tab[sizeof(SingularTable<NN>) / 8];
  __shared__ double s_S[NB * NEV];
  for (int q = threadIdx.x; q < (int)(sizeof(tab) / 8); q += blockDim.x) s_tab[q] = ((const double*)&tab)[q];
  __syncthreads();
  const SingularTable<NN>& W = *(const SingularTable<NN>*)s_tab;
  const GeomDev& g = a.g;
  Physics ph{};
  ph.k = a.k;
  const coop::Consts kc = coop::make_consts<1>(ph);
  const int l = threadIdx.x & 3;
  for (int v0 = 0; v0 < NB * NEV; v0 += 32) {
    const int v = v0 + (threadIdx.x >> 2);
    const int vn = min(v / NEV, NB - 1), ev = v - vn * NEV;
    const int i = min((int)blockIdx.x * NB + vn, g.n - 1);
    const int e = i / NN, ai = i - e * NN;
    V2 nodes[NN], pf{0.0, 0.0};
#pragma unroll
    for (int k = 0; k < NN; ++k) nodes[k] = V2{g.px[e * NN + k], g.py[e * NN + k]};
    // node coordinate c as coordinate c + 2 of the near values
    perturb<NN>(ev == 0 ? 0 : ev + 4, 1e-5 * g.elen[e], pf, nodes);
#pragma unroll
    for (int k = 0; k < NN; ++k)
      if (k == ai) pf = nodes[k];
    double X[NN], Y[NN];
#pragma unroll
    for (int k = 0; k < NN; ++k) {
      X[k] = nodes[k].x;
      Y[k] = nodes[k].y;
    }
    const double nrx = g.nx[e * NN], nry = g.ny[e * NN];
    const double lam = a.lam[i], Ti = a.T[i];
    double ch[NN], cg[NN];
#pragma unroll
    for (int k = 0; k < NN; ++k) {
      ch[k] = k == ai ? 0.0 : -lam * (a.T[e * NN + k] - Ti);
      cg[k] = lam * a.q[e * NN + k];
    }
    double S = 0.0;
    for (int q = l; q < BEM_NINTERP; q += 4) {
      double rx, ry, dx, dy;
      coop::nodal_point<NN>(X, Y, W.N[q], W.D[q], pf.x, pf.y, rx, ry, dx, dy);
      const double J2 = fma(dx, dx, dy * dy), R2 = fma(rx, rx, ry * ry);
      if (J2 < 1e-60 || R2 < 1e-60) continue;
      const double flip = dy * nrx - dx * nry < 0 ? -1.0 : 1.0;
      double U, T, wh = 0.0, wg = 0.0;
      coop::kernel_values<1>(kc, rx, ry, flip * dy, -(flip * dx), &U, &T);
#pragma unroll
      for (int k = 0; k < NN; ++k) {
        wh = fma(W.Wh[ai][q][k], ch[k], wh);
        wg = fma(W.Wg[ai][q][k], cg[k], wg);
      }
      S = fma(wh, T, fma(wg, U * f64::sqrt(J2), S));
    }
    S += __shfl_xor_sync(0xffffffffu, S, 1);
    S += __shfl_xor_sync(0xffffffffu, S, 2);
    if (l == 0 && v < NB * NEV) s_S[v] = S;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < NB * 2 * NN; t += blockDim.x) {
    const int vn = t / (2 * NN), c = t - vn * 2 * NN, i = blockIdx.x * NB + vn;
    if (i >= g.n) continue;
    const int e = i / NN;
    const double* S = s_S + vn * NEV;
    atomicAdd(a.gX + 2 * (e * NN + (c >> 1)) + (c & 1), fd_slope(S[2 * c + 2], S[0], S[2 * c + 1], 1e-5 * g.elen[e]));
  }
}

// node normal n = (t_y, -t_x) and Jacobian J = |x'| at node j from
// x'(xi_j) = sum_m D_jm X_m: chain dJ/dn, dJ/dJac to the element's nodes
__global__ void adj_chain_kernel(AdjArgs a) {
  const GeomDev& g = a.g;
  const int nn = g.nn;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= g.ne) return;
  for (int jj = 0; jj < nn; ++jj) {
    const int j = e * nn + jj;
    double da = 0.0, db = 0.0;
    for (int m = 0; m < nn; ++m) {
      da += a.R.leg_D[jj * nn + m] * g.px[e * nn + m];
      db += a.R.leg_D[jj * nn + m] * g.py[e * nn + m];
    }
    const double J = sqrt(da * da + db * db), J3 = J * J * J;
    const double gnx = a.gn[2 * j], gny = a.gn[2 * j + 1], gj = a.gJ[j];
    // n_x = b/J, n_y = -a/J
    const double ga = gj * da / J + gnx * (-da * db / J3) + gny * (-db * db / J3);
    const double gb = gj * db / J + gnx * (da * da / J3) + gny * (da * db / J3);
    for (int m = 0; m < nn; ++m) {
      a.gX[2 * (e * nn + m)] += a.R.leg_D[jj * nn + m] * ga;
      a.gX[2 * (e * nn + m) + 1] += a.R.leg_D[jj * nn + m] * gb;
    }
  }
}

// T, q from the solution u (split_sol, src/Core/Solver.jl:88-98), the
// misfit J and its gradient w.r.t. u
__global__ void adj_split_kernel(int n, const int32_t* BC, const double* BV, const double* u, const double* qt,
                                 double* T, double* q, double* dJdu, double* Jout) {
  __shared__ double s[256];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const bool dir = BC[i] == 0;
    T[i] = dir ? BV[i] : u[i];
    q[i] = dir ? u[i] : BV[i];
    const double r = dir ? u[i] - qt[i] : 0.0;
    dJdu[i] = r;
    acc += 0.5 * r * r;
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *Jout = s[0];
}

__global__ void transpose64(const double* A, int64_t lda, int N, double* At, int64_t ldt) {
  __shared__ double tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = bx + threadIdx.x, j = by + r;
    if (i < N && j < N) tile[r][threadIdx.x] = A[i + (size_t)j * lda];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = by + threadIdx.x, j = bx + r;
    if (i < N && j < N) At[i + (size_t)j * ldt] = tile[threadIdx.x][r];
  }
}

}  // namespace
}  // namespace bem

using namespace bem;

extern "C" int bem_adjoint_laplace2d(bem_ctx* c, const bem_geom2d* g, double k, const int32_t* BC,
                                     const double* BV, const double* q_target, int npg, double near_factor,
                                     double tol, int max_iter, int mem, double* J, double* grad,
                                     bem_solve_stats* stats) {
  if (!c || !g || !BC || !BV || !q_target || !J || !grad) return BEM_ERR_INVALID;
  if (mem != BEM_MEM_HOST && mem != BEM_MEM_DEVICE) return BEM_ERR_INVALID;
  if (!(k > 0) || !(tol > 0) || max_iter < 1) return BEM_ERR_INVALID;
  int rc = bem_check_geom(g, npg, near_factor);
  if (rc) return rc;
  if (g->ngeo != 0 || g->nt != g->n) {
    c->last_error = "adjoint: elements must take their geometry from the nodes (ngeo = 0), no internal points";
    return BEM_ERR_UNSUPPORTED;
  }
  CallScope cs(c);
  cudaSetDevice(c->device);
  const int n = g->n, N = n;
  const int64_t ld = (N + 3) / 4 * 4;
  Physics ph{};
  ph.kind = 0;
  ph.k = k;
  // forward: fused assembly and mixed-precision solve
  double* A = (double*)c->get(bem_ctx::SLOT_OUT0, sizeof(double) * (size_t)ld * N);
  double* At = (double*)c->get(bem_ctx::SLOT_ADJ0, sizeof(double) * (size_t)ld * N);
  // b, u, T, q, dJdu, lambda (n each) | gX, gn (2n each), gJ | J | target, BV, BC (staged inputs)
  double* v = (double*)c->get(bem_ctx::SLOT_ADJ1, sizeof(double) * (size_t)(15 * N + 64));
  if (!A || !At || !v) return BEM_ERR_NOMEM;
  double *b = v, *u = v + N, *T = v + 2 * N, *q = v + 3 * N, *dJdu = v + 4 * N, *lam = v + 5 * N;
  double *gX = v + 7 * N, *gn = v + 9 * N, *gJ = v + 11 * N, *Jd = v + 12 * N;
  double* stg = v + 12 * (size_t)N + 8;
  double* qt = stg;
  const int32_t* dBC = BC;
  const double* dBV = BV;
  if (mem == BEM_MEM_HOST) {
    // target, BV, BC up in one copy through the pinned buffer
    const size_t words = 2 * (size_t)N + ((size_t)N + 1) / 2;
    double* h = (double*)c->pinned(words * sizeof(double));
    if (!h) return BEM_ERR_NOMEM;
    std::memcpy(h, q_target, sizeof(double) * (size_t)N);
    std::memcpy(h + N, BV, sizeof(double) * (size_t)N);
    std::memcpy(h + 2 * (size_t)N, BC, sizeof(int32_t) * (size_t)N);
    cudaMemcpyAsync(stg, h, words * sizeof(double), cudaMemcpyHostToDevice, c->stream);
    c->pin_issued();
    dBV = stg + N;
    dBC = (const int32_t*)(stg + 2 * (size_t)N);
  } else {
    cudaMemcpyAsync(qt, q_target, sizeof(double) * N, cudaMemcpyDeviceToDevice, c->stream);
  }
  const int prec = (c->opt_far_df >= 1) ? 3 : 1;
  bem_solve_stats st{};
  for (int attempt = 0;; ++attempt) {
    // (the solve checks the assembly's pair count; too short a list: again)
    rc = bem_assemble_system_dev(c, g, ph, BC, BV, npg, near_factor, mem, prec, A, ld, nullptr, b,
                                 attempt == 0 && bem_pairs_fit(near_factor));
    if (rc) return rc;
    rc = bem_solve_mixed_dev(c, N, A, ld, b, tol, max_iter, 1, u, &st);
    if (rc != BEM_RETRY) break;
  }
  if (rc != BEM_OK && rc != BEM_ERR_NOT_CONVERGED) return rc;
  adj_split_kernel<<<1, 256, 0, c->stream>>>(n, dBC, dBV, u, qt, T, q, dJdu, Jd);
  // adjoint system A^T lambda = dJ/du
  transpose64<<<dim3((N + 31) / 32, (N + 31) / 32), dim3(32, 8), 0, c->stream>>>(A, ld, N, At, ld);
  count_launches(2);
  bem_solve_stats st2{};
  int rc2 = bem_solve_mixed_dev(c, N, At, ld, dJdu, tol, max_iter, 1, lam, &st2);
  if (rc2 != BEM_OK && rc2 != BEM_ERR_NOT_CONVERGED) return rc2;
  // backward: recompute, never store, the influence entries
  GeomDev gd;
  Rules R;
  rc = bem_stage_geom(c, g, npg, mem, gd, R);
  if (rc) return rc;
  const int cap = 32 * n + 1024;
  const int nev = 1 + 2 * (2 + 2 * gd.nn);
  // near pairs and their values; the candidates and records are the assembly's
  char* np = (char*)c->get(bem_ctx::SLOT_ADJ2, (sizeof(double) * nev + sizeof(int2)) * (size_t)cap);
  int* cnt = (int*)c->get(bem_ctx::SLOT_COUNTERS, 64) + 4;
  if (!np || !cnt) return BEM_ERR_NOMEM;
  cudaMemsetAsync(cnt, 0, 3 * sizeof(int), c->stream);
  cudaMemsetAsync(gX, 0, sizeof(double) * 5 * (size_t)N, c->stream);
  AdjArgs aa{};
  aa.g = gd;
  aa.R = R;
  aa.k = k;
  aa.near_factor = near_factor;
  aa.lam = lam;
  aa.T = T;
  aa.q = q;
  aa.gX = gX;
  aa.gn = gn;
  aa.gJ = gJ;
  aa.rows = (const float4*)c->slots[bem_ctx::SLOT_ROWS].p;
  aa.elems = (const ElemRec*)c->slots[bem_ctx::SLOT_ELEMS].p;
  aa.cand = (const int2*)c->slots[bem_ctx::SLOT_PAIRS].p;
  aa.ncand = cnt - 4;
  aa.ccap = (int)std::min<size_t>(c->slots[bem_ctx::SLOT_PAIRS].bytes / sizeof(int2), 0x7fffffff);
  aa.S = (double*)np;
  aa.pairs = (int2*)(np + sizeof(double) * nev * (size_t)cap);
  aa.count = cnt;
  aa.cap = cap;
  adj_pairs_kernel<<<std::min((8 * n + 127) / 128, 152 * 16), 128, 0, c->stream>>>(aa);
  adj_far_kernel<<<dim3((n + 127) / 128, (n + AF_ROWS - 1) / AF_ROWS), 128, 0, c->stream>>>(aa);
  if (R.nearfield != 0) {
    adj_near_general_kernel<<<4096, 64, 0, c->stream>>>(aa);
  } else {
    switch (gd.nn) {
      case 2: adj_near_kernel<2><<<near_ctas(near_factor), 128, 0, c->stream>>>(aa); break;
      case 3: adj_near_kernel<3><<<near_ctas(near_factor), 128, 0, c->stream>>>(aa); break;
      case 4: adj_near_kernel<4><<<near_ctas(near_factor), 128, 0, c->stream>>>(aa); break;
      case 5: adj_near_kernel<5><<<near_ctas(near_factor), 128, 0, c->stream>>>(aa); break;
      case 6: adj_near_kernel<6><<<near_ctas(near_factor), 128, 0, c->stream>>>(aa); break;
    }
  }
  adj_near_slope_kernel<<<std::min((16 * n + 127) / 128, 152 * 16), 128, 0, c->stream>>>(aa);
  switch (gd.nn) {
    case 2: adj_singular_kernel<2><<<(n + 7) / 8, 128, 0, c->stream>>>(aa, singular_table<2>(R)); break;
    case 3: adj_singular_kernel<3><<<(n + 7) / 8, 128, 0, c->stream>>>(aa, singular_table<3>(R)); break;
    case 4: adj_singular_kernel<4><<<(n + 7) / 8, 128, 0, c->stream>>>(aa, singular_table<4>(R)); break;
    case 5: adj_singular_kernel<5><<<(n + 7) / 8, 128, 0, c->stream>>>(aa, singular_table<5>(R)); break;
    case 6: adj_singular_kernel<6><<<(n + 7) / 8, 128, 0, c->stream>>>(aa, singular_table<6>(R)); break;
  }
  adj_chain_kernel<<<(g->ne + 127) / 128, 128, 0, c->stream>>>(aa);
  count_launches(6);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->cuda_fail(e, "adjoint kernels");
  // gradient, J and the pair counters back through the pinned buffer
  double* hout = (double*)c->pinned(sizeof(double) * (2 * (size_t)N + 2));
  if (!hout) return BEM_ERR_NOMEM;
  const int* hc = (const int*)(hout + 2 * (size_t)N + 1);
  cudaMemcpyAsync(hout + 2 * (size_t)N + 1, cnt, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream);
  if (mem == BEM_MEM_HOST) {
    cudaMemcpyAsync(hout, gX, sizeof(double) * 2 * (size_t)N, cudaMemcpyDeviceToHost, c->stream);
    cudaMemcpyAsync(hout + 2 * (size_t)N, Jd, sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  } else {
    cudaMemcpyAsync(grad, gX, sizeof(double) * 2 * (size_t)N, cudaMemcpyDeviceToDevice, c->stream);
    cudaMemcpyAsync(J, Jd, sizeof(double), cudaMemcpyDeviceToDevice, c->stream);
  }
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->cuda_fail(e, "adjoint");
  if (mem == BEM_MEM_HOST) {
    std::memcpy(grad, hout, sizeof(double) * 2 * (size_t)N);
    *J = hout[2 * (size_t)N];
  }
  if (hc[1] != 0) {
    c->last_error = "adjoint: near-pair list overflow";
    return BEM_ERR_INTERNAL;
  }
  if (stats) {
    *stats = st;
    stats->iterations += st2.iterations;
  }
  return (rc == BEM_ERR_NOT_CONVERGED || rc2 == BEM_ERR_NOT_CONVERGED) ? BEM_ERR_NOT_CONVERGED : BEM_OK;
}
