// Laplace potential at interior points from the solved boundary data,
// restating `interior_laplace` (src/Laplace/Lubrication.jl:399-416; the
// same sum is `_interior_T`, test/laplace.jl:36-53):
//   h_j, g_j = integrate_element over every element (closest point, then the
//              on-element Guiggiani rule if the point lies on the element,
//              else the near-field quadrature, Assembly_full.jl:262-289)
//   c = -sum_j h_j,   T(p) = (g . q - h . T) / c.
// One CTA per point; its threads take elements (and rule nodes) in a fixed
// order and the FP64 partial sums are reduced in a fixed tree, so results are
// reproducible.
//
// Most elements are far from a point, in units of their own size, and there
// the npg-point Gauss rule gives the integral to rounding, as the near-field
// map's rule with many points does; the map costs 27 000 FP64 operations a
// pair, the Gauss nodes, whose positions, weights and boundary data can be
// prepared per element, 24 each.  Which pairs those are is decided by a bound,
// not by a distance alone: with the element's geometry x(t) = x(0) + sum c_d t^d, if
//   |p - x(0)| > sum_{d >= 1} |c_d| a^d   and   |c_1| > sum_{d >= 2} d |c_d| a^(d-1)
// then log r, 1/r^2 and |x'| are analytic in the Bernstein ellipse of semi-axis
// a = (rho + 1/rho) / 2, where the field basis of degree p grows to about
// rho^p, and the Gauss error is about rho^(p - 2 npg); rho is the one that
// makes it 2^-60.  Against 64-point rules, at the edge of the bound, straight
// and curved elements of degree 1 to 5, 8 to 32 points: within 1e-14 of the
// largest integral, which is the sums' rounding (the map with 8 points: 3e-11).
// (npg >= 8 only: with fewer points the ellipse is so large that little is
// gained.)  The other pairs take the map, by warps (near_coop.cuh).  1000
// points and 341 quadratic elements: the call 15.7 -> 0.40 ms.
#include <cmath>
#include <cstring>

#include "bem_abi_internal.h"
#include "near_coop.cuh"

namespace bem {
namespace {

constexpr int IT = 128;  // threads per point
constexpr int IC = 256;  // elements per round

struct InteriorArgs {
  GeomDev g;
  Rules R;
  Physics ph;
  const double *T, *q, *xp, *yp;
  double* out;
  double a;  // semi-axis of the far rule's ellipse; 0: no far pairs
  // per element: x(0), y(0), squared reach; per element and rule node: point,
  // w times the normal of length J, and w times the interpolated T and w J
  // times the interpolated q
  double *ex, *ey, *er;
  double *nx, *ny, *nu, *nv, *nT, *nq;
};

// h . T, g . q and sum h of one pair by one thread, any option
__device__ __noinline__ void interior_pair(const InteriorArgs& a, V2 pf, int e, double& gt, double& hs) {
  const GeomDev& g = a.g;
  const int nn = g.nn;
  V2 nodes[BEM_MAXNN], geo[BEM_MAXGEO];
  load_element(g, e, nodes, geo);
  double h[BEM_MAXNN], gg[BEM_MAXNN];
  double xa, dist;
  closest_point_1d(a.R, nodes, nn, pf, xa, dist);
  const V2 nref{g.nx[e * nn], g.ny[e * nn]};
  if (dist <= 1e-12) {
    if (a.R.singular == 1)
      integrate_singular_telles<1>(a.R, a.ph, nodes, geo, pf, xa, nref, h, gg);
    else
      integrate_singular<1>(a.R, a.ph, nodes, geo, pf, xa, nref, h, gg);
  } else {
    integrate_near<1>(a.R, a.ph, nodes, geo, pf, g.elen[e], nref, h, gg);
  }
  for (int k = 0; k < nn; ++k) {
    const int j = e * nn + k;
    gt += gg[k] * a.q[j] - h[k] * a.T[j];
    hs += h[k];
  }
}

// fixed-order sums over the CTA and T(p) = (g . q - h . T) / c
__device__ __forceinline__ void interior_finish(double gt, double hs, double* out) {
  __shared__ double s_gt[IT / 32], s_h[IT / 32];
  for (int o = 16; o > 0; o >>= 1) {
    gt += __shfl_xor_sync(0xffffffffu, gt, o);
    hs += __shfl_xor_sync(0xffffffffu, hs, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_gt[threadIdx.x >> 5] = gt;
    s_h[threadIdx.x >> 5] = hs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < IT / 32; ++w) {
      a += s_gt[w];
      b += s_h[w];
    }
    *out = a / (-b);
  }
}

// near-field maps other than tanp3c, and no memory for the far rule: every
// pair by one thread
__global__ void __launch_bounds__(IT) interior_general_kernel(const __grid_constant__ InteriorArgs a) {
  const V2 pf{a.xp[blockIdx.x], a.yp[blockIdx.x]};
  double gt = 0.0, hs = 0.0;
  for (int e = threadIdx.x; e < a.g.ne; e += IT) interior_pair(a, pf, e, gt, hs);
  interior_finish(gt, hs, a.out + blockIdx.x);
}

// per-element data of the far rule, one thread per (element, rule node)
__global__ void __launch_bounds__(128) interior_setup_kernel(const __grid_constant__ InteriorArgs a) {
  const GeomDev& g = a.g;
  const Rules& R = a.R;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.ne * R.npg) return;
  const int e = t / R.npg, q = t - e * R.npg;
  V2 nodes[BEM_MAXNN], geo[BEM_MAXGEO];
  load_element(g, e, nodes, geo);
  coop::Slot s;
  // about the first node, to keep the coefficients free of the position
  const V2 o = nodes[0];
  coop::geometry(R, nodes, geo, o, s);
  const int ng = R.ngeo > 0 ? R.ngeo : R.nn;
  auto point = [&](double xi, double& x, double& y, double& dx, double& dy) {
    x = s.cx[ng - 1];
    y = s.cy[ng - 1];
    dx = dy = 0.0;
    for (int d = ng - 2; d >= 0; --d) {
      dx = fma(dx, xi, x);
      dy = fma(dy, xi, y);
      x = fma(x, xi, s.cx[d]);
      y = fma(y, xi, s.cy[d]);
    }
  };
  double x, y, dx, dy, N[BEM_MAXNN];
  point(R.qsi[0], x, y, dx, dy);
  const double flip = dy * g.nx[e * g.nn] - dx * g.ny[e * g.nn] < 0 ? -1.0 : 1.0;
  point(R.qsi[q], x, y, dx, dy);
  const double w = R.w[q];
  shapefun_prod(R.leg_x, R.leg_pw, R.leg_D, g.nn, R.qsi[q], N, nullptr);
  double Tq = 0.0, qq = 0.0;
  for (int k = 0; k < g.nn; ++k) {
    Tq += N[k] * a.T[e * g.nn + k];
    qq += N[k] * a.q[e * g.nn + k];
  }
  a.nx[t] = o.x + x;
  a.ny[t] = o.y + y;
  a.nu[t] = flip * dy * w;
  a.nv[t] = -(flip * dx * w);
  a.nT[t] = Tq;
  a.nq[t] = qq * w * sqrt(dx * dx + dy * dy);
  if (q == 0) {
    double reach = 0.0, bend = 0.0, p = 1.0, c1 = 0.0;
    for (int d = 1; d < ng; ++d) {
      const double c = sqrt(s.cx[d] * s.cx[d] + s.cy[d] * s.cy[d]);
      if (d == 1) c1 = c;
      else bend += d * c * p;
      p *= a.a;
      reach += c * p;
    }
    a.ex[e] = o.x + s.cx[0];
    a.ey[e] = o.y + s.cy[0];
    a.er[e] = a.a > 0 && c1 > bend ? reach * reach * (1 + 1e-12) : INFINITY;
  }
}

template <int NN>
__global__ void __launch_bounds__(IT) interior_laplace_kernel(const __grid_constant__ InteriorArgs a) {
  using namespace coop;
  __shared__ Slot s_slots[IT / 32][PAIRS];
  __shared__ double s_q[BEM_MAXNPG], s_w[BEM_MAXNPG];
  __shared__ unsigned char s_far[IC];
  __shared__ int s_list[IC], s_cnt[IC / 32 + 1];
  const GeomDev& g = a.g;
  const Rules& R = a.R;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const V2 pf{a.xp[blockIdx.x], a.yp[blockIdx.x]};
  const int npg = R.npg, ng = R.ngeo > 0 ? R.ngeo : NN;
  for (int q = t; q < npg; q += IT) {
    s_q[q] = R.qsi[q];
    s_w[q] = R.w[q];
  }
  const Consts kc = make_consts<1>(a.ph);
  double gt = 0.0, hs = 0.0;
  for (int e0 = 0; e0 < g.ne; e0 += IC) {
    const int nel = min(IC, g.ne - e0);
    // far elements, and the list of the others in element order
    unsigned masks[IC / IT];
#pragma unroll
    for (int r = 0; r < IC / IT; ++r) {
      const int el = r * IT + t;
      bool near = false;
      if (el < nel) {
        const double dx = pf.x - a.ex[e0 + el], dy = pf.y - a.ey[e0 + el];
        near = !(fma(dx, dx, dy * dy) > a.er[e0 + el]);
        s_far[el] = !near;
      }
      masks[r] = __ballot_sync(FULL, near);
      if (lane == 0) s_cnt[r * (IT / 32) + warp] = __popc(masks[r]);
    }
    __syncthreads();
    int cnt = 0;
#pragma unroll
    for (int b = 0; b < IC / 32; ++b) {
#pragma unroll
      for (int r = 0; r < IC / IT; ++r)
        if (b == r * (IT / 32) + warp && (masks[r] >> lane & 1u))
          s_list[cnt + __popc(masks[r] & ((1u << lane) - 1))] = e0 + r * IT + t;
      cnt += s_cnt[b];
    }
    __syncthreads();
    const size_t base = (size_t)e0 * npg;
    for (int v = t; v < nel * npg; v += IT) {
      if (!s_far[v / npg]) continue;
      const double rx = a.nx[base + v] - pf.x, ry = a.ny[base + v] - pf.y;
      const double R2 = fma(rx, rx, ry * ry);
      const double T = f64::div(fma(rx, a.nu[base + v], ry * a.nv[base + v]), R2);
      gt = fma(kc.cU * f64::log(R2), a.nq[base + v], gt);
      gt = fma(-(kc.cT * T), a.nT[base + v], gt);
      hs = fma(kc.cT, T, hs);
    }
    // the listed pairs by warps
    const int per = max(1, min(PAIRS, (cnt + IT / 32 - 1) / (IT / 32)));
    const int G = per == 1 ? 32 : (per == 2 ? 16 : 8), lg = lane & (G - 1);
    Slot* slots = s_slots[warp];
    for (int b0 = warp * per; b0 < cnt; b0 += per * (IT / 32)) {
      const int np = min(per, cnt - b0);
      if (lane < np) {
        const int e = s_list[b0 + lane];
        Slot& s = slots[lane];
        V2 nodes[NN], geo[BEM_MAXGEO];
#pragma unroll
        for (int k = 0; k < NN; ++k) nodes[k] = V2{g.px[e * NN + k], g.py[e * NN + k]};
        for (int k = 0; k < g.ngeo; ++k) geo[k] = V2{g.gx[e * g.ngeo + k], g.gy[e * g.ngeo + k]};
        geometry(R, nodes, geo, pf, s);
        s.id = e;
        s.np = 1;
        s.nrx = g.nx[e * NN];
        s.nry = g.ny[e * NN];
        // a point on the element lies within its own reach of x(0) (the
        // margin covers a field interpolant that is not the geometry)
        double own = 0.0;
        for (int d = 1; d < ng; ++d) own += sqrt(s.cx[d] * s.cx[d] + s.cy[d] * s.cy[d]);
        bool on = false;
        if (s.cx[0] * s.cx[0] + s.cy[0] * s.cy[0] <= 1.21 * own * own) {
          double xa, dist;
          closest_point_1d(R, nodes, NN, pf, xa, dist);
          on = dist <= 1e-12;
        }
        s.kind = on ? K_GENERAL : K_TANGENT;
        if (!on) complex_pole_1d(R, nodes, NN, pf, s.z0, s.e0);
      }
      __syncwarp();
      map_constants(R, slots, np, lane);
      for (int p0 = 0; p0 < np; p0 += 32 / G) {
        const int p = p0 + lane / G;
        const bool valid = p < np;
        const Slot& s = slots[valid ? p : 0];
        const int kind = valid ? s.kind : K_NONE;
        double h[NN], gg[NN];
        integrate_group<1, NN>(s, kind == K_TANGENT || kind == K_REALPOLE, npg, s_q, s_w, R, ng, kc, lg, G, h, gg);
        if (valid) {
#pragma unroll
          for (int k = 0; k < NN; ++k) {
            const int j = s.id * NN + k;
            gt += gg[k] * a.q[j] - h[k] * a.T[j];
            hs += h[k];
          }
          if (kind == K_GENERAL && lg == 0) interior_pair(a, pf, s.id, gt, hs);
        }
      }
      __syncwarp();
    }
    __syncthreads();
  }
  interior_finish(gt, hs, a.out + blockIdx.x);
}

}  // namespace
}  // namespace bem

using namespace bem;

extern "C" int bem_interior_laplace2d(bem_ctx* c, const bem_geom2d* g, double k, int npg, const double* T,
                                      const double* q, int64_t m, const double* xp, const double* yp,
                                      int mem, double* out) {
  if (!c || !g || !T || !q || m < 0 || (m > 0 && (!xp || !yp || !out))) return BEM_ERR_INVALID;
  if (mem != BEM_MEM_HOST && mem != BEM_MEM_DEVICE) return BEM_ERR_INVALID;
  if (!(k > 0)) return BEM_ERR_INVALID;
  if (m > (int64_t)0x7fffffff) return BEM_ERR_UNSUPPORTED;
  int rc = bem_check_geom(g, npg, 1.5);
  if (rc) return rc;
  if (m == 0) return BEM_OK;
  CallScope cs(c);
  cudaSetDevice(c->device);
  GeomDev gd;
  Rules R;
  rc = bem_stage_geom(c, g, npg, mem, gd, R);
  if (rc) return rc;
  Physics ph{};
  ph.kind = 0;
  ph.k = k;
  const size_t n = (size_t)g->n, mm = (size_t)m;
  const double *dT = T, *dq = q, *dx = xp, *dy = yp;
  double* dout = out;
  if (mem == BEM_MEM_HOST) {
    double* buf = (double*)c->get(bem_ctx::SLOT_OUT3, sizeof(double) * (2 * n + 3 * mm));
    if (!buf) return BEM_ERR_NOMEM;
    cudaMemcpyAsync(buf, T, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(buf + n, q, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(buf + 2 * n, xp, sizeof(double) * mm, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(buf + 2 * n + mm, yp, sizeof(double) * mm, cudaMemcpyHostToDevice, c->stream);
    dT = buf;
    dq = buf + n;
    dx = buf + 2 * n;
    dy = buf + 2 * n + mm;
    dout = buf + 2 * n + 2 * mm;
  }
  InteriorArgs ia{};
  ia.g = gd;
  ia.R = R;
  ia.ph = ph;
  ia.T = dT;
  ia.q = dq;
  ia.xp = dx;
  ia.yp = dy;
  ia.out = dout;
  // 48 bytes per element and rule node for the far rule; without them (no
  // memory left, or more than 2^30 nodes) every pair takes the map
  const size_t ne = (size_t)gd.ne, nr = ne * (size_t)npg;
  double* rec = nullptr;
  if (R.nearfield == 0 && nr <= (size_t)1 << 30)
    rec = (double*)c->get(bem_ctx::SLOT_OUT2, sizeof(double) * (3 * ne + 6 * nr));
  if (!rec) {
    interior_general_kernel<<<(unsigned)m, IT, 0, c->stream>>>(ia);
    count_launches(1);
  } else {
    const double rho = std::exp2(60.0 / (2.0 * npg - (gd.nn - 1)));
    ia.a = npg >= 8 ? 0.5 * (rho + 1.0 / rho) : 0.0;
    ia.ex = rec;
    ia.ey = rec + ne;
    ia.er = rec + 2 * ne;
    double** f[] = {&ia.nx, &ia.ny, &ia.nu, &ia.nv, &ia.nT, &ia.nq};
    for (int k = 0; k < 6; ++k) *f[k] = rec + 3 * ne + k * nr;
    interior_setup_kernel<<<(unsigned)((nr + 127) / 128), 128, 0, c->stream>>>(ia);
    switch (gd.nn) {
      case 2: interior_laplace_kernel<2><<<(unsigned)m, IT, 0, c->stream>>>(ia); break;
      case 3: interior_laplace_kernel<3><<<(unsigned)m, IT, 0, c->stream>>>(ia); break;
      case 4: interior_laplace_kernel<4><<<(unsigned)m, IT, 0, c->stream>>>(ia); break;
      case 5: interior_laplace_kernel<5><<<(unsigned)m, IT, 0, c->stream>>>(ia); break;
      case 6: interior_laplace_kernel<6><<<(unsigned)m, IT, 0, c->stream>>>(ia); break;
    }
    count_launches(2);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return c->cuda_fail(e, "interior_laplace_kernel");
  if (mem == BEM_MEM_HOST) cudaMemcpyAsync(out, dout, sizeof(double) * mm, cudaMemcpyDeviceToHost, c->stream);
  e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return c->cuda_fail(e, "interior_laplace");
  return BEM_OK;
}
