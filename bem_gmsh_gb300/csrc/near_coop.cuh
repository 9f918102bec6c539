// Near-singular element integrals by a warp (tanp3c rule, FP64).
//
// A (point, element) pair costs some 1400 FP64 operations for its map (pole,
// two arctangents, Newton for each half's p3c pole) and about 130 for each of
// its npg or 2 npg nodes.  A warp's FP64 instruction takes 64 cycles however
// few lanes it serves, so one thread per pair is slow twice over: a small
// mesh runs one pair's whole chain (700 us for 20-point rules), and the lanes
// of a warp wait for its longest pair.  Here a warp takes up to 16 pairs:
//   setup   one lane per pair: pole, element geometry as a polynomial about
//           the source point (Horner instead of Lagrange sums at each node,
//           and the difference to the source without cancellation);
//   map     two lanes per pair: one arctangent each, then one half's p3c
//           pole each;
//   nodes   8 lanes per pair (16 or 32 when the warp has only two pairs or
//           one), each lane every 8th node, sums by shuffles.
// Measured (device time, one pass): 160 linear nodes, 20-point rules 711 ->
// 54 us; N = 8193, 16-point rules 538 -> 298 us (then FP64 issue bound).
// The map's nodes and weights are the bits of nm::tanp3ctrans: the same IEEE
// operations in the same order (what does not depend on the node is done
// once).  The normal is not normalised: T J = (r . J n) / R^2 needs no
// Jacobian, only U J does.
#pragma once
#include "bem_device.cuh"
#include "fast64.cuh"

namespace bem {
namespace coop {

constexpr int PAIRS = 16;  // most pairs of a warp
constexpr unsigned FULL = 0xffffffffu;

enum Kind { K_NONE = 0, K_TANGENT = 1, K_REALPOLE = 2, K_GENERAL = 3, K_FAR = 4 };

// one pair's data in shared memory
struct Slot {
  double z0, e0, At, Bt, e0At;
  double A[2], B[2], zt[2], et2[2], mid[2], h[2];  // per half
  double cx[BEM_MAXGEO], cy[BEM_MAXGEO];           // geometry - source, coefficients of xi^d (NODAL: the nodes)
  double sx, sy;                                   // NODAL: the source
  double nrx, nry;                                 // normal of the element's first node
  int kind, np, chart, id;
};

// kernel constants
struct Consts {
  double cU, cL, cT, c;
};
template <int NC>
__device__ __forceinline__ Consts make_consts(const Physics& ph) {
  Consts k;
  if constexpr (NC == 1) {
    k.cU = -(0.5 * (1.0 / (2 * kPi)) / ph.k);  // G = cU log R2
    k.cT = 1.0 / (2 * kPi);                    // H = cT (r.n) / R2
    k.cL = k.c = 0.0;
  } else {
    const double prod1 = 4 * kPi * (1 - ph.nu);
    k.cU = 1.0 / (2 * prod1 * ph.mu);
    k.cL = -0.5 * (3 - 4 * ph.nu);
    k.cT = -1.0 / prod1;
    k.c = 1 - 2 * ph.nu;
  }
  return k;
}

// U and T of the pair at distance r, T times the length of the normal n
template <int NC>
__device__ __forceinline__ void kernel_values(const Consts& k, double rx, double ry, double nx, double ny,
                                              double* U, double* T) {
  const double R2 = fma(rx, rx, ry * ry);
  const double rn = fma(rx, nx, ry * ny);
  const double lg = f64::log(R2);
  if constexpr (NC == 1) {
    U[0] = k.cU * lg;
    T[0] = k.cT * f64::div(rn, R2);
  } else {
    const double inv = f64::rcp(R2);
    const double xi = rx * inv, yi = ry * inv;
    const double qxx = rx * xi, qxy = rx * yi, qyy = ry * yi;
    const double ul = k.cL * lg;
    U[0] = k.cU * (ul + qxx);
    U[1] = U[2] = k.cU * qxy;
    U[3] = k.cU * (ul + qyy);
    const double t = k.cT * (rn * inv);
    T[0] = t * fma(2.0, qxx, k.c);
    T[3] = t * fma(2.0, qyy, k.c);
    const double s = 2.0 * (t * qxy), w = k.cT * k.c * fma(xi, ny, -(yi * nx));
    T[1] = s - w;
    T[2] = s + w;
  }
}

// The geometry polynomial of an element about the source point.
__device__ __forceinline__ void geometry(const Rules& R, const V2* nodes, const V2* geo, V2 pf, Slot& s) {
  const int ng = R.ngeo > 0 ? R.ngeo : R.nn;
  const double* M = R.ngeo > 0 ? R.geo_mono : R.leg_mono;
  const V2* X = R.ngeo > 0 ? geo : nodes;
  double cx[BEM_MAXGEO], cy[BEM_MAXGEO];
#pragma unroll
  for (int d = 0; d < BEM_MAXGEO; ++d) cx[d] = cy[d] = 0.0;
  for (int k = 0; k < ng; ++k) {
    const double dx = X[k].x - pf.x, dy = X[k].y - pf.y;
#pragma unroll
    for (int d = 0; d < BEM_MAXGEO; ++d) {
      if (d < ng) {
        const double m = M[k * BEM_MAXGEO + d];
        cx[d] = fma(m, dx, cx[d]);
        cy[d] = fma(m, dy, cy[d]);
      }
    }
  }
#pragma unroll
  for (int d = 0; d < BEM_MAXGEO; ++d) {
    s.cx[d] = cx[d];
    s.cy[d] = cy[d];
  }
}

// The map of the warp's pairs [0, np) (slots with kind K_TANGENT and pole z0,
// e0 set), all 32 lanes: nm::tanp3ctrans's cases and constants.  Lane 2 i + s
// works on pair i, s = 0 the left half and arctangent of 1 - z0, s = 1 the right.
__device__ __forceinline__ void map_constants(const Rules& R, Slot* slots, int np, int lane) {
  using nm::ieee;
  const int i = lane >> 1, side = lane & 1;
  Slot& s = slots[i < np ? i : 0];
  const bool on = i < np && s.kind == K_TANGENT;
  const ieee z0 = s.z0;
  ieee e0 = s.e0;
  int kind = on ? K_TANGENT : K_NONE;
  if (on && nm::eq41_collinear(z0, e0, false, ieee(0.0))) kind = K_REALPOLE;
  e0 = max(e0, ieee(1e-14));
  double at = 0.0;
  if (kind == K_TANGENT) at = crm::cr_atan(((side == 0 ? ieee(1.0) - z0 : ieee(1.0) + z0) / e0).v);
  const double other = __shfl_xor_sync(FULL, at, 1);
  const ieee ap = side == 0 ? at : other, am = side == 0 ? other : at;
  const ieee den = ap + am;
  if (kind == K_TANGENT) {
    if (nm::eq41_collinear(z0, e0, true, den)) kind = K_REALPOLE;
    else if (abs(den) < ieee(1e-30)) kind = K_GENERAL;
  }
  ieee At, Bt, spole, mid, h;
  bool present = false, chart = false;
  if (kind == K_TANGENT) {
    At = ieee(2.0) / den;
    Bt = -At * (ap - am) / ieee(2.0);
    const ieee uL = Bt - At * ieee(3.141592653589793) / ieee(2.0);
    const ieee uR = Bt + At * ieee(3.141592653589793) / ieee(2.0);
    chart = abs(z0) < ieee(1.0) && ieee(-1.0) < Bt && Bt < ieee(1.0);
    if (chart) {
      const ieee lo = side == 0 ? ieee(-1.0) : Bt, hi = side == 0 ? Bt : ieee(1.0);
      mid = (hi + lo) / ieee(2.0);
      h = (hi - lo) / ieee(2.0);
      present = h > ieee(1e-14);
      if (present) spole = ((side == 0 ? uL : uR) - mid) / h;
    } else {
      present = side == 0;
      mid = 0.0;
      h = 1.0;
      spole = z0 >= ieee(1.0) ? uL : uR;
    }
  }
  ieee A, B, zt, et;
  if (present) {
    nm::p3c_inv_pole_refine(spole, ieee(1e-14), R.p3c_e, R.p3c_cb, zt, et);
    const ieee dn = ieee(1.0) + ieee(3.0) * (zt * zt) + ieee(3.0) * (et * et);
    A = ieee(3.0) / dn;
    B = (ieee(3.0) + zt * zt) * zt / dn;
  }
  const unsigned have = __ballot_sync(FULL, present);
  if (on) {
    const unsigned mine = (have >> (2 * i)) & 3u;  // the halves present
    if (side == 0) {
      s.kind = kind;
      s.e0 = e0.v;
      s.np = kind == K_TANGENT ? __popc(mine) : 1;
      s.chart = chart;
      if (kind == K_TANGENT) {
        s.At = At.v;
        s.Bt = Bt.v;
        s.e0At = (e0 / At).v;
      }
    }
    if (present) {
      const int q = (side == 1 && (mine & 1u)) ? 1 : 0;  // the order of tanp3ctrans
      s.A[q] = A.v;
      s.B[q] = B.v;
      s.zt[q] = zt.v;
      s.et2[q] = (et * et).v;
      s.mid[q] = mid.v;
      s.h[q] = h.v;
    }
  }
  __syncwarp();
}

// node q of piece k of a slot's rule: parent coordinate and weight
__device__ __forceinline__ void rule_node(const Slot& s, int k, double qsi, double w, double& xi, double& wx) {
  using nm::ieee;
  const ieee z0 = s.z0;
  if (s.kind == K_REALPOLE) {
    xi = qsi;
    wx = w;
    if (!(abs(z0) <= ieee(1.0))) {
      const ieee A = z0 * z0 - ieee(1.0), d = ieee(qsi) - (-z0);
      xi = (z0 - A / d).v;
      wx = (ieee(w) * (A / (d * d))).v;
    }
    return;
  }
  const ieee ds = ieee(qsi) - ieee(s.zt[k]);
  const ieee d2 = ds * ds, d3 = d2 * ds;
  // d3 / 3 correctly rounded: the quotient by the rounded third and its
  // remainder (Markstein; exact for a divisor whose reciprocal is rounded)
  const double third = 0.33333333333333331;
  const double q0 = crm::mul(d3.v, third);
  const ieee d33 = crm::fmaf_(crm::fmaf_(-3.0, q0, d3.v), third, q0);
  ieee ut = ieee(s.A[k]) * (d33 + ieee(s.et2[k]) * ieee(qsi)) + ieee(s.B[k]);
  ieee ws = ieee(w) * (ieee(s.A[k]) * (d2 + ieee(s.et2[k])));
  if (s.chart) {
    ut = ieee(s.mid[k]) + ieee(s.h[k]) * ut;
    ws = ws * ieee(s.h[k]);
  }
  const ieee halfpi = ieee(3.141592653589793) / ieee(2.0) - ieee(1e-8);
  const ieee th = clamp((ut - ieee(s.Bt)) / ieee(s.At), -halfpi, halfpi);
  const ieee tn = crm::cr_tan(th.v);
  xi = (z0 + ieee(s.e0) * tn).v;
  wx = (ws * (ieee(s.e0At) * (ieee(1.0) + tn * tn))).v;
}

// field basis at xi in product form
template <int NN>
__device__ __forceinline__ void basis(const double* x, const double* pw, double xi, double* N) {
  double d[NN];
#pragma unroll
  for (int i = 0; i < NN; ++i) d[i] = xi - x[i];
  double pre = 1.0;
#pragma unroll
  for (int i = 0; i < NN; ++i) {
    N[i] = i == 0 ? pw[0] : pw[i] * pre;
    pre = i == 0 ? d[0] : pre * d[i];
  }
  double suf = d[NN - 1];
#pragma unroll
  for (int i = NN - 2; i >= 0; --i) {
    N[i] *= suf;
    suf *= d[i];
  }
}

// Point (relative to the source) and tangent at the parent coordinate of
// node interpolation weights N by Lagrange sums over absolute coordinates, in
// the order of shape_geom.
template <int NN>
__device__ __forceinline__ void nodal_point(const double* X, const double* Y, const double* N, const double* dN,
                                            double sx, double sy, double& px, double& py, double& dx, double& dy) {
  px = N[0] * X[0];
  py = N[0] * Y[0];
  dx = dN[0] * X[0];
  dy = dN[0] * Y[0];
#pragma unroll
  for (int k = 1; k < NN; ++k) {
    px = fma(N[k], X[k], px);
    py = fma(N[k], Y[k], py);
    dx = fma(dN[k], X[k], dx);
    dy = fma(dN[k], Y[k], dy);
  }
  px -= sx;
  py -= sy;
}

// Sums over the rule of a slot of N_k T J w (h) and N_k U J w (g) by the
// lanes lg = 0 .. G-1 of a group of G lanes (every lane of the warp calls
// this with its own group's slot; `on` false: no work).  qs, ws: the Gauss
// rule in shared memory.  NODAL: the element's nodes are its geometry and are
// summed in absolute coordinates (nodal_point), for callers that difference
// the integrals: the rounding of the coordinates, 2^-53 of their size and not
// of the element's, then stays the one of the step-by-step rule.
template <int NC, int NN, bool NODAL = false>
__device__ __forceinline__ void integrate_group(const Slot& s, bool on, int npg, const double* qs, const double* ws,
                                                const Rules& R, int ng, const Consts& k, int lg, int G,
                                                double (&h)[NN * NC], double (&g)[NN * NC]) {
#pragma unroll
  for (int c = 0; c < NN * NC; ++c) h[c] = g[c] = 0.0;
  const int m = on ? s.np * npg : 0;
  const int lane = threadIdx.x & 31;
  double flip = 1.0;
  for (int q = lg;; q += G) {
    const bool act = q < m;
    if (!__any_sync(FULL, act)) break;
    double dx = 0.0, dy = 0.0, px = 0.0, py = 0.0, xi = 0.0, wx = 0.0;
    double N[NN];
    if (act) {
      const int piece = q >= npg ? 1 : 0;
      rule_node(s, piece, qs[q - piece * npg], ws[q - piece * npg], xi, wx);
      basis<NN>(R.leg_x, R.leg_pw, xi, N);
    }
    if (NODAL && act) {
      double dN[NN];
#pragma unroll
      for (int j = 0; j < NN; ++j) {
        dN[j] = N[0] * R.leg_D[j];
#pragma unroll
        for (int i = 1; i < NN; ++i) dN[j] = fma(N[i], R.leg_D[i * NN + j], dN[j]);
      }
      nodal_point<NN>(s.cx, s.cy, N, dN, s.sx, s.sy, px, py, dx, dy);
    }
    if (!NODAL && act) {
      // Horner for the point (relative to the source) and the tangent
      px = s.cx[ng - 1];
      py = s.cy[ng - 1];
      for (int d = ng - 2; d >= 0; --d) {
        dx = fma(dx, xi, px);
        dy = fma(dy, xi, py);
        px = fma(px, xi, s.cx[d]);
        py = fma(py, xi, s.cy[d]);
      }
    }
    if (q < G) {  // the first round: the orientation at the rule's first node
      const double side = dy * s.nrx - dx * s.nry;
      flip = __shfl_sync(FULL, side < 0 ? -1.0 : 1.0, lane - lg);
    }
    if (act) {
      const double J = f64::sqrt(fma(dx, dx, dy * dy));
      double U[4], T[4];
      kernel_values<NC>(k, px, py, flip * dy, -(flip * dx), U, T);
      const double wJ = wx * J;
#pragma unroll
      for (int j = 0; j < NN; ++j) {
        const double Nu = N[j] * wJ, Nt = N[j] * wx;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          h[j * NC + c] = fma(T[c], Nt, h[j * NC + c]);
          if (NC == 1 || c != 2) g[j * NC + c] = fma(U[c], Nu, g[j * NC + c]);
        }
      }
    }
  }
}

// sums over the group's lanes, to all of them
template <int NC, int NN>
__device__ __forceinline__ void reduce_group(int G, double (&h)[NN * NC], double (&g)[NN * NC]) {
  for (int o = G >> 1; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < NN * NC; ++c) {
      h[c] += __shfl_xor_sync(FULL, h[c], o);
      if (NC == 1 || (c & 3) != 2) g[c] += __shfl_xor_sync(FULL, g[c], o);
    }
  }
  if (NC == 4) {
#pragma unroll
    for (int j = 0; j < NN; ++j) g[j * NC + 2 % NC] = g[j * NC + 1 % NC];  // U is symmetric
  }
}

}  // namespace coop
}  // namespace bem
