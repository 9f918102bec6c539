// Near-singular, on-element and diagonal kernels of the dense 2-D BEM
// assembly (FP64).  See assemble_far.cu for the overall structure.
#include "bem_device.cuh"
#include "bem_kernels.h"
#include "near_coop.cuh"

#include <cmath>
#include <mutex>

namespace bem {

// ---------------------------------------------------------------------------
// near kernel: listed pairs, exact FP64 test, tanp3c or FP64 lumping
// ---------------------------------------------------------------------------
// store modes: 0 FP32 (H, G); 1 FP64 (H, G); 2 FP64 (A, b); 3 FP64 + FP32 (A, b)
__device__ __forceinline__ void store_hg(const NearArgs& a, size_t row, size_t col, double hv,
                                         double gv) {
  if (a.mode == 0) {
    ((float*)a.H)[row + col * a.ld] = (float)hv;
    ((float*)a.G)[row + col * a.ldg] = (float)gv;
  } else {
    ((double*)a.H)[row + col * a.ld] = hv;
    ((double*)a.G)[row + col * a.ldg] = gv;
  }
}

__device__ __forceinline__ void store_a(const NearArgs& a, size_t row, size_t col, double av) {
  ((double*)a.H)[row + col * a.ld] = av;
  if (a.mode == 3) a.A32[row + col * a.ld] = (float)av;
}

// writes the entries of pair (i, e) and adds its row sums (and b)
template <int NC>
__device__ __forceinline__ void store_pair(const NearArgs& a, int i, int e, int nn, const double* h,
                                           const double* gg) {
  constexpr int DOF = (NC == 1) ? 1 : 2;
  const bool FUSED = a.mode >= 2;
#pragma unroll
  for (int ar = 0; ar < DOF; ++ar) {
    const size_t row = (size_t)DOF * i + ar;
    double rs[DOF], bs = 0.0;
#pragma unroll
    for (int b = 0; b < DOF; ++b) rs[b] = 0.0;
#pragma unroll
    for (int k = 0; k < nn; ++k) {
      int j = e * nn + k;
#pragma unroll
      for (int b = 0; b < DOF; ++b) {
        const size_t col = (size_t)DOF * j + b;
        double hv = h[k * NC + ar * DOF + b], gv = gg[k * NC + ar * DOF + b];
        rs[b] += hv;
        if (!FUSED) {
          store_hg(a, row, col, hv, gv);
        } else {
          int bc = a.bc[col];
          double av = (bc == 0) ? -gv : hv;
          bs += (bc == 0) ? -hv * a.bv[col] : gv * a.bv[col];
          store_a(a, row, col, av);
        }
      }
    }
#pragma unroll
    for (int b = 0; b < DOF; ++b) atomicAdd(a.rowsum + row * DOF + b, rs[b]);
    if (FUSED) atomicAdd(a.b + row, bs);
  }
}

// One thread per pair, any near-field map: the maps other than tanp3c (a
// warp's threads share no work there), and the rare tanp3c pairs that take
// none of its regular branches.
template <int NC>
__device__ __noinline__ void near_general(const NearArgs& a, int i, int e) {
  const GeomDev& g = a.g;
  V2 nodes[BEM_MAXNN], geo[BEM_MAXGEO];
  load_element(g, e, nodes, geo);
  double h[BEM_MAXNN * NC], gg[BEM_MAXNN * NC];
  integrate_near<NC>(a.R, a.ph, nodes, geo, V2{g.px[i], g.py[i]}, g.elen[e], V2{g.nx[e * g.nn], g.ny[e * g.nn]}, h,
                     gg);
  store_pair<NC>(a, i, e, g.nn, h, gg);
}

template <int NC>
__global__ void __launch_bounds__(128) near_general_kernel(const __grid_constant__ NearArgs a) {
  const int count = min(*a.pair_count, a.pair_cap);
  const GeomDev& g = a.g;
  const int nn = g.nn;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
    const int2 pr = a.pairs[t];
    const int i = pr.x, e = pr.y;
    V2 nodes[BEM_MAXNN], geo[BEM_MAXGEO];
    load_element(g, e, nodes, geo);
    V2 pf{g.px[i], g.py[i]};
    if (near_element(pf, nodes, nn, g.elen[e], a.near_factor)) {
      near_general<NC>(a, i, e);
      continue;
    }
    double h[BEM_MAXNN * NC], gg[BEM_MAXNN * NC];
    for (int k = 0; k < nn; ++k) {
      int j = e * nn + k;
      double U[4], T[4];
      far_eval_f64<NC>(a.ph, g.px[j] - pf.x, g.py[j] - pf.y, g.nx[j], g.ny[j], g.jac[j] * a.R.ew[k], U, T);
      for (int c = 0; c < NC; ++c) { h[k * NC + c] = T[c]; gg[k * NC + c] = U[c]; }
    }
    store_pair<NC>(a, i, e, nn, h, gg);
  }
}

// The listed pairs by warps (near_coop.cuh).  FP64 issue bounds it: a warp
// with 16 pairs issues about 3000 FP64 instructions.  A task is as many pairs
// as spread the list over the GPU's 608 schedulers, one at least and 16 at
// most.  The kernel runs beside the far and on-element kernels, whose CTAs may
// hold any SMs when it starts: with two CTAs of four warps per SM and a fixed
// share each, they now and then stood four to an SM on half of the SMs (333 000
// pairs 5.5 or 10.5 ms).  So the warps of the first 304 CTAs have one task each
// (claimed tasks would gather on the SMs that start first: 1000 nodes 0.29 ms
// instead of 0.12), and they claim the others from a counter.  From four rounds
// of tasks on 304 CTAs more claim too, which find an SM where the first ones
// have left some free; before that they would only crowd some SMs (8193 nodes,
// 1366 tasks: H and G in FP32 0.63 ms instead of 0.59).  Even CTAs that leave at
// once change where the first ones stand (cubic and quartic elements, 1000 to
// 2600 nodes: 10 to 20 % of the call), so they are launched above a near factor
// of 3 only.
template <int NC, int NN>
__global__ void __launch_bounds__(128) near_kernel(const __grid_constant__ NearArgs a) {
  using namespace coop;
  __shared__ Slot s_slots[4][PAIRS];
  __shared__ double s_q[BEM_MAXNPG], s_w[BEM_MAXNPG];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int count = min(*a.pair_count, a.pair_cap);
  const int per = max(1, min(PAIRS, (count + 607) / 608));
  if (blockIdx.x >= NEAR_CTAS && count <= NEAR_MANY * PAIRS) return;
  auto claim = [&] {
    int t = 0;
    if (lane == 0) t = atomicAdd(a.claim, 1);
    return (4 * NEAR_CTAS + __shfl_sync(FULL, t, 0)) * per;
  };
  const GeomDev& g = a.g;
  const Rules& R = a.R;
  for (int q = threadIdx.x; q < R.npg; q += blockDim.x) {
    s_q[q] = R.qsi[q];
    s_w[q] = R.w[q];
  }
  __syncthreads();
  const Consts kc = make_consts<NC>(a.ph);
  const int ng = R.ngeo > 0 ? R.ngeo : NN;
  const int G = per == 1 ? 32 : (per == 2 ? 16 : 8);
  Slot* slots = s_slots[warp];
  for (int base = blockIdx.x < NEAR_CTAS ? (warp * NEAR_CTAS + (int)blockIdx.x) * per : claim(); base < count;
       base = claim()) {
    const int np = min(per, count - base);
    if (lane < np) {
      const int2 pr = a.pairs[base + lane];
      const int i = pr.x, e = pr.y;
      Slot& s = slots[lane];
      s.id = base + lane;
      s.kind = K_FAR;
      s.np = 1;
      V2 nodes[NN], geo[BEM_MAXGEO];
#pragma unroll
      for (int k = 0; k < NN; ++k) nodes[k] = V2{g.px[e * NN + k], g.py[e * NN + k]};
      const V2 pf{g.px[i], g.py[i]};
      if (near_element(pf, nodes, NN, g.elen[e], a.near_factor)) {
        s.kind = K_TANGENT;
        for (int k = 0; k < g.ngeo; ++k) geo[k] = V2{g.gx[e * g.ngeo + k], g.gy[e * g.ngeo + k]};
        geometry(R, nodes, geo, pf, s);
        s.nrx = g.nx[e * NN];
        s.nry = g.ny[e * NN];
        complex_pole_1d(R, nodes, NN, pf, s.z0, s.e0);
      }
    }
    __syncwarp();
    map_constants(R, slots, np, lane);
    const int lg = lane & (G - 1);
    for (int p0 = 0; p0 < np; p0 += 32 / G) {
      const int p = p0 + lane / G;
      const bool valid = p < np;
      const Slot& s = slots[valid ? p : 0];
      const int kind = valid ? s.kind : K_NONE;
      double h[NN * NC], gg[NN * NC];
      integrate_group<NC, NN>(s, kind == K_TANGENT || kind == K_REALPOLE, R.npg, s_q, s_w, R, ng, kc, lg, G, h, gg);
      int i = 0, e = 0;
      if (valid) {
        const int2 pr = a.pairs[s.id];
        i = pr.x;
        e = pr.y;
      }
      if (kind == K_FAR && lg < NN) {
        // far after all: nodal lumping, lane k taking node k
        const int j = e * NN + lg;
        double U[4], T[4];
        far_eval_f64<NC>(a.ph, g.px[j] - g.px[i], g.py[j] - g.py[i], g.nx[j], g.ny[j], g.jac[j] * R.ew[lg], U, T);
#pragma unroll
        for (int k = 0; k < NN; ++k)
          if (k == lg) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              h[k * NC + c] = T[c];
              gg[k * NC + c] = U[c];
            }
          }
      }
      reduce_group<NC, NN>(G, h, gg);
      if (lg == 0 && valid) {
        if (kind == K_GENERAL) near_general<NC>(a, i, e);
        else store_pair<NC>(a, i, e, NN, h, gg);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// on-element kernels: collocation node i on its own element
// ---------------------------------------------------------------------------
template <int NC>
__device__ __forceinline__ void store_own(const NearArgs& a, int i, int e, int nn, const double* h,
                                          const double* gg) {
  constexpr int DOF = (NC == 1) ? 1 : 2;
  const bool FUSED = a.mode >= 2;
#pragma unroll
  for (int ar = 0; ar < DOF; ++ar) {
    const size_t row = (size_t)DOF * i + ar;
    double rs[DOF], bs = 0.0;
#pragma unroll
    for (int b = 0; b < DOF; ++b) rs[b] = 0.0;
#pragma unroll
    for (int k = 0; k < nn; ++k) {
      int j = e * nn + k;
#pragma unroll
      for (int b = 0; b < DOF; ++b) {
        const size_t col = (size_t)DOF * j + b;
        double hv = h[k * NC + ar * DOF + b], gv = gg[k * NC + ar * DOF + b];
        const bool diag_blk = (j == i);
        if (!FUSED) {
          if (!diag_blk) {
            rs[b] += hv;
            store_hg(a, row, col, hv, gv);
          } else {
            if (a.mode == 0) ((float*)a.G)[row + col * a.ldg] = (float)gv;
            else ((double*)a.G)[row + col * a.ldg] = gv;
          }
        } else {
          int bc = a.bc[col];
          if (!diag_blk) {
            rs[b] += hv;
            double av = (bc == 0) ? -gv : hv;
            bs += (bc == 0) ? -hv * a.bv[col] : gv * a.bv[col];
            store_a(a, row, col, av);
          } else {
            // the diagonal block's H comes from the row sum (finalize); its
            // G part is final here.
            a.gdiag[(size_t)DOF * DOF * i + ar * DOF + b] = gv;
            if (bc != 0) bs += gv * a.bv[col];
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < DOF; ++b) atomicAdd(a.rowsum + row * DOF + b, rs[b]);
    if (FUSED) atomicAdd(a.b + row, bs);
  }
}

// Telles rule: one thread per node
template <int NC>
__global__ void __launch_bounds__(64) singular_telles_kernel(NearArgs a) {
  const GeomDev& g = a.g;
  const int nn = g.nn;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const int e = i / nn;
  V2 nodes[BEM_MAXNN], geo[BEM_MAXGEO];
  load_element(g, e, nodes, geo);
  V2 pf{g.px[i], g.py[i]};
  double xa, dist;
  closest_point_1d(a.R, nodes, nn, pf, xa, dist);
  V2 nref{g.nx[e * nn], g.ny[e * nn]};
  double h[BEM_MAXNN * NC], gg[BEM_MAXNN * NC];
  integrate_singular_telles<NC>(a.R, a.ph, nodes, geo, pf, xa, nref, h, gg);
  store_own<NC>(a, i, e, nn, h, gg);
}

// Interpolated Guiggiani.  A collocation node is a field node of its
// element, so its parent coordinate, the rule's interpolation weights, pole
// and logarithm corrections are constants of the element type, and the whole
// rule is one fixed linear functional of the 20 samples (singular_weights
// below): h = sum_i Wh[node][i][k] T_i J_i, g alike.  What is left per sample
// is the geometry, one square root, quotient and logarithm (45 FP64
// operations; the step-by-step rule with its Newton search for the known
// source took 4200 per node).  Four lanes per node, five samples each: 427 ->
// 34 us at N = 8193, 370 -> 19 us at N = 160, bound by the samples' latency
// and the table's copy to shared memory.
constexpr int OWN_LANES = 4;

template <int NC, int NN>
__global__ void __launch_bounds__(64) singular_kernel(const __grid_constant__ NearArgs a,
                                                      const __grid_constant__ SingularTable<NN> tab) {
  __shared__ double s_tab[sizeof(SingularTable<NN>) / 8];
  for (int q = threadIdx.x; q < (int)(sizeof(tab) / 8); q += blockDim.x) s_tab[q] = ((const double*)&tab)[q];
  __syncthreads();
  const SingularTable<NN>& W = *(const SingularTable<NN>*)s_tab;
  const GeomDev& g = a.g;
  const Rules& R = a.R;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int l = t & (OWN_LANES - 1);
  const bool valid = t / OWN_LANES < g.n;
  const int i = valid ? t / OWN_LANES : g.n - 1;
  const int e = i / NN, ai = i - e * NN;
  const int ng = R.ngeo > 0 ? R.ngeo : NN;
  const double sx = g.px[i], sy = g.py[i];
  // element nodes relative to the source
  double X[BEM_MAXGEO], Y[BEM_MAXGEO];
#pragma unroll
  for (int k = 0; k < BEM_MAXGEO; ++k)
    if (k < ng) {
      X[k] = (R.ngeo > 0 ? g.gx[e * ng + k] : g.px[e * NN + k]) - sx;
      Y[k] = (R.ngeo > 0 ? g.gy[e * ng + k] : g.py[e * NN + k]) - sy;
    }
  const double nrx = g.nx[e * NN], nry = g.ny[e * NN];
  const coop::Consts kc = coop::make_consts<NC>(a.ph);
  double h[NN * NC], gg[NN * NC];
#pragma unroll
  for (int c = 0; c < NN * NC; ++c) h[c] = gg[c] = 0.0;
  for (int q = l; q < BEM_NINTERP; q += OWN_LANES) {
    double rx = 0.0, ry = 0.0, dx = 0.0, dy = 0.0;
#pragma unroll
    for (int k = 0; k < BEM_MAXGEO; ++k)
      if (k < ng) {
        const double N = W.N[q][k], D = W.D[q][k];
        rx = fma(N, X[k], rx);
        ry = fma(N, Y[k], ry);
        dx = fma(D, X[k], dx);
        dy = fma(D, Y[k], dy);
      }
    const double J2 = fma(dx, dx, dy * dy), R2 = fma(rx, rx, ry * ry);
    if (J2 < 1e-60 || R2 < 1e-60) continue;
    const double J = f64::sqrt(J2);
    const double flip = dy * nrx - dx * nry < 0 ? -1.0 : 1.0;
    double U[4], T[4];
    coop::kernel_values<NC>(kc, rx, ry, flip * dy, -(flip * dx), U, T);
#pragma unroll
    for (int j = 0; j < NN; ++j) {
      const double wh = W.Wh[ai][q][j], wg = W.Wg[ai][q][j] * J;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        h[j * NC + c] = fma(wh, T[c], h[j * NC + c]);
        gg[j * NC + c] = fma(wg, U[c], gg[j * NC + c]);
      }
    }
  }
#pragma unroll
  for (int o = 1; o < OWN_LANES; o <<= 1)
#pragma unroll
    for (int c = 0; c < NN * NC; ++c) {
      h[c] += __shfl_xor_sync(0xffffffffu, h[c], o);
      gg[c] += __shfl_xor_sync(0xffffffffu, gg[c], o);
    }
  if (valid && l == 0) store_own<NC>(a, i, e, NN, h, gg);
}

// The rule of integrate_singular for a source on field node a of the
// element, as weights of the samples F_i: with d_i = x_i - a, the
// interpolation weights N_i at a, the pole coefficient F_p = sum N_i d_i F_i
// and the logarithm's least-squares coefficient F_l = sum u_i (F_i - F_p / d_i),
//   h = sum w_i (F_i - F_p / d_i) + F_p P,
//   g = sum w_i (F_i - F_p / d_i - F_l log|d_i|) + F_p P + F_l Q.
template <int NN>
static void singular_weights(const Rules& R, SingularTable<NN>& W) {
  constexpr int M = BEM_NINTERP;
  using T = long double;
  // geometry basis at the samples: the operations of shapefun_prod (its
  // derivative sums contracted as the compiler does on the device)
  const int ng = R.ngeo > 0 ? R.ngeo : NN;
  const double* gx = R.ngeo > 0 ? R.geo_x : R.leg_x;
  const double* gpw = R.ngeo > 0 ? R.geo_pw : R.leg_pw;
  const double* gD = R.ngeo > 0 ? R.geo_D : R.leg_D;
  for (int q = 0; q < M; ++q) {
    double* N = W.N[q];
    double pre = 1.0, suf = 1.0;
    for (int k = 0; k < ng; ++k) {
      N[k] = gpw[k] * pre;
      pre *= R.gi_x[q] - gx[k];
    }
    for (int k = ng - 1; k >= 0; --k) {
      N[k] *= suf;
      suf *= R.gi_x[q] - gx[k];
    }
    for (int k = 0; k < ng; ++k) {
      double d = N[0] * gD[k];
      for (int i = 1; i < ng; ++i) d = std::fma(N[i], gD[i * ng + k], d);
      W.D[q][k] = d;
    }
  }
  for (int ai = 0; ai < NN; ++ai) {
    const T a = R.leg_x[ai];
    T d[M], Ni[M], lg[M], sum = 0, sL = 0, sL2 = 0, sWd = 0, sWL = 0;
    for (int i = 0; i < M; ++i) {
      d[i] = R.gi_x[i] - a;
      Ni[i] = -R.gi_bw[i] / d[i];
      sum += Ni[i];
      lg[i] = logl(fabsl(d[i]));
      sL += lg[i];
      sL2 += lg[i] * lg[i];
      sWd += R.gi_w[i] / d[i];
      sWL += R.gi_w[i] * lg[i];
    }
    const T det = sL2 * M - sL * sL;
    const T P = logl((1 - a) / (1 + a));
    const T Q = (1 - a) * logl(1 - a) + (1 + a) * logl(1 + a) - 2;
    T ud = 0;
    for (int i = 0; i < M; ++i) ud += (M * lg[i] - sL) / det / d[i];
    for (int i = 0; i < M; ++i) {
      const T pole = Ni[i] / sum * d[i];
      const T wh = R.gi_w[i] + pole * (P - sWd);
      const T u = (M * lg[i] - sL) / det - pole * ud;
      const T wg = wh + u * (Q - sWL);
      for (int j = 0; j < NN; ++j) {
        T N = 1;
        for (int m = 0; m < NN; ++m)
          if (m != j) N *= (R.gi_x[i] - R.leg_x[m]) / ((T)R.leg_x[j] - R.leg_x[m]);
        W.Wh[ai][i][j] = (double)(wh * N);
        W.Wg[ai][i][j] = (double)(wg * N);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// finalize: diagonal (block) from the row sums
// ---------------------------------------------------------------------------
__device__ __forceinline__ void store_diag(const FinalArgs& a, size_t row, size_t col, double v) {
  if (a.mode == 0) ((float*)a.H)[row + col * a.ld] = (float)v;
  else ((double*)a.H)[row + col * a.ld] = v;
  if (a.mode == 3) a.A32[row + col * a.ld] = (float)v;
}

template <int NC>
__global__ void finalize_kernel(FinalArgs a) {
  constexpr int DOF = (NC == 1) ? 1 : 2;
  const bool FUSED = a.mode >= 2;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nt) return;
  if constexpr (DOF == 1) {
    double hii = -a.rowsum[i];
    if (!FUSED) {
      store_diag(a, i, i, hii);
    } else {
      double av = hii;
      if (i < a.n && a.bc[i] == 0) {
        av = -a.gdiag[i];
        a.b[i] += -hii * a.bv[i];
      }
      store_diag(a, i, i, av);
    }
  } else {
    // rigid-body row-sum (_vectorial_free_term!): block (2i+a, 2i+b) =
    // -sum of row 2i+a over columns of dof b, other blocks excluded.  The
    // row sums were accumulated per row over all columns; split by column
    // dof with the per-dof accumulators.
    for (int ar = 0; ar < 2; ++ar)
      for (int b = 0; b < 2; ++b) {
        size_t row = 2 * (size_t)i + ar, col = 2 * (size_t)i + b;
        double hv = -a.rowsum[(2 * (size_t)i + ar) * 2 + b];
        if (!FUSED) {
          store_diag(a, row, col, hv);
        } else {
          double av = hv;
          if ((size_t)i < (size_t)a.n && a.bc[col] == 0) {
            av = -a.gdiag[4 * (size_t)i + ar * 2 + b];
            a.b[row] += -hv * a.bv[col];
          }
          store_diag(a, row, col, av);
        }
      }
  }
}




template <int NC>
static void launch_near_nc(const NearArgs& na, cudaStream_t st) {
  if (na.R.nearfield != 0) {
    int nblk = (na.pair_cap + 127) / 128;
    if (nblk > 152 * 16) nblk = 152 * 16;
    if (nblk < 1) nblk = 1;
    near_general_kernel<NC><<<nblk, 128, 0, st>>>(na);
    return;
  }
  const int nblk = near_ctas(na.near_factor);
  switch (na.R.nn) {
    case 2: near_kernel<NC, 2><<<nblk, 128, 0, st>>>(na); break;
    case 3: near_kernel<NC, 3><<<nblk, 128, 0, st>>>(na); break;
    case 4: near_kernel<NC, 4><<<nblk, 128, 0, st>>>(na); break;
    case 5: near_kernel<NC, 5><<<nblk, 128, 0, st>>>(na); break;
    case 6: near_kernel<NC, 6><<<nblk, 128, 0, st>>>(na); break;
  }
}

void launch_near_pairs(const NearArgs& na, int nc, cudaStream_t st) {
  if (nc == 1) launch_near_nc<1>(na, st);
  else launch_near_nc<4>(na, st);
}

template <int NN>
const SingularTable<NN>& singular_table(const Rules& R) {
  static SingularTable<NN> tab[BEM_MAXGEO + 1];
  static std::once_flag once[BEM_MAXGEO + 1];
  std::call_once(once[R.ngeo], [&] { singular_weights<NN>(R, tab[R.ngeo]); });
  return tab[R.ngeo];
}
template const SingularTable<2>& singular_table<2>(const Rules&);
template const SingularTable<3>& singular_table<3>(const Rules&);
template const SingularTable<4>& singular_table<4>(const Rules&);
template const SingularTable<5>& singular_table<5>(const Rules&);
template const SingularTable<6>& singular_table<6>(const Rules&);

template <int NC, int NN>
static void launch_singular_nn(const NearArgs& na, int n, cudaStream_t st) {
  const int nblk = (int)(((int64_t)n * OWN_LANES + 63) / 64);
  singular_kernel<NC, NN><<<nblk, 64, 0, st>>>(na, singular_table<NN>(na.R));
}

template <int NC>
static void launch_singular_nc(const NearArgs& na, int n, cudaStream_t st) {
  if (na.R.singular == 1) {
    singular_telles_kernel<NC><<<(n + 63) / 64, 64, 0, st>>>(na);
    return;
  }
  switch (na.R.nn) {
    case 2: launch_singular_nn<NC, 2>(na, n, st); break;
    case 3: launch_singular_nn<NC, 3>(na, n, st); break;
    case 4: launch_singular_nn<NC, 4>(na, n, st); break;
    case 5: launch_singular_nn<NC, 5>(na, n, st); break;
    case 6: launch_singular_nn<NC, 6>(na, n, st); break;
  }
}

void launch_singular(const NearArgs& na, int nc, int n, cudaStream_t st) {
  if (n <= 0) return;
  if (nc == 1) launch_singular_nc<1>(na, n, st);
  else launch_singular_nc<4>(na, n, st);
}

void launch_finalize(const FinalArgs& fi, int nc, int nt, cudaStream_t st) {
  if (nc == 1) finalize_kernel<1><<<(nt + 255) / 256, 256, 0, st>>>(fi);
  else finalize_kernel<4><<<(nt + 255) / 256, 256, 0, st>>>(fi);
}

}  // namespace bem
