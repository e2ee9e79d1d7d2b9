// Device functions that both forms of the fused kernel share: the stress
// updates of the materials, the node-block flags of a window, and the
// order-independent sums of the deterministic form.
#pragma once

#include "geom.cuh"
#include "state.cuh"

namespace mpmb200 {

// Marks the node blocks covered by a point's window.
template <int DIM, typename R>
__device__ __forceinline__ void mark_blocks(const Geom& g, const PointMapT<R>& pm, uint32_t* flags) {
  const int i0 = pm.ax[0].base >> g.bsh[0], i1 = (pm.ax[0].base + pm.ax[0].span - 1) >> g.bsh[0];
  const int j0 = pm.ax[1].base >> g.bsh[1], j1 = (pm.ax[1].base + pm.ax[1].span - 1) >> g.bsh[1];
  int k0 = 0, k1 = 0;
  if (DIM == 3) {
    k0 = pm.ax[2].base >> g.bsh[2];
    k1 = (pm.ax[2].base + pm.ax[2].span - 1) >> g.bsh[2];
  }
  for (int k = k0; k <= k1; k++)
    for (int j = j0; j <= j1; j++)
      for (int i = i0; i <= i1; i++) flags[i + (int64_t)g.nb[0] * (j + (int64_t)g.nb[1] * k)] = 1u;
}

// Jaumann update of IsotropicLinearElasticity (isolin.cpp:62-74) on the 6
// stored components. For symmetric T and W = -W^T, (T W)_ab = -(W T)_ba, so
// W T - T W = (W T)_ab + (W T)_ba.
template <int DIM, typename R>
__device__ __forceinline__ void jaumann_update(const R L[3][3], R* s6, R G, R lambda, R dt) {
  R D[3][3], W[3][3];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      D[a][b] = R(0.5) * (L[a][b] + L[b][a]);
      W[a][b] = R(0.5) * (L[a][b] - L[b][a]);
    }
  const R trD = D[0][0] + D[1][1] + D[2][2];
  const R T[3][3] = {{s6[0], s6[3], s6[5]}, {s6[3], s6[1], s6[4]}, {s6[5], s6[4], s6[2]}};
  R WT[3][3];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) WT[a][b] = W[a][0] * T[0][b] + W[a][1] * T[1][b] + W[a][2] * T[2][b];
  const R twoG = R(2.0) * G;
  const R ltr = lambda * trD;
  const int ia[6] = {0, 1, 2, 0, 1, 0};
  const int ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int c = 0; c < 6; c++) {
    const int a = ia[c], b = ib[c];
    const R rate = ((twoG * D[a][b] + (a == b ? ltr : R(0.0))) + WT[a][b]) + WT[b][a];
    s6[c] = s6[c] + dt * rate;
  }
}

// The Jaumann update of one point in its form. The mixed form keeps its
// stress and velocity gradient in FP32 but runs the update in FP64 and
// rounds the result once (measured on the block-drop ensemble: the FP32
// update's rounding, amplified by a soft block's dynamics, reached 1.9e-4
// of the stress after 500 steps; in FP64 arithmetic 8.3e-5).
template <int DIM, typename R>
__device__ __forceinline__ void jaumann_point(const R L[3][3], R* s6, const MaterialParams& mp, double dt) {
  if constexpr (sizeof(R) == 4) {
    double Ld[3][3], sd[6];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int b = 0; b < 3; b++) Ld[a][b] = (double)L[a][b];
#pragma unroll
    for (int k = 0; k < 6; k++) sd[k] = (double)s6[k];
    jaumann_update<DIM, double>(Ld, sd, mp.G, mp.lambda, dt);
#pragma unroll
    for (int k = 0; k < 6; k++) s6[k] = (R)sd[k];
  } else {
    jaumann_update<DIM, R>(L, s6, (R)mp.G, (R)mp.lambda, (R)dt);
  }
}

// CompressibleNeohookeanElasticity::calculateStress
// (compressible_neohookean_elasticity.cpp:44-62) for one point. The
// reference advances F += (L F) dt and sets T = G/J (B - I) + lambda ln(J)/J I
// with B = F F^T, J = sqrt(det B), lambda = K - 2G/3. Here the deformation
// gradient is kept as H = F - I (global memory, row-major components
// H[0..8]), so the same quantities come without the cancellation of B - I
// and ln J near the identity (which costs FP32 most of its digits at small
// strains): H += (L + L H) dt, B - I = H + H^T + H H^T,
// J - 1 = det(I + H) - 1 = tr H + ((tr H)^2 - tr(H H))/2 + det H, and
// ln J = log1p(J - 1). Returns the 6 stored stress components.
template <typename R, typename PT>
__device__ __forceinline__ void neohookean_update(PT* const* Hp, int64_t p, const R L[3][3], R* s6, R G, R lambda,
                                                  R dt) {
  R H[3][3];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) H[a][b] = (R)Hp[3 * a + b][p];
  R LH[3][3];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) LH[a][b] = L[a][0] * H[0][b] + L[a][1] * H[1][b] + L[a][2] * H[2][b];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      H[a][b] = H[a][b] + (L[a][b] + LH[a][b]) * dt;
      Hp[3 * a + b][p] = (PT)H[a][b];
    }
  const R trH = H[0][0] + H[1][1] + H[2][2];
  R trHH = R(0);
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) trHH += H[a][b] * H[b][a];
  const R detH = H[0][0] * (H[1][1] * H[2][2] - H[2][1] * H[1][2]) - H[0][1] * (H[1][0] * H[2][2] - H[2][0] * H[1][2]) +
                 H[0][2] * (H[1][0] * H[2][1] - H[2][0] * H[1][1]);
  const R Jm1 = trH + R(0.5) * (trH * trH - trHH) + detH;
  const R J = R(1) + Jm1;
  const R s1 = G / J;
  const R s2 = lambda * log1p(Jm1) / J;
  const int ia[6] = {0, 1, 2, 0, 1, 0};
  const int ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int c = 0; c < 6; c++) {
    const int a = ia[c], b = ib[c];
    const R bmi = H[a][b] + H[b][a] + (H[a][0] * H[b][0] + H[a][1] * H[b][1] + H[a][2] * H[b][2]);
    s6[c] = s1 * bmi + (a == b ? s2 : R(0));
  }
}

// Sand_SachithLocal::calculateStress (sand_sachithlocal.cpp:140-215) for one
// point, cohesion 0, on the 6 stored components. The trial stress s_tr is
// the Jaumann update above; p_tr = -tr(s_tr)/3 (or K (rho/rho_c - 1) with
// USE_DENSITY_FOR_PRESSURE), t0 = s_tr + p_tr I, tau_tr = |t0|/sqrt(2) with
// |t0|^2 summed in the reference's row-major order. Below the critical
// density, or at p_tr <= 0, the stress is zero and the shear rate is
// tau_tr/(G dt). Inside the cone tau_tr <= mu_s p_tr the trial stress stays.
// Otherwise tau is the smaller root of tau^2 - (S2 + tau_tr + alpha) tau +
// S2 tau_tr + S0 alpha (S0 = mu_s p_tr, S2 = mu_2 p_tr, alpha = G I_0 dt
// sqrt(p_tr/grains_rho)/grains_d), taken as in negative_root (44-53), and
// T = (tau/tau_tr) t0 - p_tr I. A NaN p_tr leaves T as it was. gammap
// (st[0]) advances by the shear rate times dt and gammap_dot (st[1]) takes
// the rate. rho = m/V with V already updated this step (updateDensity runs
// before the stress, explicit_usl.cpp:332-352).
template <int DIM, typename R, typename PT>
__device__ __forceinline__ void sand_update(PT* const* st, int64_t p, const R L[3][3], R* s6, R m, R vol,
                                            const MaterialParams& mp, R dt) {
  R t0[6];
#pragma unroll
  for (int k = 0; k < 6; k++) t0[k] = s6[k];
  jaumann_update<DIM, R>(L, t0, (R)mp.G, (R)mp.lambda, dt);
  R p_tr = -((t0[0] + t0[1]) + t0[2]) / R(3.0);
#pragma unroll
  for (int k = 0; k < 3; k++) t0[k] = t0[k] + p_tr;
  // xx xy xz yx yy yz zx zy zz
  R nn = t0[0] * t0[0];
  nn += t0[3] * t0[3];
  nn += t0[5] * t0[5];
  nn += t0[3] * t0[3];
  nn += t0[1] * t0[1];
  nn += t0[4] * t0[4];
  nn += t0[5] * t0[5];
  nn += t0[4] * t0[4];
  nn += t0[2] * t0[2];
  const R tau_tr = sqrt(nn) / sqrt(R(2.0));
  const R G = (R)mp.G;
  const R rho = m / vol;
  const R rho_c = (R)mp.rho_critical;
  if (mp.use_density) p_tr = (R)mp.K * ((rho - rho_c) / rho_c);
  R nup;
  if (rho < rho_c || p_tr <= R(0)) {
    nup = tau_tr / (G * dt);
#pragma unroll
    for (int k = 0; k < 6; k++) s6[k] = R(0);
  } else if (p_tr > R(0)) {
    const R S0 = (R)mp.mu_s * p_tr;
    R tau = tau_tr, scale = R(1);
    if (!(tau_tr <= S0)) {
      const R S2 = (R)mp.mu_2 * p_tr;
      const R alpha = G * (R)mp.i_0 * dt * sqrt(p_tr / (R)mp.grains_rho) / (R)mp.grains_d;
      const R b = -(S2 + tau_tr + alpha);
      const R c = S2 * tau_tr + S0 * alpha;
      const R disc = sqrt(b * b - R(4) * c);
      tau = b > R(0) ? (-b - disc) / R(2) : (R(2) * c) / (-b + disc);
      scale = tau / tau_tr;
    }
    nup = ((tau_tr - tau) / G) / dt;
#pragma unroll
    for (int k = 0; k < 6; k++) s6[k] = scale * t0[k] - (k < 3 ? p_tr : R(0));
  } else {
    nup = R(0);
  }
  st[0][p] = (PT)((R)st[0][p] + nup * dt);
  st[1][p] = (PT)nup;
}

// Order-independent nodal sums of the deterministic form (pre-rounded
// two-level summation after Demmel and Nguyen, "Fast reproducible
// floating-point summation", ARITH 2013). With M bounding every partial sum
// of |contributions| to a node (n contributions of at most maxc each), a
// contribution x splits exactly into q0 + q1 + e: q0 is x rounded to a
// multiple of 2^(E0-52) with 2^E0 > 2M, q1 the remainder rounded to a
// multiple of 2^(E1-52) with E1 = E0 - 52 + L, 2^L > 2n, and |e| <
// 2^(E1-53). Sums of q0 (of q1) stay below 2^E0 (2^E1) in any order, so
// every addition is exact and the two sums are the same bits whatever the
// order; the nodal value is level0 + level1 rounded once.
struct Split2 {
  double s0;  // 1.5 * 2^E0
  double s1;  // 1.5 * 2^E1
};

__device__ __forceinline__ Split2 make_split(double maxc, int64_t n) {
  Split2 k{0.0, 0.0};
  if (!(maxc > 0.0) || n < 1) return k;  // all contributions are zero
  const int L = ilogb((double)n) + 2;
  const int E0 = ilogb(maxc) + L + 1;
  const int E1 = E0 - 52 + L;
  k.s0 = ldexp(1.5, E0);
  k.s1 = ldexp(1.5, E1);
  return k;
}

__device__ __forceinline__ void presplit(double x, const Split2& k, double& q0, double& q1) {
  q0 = __dsub_rn(__dadd_rn(k.s0, x), k.s0);
  const double r = __dsub_rn(x, q0);
  q1 = __dsub_rn(__dadd_rn(k.s1, r), k.s1);
}

}  // namespace mpmb200
