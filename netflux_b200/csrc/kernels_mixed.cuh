// Mixed-precision form in difference variables: FP64 state, primitives,
// ghosts, boundary fluxes and update; FP32 gradient, limiter, reconstruction
// and interior Rusanov fluxes, computed from differences to the cell's own
// FP64 primitives so that FP32 rounding is relative to those differences.
//
// With the face normals of a closed cell summing to zero,
//   grad V_c = 1/vol sum_f 0.5 (V_c + V_f) S_f = 0.5/vol sum_f (V_f - V_c) S_f
//   R_c = -sum_f F(V_L, V_R; S_f) = -sum_f [F(V_L, V_R; S_f) - F(V_c) . S_f]
// (calc_green_gauss_gradient Numerics.hpp:86-128, evaluate_inviscid_fluxes
// Solver.cpp:144-230): the same operator as the FP64 forms in exact
// arithmetic. Storing FP32 copies of V and of the face states instead rounds
// at |V| * 2^-24, which puts a floor under the steady residual (near a 1e-5
// drop); here everything FP32 carries is small near a steady state: V_f - V_c,
// the reconstruction increments phi grad V . r and the flux differences
// F - F(V_c), so the residual keeps converging.
#pragma once

#include "kernels.cuh"

namespace nf {

// F(V_c + dL, V_c + dR; n, area) - area F(V_c) . n for the Rusanov flux
// (rusanov Numerics.cpp:10-18, inviscid_flux SolverData.hpp:239-255), expanded
// so every term is a difference times an O(1) factor:
//   rho_X q_X - rho_c q_c            = d_rho q_c + rho_X dq
//   rho_X u_X q_X - rho_c u_c q_c    = (d_rho u_c + rho_X du) q_c + rho_X u_X dq
//   H_X q_X - H_c q_c                = (dE + dp) q_c + H_X dq
//   E_X - E_c = dp/(g-1) + 0.5 (d_rho |u_c|^2 + rho_X (2 u_c . du + |du|^2))
struct DeltaSide {
  float dU[5];  // U(V_c + d) - U(V_c)
  float dF[5];  // (F(V_c + d) - F(V_c)) . n
  float s;      // |q| + c of the state
};

__device__ __forceinline__ DeltaSide delta_side(const float vc[5], float q_c, float uu_c, const float d[5],
                                                const float n[3]) {
  constexpr float g1i = Gas<float>::g1_inv;
  DeltaSide o;
  const float rho = vc[0] + d[0], p = vc[4] + d[4];
  const float u[3] = {vc[1] + d[1], vc[2] + d[2], vc[3] + d[3]};
  const float dq = fmaf(d[3], n[2], fmaf(d[2], n[1], d[1] * n[0]));
  const float udu = fmaf(vc[3], d[3], fmaf(vc[2], d[2], vc[1] * d[1]));
  const float dudu = fmaf(d[3], d[3], fmaf(d[2], d[2], d[1] * d[1]));
  const float dE = fmaf(d[4], g1i, 0.5f * fmaf(d[0], uu_c, rho * fmaf(2.0f, udu, dudu)));
  o.dU[0] = d[0];
  o.dF[0] = fmaf(d[0], q_c, rho * dq);
#pragma unroll
  for (int e = 0; e < 3; e++) {
    o.dU[e + 1] = fmaf(d[0], vc[e + 1], rho * d[e + 1]);
    o.dF[e + 1] = fmaf(o.dU[e + 1], q_c, fmaf(rho * u[e], dq, d[4] * n[e]));
  }
  const float uu = fmaf(u[2], u[2], fmaf(u[1], u[1], u[0] * u[0]));
  const float H = fmaf(p, g1i, fmaf(0.5f * rho, uu, p));  // E + p
  o.dU[4] = dE;
  o.dF[4] = fmaf(dE + d[4], q_c, H * dq);
  o.s = fabsf(q_c + dq) + sound_speed_fast(rho, p);
  return o;
}

__device__ __forceinline__ void rusanov_delta(const float vc[5], const float dL[5], const float dR[5],
                                              const float n[3], float area, float F[5]) {
  const float q_c = fmaf(vc[3], n[2], fmaf(vc[2], n[1], vc[1] * n[0]));
  const float uu_c = fmaf(vc[3], vc[3], fmaf(vc[2], vc[2], vc[1] * vc[1]));
  const DeltaSide L = delta_side(vc, q_c, uu_c, dL, n);
  const DeltaSide R = delta_side(vc, q_c, uu_c, dR, n);
  const float smax = fmaxf(R.s, L.s);
  const float h = 0.5f * area;
#pragma unroll
  for (int k = 0; k < 5; k++) F[k] = h * fmaf(-smax, R.dU[k] - L.dU[k], L.dF[k] + R.dF[k]);
}

}  // namespace nf
