// The form with FP32 copies under the Barth limiter: a limiter kernel that writes
// 20 FP32 face states a cell and a flux kernel that reads them, in the operations
// (and roundings) this form has always used. Its rounding errors are amplified by
// the limiter's switches (a hundred steps turn 2e-8 into some 1e-6 of the state's
// norm, and a thousand times that in single cells), so another arrangement of the
// same reconstruction, such as the stage kernel's, gives results that differ from
// these by up to 1e-3 in a cell after a hundred steps. Which of the two is nearer to
// FP64 has not been measured; until it is, the form keeps its operations. The other
// forms, and this one without the limiter or in first order, have no such
// amplification. At 3.1M tets 140 and 186 us a launch.
#pragma once

#include "kernels_cell.cuh"

namespace nf {

// kPipe: 0 one variable's loads at a time; 1 the next variable's loads in
// flight during this one's arithmetic; 2 all five variables' loads issued
// together before any arithmetic; 3 as 0, with the cell's own rows prefetched
// into L2 first.
template <int kPipe>
__device__ __forceinline__ void gradient_copy_cell(const MeshView<float>& m, const StageArgs& a, int c) {
  using T = float;
  const int st = m.stride;
  const T* __restrict__ Vin = a.Vin32;
  const T* __restrict__ Vg = a.vg32;
  T* __restrict__ fsc = a.fs32 + c;  // this cell's column of the face states
  int nb[4];
#pragma unroll
  for (int q = 0; q < 4; q++) nb[q] = checked_nb(m.nbvf[q * st + c], 0, m.n, m.nb, c, a.status);
  // each face's row base and row stride (a cell's or a ghost's) chosen once,
  // so a variable's neighbour load is one address computation
  const T* qb[4];
  int qs[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const bool cell = nb[q] >= 0;
    qb[q] = cell ? Vin + nb[q] : Vg + (-nb[q] - 1);
    qs[q] = cell ? st : m.bstride;
  }
  auto fetch = [&](int k, T& vc, T vo[4]) {
    vc = Vin[size_t(k) * st + c];
#pragma unroll
    for (int q = 0; q < 4; q++) vo[q] = qb[q][k * qs[q]];
  };
  if constexpr (kPipe == 3) {
#pragma unroll
    for (int k = 0; k < 5; k++) prefetch_l2(Vin + size_t(k) * st + c);
  }
  [[maybe_unused]] T vcN, voN[4];
  [[maybe_unused]] T vcA[5], voA[5][4];
  if constexpr (kPipe == 2) {
    // the same loads as fetch(), all five variables' at once
#pragma unroll
    for (int k = 0; k < 5; k++) vcA[k] = Vin[size_t(k) * st + c];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const bool cell = nb[q] >= 0;
      const auto* p = cell ? Vin + nb[q] : Vg + (-nb[q] - 1);
      const size_t rs = cell ? size_t(st) : size_t(m.bstride);
#pragma unroll
      for (int k = 0; k < 5; k++) voA[k][q] = p[k * rs];
    }
  } else if (kPipe == 1) {
    fetch(0, vcN, voN);
  }
  const int code = m.gcode[c];
  T S[4][3], d[4][3];  // outward normals; (centroid - P_m) / 3
  {
    T P[4][3];
    load_vertices(m, c, P, a.status);
    face_normals(P, S);
    const T cen[3] = {T(0.25) * ((P[0][0] + P[1][0]) + (P[2][0] + P[3][0])),
                      T(0.25) * ((P[0][1] + P[1][1]) + (P[2][1] + P[3][1])),
                      T(0.25) * ((P[0][2] + P[1][2]) + (P[2][2] + P[3][2]))};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int bits = code >> (3 * q);
      const T sgn = (bits & 1) == 0 ? T(0) : ((bits & 2) ? T(-1) : T(1));  // 0: no face
#pragma unroll
      for (int e = 0; e < 3; e++) {
        S[q][e] *= sgn;
        d[q][e] = (bits & 1) ? (cen[e] - P[q][e]) * T(1.0 / 3.0) : T(0);
      }
    }
  }
  const T ssum[3] = {(S[0][0] + S[1][0]) + (S[2][0] + S[3][0]), (S[0][1] + S[1][1]) + (S[2][1] + S[3][1]),
                     (S[0][2] + S[1][2]) + (S[2][2] + S[3][2])};
  const T hv = T(0.5) * nr_rcp(T(m.vol[c]));
  const bool rat = ratchet_on(a, c);
  auto variable = [&](int k, T vc, const T vo[4]) {
    T acc[3];
#pragma unroll
    for (int e = 0; e < 3; e++) {
      acc[e] = vc * ssum[e];
#pragma unroll
      for (int q = 0; q < 4; q++) acc[e] = fma(vo[q], S[q][e], acc[e]);
    }
    const T g[3] = {hv * acc[0], hv * acc[1], hv * acc[2]};
    const T vmax = fmax(fmax(fmax(vc, vo[0]), fmax(vo[1], vo[2])), vo[3]);
    const T vmin = fmin(fmin(fmin(vc, vo[0]), fmin(vo[1], vo[2])), vo[3]);
    T gr[4];
#pragma unroll
    for (int q = 0; q < 4; q++) gr[q] = fma(g[2], d[q][2], fma(g[1], d[q][1], g[0] * d[q][0]));
    T An = T(1), Dn = T(1);  // best ratio so far, starting at 1
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const T d2 = gr[q];
      const T A = d2 > T(0) ? vmax - vc : vc - vmin;
      const T D = fabs(d2) + Gas<T>::eps;
      const bool better = (d2 != T(0)) && (A * Dn < An * D);
      An = better ? A : An;
      Dn = better ? D : Dn;
    }
    T phi = An * nr_rcp(Dn);
    if (rat) phi = ratchet(a, size_t(k) * st + c, phi);
#pragma unroll
    for (int q = 0; q < 4; q++) fsc[size_t(q * 5 + k) * st] = fma(phi, gr[q], vc);
    if (a.phi32) a.phi32[k * st + c] = phi;
  };
  if constexpr (kPipe == 2) {
#pragma unroll
    for (int k = 0; k < 5; k++) variable(k, vcA[k], voA[k]);
  } else {
#pragma unroll 1
    for (int k = 0; k < 5; k++) {
      T vc, vo[4];
      if (kPipe == 1) {
        vc = vcN;
#pragma unroll
        for (int q = 0; q < 4; q++) vo[q] = voN[q];
        if (k < 4) fetch(k + 1, vcN, voN);  // next variable's loads overlap this one's arithmetic
      } else {
        fetch(k, vc, vo);
      }
      variable(k, vc, vo);
    }
  }
}

template <int kPipe, int kMinBlocks>
__global__ void __launch_bounds__(128, kMinBlocks) gradient_copy_kernel(MeshView<float> m, StageArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait_previous();
  if (c < m.n && !frozen_cell(a, c)) gradient_copy_cell<kPipe>(m, a, c);
}

// Flux balance and stage update of one cell per thread. Each interior face's
// flux is evaluated with the reference's owner on the left and the
// owner-to-neighbour unit normal, which both cells rebuild to the same bits, so
// both add exactly opposite contributions; boundary faces add the flux
// boundary_flux_copy_kernel computed.
template <typename T>
struct FaceIn {
  T s[5];      // this cell's face state, or the boundary flux
  T x[5];      // the other side's face state
  int kind;    // 0 no face, 1 interior (owner), 2 interior (neighbour side), 3 boundary
};

// kPipe: 0 one face's loads at a time, 1 the next face's loads in flight
// during this face's flux, 2 all four faces' loads issued together, 3 as 0
// with the cell's own face states and update rows prefetched into L2 first.
template <int kPipe, int kMinBlocks>
__global__ void __launch_bounds__(128, kMinBlocks) flux_copy_kernel(MeshView<float> m, StageArgs a) {
  using T = float;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait_previous();
  double dt_next = DBL_MAX;
  const bool act = c < m.n && !frozen_cell(a, c);
  if (c < m.n && !act && a.dt_next_min && a.dt_next) a.dt_next[c] = 0.0;  // a converged case keeps its state
  if (act) {
  const int st = m.stride;
  const T* __restrict__ fsb = a.fs32;
  const T* __restrict__ fb = a.fb32;
  const int code = m.gcode[c];
  int ns[4];
#pragma unroll
  for (int q = 0; q < 4; q++) ns[q] = checked_nb(m.nbsf[q * st + c], 2, m.n, m.nb, c << 2 | q, a.status);
  auto fetch = [&](int q, FaceIn<T>& in) {
    const int bits = code >> (3 * q);
    if ((bits & 1) == 0) {
      in.kind = 0;
    } else if (ns[q] < 0) {
      in.kind = 3;
      const int b = -ns[q] - 1;
#pragma unroll
      for (int k = 0; k < 5; k++) in.s[k] = fb[k * m.bstride + b];
    } else {
      const int o = ns[q] >> 2, q2 = ns[q] & 3;
      in.kind = (bits & 4) ? 2 : 1;
#pragma unroll
      for (int k = 0; k < 5; k++) {
        in.s[k] = fsb[(q * 5 + k) * st + c];
        in.x[k] = fsb[(q2 * 5 + k) * st + o];
      }
    }
  };
  if constexpr (kPipe == 3) {
#pragma unroll
    for (int r = 0; r < 20; r++) prefetch_l2(fsb + size_t(r) * st + c);
    prefetch_update_rows(a, c, st);
  }
  [[maybe_unused]] FaceIn<T> nxt;
  [[maybe_unused]] FaceIn<T> all[4];
  if constexpr (kPipe == 2) {
#pragma unroll
    for (int q = 0; q < 4; q++) fetch(q, all[q]);
  } else if (kPipe == 1) {
    fetch(0, nxt);
  }
  T S[4][3];
  {
    T P[4][3];
    load_vertices(m, c, P, a.status);
    face_normals(P, S);
  }
  // the FP32 fluxes summed in FP32, the sum to the FP64 update
  using Acc = float;
  Acc R[5] = {Acc(0), Acc(0), Acc(0), Acc(0), Acc(0)};
#pragma unroll
  for (int q = 0; q < 4; q++) {
    FaceIn<T> cur;
    if constexpr (kPipe == 2) {
      cur = all[q];
    } else if (kPipe == 1) {
      cur = nxt;
      if (q < 3) fetch(q + 1, nxt);  // next face's loads overlap this face's flux
    } else {
      fetch(q, cur);
    }
    if (cur.kind == 3) {
#pragma unroll
      for (int k = 0; k < 5; k++) R[k] -= Acc(cur.s[k]);
    } else if (cur.kind != 0) {
      const int bits = code >> (3 * q);
      const bool own = cur.kind == 1;
      // owner-to-neighbour normal: this cell's outward normal on the owner side
      const bool flip = own ? (bits & 2) != 0 : (bits & 2) == 0;
      const T a2 = (S[q][0] * S[q][0] + S[q][1] * S[q][1]) + S[q][2] * S[q][2];
      const T inv = nr_rsqrt(a2);  // 1 / |S|
      const T area = a2 * inv;
      const T sg = flip ? -inv : inv;
      const T nh[3] = {S[q][0] * sg, S[q][1] * sg, S[q][2] * sg};
      T Fl[5];
      if (own) rusanov_fast<T>(cur.s, cur.x, nh, area, Fl);
      else rusanov_fast<T>(cur.x, cur.s, nh, area, Fl);
#pragma unroll
      for (int k = 0; k < 5; k++) R[k] = own ? R[k] - Acc(Fl[k]) : R[k] + Acc(Fl[k]);
    }
  }
  const double Rd[5] = {double(R[0]), double(R[1]), double(R[2]), double(R[3]), double(R[4])};
  double Vn[5];
  dt_next = stage_update(a, c, st, Rd, 1.0, m.vol[c], Vn);
  }
  if (a.dt_next_min) warp_min_to(dt_next, a.dt_next_min);
}

// Boundary fluxes from the owner's face state and the ghost of that state, in FP64
// from the FP32 face states, stored in FP32.
__global__ void __launch_bounds__(256) boundary_flux_copy_kernel(MeshView<double> m, TileView tv, StageArgs a) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait_previous();
  if (b >= m.nb) return;
  const int2 ref = tv.b_ref[b];
  const double4 geo = tv.b_geo[b];
  const int c = checked(ref.x >> 2, m.n, a.status), q = ref.x & 3, st = m.stride;
  double VL[5], VR[5], Fl[5];
#pragma unroll
  for (int k = 0; k < 5; k++) VL[k] = double(a.fs32[(q * 5 + k) * st + c]);
  const double nh[3] = {geo.x, geo.y, geo.z};
  ghost_state<double>(m.patches[checked(ref.y, m.n_patches, a.status)], VL, nh, VR);
  rusanov_fast<double>(VL, VR, nh, geo.w, Fl);
#pragma unroll
  for (int k = 0; k < 5; k++) a.fb32[k * m.bstride + b] = float(Fl[k]);
}

}  // namespace nf
