// Per-cell gather kernels of one explicit step on the device mesh: the
// reference-order form whole, and what the fast forms' stage kernel
// (kernels_tile.cuh) is made of.
//
// Layout (all arrays resident in HBM for the whole run; cell c is the c-th
// cell along the Hilbert curve):
//   cell SoA    U, W, V[2], phi : [5][stride], grad : [15][stride] (k*3+d)
//               vol, dt_local   : [stride], dS : [3][stride]
//   cell slots  slot : [4][stride] = face << 1 | side (side 0: the cell is the
//               face's owner i, side 1: its neighbour j), -1 = no face. The 4
//               slots of a cell list its faces in the reference's global face
//               order, which is the order the reference accumulates the
//               gradient and the flux balance of that cell in
//               (FV_Grid.cpp:135-137, 207-227), so every per-cell sum below
//               adds the same terms in the same order as the face loops of
//               Numerics.hpp:112-127 and Solver.cpp:171-229.
//               nbslot : [4][stride] = neighbour << 2 | the neighbour's slot
//               of the same face, or -(1 + patch) at a boundary face
//   face states fs : [4][5][stride], the limited reconstruction of the cell's
//               primitives at each of its faces (written by the gradient
//               kernel, read by the flux kernel of both adjacent cells)
//   face SoA    S, nhat : [3][F]; area : [F]
//   slot SoA    rs : [3][4][stride], the vector from the cell centroid to the
//               centroid of each of its faces (r_i or r_j of the face)
//   boundary    b_cell, b_slot, b_face, b_patch : [nb]; ghost states vg and
//               boundary fluxes fb : [5][bstride]
// The slots, face states, face arrays and boundary fluxes are the
// reference-order form's. Each face's flux is evaluated by both of its cells, so
// that both see bit-identical values; no atomics, deterministic results. The
// reference-order gradient kernel runs one thread per (cell, variable), its flux
// kernel four threads per cell (one per face slot).
#pragma once

#include <type_traits>

#include <cuda_runtime.h>

#include "euler.cuh"

namespace nf {

// Geometry and topology of the device mesh (T: double, or float for the
// mixed-precision face work).
template <typename T>
struct MeshView {
  int n;          // interior cells
  int stride;     // SoA stride of cell arrays
  int n_faces;
  const int* __restrict__ slot;    // [4][stride] face << 1 | side
  const int* __restrict__ nbslot;  // [4][stride] neighbour << 2 | its slot, or -(1 + boundary face)
  const T* __restrict__ S;         // [3][F]
  const T* __restrict__ nhat;      // [3][F]
  const T* __restrict__ area;      // [F]
  const T* __restrict__ rs;        // [3][4][stride] centroid-to-face vector of each slot
  // node-based geometry of the fast forms (face m = the face opposite vertex m)
  const T* __restrict__ nodes;     // [n_nodes][4] x, y, z, 0
  const int* __restrict__ cnode;   // [4][stride] vertices of each cell, ascending node id
  const int* __restrict__ gcode;   // [stride] per face m, bits 3m..3m+2: present, outward flip, neighbour side
  const int* __restrict__ nbvf;    // [4][stride] neighbour cell of face m, -(1 + boundary face), or the cell itself
  const int* __restrict__ nbsf;    // [4][stride] neighbour << 2 | its face index, or -(1 + boundary face)
  const double* __restrict__ vol;
  const double* __restrict__ dS;
  const PatchBC* __restrict__ patches;
  // boundary faces, ordered by owner cell
  int nb;                          // number of boundary faces
  int bstride;                     // SoA stride of boundary arrays
  const int* __restrict__ b_cell;  // owner cell
  const int* __restrict__ b_slot;  // owner's slot of the face
  const int* __restrict__ b_face;  // face id (geometry)
  const int* __restrict__ b_patch; // patch
  int n_nodes;                     // for the index checks of NF_DEBUG builds
  int n_patches;
};

// Index checks of NF_DEBUG builds (make debug): every index a kernel reads
// from the mesh arrays or a tile's lists is checked before it is used (the lists'
// own bounds, TileHead, are not); an index out of range
// sets kErrIndex in the status word and is replaced by a valid one (0, or the
// cell itself), so the access stays in bounds and the host reports the error.
// In the release build these are the identity.
__device__ __forceinline__ int checked(int idx, int limit, unsigned* status) {
#ifdef NF_DEBUG
  if (idx < 0 || idx >= limit) {
    atomicOr(status, kErrIndex);
    return 0;
  }
#endif
  return idx;
}
// a neighbour code: cell << shift (| slot) below n cells, or -(1 + boundary face) below nb
__device__ __forceinline__ int checked_nb(int code, int shift, int n, int nb, int self, unsigned* status) {
#ifdef NF_DEBUG
  const bool ok = code >= 0 ? (code >> shift) < n : (-code - 1) < nb;
  if (!ok) {
    atomicOr(status, kErrIndex);
    return self;
  }
#endif
  return code;
}

struct StageArgs {
  int second_order;      // SpatialOrder::Second
  int barth;             // Limiter::Barth
  int scheme;            // 0 explicit Euler, 1 TVD-RK3
  int stage;             // 0, 1, 2
  int local_dt;
  int freeze;            // a cell with dt == 0 keeps its state exactly (converged case)
  const double* Vin;     // primitives of the stage input [5][stride]
  double* fs;            // reconstructed face states [4 slots][5][stride]
  double* grad;          // optional copy of the gradient [15][stride] (k*3+d)
  double* phi;           // optional copy of the limiter [5][stride]
  const double* Uin;     // stage input state (own cell)
  const double* Un;      // U^n (stages 1, 2)
  double* Uout;          // may alias Uin
  double* Vout;          // primitives of Uout
  double* R;             // optional flux-balance dump [5][stride]
  double* res_cell;      // optional R_rho / vol per cell (first stage)
  const double* dt_local;
  const double* scal;    // device scalars: [0] dt (min target), [1] time, [2] t_end
  unsigned* status;
  // mixed forms: kept stage fields; FP32 copies under the limiter: face states
  // [4][5][stride] and boundary fluxes [5][bstride]
  float* fs32;
  float* fb32;
  float* grad32;
  float* phi32;
  // boundary faces: cell-centre ghost states [5][bstride] and boundary fluxes
  // [5][bstride] (reference-order form)
  double* vg;
  double* fb;
  // mixed form with FP32 copies (NF_PREC_MIXED32): the FP32 primitives of
  // the stage input and of its result, and FP32 ghost states [5][bstride].
  // Vout (FP64) is written only where a later time step reads it (null otherwise).
  const float* Vin32;
  float* Vout32;
  float* vg32;
  // fast forms, second order: where the stage kernel puts the cell-centre ghosts
  // of its result, the next stage's (the other of two buffers; null: not needed)
  double* vg_next;
  float* vg_next32;
  // fast forms: a stage that has the primitives the reference's calc_timestep
  // reads (those of the last stage's input, Solver.cpp:250) also computes the
  // next step's time step from them: the last stage from its input
  // (dt_from_input; after the halo exchange of a split mesh), and the form with
  // FP32 copies, which stages no FP64 primitives, under TVD-RK3 stage 2 of 3 from
  // its FP64 result. Per cell into dt_next (local time stepping, else null) and
  // the minimum into *dt_next_min (null: not this stage)
  int dt_from_input;
  double* dt_next;
  unsigned long long* dt_next_min;
  const double* dS;  // [3][stride] projected areas (calc_Delta_S)
  double cfl;
  // converged cases of a steady solve (null: none); their cells are skipped
  // by the fast kernels (cases share no faces, and U is left untouched)
  const int* case_frozen;
  // limiter ratchet (extension): per-cell case, per-case switch (null: off)
  // and the kept limiter values [5][stride] (FP64 or FP32 with the state form)
  const int* cell_case;
  const int* lim_ratchet;
  double* phi_keep;
  float* phi_keep32;
};

// Programmatic dependent launch (the fast forms' stage kernels are launched
// with programmatic stream serialization, solver.cu): a kernel lets the next
// one in the stream launch once all of its blocks have started, and waits for
// the previous one to complete (its writes visible) before reading anything
// that kernel wrote. The next kernel's launch and block set-up then overlap
// this one's last wave. Launched without the attribute, both are no-ops.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Once a case's ratchet is on, a cell's limiter value is the minimum of the
// live value and the kept one, and is kept: it only tightens, so it settles
// and the steady residual can converge (the live Barth limiter makes it stall).
// Where another tile needs the cell's limiter in the same stage it evaluates the
// same live value and takes the minimum with the kept one without writing it
// (ratchet_seen): the same result whether it reads the kept value before or
// after the owner's update, as that is the minimum with the same live value.
__device__ __forceinline__ bool frozen_cell(const StageArgs& a, int c) {
  return a.case_frozen != nullptr && a.case_frozen[a.cell_case[c]] != 0;
}
__device__ __forceinline__ bool ratchet_on(const StageArgs& a, int c) {
  return a.lim_ratchet != nullptr && a.lim_ratchet[a.cell_case[c]] != 0;
}
template <typename T>
__device__ __forceinline__ T ratchet_seen(const StageArgs& a, size_t at, T phi) {
  const volatile T* keep;
  if constexpr (sizeof(T) == 8) keep = a.phi_keep;
  else keep = a.phi_keep32;
  const T v = keep[at];
  return (v < phi) ? v : phi;  // std::min(phi, kept)
}
template <typename T>
__device__ __forceinline__ T ratchet(const StageArgs& a, size_t at, T phi) {
  volatile T* keep;
  if constexpr (sizeof(T) == 8) keep = a.phi_keep;
  else keep = a.phi_keep32;
  const T v = ratchet_seen(a, at, phi);
  keep[at] = v;
  return v;
}

// device scalars: the step's dt (minimum), the time, t_end, the dt last used,
// and the next step's dt while the last stage computes it
enum : int { kScalDtMin = 0, kScalTime = 1, kScalTEnd = 2, kScalDtUsed = 3, kScalDtNext = 4, kScalCount = 8 };

__device__ __forceinline__ double stage_dt(const double* scal) {
  double dt = scal[kScalDtMin];
  const double t_end = scal[kScalTEnd];
  if (t_end > 0.0) {
    const double left = t_end - scal[kScalTime];
    dt = (left < dt) ? left : dt;
  }
  return dt;
}

// The reference-order kernels run in FP64 (T = double).
template <typename T>
__device__ __forceinline__ T ld_v(const StageArgs& a, int idx) {
  static_assert(sizeof(T) == 8, "FP64 kernels");
  return a.Vin[idx];
}

// Four threads per cell: lane q of a quad owns the cell's face slot q. A
// cell's per-face terms are combined across its quad with shuffles, folded in
// slot order q = 0, 1, 2, 3, so sums keep the reference's order. A missing
// slot contributes -0.0, which leaves any IEEE sum unchanged.
constexpr unsigned kFull = 0xffffffffu;

template <typename T>
__device__ __forceinline__ T quad_sum_ordered(T v) {
  T s = T(0);
#pragma unroll
  for (int p = 0; p < 4; p++) s = s + __shfl_sync(kFull, v, p, 4);
  return s;
}

// ---------------------------------------------------------------------------
// Green-Gauss gradient + min/max + Barth limiter
// (calc_green_gauss_gradient, calc_max_and_min_values, calc_barth_limiter,
//  Numerics.hpp:86-292), then the limited reconstruction at each face
// (calc_limited_reconstruction, Numerics.hpp:135-145), which is what the flux
// kernel consumes. Ghost states at boundary faces are the cell-centre ghosts
// of set_constant_ghost_values (Solver.cpp:300-330).
//
// One thread per (cell, primitive variable k): every step of this kernel acts
// on one variable at a time, so the five threads of a cell share nothing but
// the cell's geometry (same addresses, served once per warp). Each thread
// folds its cell's faces in slot order, exactly as the reference's face loops
// reach that cell.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) gradient_limiter_kernel(MeshView<T> m, StageArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = t / 5;
  const int k = t - 5 * c;
  if (c >= m.n) return;
  const int st = m.stride;
  const int F = m.n_faces;
  int sl[4], ns[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    sl[q] = m.slot[q * st + c];
    sl[q] = sl[q] < 0 ? -1 : (checked(sl[q] >> 1, F, a.status) << 1 | (sl[q] & 1));
    ns[q] = checked_nb(m.nbslot[q * st + c], 2, m.n, m.nb, c << 2, a.status);
  }
  const T vc = ld_v<T>(a, k * st + c);
  const T vol = T(m.vol[c]);
  T g[3] = {T(0), T(0), T(0)};
  T vmax = -std::numeric_limits<T>::max(), vmin = std::numeric_limits<T>::max();
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (sl[q] < 0) continue;
    const int f = sl[q] >> 1;
    const bool own = (sl[q] & 1) == 0;
    T vo;
    if (ns[q] >= 0) vo = ld_v<T>(a, k * st + (ns[q] >> 2));
    else vo = a.vg[k * m.bstride + (-ns[q] - 1)];
    // the neighbour side subtracts its term: (-x)/v == -(x/v) and
    // g + (-y) == g - y exactly, so a signed normal reproduces both branches
    const T s0 = m.S[f], s1 = m.S[F + f], s2 = m.S[2 * F + f];
    const T Sg[3] = {own ? s0 : -s0, own ? s1 : -s1, own ? s2 : -s2};
    const T uf = T(0.5) * (vc + vo);  // 0.5 (V_i + V_j); the sum commutes exactly
#pragma unroll
    for (int d = 0; d < 3; d++) g[d] = g[d] + uf * Sg[d] / vol;
    const T vi = own ? vc : vo, vj = own ? vo : vc;  // max(V_i, V_j) in the face's operand order
    vmax = rmax(vmax, rmax(vi, vj));
    vmin = rmin(vmin, rmin(vi, vj));
  }
  // grad V_k . r at each face: the limiter's Delta_2 before its sign/epsilon
  // adjustment, and the increment of the reconstruction
  T gr[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const T* r = m.rs + q * st + c;  // [d][q][cell]
    gr[q] = (g[0] * r[0] + g[1] * r[4 * st]) + g[2] * r[8 * st];
  }
  T phi = T(1);
  if (a.barth) {
    phi = std::numeric_limits<T>::max();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (sl[q] < 0) continue;
      T d2 = gr[q];
      const T sg = (d2 > T(0)) ? T(1) : ((d2 < T(0)) ? T(-1) : T(0));
      d2 = sg * (fabs(d2) + Gas<T>::eps);
      T fc = T(1);
      if (d2 != T(0)) {
        const T num = (d2 > T(0)) ? vmax - vc : vmin - vc;
        fc = rmin(T(1), num / d2);
      }
      phi = rmin(phi, fc);
    }
    if (ratchet_on(a, c)) phi = ratchet(a, size_t(k) * st + c, phi);
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (sl[q] < 0) continue;
    a.fs[(q * 5 + k) * st + c] = vc + phi * gr[q];
  }
  if (a.grad) {
#pragma unroll
    for (int d = 0; d < 3; d++) a.grad[(k * 3 + d) * st + c] = g[d];
    a.phi[k * st + c] = phi;
  }
}

// ---------------------------------------------------------------------------
// Face fluxes, flux balance R and the stage update of one cell
// (evaluate_inviscid_fluxes Solver.cpp:144-230, rusanov Numerics.cpp:10-18,
//  TVD_RK3 Solver.cpp:103-133, explicit_euler 83-101), then the primitives of
// the new state for the next stage (set_primvars, SolverData.cpp:37-48).
// The face states come from gradient_limiter_kernel (second order) or are the
// cell primitives (first order). Lane q evaluates the flux of face slot q.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) flux_update_kernel(MeshView<T> m, StageArgs a) {
  const int q = threadIdx.x & 3;
  int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  const bool valid = c < m.n;
  if (!valid) c = m.n - 1;
  const int st = m.stride;
  const int F = m.n_faces;
  const bool second = a.second_order != 0;
  int sl = m.slot[q * st + c];
  sl = sl < 0 ? -1 : (checked(sl >> 1, F, a.status) << 1 | (sl & 1));
  const int ns = checked_nb(m.nbslot[q * st + c], 2, m.n, m.nb, c << 2 | q, a.status);
  const bool has = sl >= 0;
  const bool own = (sl & 1) == 0;
  // this face's contribution to R: -F on the owner side, +F on the other
  double contrib[5] = {-0.0, -0.0, -0.0, -0.0, -0.0};
  if (has && ns < 0) {
    // boundary face (this cell is its owner): flux from boundary_flux_kernel
    const int b = -ns - 1;
#pragma unroll
    for (int k = 0; k < 5; k++) contrib[k] = -a.fb[k * m.bstride + b];
  } else if (has) {
    const int f = sl >> 1;
    const T nh[3] = {m.nhat[f], m.nhat[F + f], m.nhat[2 * F + f]};
    const T area = m.area[f];
    T Vs[5], Vx[5];  // this cell's face state, the other side's
    const int o = ns >> 2, q2 = ns & 3;
#pragma unroll
    for (int k = 0; k < 5; k++) {
      if (second) {
        Vs[k] = a.fs[(q * 5 + k) * st + c];
        Vx[k] = a.fs[(q2 * 5 + k) * st + o];
      } else {
        Vs[k] = ld_v<T>(a, k * st + c);
        Vx[k] = ld_v<T>(a, k * st + o);
      }
    }
    const T* VL = own ? Vs : Vx;
    const T* VR = own ? Vx : Vs;
    T Fl[5], UL[5], UR[5];
    prim_to_cons<T, true>(VL, UL);
    prim_to_cons<T, true>(VR, UR);
    rusanov_ref<T>(UL, UR, nh, area, Fl);
#pragma unroll
    for (int k = 0; k < 5; k++) contrib[k] = own ? -double(Fl[k]) : double(Fl[k]);
  }
  // flux balance, accumulated in face-slot order: ((0 + c0) + c1) + ...
  double R[5];
#pragma unroll
  for (int k = 0; k < 5; k++) R[k] = quad_sum_ordered(contrib[k]);

  // ---- stage update (FP64); every lane computes it, lanes store by component ----
  const double vol = m.vol[c];
  const double dt = a.local_dt ? a.dt_local[c] : stage_dt(a.scal);
  double U[5], Uo[5];
#pragma unroll
  for (int k = 0; k < 5; k++) U[k] = a.Uin[k * st + c];
  if (a.scheme == 1 && a.stage > 0) {
#pragma unroll
    for (int k = 0; k < 5; k++) Uo[k] = a.Un[k * st + c];
  }
  double Unew[5];
  if (a.scheme == 0 || a.stage == 0) {
    const double qf = dt / vol;
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = U[k] + qf * R[k];
  } else if (a.stage == 1) {
    const double qf = 1.0 / 4.0 * dt / vol;
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = 3.0 / 4.0 * Uo[k] + 1.0 / 4.0 * U[k] + qf * R[k];
  } else {
    const double qf = 2.0 / 3.0 * dt / vol;
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = 1.0 / 3.0 * Uo[k] + 2.0 / 3.0 * U[k] + qf * R[k];
  }
  if (a.freeze && dt == 0.0) {
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = U[k];
  }
  double Vn[5];
  cons_to_prim<double, true>(Unew, Vn);
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    if (k == q || (k == 4 && q == 0)) {
      a.Uout[k * st + c] = Unew[k];
      a.Vout[k * st + c] = Vn[k];
        if (a.R) a.R[k * st + c] = R[k];
    }
  }
  if (q == 0) {
    if (a.res_cell) a.res_cell[c] = R[0] / vol;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 5; k++) finite = finite && isfinite(R[k]) && isfinite(Unew[k]);
    if (!finite) atomicOr(a.status, kErrNonFinite);
    else if (!(Vn[0] > 0.0) || !(Vn[4] > 0.0)) atomicOr(a.status, kErrNonPhysical);
  }
}

// Per-cell CFL time step of EulerSolver::calc_timestep (Solver.cpp:232-274) on
// one cell's primitives, every operation rounded on its own (no contraction)
// in the reference's order, so the result is the reference's bit for bit in
// every translation unit.
__device__ __forceinline__ double dt_of_cell(const double V[5], double dS0, double dS1, double dS2, double vol,
                                             double cfl) {
  const double cs = __dsqrt_rn(__ddiv_rn(__dmul_rn(Gas<double>::gamma, V[4]), V[0]));
  const double sx = __dmul_rn(__dadd_rn(fabs(V[1]), cs), dS0);
  const double sy = __dmul_rn(__dadd_rn(fabs(V[2]), cs), dS1);
  const double sz = __dmul_rn(__dadd_rn(fabs(V[3]), cs), dS2);
  return __ddiv_rn(__dmul_rn(cfl, vol), __dadd_rn(__dadd_rn(sx, sy), sz));
}

// Minimum of v over the warp, then one atomicMin on the bit pattern (exact
// and order-free for positive doubles), skipped when the warp's minimum is not
// below the current one (the value only decreases, so the result is the same
// exact minimum); no block barrier. Every lane of the warp calls it.
__device__ __forceinline__ void warp_min_to(double v, unsigned long long* target) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0 && v < DBL_MAX &&
      v < __longlong_as_double(static_cast<long long>(*reinterpret_cast<volatile unsigned long long*>(target))))
    atomicMin(target, (unsigned long long)__double_as_longlong(v));
}

// ---------------------------------------------------------------------------
// Fast forms (FP64 with contraction, and mixed FP32): one thread per cell, the
// cell's faces indexed by the vertex they face, geometry rebuilt from the
// vertices (the node array stays in L2):
//   * the vertices of a cell are stored sorted by node id, so face m's three
//     vertices, taken in that order, are the same ordered triple in both cells
//     of the face and give bit-identical normals S = 0.5 (B - A) x (C - A);
//     a per-face bit turns S outward;
//   * the vector from the centroid to the centroid of face m is
//     (centroid - P_m) / 3.
// The reconstruction of a tetrahedron needs no geometry. With lambda_m the
// barycentric coordinate of vertex m, the outward normal of the face opposite it
// is S_m = -3 vol grad(lambda_m), and r_m = (centroid - P_m) / 3, so for the
// Green-Gauss gradient (Numerics.hpp:86-128) of the neighbours' values V_p
//   grad V . r_m = -1/2 sum_p (V_p + V_c) grad(lambda_p) . (centroid - P_m)
//                = -1/2 sum_p (V_p + V_c) (1/4 - [p = m]) = 1/2 (V_m - M),
//   M = mean of the four neighbours' values.
// So it takes only the cell's own and its neighbours' primitives: no vertices,
// normals, volume or face codes (agreement with the reference form to
// round-off). A missing face (a boundary face no marker
// lists, FV_Grid.cpp:79-85) has S = r = 0 and names the cell itself; the sum
// then runs over the listed faces, M = 1/4 sum_listed (V_p + V_c) - V_c.
// The Barth limiter (Numerics.hpp:148-250) is
//   phi = min(1, min_m A_m / D_m), A_m = (V_max - V_c) or (V_c - V_min) by the
//   sign of grad V . r_m, D_m = |grad V . r_m| + eps;
// A_m is the same for all faces of one sign, so only the largest and the
// smallest increment count, and with the formula above those are the largest
// and the smallest neighbour value. One division per variable.
// ---------------------------------------------------------------------------
// Node records are 4 values (x, y, z, pad) from a 256-byte aligned buffer, so
// a record starts on 32 bytes (FP64) or 16 bytes (FP32): x and y come in one
// 16-byte load (FP64), or the whole record in one (FP32).
template <typename T>
__device__ __forceinline__ void load_vertices(const MeshView<T>& m, int c, T P[4][3], unsigned* status) {
#pragma unroll
  for (int v = 0; v < 4; v++) {
    const int id = checked(m.cnode[v * m.stride + c], m.n_nodes, status);
    const T* p = m.nodes + 4 * size_t(id);
    if constexpr (sizeof(T) == 8) {
      const double2 xy = *reinterpret_cast<const double2*>(p);
      P[v][0] = xy.x;
      P[v][1] = xy.y;
      P[v][2] = p[2];
    } else {
      const float4 r = *reinterpret_cast<const float4*>(p);
      P[v][0] = r.x;
      P[v][1] = r.y;
      P[v][2] = r.z;
    }
  }
}

// normal of face fm (opposite vertex fm) from its vertices in ascending order
template <typename T, int fm>
__device__ __forceinline__ void face_normal(const T P[4][3], T S[3]) {
  constexpr int a = fm == 0 ? 1 : 0;
  constexpr int b = fm <= 1 ? 2 : 1;
  constexpr int cc = fm == 3 ? 2 : 3;
  const T e1[3] = {P[b][0] - P[a][0], P[b][1] - P[a][1], P[b][2] - P[a][2]};
  const T e2[3] = {P[cc][0] - P[a][0], P[cc][1] - P[a][1], P[cc][2] - P[a][2]};
  S[0] = T(0.5) * (e1[1] * e2[2] - e1[2] * e2[1]);
  S[1] = T(0.5) * (e1[2] * e2[0] - e1[0] * e2[2]);
  S[2] = T(0.5) * (e1[0] * e2[1] - e1[1] * e2[0]);
}

template <typename T>
__device__ __forceinline__ void face_normals(const T P[4][3], T S[4][3]) {
  face_normal<T, 0>(P, S[0]);
  face_normal<T, 1>(P, S[1]);
  face_normal<T, 2>(P, S[2]);
  face_normal<T, 3>(P, S[3]);
}

// max(v, 0) by the sign bit, off the FP64 pipe; FP32 minima and maxima are one
// instruction. (A NaN anywhere in a cell's neighbourhood reaches the states
// through the mean.)
__device__ __forceinline__ double positive_part(double v) { return __double2hiint(v) < 0 ? 0.0 : v; }
__device__ __forceinline__ float positive_part(float v) { return fmaxf(v, 0.f); }
__device__ __forceinline__ void order_pair(double a, double b, double& lo, double& hi) {
  const bool s = a < b;
  lo = s ? a : b;
  hi = s ? b : a;
}
__device__ __forceinline__ void order_pair(float a, float b, float& lo, float& hi) {
  lo = fminf(a, b);
  hi = fmaxf(a, b);
}
__device__ __forceinline__ double larger(double a, double b) { return a < b ? b : a; }
__device__ __forceinline__ float larger(float a, float b) { return fmaxf(a, b); }

// The limiter value of one variable (1 without a limiter) from the neighbours'
// values minus the cell's own, d; *mean receives M - V_c, so the increment at
// face m is 1/2 (d_m - *mean). none: bit m set where face m is not listed (its d
// is 0 then); vc is the cell's own value. The operations are spelled out (fma)
// so that every place that evaluates a cell gets the same bits.
template <typename T>
__device__ __forceinline__ T limiter_value(const T d[4], unsigned none, T vc, bool barth, T* mean) {
  const T sum = (d[0] + d[1]) + (d[2] + d[3]);
  T mu = T(0.25) * sum;
  // faces not listed add -1/2 V_c each to M - V_c
  if (none) mu = fma(T(0.25), sum, T(-0.5) * T(__popc(none)) * vc);
  *mean = mu;
  if (!barth) return T(1);
  T l0, h0, l1, h1;
  order_pair(d[0], d[1], l0, h0);
  order_pair(d[2], d[3], l1, h1);
  const T dmax = larger(h0, h1), dmin = -larger(-l0, -l1);
  T gh = dmax - mu, gl = mu - dmin;  // twice the largest and the smallest increment's size
  if (none) {  // listed faces only
    gh = gl = T(0);
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (!(none >> q & 1)) {
        gh = larger(gh, d[q] - mu);
        gl = larger(gl, mu - d[q]);
      }
  }
  T An = T(1), Dn = T(1);  // best ratio so far, starting at 1
  const T Ah = positive_part(dmax), Dh = fma(T(0.5), gh, Gas<T>::eps);   // V_max - V_c
  const T Al = positive_part(-dmin), Dl = fma(T(0.5), gl, Gas<T>::eps);  // V_c - V_min
  if (gh > T(0) && Ah < Dh) {
    An = Ah;
    Dn = Dh;
  }
  const bool better = gl > T(0) && Al * Dn < An * Dl;
  An = better ? Al : An;
  Dn = better ? Dl : Dn;
  return An * nr_rcp(Dn);
}

// CFL time step of one cell from its primitives with the fast forms'
// reciprocal and reciprocal square root (within 2 ulp of dt_of_cell).
__device__ __forceinline__ double dt_of_cell_fast(const double V[5], double dS0, double dS1, double dS2, double vol,
                                                  double cfl) {
  const double g = Gas<double>::gamma * V[4];
  const double cs = g * nr_rsqrt(g * V[0]);  // sqrt(gamma p / rho)
  const double sum = fma(fabs(V[3]) + cs, dS2, fma(fabs(V[2]) + cs, dS1, (fabs(V[1]) + cs) * dS0));
  return cfl * vol * nr_rcp(sum);
}

// The Green-Gauss gradient itself (calc_green_gauss_gradient, Numerics.hpp:86-128)
// for nf_get_field: the step never reads it, so it is computed apart, only
// where the stage fields are kept. One thread per cell, from the primitives V
// and ghosts Vg in FP64 or FP32, into out [15][stride] (k*3+d).
template <typename T, typename Vt>
__global__ void __launch_bounds__(128) gradient_field_kernel(MeshView<T> m, StageArgs a, const Vt* __restrict__ V,
                                                             const Vt* __restrict__ Vg, T* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n || frozen_cell(a, c)) return;
  const int st = m.stride;
  const int code = m.gcode[c];
  T P[4][3], S[4][3], ssum[3] = {T(0), T(0), T(0)};
  load_vertices(m, c, P, a.status);
  face_normals(P, S);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int bits = code >> (3 * q);
    const T sgn = (bits & 1) == 0 ? T(0) : ((bits & 2) ? T(-1) : T(1));  // 0: no face
#pragma unroll
    for (int e = 0; e < 3; e++) ssum[e] += (S[q][e] *= sgn);
  }
  const bool closed = (code & 0x249) == 0x249;  // the listed normals sum to zero
  const double ivol = 1.0 / m.vol[c];
  for (int k = 0; k < 5; k++) {
    const Vt vc = V[size_t(k) * st + c];
    T g[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int nb = checked_nb(m.nbvf[q * st + c], 0, m.n, m.nb, c, a.status);
      const T d = T((nb >= 0 ? V[size_t(k) * st + nb] : Vg[size_t(k) * m.bstride + (-nb - 1)]) - vc);
#pragma unroll
      for (int e = 0; e < 3; e++) g[e] = fma(d, S[q][e], g[e]);
    }
#pragma unroll
    for (int e = 0; e < 3; e++)
      out[size_t(k * 3 + e) * st + c] =
          T(0.5 * ivol) * g[e] + (closed ? T(0) : T(double(vc) * double(ssum[e]) * ivol));
  }
}

// The next step's time step of one cell from the primitives the reference's
// calc_timestep reads (a.dt_next_min set): written where local time stepping
// keeps it; returns its part of the minimum. A frozen cell keeps its state (dt 0).
// kRef: with the reference's operations and rounding, as timestep_kernel.
template <bool kRef>
__device__ __forceinline__ double cell_next_dt(const StageArgs& a, int c, int st, const double V[5], double vol,
                                               bool frozen) {
  if (frozen) {
    if (a.dt_next) a.dt_next[c] = 0.0;
    return DBL_MAX;
  }
  double d;
  if constexpr (kRef) d = dt_of_cell(V, a.dS[c], a.dS[st + c], a.dS[2 * st + c], vol, a.cfl);
  else d = dt_of_cell_fast(V, a.dS[c], a.dS[st + c], a.dS[2 * st + c], vol, a.cfl);
  if (a.dt_next) a.dt_next[c] = d;
  if (!(d > 0.0) && !isnan(d)) atomicOr(a.status, kErrDt);
  return d > 0.0 ? d : DBL_MAX;  // std::min skips NaN (comparisons with NaN are false)
}

// Stage update of one cell from its flux balance rs * R (TVD_RK3
// Solver.cpp:103-133, explicit_euler 83-101) in FP64, then the primitives of the
// new state (set_primvars, SolverData.cpp:37-48), the optional dumps and the
// status. Returns the cell's part of the next step's minimum time step where
// this stage computes it from its result, DBL_MAX otherwise. rs is a power of
// two; Vn receives the new primitives.
__device__ __forceinline__ double stage_update(const StageArgs& a, int c, int st, const double R[5], double rs,
                                               double vol, double Vn[5]) {
  const double dt = a.local_dt ? a.dt_local[c] : stage_dt(a.scal);
  double Unew[5];
  const double ivol = rs * nr_rcp(vol);
  if (a.scheme == 0 || a.stage == 0) {
    const double qf = dt * ivol;
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = fma(qf, R[k], a.Uin[k * st + c]);
  } else if (a.stage == 1) {
    const double qf = 0.25 * dt * ivol;
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = 0.75 * a.Un[k * st + c] + 0.25 * a.Uin[k * st + c] + qf * R[k];
  } else {
    const double qf = 2.0 / 3.0 * dt * ivol;
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = 1.0 / 3.0 * a.Un[k * st + c] + 2.0 / 3.0 * a.Uin[k * st + c] + qf * R[k];
  }
  if (a.freeze && dt == 0.0) {
#pragma unroll
    for (int k = 0; k < 5; k++) Unew[k] = a.Uin[k * st + c];
  }
  cons_to_prim<double, false>(Unew, Vn);
  // a non-finite R makes Unew non-finite (dt / vol is finite), so Unew alone is
  // checked, by the exponents
  int top = 0;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    a.Uout[k * st + c] = Unew[k];
    top = max(top, __double2hiint(Unew[k]) & 0x7fffffff);
  }
  if (a.Vout) {
#pragma unroll
    for (int k = 0; k < 5; k++) a.Vout[k * st + c] = Vn[k];
  }
  if (a.Vout32) {
#pragma unroll
    for (int k = 0; k < 5; k++) a.Vout32[k * st + c] = float(Vn[k]);
  }
  if (a.R) {
#pragma unroll
    for (int k = 0; k < 5; k++) a.R[k * st + c] = rs * R[k];
  }
  if (a.res_cell) a.res_cell[c] = R[0] * ivol;
  if (top >= 0x7ff00000) atomicOr(a.status, kErrNonFinite);
  else if (!(Vn[0] > 0.0) || !(Vn[4] > 0.0)) atomicOr(a.status, kErrNonPhysical);
  return a.dt_next_min && !a.dt_from_input ? cell_next_dt<false>(a, c, st, Vn, vol, a.freeze && dt == 0.0) : DBL_MAX;
}

// ---------------------------------------------------------------------------
// Boundary faces of the reference-order form. ghost_kernel: the cell-centre ghost
// state of every boundary face (set_constant_ghost_values, Solver.cpp:300-330),
// read by the gradient kernel like a neighbour's primitives.
// boundary_flux_kernel: the flux through every boundary face, from the owner's
// reconstructed face state and the ghost built from that state
// (Solver.cpp:197-229), read by the flux kernel at the face's slot. One thread
// per boundary face; the other kernels carry no boundary-condition code.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) ghost_kernel(MeshView<T> m, StageArgs a) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= m.nb) return;
  const int c = checked(m.b_cell[b], m.n, a.status), f = checked(m.b_face[b], m.n_faces, a.status);
  const int F = m.n_faces, st = m.stride;
  T V[5], G[5];
#pragma unroll
  for (int k = 0; k < 5; k++) V[k] = ld_v<T>(a, k * st + c);
  const T nh[3] = {m.nhat[f], m.nhat[F + f], m.nhat[2 * F + f]};
  ghost_state<T>(m.patches[checked(m.b_patch[b], m.n_patches, a.status)], V, nh, G);
#pragma unroll
  for (int k = 0; k < 5; k++) a.vg[k * m.bstride + b] = G[k];
}

template <typename T>
__global__ void __launch_bounds__(256) boundary_flux_kernel(MeshView<T> m, StageArgs a) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= m.nb) return;
  const int c = checked(m.b_cell[b], m.n, a.status), q = checked(m.b_slot[b], 4, a.status),
            f = checked(m.b_face[b], m.n_faces, a.status);
  const int F = m.n_faces, st = m.stride;
  T VL[5], VR[5];
#pragma unroll
  for (int k = 0; k < 5; k++) VL[k] = a.second_order ? a.fs[(q * 5 + k) * st + c] : ld_v<T>(a, k * st + c);
  const T nh[3] = {m.nhat[f], m.nhat[F + f], m.nhat[2 * F + f]};
  ghost_state<T>(m.patches[checked(m.b_patch[b], m.n_patches, a.status)], VL, nh, VR);
  T Fl[5], UL[5], UR[5];
  prim_to_cons<T, true>(VL, UL);
  prim_to_cons<T, true>(VR, UR);
  rusanov_ref<T>(UL, UR, nh, m.area[f], Fl);
#pragma unroll
  for (int k = 0; k < 5; k++) a.fb[k * m.bstride + b] = Fl[k];
}

// ---------------------------------------------------------------------------
// Time step (EulerSolver::calc_timestep, Solver.cpp:232-274): per cell
// CFL*vol / sum_d (|u_d| + c) dS_d from the given primitives; the global dt
// is their minimum (atomicMin on the bit pattern, exact and order-free for
// positive doubles).
// ---------------------------------------------------------------------------
struct DtArgs {
  const double* V;
  double cfl;
  double* dt_local;  // per-cell dt, or nullptr
  unsigned long long* dt_min_bits;
  unsigned* status;
  const int* cell_case;    // case of each cell (batched meshes)
  const int* case_frozen;  // nonzero: the case has converged; its cells get dt = 0
};

template <bool kRef>
__global__ void __launch_bounds__(256) timestep_kernel(MeshView<double> m, DtArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  double dtc = DBL_MAX;
  if (c < m.n) {
    const int st = m.stride;
    double V[5];
#pragma unroll
    for (int k = 0; k < 5; k++) V[k] = a.V[k * st + c];
    const double d = dt_of_cell(V, m.dS[c], m.dS[st + c], m.dS[2 * st + c], m.vol[c], a.cfl);
    const bool frozen = a.case_frozen && a.case_frozen[a.cell_case[c]];
    if (a.dt_local) a.dt_local[c] = frozen ? 0.0 : d;
    if (!frozen) {
      if (!(d > 0.0) && !isnan(d)) atomicOr(a.status, kErrDt);
      if (d > 0.0) dtc = d;  // std::min skips NaN (comparisons with NaN are false)
    }
  }
  // warp then block minimum, one atomic per block
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) dtc = fmin(dtc, __shfl_xor_sync(0xffffffffu, dtc, off));
  __shared__ double wmin[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) wmin[warp] = dtc;
  __syncthreads();
  if (warp == 0) {
    dtc = (lane < (blockDim.x + 31) / 32) ? wmin[lane] : DBL_MAX;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dtc = fmin(dtc, __shfl_xor_sync(0xffffffffu, dtc, off));
    if (lane == 0) atomicMin(a.dt_min_bits, (unsigned long long)__double_as_longlong(dtc));
  }
}

}  // namespace nf
