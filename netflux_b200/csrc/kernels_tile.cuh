// The stage kernel of the fast forms: one launch per stage does the limiter, the
// reconstruction, the boundary and interior fluxes and the stage update.
//
// A block takes one tile of TC consecutive cells of the device order (compact,
// that order being a space-filling curve) and works in shared memory:
//   1. stage the primitives of the tile's cells, of the outside cell of every
//      face that leaves the tile (a cut face), of the tile's ghosts, and of the
//      cells and ghosts those outside cells touch (the far list);
//   2. a pair of variables at a time: limiter and face states of the tile's cells, and
//      of each cut face's outside cell at that face, written over the pair's
//      staged values once every thread has read them;
//   3. boundary faces: ghost of the reconstructed state and its flux, each by the
//      warp of its cell;
//   4. per cell: four fluxes, the balance, the stage update;
//   5. the ghosts of the result, for the next stage.
// Nothing between the primitives and the updated state goes through HBM, and a
// stage is one launch (two where the ghosts have their own kernel). Separate
// limiter and flux kernels wrote and re-read 20 face states a cell (160 B out and
// 160 B in, FP64) in four launches. The price is the limiter of the cut faces'
// outside cells, 0.7 to 0.9 a cell at 256 cells a tile on meshes of compact cells (0.70
// at 393,216 tets of the channel, 0.74 at 3.1M, 0.80 in the cube of 48,000), more where
// cells are flat or stretched: those meshes go by one thread a cell (kernels_cell.cuh;
// solver.cu has the rule).
//
// A step, against those kernels: FP64 48,000 tets 62 -> 42 us, 3.1M tets 1.218 ->
// 1.100 ms; FP32 copies without the limiter, 3.1M, 0.80 -> 0.73 ms; difference form 96,000 tets 74 -> 49 us, 393,216 183 -> 159
// us, 3.1M 1.051 -> 1.050 ms. Bound by latency: about 1,860 instructions a cell at 24
// warps an SM (80 registers, three blocks), 43 % of issue slots and 33 % of the
// FP64 pipe busy; of 12.5 cycles between a warp's instructions 3 wait for global
// loads and 2.6 at barriers (393,216 tets, FP64). Loads of the tile that an SM
// takes a wave later are asked into L2 in bulk, which took 8 % off.
//
// Both cells of a face evaluate its flux from the same two states and opposite
// normals of the same bits, with exactly antisymmetric arithmetic (rusanov_raw) or
// with the owner on the left (FP32), and the outside cells' limiters are recomputed
// with the same operations on the same values, so the two contributions cancel
// exactly, inside a tile or across tiles, and a case gives the same bits alone or
// in a batch.
#pragma once

#include <type_traits>

#include "kernels_mixed.cuh"
#include "tiles.hpp"

namespace nf {

enum : int { kFormFp64 = 0, kFormDelta = 1, kFormCopy = 2 };
// what the stage kernel is compiled for: first order; second order, and the same
// with the result's ghosts; or everything (the limiter ratchet, kept limiter
// values, faces no marker lists, and the ghosts where asked for). At 3.1M tets the
// FP64 launch takes 17 us more when it leaves the ghosts (a kernel of their own 9.5
// us), and took 15 us more with the ratchet's code in it, unused.
enum : int { kModeFirst = 0, kModePlain = 1, kModeGhosts = 2, kModeGeneral = 3 };
// staged primitives V, face states S (increments in the difference form) and
// geometry G of each form
template <int kForm>
struct FormTypes {
  using V = double;
  using S = double;
  using G = double;
};
template <>
struct FormTypes<kFormDelta> {
  using V = double;
  using S = float;
  using G = float;
};
template <>
struct FormTypes<kFormCopy> {
  using V = float;
  using S = float;
  using G = float;
};

struct TileView {
  const TileHead* __restrict__ head;
  const uint2* __restrict__ code;  // per cell, four of 16 bits
  const uint2* __restrict__ vert;
  const int* __restrict__ cut_cell;
  const ushort4* __restrict__ cut_nb;
  const int* __restrict__ far_id;
  const int* __restrict__ node_id;
  const void* __restrict__ nodes;  // [n_nodes][4] of the form's geometry type
  const double4* __restrict__ b_geo;  // per boundary face: unit normal and area
  const int2* __restrict__ b_ref;     // owner cell << 2 | its face, and patch
  int n_tiles;
  int ahead;  // blocks the device holds at once
};

// Shared memory of a block: five rows of kRow values, a variable each (the
// staged values, in second order the face states in their place), then the
// tile's vertices. A row's length is fixed so that addresses within it are
// immediates.
template <int kForm, int kRow>
inline size_t tile_smem_bytes(int max_nodes) {
  using F = FormTypes<kForm>;
  return 5 * size_t(kRow) * sizeof(typename F::V) + 3 * size_t(max_nodes) * sizeof(typename F::G);
}

// raw normal 2 S of face fm (opposite vertex fm) from its vertices in ascending
// order (FP64); FP32: the normal S
template <int fm>
__device__ __forceinline__ void tile_normal(const float P[4][3], float X[3]) {
  face_normal<float, fm>(P, X);
}
template <int fm>
__device__ __forceinline__ void tile_normal(const double P[4][3], double X[3]) {
  using T = double;
  constexpr int a = fm == 0 ? 1 : 0;
  constexpr int b = fm <= 1 ? 2 : 1;
  constexpr int cc = fm == 3 ? 2 : 3;
  const T e1[3] = {P[b][0] - P[a][0], P[b][1] - P[a][1], P[b][2] - P[a][2]};
  const T e2[3] = {P[cc][0] - P[a][0], P[cc][1] - P[a][1], P[cc][2] - P[a][2]};
  X[0] = fma(e1[1], e2[2], -(e1[2] * e2[1]));
  X[1] = fma(e1[2], e2[0], -(e1[0] * e2[2]));
  X[2] = fma(e1[0], e2[1], -(e1[1] * e2[0]));
}

// v with its sign flipped where flip is set: an integer operation, off the FP64 pipe
__device__ __forceinline__ double flip_sign(double v, bool flip) {
  return __hiloint2double(__double2hiint(v) ^ (flip ? int(0x80000000u) : 0), __double2loint(v));
}
__device__ __forceinline__ float flip_sign(float v, bool flip) {
  return __int_as_float(__float_as_int(v) ^ (flip ? int(0x80000000u) : 0));
}

// products and sums rounded one by one (never contracted)
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// Four times the Rusanov flux (Numerics.cpp:10-18) out of a cell through a face
// of raw outward normal X = 2 S, from the primitive states of its own side s and
// the other side x. With q = V . X the factors of 2 stay out of the arithmetic
// (the update's scale takes them), and the spectral radius times |X| needs no
// normalised normal: c |X| = sqrt(gamma p |X|^2 / rho). Every step is exactly
// antisymmetric under exchange of the sides (the two sides' terms are added
// without contraction), so the two cells of a face get opposite bits and need
// not agree on an order.
__device__ __forceinline__ void rusanov_raw(const double s[5], const double x[5], const double X[3], double F[5]) {
  const double a2 = fma(X[2], X[2], fma(X[1], X[1], mul_rn(X[0], X[0])));
  const double qs = fma(s[3], X[2], fma(s[2], X[1], mul_rn(s[1], X[0])));
  const double qx = fma(x[3], X[2], fma(x[2], X[1], mul_rn(x[1], X[0])));
  const double ga = mul_rn(Gas<double>::gamma, a2);
  const double ts = mul_rn(ga, s[4]), tx = mul_rn(ga, x[4]);
  const double cs = mul_rn(ts, nr_rsqrt(mul_rn(ts, s[0]))), cx = mul_rn(tx, nr_rsqrt(mul_rn(tx, x[0])));
  const double lam = larger(add_rn(fabs(qs), cs), add_rn(fabs(qx), cx));
  const double ms = mul_rn(s[0], qs), mx = mul_rn(x[0], qx), ps = add_rn(s[4], x[4]);
  F[0] = fma(-lam, add_rn(x[0], -s[0]), add_rn(ms, mx));
  double ks = 0.0, kx = 0.0;
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const double ws = mul_rn(s[0], s[1 + e]), wx = mul_rn(x[0], x[1 + e]);
    ks = fma(ws, s[1 + e], ks);
    kx = fma(wx, x[1 + e], kx);
    F[1 + e] = fma(-lam, add_rn(wx, -ws), fma(ps, X[e], add_rn(mul_rn(ms, s[1 + e]), mul_rn(mx, x[1 + e]))));
  }
  const double Es = fma(Gas<double>::g1_inv, s[4], mul_rn(0.5, ks)), Ex = fma(Gas<double>::g1_inv, x[4], mul_rn(0.5, kx));
  F[4] = fma(-lam, add_rn(Ex, -Es), add_rn(mul_rn(qs, add_rn(Es, s[4])), mul_rn(qx, add_rn(Ex, x[4]))));
}

// Ask for `bytes` (a multiple of 16) from a 16-byte aligned address in L2, without waiting.
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

struct FiveValues {
  double v[5];
};
// The ghost state of a boundary face of unit normal and area geo from the
// owner's primitives (set_constant_ghost_values, Solver.cpp:300-330), and the
// flux through it from the owner's face state and the ghost of that state
// (Solver.cpp:197-229), then Rusanov. Out of line: few warps have a boundary
// face, and the far field's square roots would cost every warp registers.
static __device__ __noinline__ FiveValues boundary_ghost(const PatchBC* bc, double4 geo, FiveValues V) {
  const double nh[3] = {geo.x, geo.y, geo.z};
  FiveValues o;
  ghost_state<double, false>(*bc, V.v, nh, o.v);
  return o;
}
static __device__ __noinline__ FiveValues boundary_flux(const PatchBC* bc, double4 geo, FiveValues V) {
  const double nh[3] = {geo.x, geo.y, geo.z};
  double G[5];
  ghost_state<double, false>(*bc, V.v, nh, G);
  FiveValues o;
  rusanov_fast<double>(V.v, G, nh, geo.w, o.v);
  return o;
}

// TC cells a tile, rows of kRow values; variable k's staged value i is rv[k * kRow + i].
template <int kForm, int TC, int kRow, int kMinBlocks, int kMode>
__global__ void __launch_bounds__(TC, kMinBlocks) stage_kernel(MeshView<double> m, TileView tv, StageArgs a) {
  using V = typename FormTypes<kForm>::V;
  using S = typename FormTypes<kForm>::S;
  using G = typename FormTypes<kForm>::G;
  constexpr bool kSecond = kMode != kModeFirst, kGeneral = kMode == kModeGeneral;
  constexpr int kRowS = kRow * int(sizeof(V) / sizeof(S));  // a row's length in face states
  constexpr double kFluxScale = kForm == kFormFp64 ? 4.0 : 1.0;  // of the flux sums (rusanov_raw)
  constexpr int kDiff = kRowS - 4 * TC;                     // difference form: the own faces' V_o - V_c
  extern __shared__ __align__(16) unsigned char smem[];
  V* const rv = reinterpret_cast<V*>(smem);
  S* const rs = reinterpret_cast<S*>(smem);
  G* const nodes = reinterpret_cast<G*>(smem + 5 * kRow * sizeof(V));  // [nnode][3]
  const int t = threadIdx.x, c = blockIdx.x * TC + t, st = m.stride;
  const bool in = c < m.n;
  pdl_launch_dependents();
  // the mesh does not change: its lists are read before the previous kernel is done
  const TileHead h = tv.head[blockIdx.x];
  const uint2 code4 = tv.code[c], vert4 = tv.vert[c];  // padded to whole tiles
  const int cut0 = t < h.ncut ? checked(tv.cut_cell[h.cut0 + t], m.n, a.status) : 0;
  const int far0 = kSecond && t < h.nfar ? checked_nb(tv.far_id[h.far0 + t], 0, m.n, m.nb, 0, a.status) : 0;
  for (int i = t; i < h.nnode; i += TC) {
    const G* p = static_cast<const G*>(tv.nodes) + 4 * size_t(checked(tv.node_id[h.node0 + i], m.n_nodes, a.status));
#pragma unroll
    for (int e = 0; e < 3; e++) nodes[3 * i + e] = p[e];
  }
  // two spellings: the checked one, though checked() is the identity in the release
  // build, made first order 4 % slower there (745 against 716 us a step of 3.1M tets)
#ifdef NF_DEBUG
  auto code = [&](int q) {
    const int v = int(((q & 2) ? code4.y : code4.x) >> (16 * (q & 1)) & 0xffffu);
    return v == kFaceNone ? v : checked(v, 4 * TC + h.ncut + h.nb, a.status);
  };
#else
  auto code = [&](int q) { return int(((q & 2) ? code4.y : code4.x) >> (16 * (q & 1)) & 0xffffu); };
#endif
  auto vert = [&](int q) { return int(((q & 2) ? vert4.y : vert4.x) >> (16 * (q & 1)) & 0xffffu); };
  pdl_wait_previous();
  const bool act = in && !(a.case_frozen != nullptr && a.case_frozen[h.case_id >= 0 ? h.case_id : a.cell_case[c]] != 0);
  if (a.case_frozen != nullptr && !__syncthreads_or(act)) {  // every case of the tile has converged
    if (in && a.dt_next_min && a.dt_next) a.dt_next[c] = 0.0;
    return;
  }

  // ---- 1. stage ----
  const V* __restrict__ Vin;
  const V* __restrict__ Vg;
  if constexpr (kForm == kFormCopy) {
    Vin = a.Vin32;
    Vg = a.vg32;
  } else {
    Vin = a.Vin;
    Vg = a.vg;
  }
  const int n1 = TC + h.ncut, n2 = n1 + h.nb;  // staged numbers of the first ghost and far value
  {
    V own[5], cut[5], far[5];
    const V* pf = far0 >= 0 ? Vin + far0 : Vg + (-far0 - 1);
    const int sf = far0 >= 0 ? st : m.bstride;
#pragma unroll
    for (int k = 0; k < 5; k++) {
      own[k] = in ? Vin[k * st + c] : V(0);
      cut[k] = t < h.ncut ? Vin[k * st + cut0] : V(0);
      if (kSecond) far[k] = t < h.nfar ? pf[k * sf] : V(0);
    }
#pragma unroll
    for (int k = 0; k < 5; k++) rv[k * kRow + t] = own[k];
    if constexpr (kForm != kFormCopy) {
      if (a.dt_from_input) {
        const double d = in ? cell_next_dt<kForm == kFormFp64 && !kSecond>(a, c, st, own, m.vol[c], !act) : DBL_MAX;
        warp_min_to(d, a.dt_next_min);
      }
    }
    if (t < h.ncut) {
#pragma unroll
      for (int k = 0; k < 5; k++) rv[k * kRow + TC + t] = cut[k];
    }
    if (kSecond && t < h.nfar) {
#pragma unroll
      for (int k = 0; k < 5; k++) rv[k * kRow + n2 + t] = far[k];
    }
  }
  for (int i = t + TC; i < h.ncut; i += TC) {
    const int id = checked(tv.cut_cell[h.cut0 + i], m.n, a.status);
#pragma unroll
    for (int k = 0; k < 5; k++) rv[k * kRow + TC + i] = Vin[k * st + id];
  }
  if constexpr (kSecond) {
    for (int i = t; i < h.nb; i += TC) {
#pragma unroll
      for (int k = 0; k < 5; k++) rv[k * kRow + n1 + i] = Vg[k * m.bstride + h.b0 + i];
    }
    for (int i = t + TC; i < h.nfar; i += TC) {
      const int id = checked_nb(tv.far_id[h.far0 + i], 0, m.n, m.nb, 0, a.status);
      const V* p = id >= 0 ? Vin + id : Vg + (-id - 1);
      const int s = id >= 0 ? st : m.bstride;
#pragma unroll
      for (int k = 0; k < 5; k++) rv[k * kRow + n2 + i] = p[k * s];
    }
  }
  // the rows and lists of the tile this multiprocessor takes about one wave of
  // blocks later, so its loads find them in L2
  const int tn = int(blockIdx.x) + tv.ahead;
  if (t < 32 && tn < tv.n_tiles) {
    const int cn = tn * TC;
    const unsigned cells = unsigned(min(TC, st - cn));
    if (t < 5) prefetch_l2_bulk(Vin + size_t(t) * st + cn, cells * unsigned(sizeof(V)));
    else if (t < 10) prefetch_l2_bulk(a.Uin + size_t(t - 5) * st + cn, cells * 8u);
    else if (t < 15 && a.scheme != 0 && a.stage != 0) prefetch_l2_bulk(a.Un + size_t(t - 10) * st + cn, cells * 8u);
    else if (t == 15) prefetch_l2_bulk(m.vol + cn, cells * 8u);
    else if (t == 16 && a.local_dt) prefetch_l2_bulk(a.dt_local + cn, cells * 8u);
    else if (t == 17) prefetch_l2_bulk(tv.code + cn, TC * 8u);
    else if (t == 18) prefetch_l2_bulk(tv.vert + cn, TC * 8u);
    else if (t == 19) {
      const TileHead f = tv.head[tn];
      if (f.ncut) {
        prefetch_l2_bulk(tv.cut_cell + f.cut0, unsigned(f.ncut + 3) / 4u * 16u);
        if (kSecond) prefetch_l2_bulk(tv.cut_nb + f.cut0, unsigned(f.ncut + 1) / 2u * 16u);
      }
      if (kSecond && f.nfar) prefetch_l2_bulk(tv.far_id + f.far0, unsigned(f.nfar + 3) / 4u * 16u);
      if (f.nnode) prefetch_l2_bulk(tv.node_id + f.node0, unsigned(f.nnode + 3) / 4u * 16u);
    }
  }
  int nb[4];  // staged number of each neighbour (the cell itself: no face)
  unsigned none = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    nb[q] = staged_of(code(q), TC);
    if (code(q) == kFaceNone) {
      nb[q] = t;
      none |= 1u << q;
    }
  }
  constexpr int kRounds = kRow / TC - 4 < 4 ? kRow / TC - 4 : 4;  // of cut faces: at most four a cell
  [[maybe_unused]] ushort4 cn[kRounds];
  if constexpr (kSecond) {
#pragma unroll
    for (int r = 0; r < kRounds; r++)
      if (r * TC < h.ncut && r * TC + t < h.ncut) cn[r] = tv.cut_nb[h.cut0 + r * TC + t];
  }
  __syncthreads();

  // ---- 2. limiter and face states, a pair of variables at a time ----
  const int n_states = 4 * TC + h.ncut;
  if constexpr (kSecond) {
    const bool barth = a.barth != 0;
    // the ratchet of a tile within one case is on or off for the whole block
    const bool rat_tile = kGeneral && barth && a.lim_ratchet != nullptr && h.case_id >= 0 && a.lim_ratchet[h.case_id] != 0;
    const bool rat = kGeneral && act && (rat_tile || (barth && h.case_id < 0 && in && ratchet_on(a, c)));
    S* pdump;
    if constexpr (sizeof(S) == 8) pdump = a.phi;
    else pdump = a.phi32;
    // kLean: every face listed, one case, no kept fields (uniform over the block)
    auto variables = [&](auto lean, auto first, auto count) {
      constexpr bool kLean = decltype(lean)::value;
      constexpr int k0 = decltype(first)::value, nk = decltype(count)::value;
      S d[nk][4], s[nk][4], sc[nk][kRounds];
#pragma unroll
      for (int j = 0; j < nk; j++) {
        const V* Vk = rv + (k0 + j) * kRow;
        const V vc = Vk[t];
#pragma unroll
        for (int q = 0; q < 4; q++) d[j][q] = S(Vk[nb[q]] - vc);
        S mean;
        S phi = limiter_value(d[j], kLean ? 0u : none, S(vc), barth, &mean);
        if (rat) phi = ratchet(a, size_t(k0 + j) * st + c, phi);
        if constexpr (!kLean) {
          if (pdump && act) pdump[size_t(k0 + j) * st + c] = phi;
        }
        const S hp = S(0.5) * phi;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if constexpr (kForm == kFormDelta) s[j][q] = hp * (d[j][q] - mean);
          else s[j][q] = fma(hp, d[j][q] - mean, S(vc));
        }
      }
#pragma unroll
      for (int r = 0; r < kRounds; r++) {
        const int i = r * TC + t;
        if (r * TC < h.ncut && i < h.ncut) {
          const int slot = cn[r].x >> 14;
          const int n_staged = n2 + h.nfar;
          const int nc[4] = {checked(cn[r].x & 0x3fff, n_staged, a.status), checked(cn[r].y, n_staged, a.status),
                             checked(cn[r].z, n_staged, a.status), checked(cn[r].w, n_staged, a.status)};
          unsigned nn = 0;
          if constexpr (!kLean) {
#pragma unroll
            for (int q = 0; q < 4; q++)
              if (nc[q] == TC + i) nn |= 1u << q;
          }
#pragma unroll
          for (int j = 0; j < nk; j++) {
            const V* Vk = rv + (k0 + j) * kRow;
            const V vc = Vk[TC + i];
            S dc[4];
#pragma unroll
            for (int q = 0; q < 4; q++) dc[q] = S(Vk[nc[q]] - vc);
            S mean;
            S phi = limiter_value(dc, nn, S(vc), barth, &mean);
            if (rat_tile || (!kLean && barth && a.lim_ratchet != nullptr && h.case_id < 0)) {
              const int id = r == 0 ? cut0 : checked(tv.cut_cell[h.cut0 + i], m.n, a.status);
              if (rat_tile || ratchet_on(a, id)) phi = ratchet_seen(a, size_t(k0 + j) * st + id, phi);
            }
            const S ds = slot & 2 ? (slot & 1 ? dc[3] : dc[2]) : (slot & 1 ? dc[1] : dc[0]), hp = S(0.5) * phi;
            if constexpr (kForm == kFormDelta) sc[j][r] = hp * (ds - mean);
            else sc[j][r] = fma(hp, ds - mean, S(vc));
          }
        }
      }
      __syncthreads();  // the staged values of these variables are no longer needed
#pragma unroll
      for (int j = 0; j < nk; j++) {
        S* Sk = rs + (k0 + j) * kRowS;
#pragma unroll
        for (int q = 0; q < 4; q++) Sk[q * TC + t] = s[j][q];
        if constexpr (kForm == kFormDelta) {
#pragma unroll
          for (int q = 0; q < 4; q++) Sk[kDiff + q * TC + t] = d[j][q];
        }
#pragma unroll
        for (int r = 0; r < kRounds; r++)
          if (r * TC < h.ncut && r * TC + t < h.ncut) Sk[4 * TC + r * TC + t] = sc[j][r];
      }
    };
    auto all = [&](auto lean) {
      using std::integral_constant;
      variables(lean, integral_constant<int, 0>(), integral_constant<int, 2>());
      variables(lean, integral_constant<int, 2>(), integral_constant<int, 2>());
      variables(lean, integral_constant<int, 4>(), integral_constant<int, 1>());
    };
    if constexpr (kGeneral) {
      if (h.open == 0 && (h.case_id >= 0 || a.lim_ratchet == nullptr) && pdump == nullptr) all(std::true_type());
      else all(std::false_type());
    } else {
      all(std::true_type());
    }
    __syncthreads();
  }

  // ---- 3. boundary faces: their fluxes after the face states, or (first order)
  // in the place of their ghosts. They lie in the order of their cells, so in second
  // order a warp does those of its own cells, a range, and no other waits for it
  // (a step of 48,000 tets 42.8 -> 41.6 us, of 393,216 in the difference form 168 ->
  // 163 us, of 3.1M 1.118 -> 1.102 ms). In first order the block shares them: the
  // kernel has little else to do (178,000 tets 1.1 % slower by warps) ----
  [[maybe_unused]] int b_first = 1 << 30, b_end = 0;  // of this warp's cells (none: empty)
  if (h.nb > 0) {
    if constexpr (kSecond) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (code(q) >= n_states && code(q) != kFaceNone) {
          b_first = min(b_first, code(q) - n_states);
          b_end = max(b_end, code(q) - n_states + 1);
        }
      }
      b_first = __reduce_min_sync(0xffffffffu, b_first);
      b_end = __reduce_max_sync(0xffffffffu, b_end);
    } else {
      b_first = 0;
      b_end = h.nb;
    }
    for (int i = b_first + (kSecond ? t & 31 : t); i < b_end; i += kSecond ? 32 : TC) {
      const int2 ref = tv.b_ref[h.b0 + i];
      const double4 geo = tv.b_geo[h.b0 + i];
      const int cb = checked(ref.x >> 2, m.n, a.status), q = ref.x & 3;
      const int lc = checked(cb - int(blockIdx.x) * TC, TC, a.status);
      const PatchBC* bc = m.patches + checked(ref.y, m.n_patches, a.status);
      FiveValues VL;
      [[maybe_unused]] double Vc[5];
#pragma unroll
      for (int k = 0; k < 5; k++) {
        if constexpr (kForm == kFormDelta) {
          Vc[k] = a.Vin[k * st + cb];
          VL.v[k] = kSecond ? Vc[k] + double(rs[k * kRowS + q * TC + lc]) : Vc[k];
        } else {
          VL.v[k] = double(kSecond ? rs[k * kRowS + q * TC + lc] : S(rv[k * kRow + lc]));
        }
      }
      FiveValues fl = boundary_flux(bc, geo, VL);
      if constexpr (kForm == kFormDelta) {
        // minus the owner's physical flux through the face, area F(V_c) . n
        const double nh[3] = {geo.x, geo.y, geo.z}, area = geo.w;
        const double qn = (Vc[1] * nh[0] + Vc[2] * nh[1]) + Vc[3] * nh[2];
        const double m0 = Vc[0] * qn;
        const double E =
            Gas<double>::g1_inv * Vc[4] + 0.5 * Vc[0] * ((Vc[1] * Vc[1] + Vc[2] * Vc[2]) + Vc[3] * Vc[3]);
        const double Fc[5] = {m0, m0 * Vc[1] + Vc[4] * nh[0], m0 * Vc[2] + Vc[4] * nh[1], m0 * Vc[3] + Vc[4] * nh[2],
                              qn * (E + Vc[4])};
#pragma unroll
        for (int k = 0; k < 5; k++) fl.v[k] -= area * Fc[k];
      } else {
#pragma unroll
        for (int k = 0; k < 5; k++) fl.v[k] *= kFluxScale;
      }
#pragma unroll
      for (int k = 0; k < 5; k++) {
        if constexpr (kSecond) rs[k * kRowS + n_states + i] = S(fl.v[k]);
        else rv[k * kRow + n1 + i] = V(S(fl.v[k]));
      }
    }
    if constexpr (kSecond) __syncwarp();
    else __syncthreads();
  }

  // ---- 4. fluxes and update ----
  double dt_next = DBL_MAX, Vn[5];
  if (!act) {
    if (in && a.dt_next_min && a.dt_next) a.dt_next[c] = 0.0;  // a converged case keeps its state
  } else {
    G P[4][3];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int e = 0; e < 3; e++) P[q][e] = nodes[3 * checked(vert(q) & kVertIndex, h.nnode, a.status) + e];
    // a boundary face's flux, or nothing for a face not listed; true: an interior face
    using Acc = typename std::conditional<kForm == kFormDelta, double, S>::type;
    Acc R[5] = {Acc(0), Acc(0), Acc(0), Acc(0), Acc(0)};
    auto interior = [&](int q) {
      if (code(q) < n_states) return true;
      if (code(q) != kFaceNone) {
#pragma unroll
        for (int k = 0; k < 5; k++)
          R[k] -= kSecond ? Acc(rs[k * kRowS + code(q)]) : Acc(rv[k * kRow + nb[q]]);
      }
      return false;
    };
    G X[3] = {G(0), G(0), G(0)};
    if constexpr (kForm == kFormDelta) {
      double vcd[5];
      float vc[5], slist[3] = {0.f, 0.f, 0.f};  // sum of the listed faces' outward normals
#pragma unroll
      for (int k = 0; k < 5; k++) {
        vcd[k] = a.Vin[k * st + c];
        vc[k] = float(vcd[k]);
      }
      auto face = [&](int q) {
        const bool inward = (vert(q) & kVertFlip) != 0;
        const float Sn[3] = {flip_sign(X[0], inward), flip_sign(X[1], inward), flip_sign(X[2], inward)};
        if ((kGeneral || !kSecond) && none && !(none >> q & 1)) {
#pragma unroll
          for (int e = 0; e < 3; e++) slist[e] += Sn[e];
        }
        if (!interior(q)) return;
        float s[5], x[5], Fl[5];
#pragma unroll
        for (int k = 0; k < 5; k++) {
          if constexpr (kSecond) {
            s[k] = rs[k * kRowS + q * TC + t];
            x[k] = rs[k * kRowS + kDiff + q * TC + t] + rs[k * kRowS + code(q)];
          } else {
            s[k] = 0.f;
            x[k] = float(rv[k * kRow + nb[q]] - vcd[k]);
          }
        }
        const float a2 = fmaf(Sn[2], Sn[2], fmaf(Sn[1], Sn[1], Sn[0] * Sn[0]));
        const float inv = nr_rsqrt(a2);  // 1 / |S|
        const float nh[3] = {Sn[0] * inv, Sn[1] * inv, Sn[2] * inv};
        rusanov_delta(vc, s, x, nh, a2 * inv, Fl);
#pragma unroll
        for (int k = 0; k < 5; k++) R[k] -= double(Fl[k]);
      };
      tile_normal<0>(P, X);
      face(0);
      tile_normal<1>(P, X);
      face(1);
      tile_normal<2>(P, X);
      face(2);
      tile_normal<3>(P, X);
      face(3);
      if ((kGeneral || !kSecond) && none) {
        // A boundary face that no marker lists is dropped (FV_Grid.cpp:79-85), so
        // the listed normals do not sum to zero: R = R_diff - F(V_c) . sum_listed S.
        const double sx = slist[0], sy = slist[1], sz = slist[2];
        const double qs = (vcd[1] * sx + vcd[2] * sy) + vcd[3] * sz;
        const double m0 = vcd[0] * qs;
        const double E =
            Gas<double>::g1_inv * vcd[4] + 0.5 * vcd[0] * ((vcd[1] * vcd[1] + vcd[2] * vcd[2]) + vcd[3] * vcd[3]);
        R[0] -= m0;
        R[1] -= m0 * vcd[1] + vcd[4] * sx;
        R[2] -= m0 * vcd[2] + vcd[4] * sy;
        R[3] -= m0 * vcd[3] + vcd[4] * sz;
        R[4] -= qs * (E + vcd[4]);
      }
      dt_next = stage_update(a, c, st, R, 1.0, m.vol[c], Vn);
    } else {
      auto face = [&](int q) {
        if (!interior(q)) return;
        const bool inward = (vert(q) & kVertFlip) != 0;
        S s[5], x[5], Fl[5];
        if constexpr (kForm == kFormFp64) {
          const S Xo[3] = {flip_sign(X[0], inward), flip_sign(X[1], inward), flip_sign(X[2], inward)};
          const S* ps = rs + t;
          const S* px = rs + (kSecond ? code(q) : nb[q]);
#pragma unroll
          for (int k = 0; k < 5; k++) {
            s[k] = ps[k * kRowS + (kSecond ? q * TC : 0)];
            x[k] = px[k * kRowS];
          }
          rusanov_raw(s, x, Xo, Fl);
#pragma unroll
          for (int k = 0; k < 5; k++) R[k] -= Fl[k];
        } else {
          // FP32: the reference's owner on the left and its unit normal, in the
          // operations the form has always used (its rounding, amplified by the
          // limiter's switches, shows in long runs)
          const bool side = (vert(q) & kVertSide) != 0;
          const int own = kSecond ? q * TC + t : t, other = kSecond ? code(q) : nb[q];
          const S* pL = rs + (side ? other : own);
          const S* pR = rs + (side ? own : other);
#pragma unroll
          for (int k = 0; k < 5; k++) {
            s[k] = pL[k * kRowS];
            x[k] = pR[k * kRowS];
          }
          const S a2 = (X[0] * X[0] + X[1] * X[1]) + X[2] * X[2];
          const S inv = nr_rsqrt(a2);  // 1 / |S|
          const S sg = inward != side ? -inv : inv;
          const S nh[3] = {X[0] * sg, X[1] * sg, X[2] * sg};
          rusanov_fast<S>(s, x, nh, a2 * inv, Fl);
#pragma unroll
          for (int k = 0; k < 5; k++) R[k] = side ? R[k] + Fl[k] : R[k] - Fl[k];
        }
      };
      tile_normal<0>(P, X);
      face(0);
      tile_normal<1>(P, X);
      face(1);
      tile_normal<2>(P, X);
      face(2);
      tile_normal<3>(P, X);
      face(3);
      const double Rd[5] = {double(R[0]), double(R[1]), double(R[2]), double(R[3]), double(R[4])};
      dt_next = stage_update(a, c, st, Rd, 1.0 / kFluxScale, m.vol[c], Vn);
    }
  }
  if (a.dt_next_min && !a.dt_from_input) warp_min_to(dt_next, a.dt_next_min);

  // ---- 5. the result's ghosts, which the next stage stages ----
  if constexpr (kMode == kModeGhosts || kGeneral) {
    if (h.nb > 0 && (kForm == kFormCopy ? a.vg_next32 != nullptr : a.vg_next != nullptr)) {
      for (int i0 = b_first; i0 < b_end; i0 += 32) {
        const int i = i0 + (t & 31);
        const bool mine = i < b_end;
        int2 ref = make_int2(0, 0);
        if (mine) ref = tv.b_ref[h.b0 + i];
        const int src = checked(ref.x >> 2, m.n, a.status) & 31;  // its cell's lane
        FiveValues v;
#pragma unroll
        for (int k = 0; k < 5; k++) v.v[k] = double(V(__shfl_sync(0xffffffffu, Vn[k], src)));
        const bool moved = __shfl_sync(0xffffffffu, int(act), src) != 0;
        if (!mine || !moved) continue;  // a converged case keeps its state and its ghosts
        const FiveValues g = boundary_ghost(m.patches + checked(ref.y, m.n_patches, a.status), tv.b_geo[h.b0 + i], v);
#pragma unroll
        for (int k = 0; k < 5; k++) {
          if constexpr (kForm == kFormCopy) a.vg_next32[k * m.bstride + h.b0 + i] = float(g.v[k]);
          else a.vg_next[k * m.bstride + h.b0 + i] = g.v[k];
        }
      }
    }
  }
}

}  // namespace nf
