// The fast forms' stage as kernels of one thread a cell, for meshes whose tiles are
// cut through too often for the stage kernel (kernels_tile.cuh; solver.cu has the
// rule): flat or stretched cells, whose device order (a curve through the centroids)
// gives thin tiles, cells in no order, and first order on large meshes. In second
// order the limiter kernel writes four face states a cell, the boundary kernel the
// boundary fluxes, and the flux kernel reads both, own and opposite, from HBM: 320 B a
// cell more than the stage kernel in FP64, but nothing twice for a cut face. Bound by
// the latency of their gathered reads.
//
// Every operation is the stage kernel's, in its order, so a case gives the same bits
// whichever of the two a mesh, or a batch that it is part of, takes.
//
// Per launch at 1.3M tets, limiter / flux kernel: FP64 69 / 110 us, differences 51 /
// 111, FP32 copies 35 / 85; first order 89 (FP64). A step of a mesh flat 50:1, against
// limiter and flux kernels of before the stage kernel and against the stage kernel:
// FP64 643 and 2,034 -> 503 us, differences 541 and 1,651 -> 453, FP32 copies 430 and
// 796 -> 340, FP64 first order 323 and 403 -> 279.
#pragma once

#include "kernels_tile.cuh"

namespace nf {

template <int kForm>
struct CellIO {  // where a form keeps primitives, ghosts, face states and boundary fluxes
  using F = FormTypes<kForm>;
  using V = typename F::V;
  using S = typename F::S;
  static __device__ __forceinline__ const V* vin(const StageArgs& a) {
    if constexpr (kForm == kFormCopy) return a.Vin32;
    else return a.Vin;
  }
  static __device__ __forceinline__ const V* vg(const StageArgs& a) {
    if constexpr (kForm == kFormCopy) return a.vg32;
    else return a.vg;
  }
  static __device__ __forceinline__ S* fs(const StageArgs& a) {
    if constexpr (sizeof(S) == 8) return a.fs;
    else return a.fs32;
  }
  static __device__ __forceinline__ S* fb(const StageArgs& a) {
    if constexpr (sizeof(S) == 8) return a.fb;
    else return a.fb32;
  }
  static __device__ __forceinline__ S* phi(const StageArgs& a) {
    if constexpr (sizeof(S) == 8) return a.phi;
    else return a.phi32;
  }
};

// Ask the memory system to bring a line into L2 without holding a register;
// the later load of the same address then waits on an L2 hit, not on DRAM.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The own-cell rows the stage update reads (Uin, Un, the local dt).
__device__ __forceinline__ void prefetch_update_rows(const StageArgs& a, int c, int st) {
#pragma unroll
  for (int k = 0; k < 5; k++) prefetch_l2(a.Uin + size_t(k) * st + c);
  if (a.scheme != 0 && a.stage != 0) {
#pragma unroll
    for (int k = 0; k < 5; k++) prefetch_l2(a.Un + size_t(k) * st + c);
  }
  if (a.local_dt) prefetch_l2(a.dt_local + c);
}

// Limiter and face states (increments in the difference form) of a cell, and the
// next step's dt where the stage computes it from its input.
template <int kForm>
__global__ void __launch_bounds__(128) face_state_kernel(MeshView<double> m, StageArgs a) {
  using IO = CellIO<kForm>;
  using V = typename IO::V;
  using S = typename IO::S;
  const int c = blockIdx.x * blockDim.x + threadIdx.x, st = m.stride;
  const bool in = c < m.n;
  pdl_launch_dependents();
  int nb[4] = {0, 0, 0, 0};  // the mesh does not change: read before the previous kernel is done
  unsigned none = 0;
  if (in) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      nb[q] = checked_nb(m.nbvf[q * st + c], 0, m.n, m.nb, c, a.status);
      if (nb[q] == c) none |= 1u << q;
    }
  }
  pdl_wait_previous();
  const bool act = in && !frozen_cell(a, c);
  double own[5];
  if (act) {
    const V* __restrict__ Vin = IO::vin(a);
    const V* __restrict__ Vg = IO::vg(a);
    S* __restrict__ fsc = IO::fs(a) + c;
    const V* qb[4];
    int qs[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const bool cell = nb[q] >= 0;
      qb[q] = cell ? Vin + nb[q] : Vg + (-nb[q] - 1);
      qs[q] = cell ? st : m.bstride;
    }
    const bool barth = a.barth != 0, rat = barth && ratchet_on(a, c);
    S* const pdump = IO::phi(a);
    auto fetch = [&](int k, V& vc, V vo[4]) {
      vc = Vin[size_t(k) * st + c];
#pragma unroll
      for (int q = 0; q < 4; q++) vo[q] = qb[q][k * qs[q]];
    };
    auto variable = [&](int k, V vc, const V vo[4]) {
      S d[4], mean;
#pragma unroll
      for (int q = 0; q < 4; q++) d[q] = S(vo[q] - vc);
      S phi = limiter_value(d, none, S(vc), barth, &mean);
      if (rat) phi = ratchet(a, size_t(k) * st + c, phi);
      if (pdump) pdump[size_t(k) * st + c] = phi;
      const S hp = S(0.5) * phi;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        S s;
        if constexpr (kForm == kFormDelta) s = hp * (d[q] - mean);
        else s = fma(hp, d[q] - mean, S(vc));
        fsc[size_t(q * 5 + k) * st] = s;
      }
    };
    // every load before any arithmetic: one wait for memory instead of five
    V vc[5], vo[5][4];
#pragma unroll
    for (int k = 0; k < 5; k++) fetch(k, vc[k], vo[k]);
#pragma unroll
    for (int k = 0; k < 5; k++) {
      own[k] = double(vc[k]);
      variable(k, vc[k], vo[k]);
    }
  }
  if constexpr (kForm != kFormCopy) {
    if (a.dt_from_input) {
      if (!act)
#pragma unroll
        for (int k = 0; k < 5; k++) own[k] = 1.0;  // not read
      const double d = in ? cell_next_dt<false>(a, c, st, own, m.vol[c], !act) : DBL_MAX;
      warp_min_to(d, a.dt_next_min);
    }
  }
}

// Flux through each boundary face from its owner's face state (primitives in first
// order); in the difference form minus the owner's physical flux through it.
template <int kForm, bool kSecond>
__global__ void __launch_bounds__(128) boundary_face_kernel(MeshView<double> m, TileView tv, StageArgs a) {
  using IO = CellIO<kForm>;
  using S = typename IO::S;
  constexpr double kFluxScale = kForm == kFormFp64 ? 4.0 : 1.0;
  const int b = blockIdx.x * blockDim.x + threadIdx.x, st = m.stride;
  pdl_launch_dependents();
  pdl_wait_previous();
  if (b >= m.nb) return;
  const int2 ref = tv.b_ref[b];
  const double4 geo = tv.b_geo[b];
  const int cb = checked(ref.x >> 2, m.n, a.status), q = ref.x & 3;
  const PatchBC* bc = m.patches + checked(ref.y, m.n_patches, a.status);
  FiveValues VL;
  [[maybe_unused]] double Vc[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const S s = kSecond ? IO::fs(a)[size_t(q * 5 + k) * st + cb] : S(0);
    if constexpr (kForm == kFormDelta) {
      Vc[k] = a.Vin[k * st + cb];
      VL.v[k] = kSecond ? Vc[k] + double(s) : Vc[k];
    } else {
      VL.v[k] = double(kSecond ? s : S(IO::vin(a)[k * st + cb]));
    }
  }
  FiveValues fl = boundary_flux(bc, geo, VL);
  if constexpr (kForm == kFormDelta) {
    const double nh[3] = {geo.x, geo.y, geo.z}, area = geo.w;
    const double qn = (Vc[1] * nh[0] + Vc[2] * nh[1]) + Vc[3] * nh[2];
    const double m0 = Vc[0] * qn;
    const double E = Gas<double>::g1_inv * Vc[4] + 0.5 * Vc[0] * ((Vc[1] * Vc[1] + Vc[2] * Vc[2]) + Vc[3] * Vc[3]);
    const double Fc[5] = {m0, m0 * Vc[1] + Vc[4] * nh[0], m0 * Vc[2] + Vc[4] * nh[1], m0 * Vc[3] + Vc[4] * nh[2],
                          qn * (E + Vc[4])};
#pragma unroll
    for (int k = 0; k < 5; k++) fl.v[k] -= area * Fc[k];
  } else {
#pragma unroll
    for (int k = 0; k < 5; k++) fl.v[k] *= kFluxScale;
  }
#pragma unroll
  for (int k = 0; k < 5; k++) IO::fb(a)[k * m.bstride + b] = S(fl.v[k]);
}

// Four fluxes, the balance and the stage update of a cell.
template <int kForm, bool kSecond, int kMinBlocks>
__global__ void __launch_bounds__(128, kMinBlocks)
    cell_flux_kernel(MeshView<typename FormTypes<kForm>::G> m, StageArgs a) {
  using IO = CellIO<kForm>;
  using V = typename IO::V;
  using S = typename IO::S;
  using G = typename FormTypes<kForm>::G;
  constexpr double kFluxScale = kForm == kFormFp64 ? 4.0 : 1.0;
  const int c = blockIdx.x * blockDim.x + threadIdx.x, st = m.stride;
  const bool in = c < m.n;
  pdl_launch_dependents();
  int ns[4] = {0, 0, 0, 0}, code = 0;
  G P[4][3];
  if (in) {
    code = m.gcode[c];
#pragma unroll
    for (int q = 0; q < 4; q++) ns[q] = checked_nb(m.nbsf[q * st + c], 2, m.n, m.nb, c << 2 | q, a.status);
    load_vertices(m, c, P, a.status);
  }
  pdl_wait_previous();
  const bool act = in && !frozen_cell(a, c);
  const V* __restrict__ Vin = IO::vin(a);
  const S* __restrict__ fsb = IO::fs(a);
  const S* __restrict__ fb = IO::fb(a);
  [[maybe_unused]] double vcd[5];
  double dt_next = DBL_MAX, Vn[5];
  if (!act) {
    if (in && a.dt_next_min && a.dt_next) a.dt_next[c] = 0.0;  // a converged case keeps its state
  } else {
    if constexpr (kSecond) {
#pragma unroll
      for (int r = 0; r < 20; r++) prefetch_l2(fsb + size_t(r) * st + c);
    }
    prefetch_update_rows(a, c, st);
    using Acc = typename std::conditional<kForm == kFormDelta, double, S>::type;
    Acc R[5] = {Acc(0), Acc(0), Acc(0), Acc(0), Acc(0)};
    [[maybe_unused]] V vc[5];
    if constexpr (!kSecond || kForm == kFormDelta) {
#pragma unroll
      for (int k = 0; k < 5; k++) {
        vc[k] = Vin[k * st + c];
        vcd[k] = double(vc[k]);
      }
    }
    // both sides' states (differences to the cell's own primitives in the difference form)
    auto sides = [&](int q, S s[5], S x[5]) {
      const int o = ns[q] >> 2, q2 = ns[q] & 3;
#pragma unroll
      for (int k = 0; k < 5; k++) {
        if constexpr (kForm == kFormDelta) {
          const S d = S(Vin[size_t(k) * st + o] - vc[k]);
          s[k] = kSecond ? fsb[size_t(q * 5 + k) * st + c] : S(0);
          x[k] = kSecond ? d + fsb[size_t(q2 * 5 + k) * st + o] : d;
        } else {
          s[k] = kSecond ? fsb[size_t(q * 5 + k) * st + c] : S(vc[k]);
          x[k] = kSecond ? fsb[size_t(q2 * 5 + k) * st + o] : S(Vin[size_t(k) * st + o]);
        }
      }
    };
    // a boundary face's flux, or nothing for a face not listed; true: an interior face
    auto interior = [&](int q) {
      if ((code >> (3 * q) & 1) == 0) return false;
      if (ns[q] >= 0) return true;
      const int b = -ns[q] - 1;
#pragma unroll
      for (int k = 0; k < 5; k++) R[k] -= Acc(fb[k * m.bstride + b]);
      return false;
    };
    G X[3] = {G(0), G(0), G(0)};
    if constexpr (kForm == kFormDelta) {
      float vcf[5], slist[3] = {0.f, 0.f, 0.f};  // sum of the listed faces' outward normals
#pragma unroll
      for (int k = 0; k < 5; k++) vcf[k] = float(vcd[k]);
      const bool open = (code & 0x249) != 0x249;
      auto face = [&](int q) {
        const bool inward = (code >> (3 * q) & 2) != 0;
        const float Sn[3] = {flip_sign(X[0], inward), flip_sign(X[1], inward), flip_sign(X[2], inward)};
        if (open && (code >> (3 * q) & 1)) {
#pragma unroll
          for (int e = 0; e < 3; e++) slist[e] += Sn[e];
        }
        if (!interior(q)) return;
        float s[5], x[5], Fl[5];
        sides(q, s, x);
        const float a2 = fmaf(Sn[2], Sn[2], fmaf(Sn[1], Sn[1], Sn[0] * Sn[0]));
        const float inv = nr_rsqrt(a2);  // 1 / |S|
        const float nh[3] = {Sn[0] * inv, Sn[1] * inv, Sn[2] * inv};
        rusanov_delta(vcf, s, x, nh, a2 * inv, Fl);
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
      if (open) {  // R = R_diff - F(V_c) . sum_listed S (kernels_tile.cuh)
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
    } else {
      auto face = [&](int q) {
        if (!interior(q)) return;
        const bool inward = (code >> (3 * q) & 2) != 0;
        S s[5], x[5], Fl[5];
        sides(q, s, x);
        if constexpr (kForm == kFormFp64) {
          const S Xo[3] = {flip_sign(X[0], inward), flip_sign(X[1], inward), flip_sign(X[2], inward)};
          rusanov_raw(s, x, Xo, Fl);
#pragma unroll
          for (int k = 0; k < 5; k++) R[k] -= Fl[k];
        } else {  // the reference's owner on the left
          const bool side = (code >> (3 * q) & 4) != 0;
          S sL[5], sR[5];
#pragma unroll
          for (int k = 0; k < 5; k++) {
            sL[k] = side ? x[k] : s[k];
            sR[k] = side ? s[k] : x[k];
          }
          const S a2 = (X[0] * X[0] + X[1] * X[1]) + X[2] * X[2];
          const S inv = nr_rsqrt(a2);  // 1 / |S|
          const S sg = inward != side ? -inv : inv;
          const S nh[3] = {X[0] * sg, X[1] * sg, X[2] * sg};
          rusanov_fast<S>(sL, sR, nh, a2 * inv, Fl);
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
    }
    const double Rd[5] = {double(R[0]), double(R[1]), double(R[2]), double(R[3]), double(R[4])};
    dt_next = stage_update(a, c, st, Rd, 1.0 / kFluxScale, m.vol[c], Vn);
  }
  if (a.dt_next_min && (!a.dt_from_input || !kSecond)) {
    if constexpr (!kSecond && kForm != kFormCopy) {
      if (a.dt_from_input) {
        if (!act)
#pragma unroll
          for (int k = 0; k < 5; k++) vcd[k] = 1.0;  // not read
        dt_next = in ? cell_next_dt<kForm == kFormFp64>(a, c, st, vcd, m.vol[c], !act) : DBL_MAX;
      }
    }
    warp_min_to(dt_next, a.dt_next_min);
  }
}

}  // namespace nf
