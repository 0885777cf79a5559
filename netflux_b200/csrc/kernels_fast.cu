// Launchers of the forms with reciprocals and fused multiply-adds: FP64, and the
// mixed forms (FP32 face work; FP64 state, ghosts, boundary fluxes and update).
#include <type_traits>
#include <utility>

#include "kernels_copy.cuh"
#include "launch.hpp"

namespace nf {

template <bool kRef>
__global__ void __launch_bounds__(256) prim_kernel_fast(int n, int st, const double* __restrict__ U,
                                                       double* __restrict__ V, float* __restrict__ V32) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double u[5], v[5];
#pragma unroll
  for (int k = 0; k < 5; k++) u[k] = U[k * st + c];
  cons_to_prim<double, kRef>(u, v);
#pragma unroll
  for (int k = 0; k < 5; k++) {
    V[k * st + c] = v[k];
    if (V32) V32[k * st + c] = float(v[k]);
  }
}

static inline int grid_for(int n, int block) { return (n + block - 1) / block; }

// Launch with programmatic stream serialization: the kernel may start while
// the previous kernel in the stream finishes (it waits for it on the device
// before reading its results, pdl_wait_previous). Captured into the step's
// CUDA graph as a programmatic dependency.
template <typename... P, typename... A>
static void launch_pdl(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// ---- the stage kernel ----
// Threads an SM should hold, which caps a thread's registers: three blocks of 256
// at 80 registers (also what their shared memory allows), four at 64 for the form
// with FP32 copies. Per launch at 3.1M tets: FP64 455 us with two blocks at 128
// registers, 369 us with three; FP32 copies 291 us with three, 251 us with four;
// difference form 374 us with three, 408 us with four (spills).
template <int kForm>
constexpr int kThreadsPerSm = kForm == kFormCopy ? 1024 : 768;

// f(kernel, form, row length) for the form, tile size and mode
template <typename Fn>
static void with_stage_kernel(int form, int tile, int mode, Fn&& f) {
  auto order = [&](auto frm, auto tc, auto row) {
    constexpr int kF = decltype(frm)::value, kT = decltype(tc)::value, kR = decltype(row)::value;
    constexpr int kB = kThreadsPerSm<kF> / kT;
    if (mode == kModeFirst) f(stage_kernel<kF, kT, kR, kB, kModeFirst>, frm, row);
    else if (mode == kModePlain) f(stage_kernel<kF, kT, kR, kB, kModePlain>, frm, row);
    else if (mode == kModeGhosts) f(stage_kernel<kF, kT, kR, kB, kModeGhosts>, frm, row);
    else f(stage_kernel<kF, kT, kR, kB, kModeGeneral>, frm, row);
  };
  auto size = [&](auto frm) {
    using std::integral_constant;
    // 256 threads: the largest tile whose lists fit three times in an SM's shared
    // memory (at 3.1M tets FP64 369 us a launch, 379 us at 192, 413 us at 160,
    // 520 us or more at 128). Small meshes whose tiles touch more than its rows hold
    // (thin or flat ones) take 128 with longer rows.
    if (tile == 256) order(frm, integral_constant<int, 256>(), integral_constant<int, 6 * 256>());
    else order(frm, integral_constant<int, 128>(), integral_constant<int, 8 * 128>());
  };
  if (form == kFormFp64) size(std::integral_constant<int, kFormFp64>());
  else if (form == kFormDelta) size(std::integral_constant<int, kFormDelta>());
  else size(std::integral_constant<int, kFormCopy>());
}

size_t stage_smem(int form, const Tiles& t, bool second) {
  size_t bytes = 0;
  with_stage_kernel(form, t.tile, second ? kModePlain : kModeFirst, [&](auto, auto frm, auto row) {
    constexpr int kR = decltype(row)::value;
    const bool fits = (second ? t.max_staged2 : t.max_staged1) <= kR && (!second || t.max_states <= kR);
    bytes = fits ? tile_smem_bytes<decltype(frm)::value, kR>(t.max_nodes) : 0;
  });
  return bytes;
}
cudaError_t stage_setup(int form, int tile, int mode, int max_smem, size_t smem, int* blocks) {
  cudaError_t e = cudaSuccess;
  with_stage_kernel(form, tile, mode, [&](auto k, auto, auto) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, tile, smem);
  });
  return e;
}
void launch_stage(int form, int tile, int mode, const MeshView<double>& m, const TileView& tv, const StageArgs& a,
                  size_t smem, cudaStream_t st) {
  with_stage_kernel(form, tile, mode, [&](auto k, auto, auto) { launch_pdl(k, tv.n_tiles, tile, smem, st, m, tv, a); });
}
// ---- the same stage by one thread a cell ----
// f(form) or f(form, second order) with compile-time values
template <typename Fn>
static void with_form(int form, Fn&& f) {
  using std::integral_constant;
  if (form == kFormFp64) f(integral_constant<int, kFormFp64>());
  else if (form == kFormDelta) f(integral_constant<int, kFormDelta>());
  else f(integral_constant<int, kFormCopy>());
}
template <typename Fn>
static void with_form_order(int form, bool second, Fn&& f) {
  with_form(form, [&](auto frm) {
    if (second) f(frm, std::true_type());
    else f(frm, std::false_type());
  });
}
void launch_cell_states(int form, const MeshView<double>& m, const StageArgs& a, cudaStream_t st) {
  with_form(form, [&](auto f) {
    launch_pdl(face_state_kernel<decltype(f)::value>, grid_for(m.n, 64), 64, 0, st, m, a);
  });
}
void launch_cell_boundary(int form, bool second, const MeshView<double>& m, const TileView& tv, const StageArgs& a,
                          cudaStream_t st) {
  if (m.nb == 0) return;
  with_form_order(form, second, [&](auto f, auto sec) {
    launch_pdl(boundary_face_kernel<decltype(f)::value, decltype(sec)::value>, grid_for(m.nb, 128), 128, 0, st, m, tv, a);
  });
}
// Blocks of 128 an SM should hold, which caps a thread's registers. Per launch at 1.3M
// tets: FP64 second order 110 us at 6, 116 at 7, 125 at 8, 123 without a cap (first
// order 91, 89, 95, 113); differences 121, 122, 111, 131 (first order 92, 87, 89, 103);
// FP32 copies 92, 88, 85, 92.
template <int kForm, bool kSecond>
constexpr int kCellBlocks = kForm != kFormFp64 ? 8 : kSecond ? 6 : 7;
void launch_cell_fluxes(int form, bool second, const MeshView<double>& m, const MeshView<float>& m32,
                        const StageArgs& a, cudaStream_t st) {
  with_form_order(form, second, [&](auto f, auto sec) {
    constexpr int kF = decltype(f)::value;
    constexpr bool kS = decltype(sec)::value;
    auto* k = cell_flux_kernel<kF, kS, kCellBlocks<kF, kS>>;
    if constexpr (kF == kFormFp64) launch_pdl(k, grid_for(m.n, 128), 128, 0, st, m, a);
    else launch_pdl(k, grid_for(m.n, 128), 128, 0, st, m32, a);
  });
}
// The form with FP32 copies under the Barth limiter: launch variants the tuner
// times. 0 plain, 1 software-pipelined, 2 and 3 the same with registers capped
// for 8 resident 128-thread blocks an SM, 4 and 5 for 9, 6 and 7 with every load
// issued before the arithmetic, uncapped and capped for 5, 8 and 9 plain with the
// cell's own rows prefetched into L2, capped as 2 and 4.
template <typename Fn>
static void with_variant(int variant, Fn&& f) {
  using std::integral_constant;
  auto go = [&](auto pipe, auto blocks) { f(pipe, blocks); };
  using P0 = integral_constant<int, 0>;
  using P1 = integral_constant<int, 1>;
  using P2 = integral_constant<int, 2>;
  using P3 = integral_constant<int, 3>;
  switch (variant) {
    case 1: go(P1(), integral_constant<int, 1>()); break;
    case 2: go(P0(), integral_constant<int, 8>()); break;
    case 3: go(P1(), integral_constant<int, 8>()); break;
    case 4: go(P0(), integral_constant<int, 9>()); break;
    case 5: go(P1(), integral_constant<int, 9>()); break;
    case 6: go(P2(), integral_constant<int, 1>()); break;
    case 7: go(P2(), integral_constant<int, 5>()); break;
    case 8: go(P3(), integral_constant<int, 8>()); break;
    case 9: go(P3(), integral_constant<int, 9>()); break;
    default: go(P0(), integral_constant<int, 1>()); break;
  }
}
void launch_gradient_copy(const MeshView<float>& m, const StageArgs& a, Launch l, int variant) {
  const int b = l.block > 128 ? 128 : l.block;
  with_variant(variant, [&](auto pipe, auto blocks) {
    launch_pdl(gradient_copy_kernel<decltype(pipe)::value, decltype(blocks)::value>, grid_for(m.n, b), b, 0, l.stream,
               m, a);
  });
}
void launch_flux_copy(const MeshView<float>& m, const StageArgs& a, Launch l, int variant) {
  const int b = l.block > 128 ? 128 : l.block;
  with_variant(variant, [&](auto pipe, auto blocks) {
    launch_pdl(flux_copy_kernel<decltype(pipe)::value, decltype(blocks)::value>, grid_for(m.n, b), b, 0, l.stream, m, a);
  });
}
void launch_bflux_copy(const MeshView<double>& m, const TileView& tv, const StageArgs& a, Launch l) {
  if (m.nb > 0) launch_pdl(boundary_flux_copy_kernel, grid_for(m.nb, l.block), l.block, 0, l.stream, m, tv, a);
}
void launch_gradient_field(int form, const MeshView<double>& m, const MeshView<float>& m32, const StageArgs& a,
                           cudaStream_t st) {
  const int g = grid_for(m.n, 128);
  if (form == kFormFp64) gradient_field_kernel<double, double><<<g, 128, 0, st>>>(m, a, a.Vin, a.vg, a.grad);
  else if (form == kFormDelta) gradient_field_kernel<float, double><<<g, 128, 0, st>>>(m32, a, a.Vin, a.vg, a.grad32);
  else gradient_field_kernel<float, float><<<g, 128, 0, st>>>(m32, a, a.Vin32, a.vg32, a.grad32);
}

// The cell-centre ghost state of every boundary face from the stage input's
// primitives (set_constant_ghost_values, Solver.cpp:300-330), where the previous
// stage kernel did not leave it, by the function the stage kernel calls, so that it
// is the same state wherever it is computed. kCopy: from the FP32 primitives,
// computed in FP64 (boundary faces are a few percent of the faces), stored in FP32.
// kPowers: for the kernels of kernels_copy.cuh, with the powers as ever.
template <bool kCopy, bool kPowers>
__global__ void __launch_bounds__(256) ghost_kernel_fast(MeshView<double> m, TileView tv, StageArgs a) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait_previous();
  if (b >= m.nb) return;
  const int2 ref = tv.b_ref[b];
  const double4 geo = tv.b_geo[b];
  const int c = checked(ref.x >> 2, m.n, a.status), st = m.stride;
  const PatchBC* bc = m.patches + checked(ref.y, m.n_patches, a.status);
  FiveValues V, G;
#pragma unroll
  for (int k = 0; k < 5; k++) V.v[k] = kCopy ? double(a.Vin32[k * st + c]) : a.Vin[k * st + c];
  if constexpr (kPowers) {
    const double nh[3] = {geo.x, geo.y, geo.z};
    ghost_state<double, true>(*bc, V.v, nh, G.v);
  } else {
    G = boundary_ghost(bc, geo, V);
  }
#pragma unroll
  for (int k = 0; k < 5; k++) {
    if constexpr (kCopy) a.vg32[k * m.bstride + b] = float(G.v[k]);
    else a.vg[k * m.bstride + b] = G.v[k];
  }
}
void launch_ghost(int form, bool powers, const MeshView<double>& m, const TileView& tv, const StageArgs& a, Launch l) {
  if (m.nb == 0) return;
  auto* k = form != kFormCopy ? ghost_kernel_fast<false, false>
            : powers          ? ghost_kernel_fast<true, true>
                              : ghost_kernel_fast<true, false>;
  launch_pdl(k, grid_for(m.nb, l.block), l.block, 0, l.stream, m, tv, a);
}
__global__ void fastmath_kernel(const double* x, int n, double* rcp, double* rsq) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  rcp[i] = nr_rcp(x[i]);
  rsq[i] = nr_rsqrt(x[i]);
}
void launch_fastmath(const double* x, int n, double* rcp, double* rsq, Launch l) {
  fastmath_kernel<<<grid_for(n, l.block), l.block, 0, l.stream>>>(x, n, rcp, rsq);
}

void launch_prim_fast(int n, int stride, const double* U, double* V, float* V32, Launch l) {
  prim_kernel_fast<false><<<grid_for(n, l.block), l.block, 0, l.stream>>>(n, stride, U, V, V32);
}

}  // namespace nf
