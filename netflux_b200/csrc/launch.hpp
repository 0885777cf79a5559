// Host-callable launchers of the device kernels. Each arithmetic form lives
// in its own translation unit: kernels_ref.cu is compiled with -fmad=false
// (reference rounding), kernels_fast.cu with contraction on.
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace nf {

struct Launch {
  int block;
  cudaStream_t stream;
};

// reference-order FP64 (kernels_ref.cu)
void launch_gradient_ref(const MeshView<double>& m, const StageArgs& a, Launch l);
void launch_flux_ref(const MeshView<double>& m, const StageArgs& a, Launch l);
void launch_ghost_ref(const MeshView<double>& m, const StageArgs& a, Launch l);
void launch_bflux_ref(const MeshView<double>& m, const StageArgs& a, Launch l);
void launch_timestep(const MeshView<double>& m, const DtArgs& a, Launch l);
void launch_prim_ref(int n, int stride, const double* U, double* V, float* V32, Launch l);

// fast forms (kernels_fast.cu): the stage kernel (kernels_tile.cuh) of a form
// (kFormFp64, kFormDelta, kFormCopy) over the tiles of a mesh
struct Tiles;
struct TileView;
size_t stage_smem(int form, const Tiles& t, bool second);  // shared memory of a block; 0: the tiles' lists are too long
// once per device before a launch of a mode (kModeFirst ...); *blocks: blocks a multiprocessor holds
cudaError_t stage_setup(int form, int tile, int mode, int max_smem, size_t smem, int* blocks);
void launch_stage(int form, int tile, int mode, const MeshView<double>& m, const TileView& tv, const StageArgs& a,
                  size_t smem, cudaStream_t st);
// the same stage by one thread a cell (kernels_cell.cuh): limiter and face states
// (second order), then boundary fluxes, fluxes and update
void launch_cell_states(int form, const MeshView<double>& m, const StageArgs& a, cudaStream_t st);
void launch_cell_boundary(int form, bool second, const MeshView<double>& m, const TileView& tv, const StageArgs& a,
                          cudaStream_t st);
void launch_cell_fluxes(int form, bool second, const MeshView<double>& m, const MeshView<float>& m32,
                        const StageArgs& a, cudaStream_t st);
// the form with FP32 copies under the Barth limiter (kernels_copy.cuh)
void launch_gradient_copy(const MeshView<float>& m, const StageArgs& a, Launch l, int variant);
void launch_flux_copy(const MeshView<float>& m, const StageArgs& a, Launch l, int variant);
void launch_bflux_copy(const MeshView<double>& m, const TileView& tv, const StageArgs& a, Launch l);
// the gradient field of a stage's input (keep_stage_fields)
void launch_gradient_field(int form, const MeshView<double>& m, const MeshView<float>& m32, const StageArgs& a,
                           cudaStream_t st);
// cell-centre ghost states of the stage's input, FP64 or (FP32 copies) FP32;
// powers: the far field's by pow (FP32 copies under the Barth limiter)
void launch_ghost(int form, bool powers, const MeshView<double>& m, const TileView& tv, const StageArgs& a, Launch l);
void launch_prim_fast(int n, int stride, const double* U, double* V, float* V32, Launch l);
// the fast forms' reciprocal and reciprocal square root, elementwise (self-test)
void launch_fastmath(const double* x, int n, double* rcp, double* rsq, Launch l);

}  // namespace nf
