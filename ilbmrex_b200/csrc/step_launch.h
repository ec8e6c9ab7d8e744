// Launches of the level-step kernels.  The templates are defined in
// level_step.cuh and instantiated per lattice and storage form in step_q*.cu,
// which compile beside one another.
#pragma once

#include "ilbm_common.cuh"
#include "step_args.cuh"

namespace ilbm {

// lanes of a warp that own columns in the vector form (lanes 1 .. kOwned; the
// first and last lane hold the neighbours' cells)
constexpr int kOwned = 30;
// vectors (V > 1) or cells (V = 1) a block of n threads takes
__host__ __device__ constexpr uint32_t step_vectors_per_block(int V, uint32_t n) {
  return V > 1 ? n / 32u * kOwned : n;
}

// cells of one launch: its vectors are counted in 32 bits and divided as
// numbers below 2^31 (fast_div), the halo lanes' and ghost blocks' included
constexpr int64_t kMaxLaunchCells = 1 << 30;

// magic of a division by d (1 <= d < 2^31) of numbers below 2^31 (fast_div)
DivMagic div_magic(uint32_t d);
// the cells [rlo, rhi] of a launch as a sequence of V-cell vectors; false: empty
bool plan_vectors(StepArgs &a, int dim, int V);

// the cells a thread takes at once for these arrays
template <class L, int S>
int vec_width(const StepArgs &a);

// k_step over [rlo, rhi] (minus the skip box), with the ghost shell push or
// not; singly: in the cell form whatever the layout
template <class L, int S>
void launch_cells(ilbm_ctx *ctx, const StepArgs &a, cudaStream_t st, bool with_ghosts, bool singly = false);

// the boxes of a level (whole, with their ghost shells) in one launch; false,
// with nothing launched: they hold more than kMaxLaunchCells cells
template <class L, int S>
bool launch_step_boxes(ilbm_ctx *ctx, StepBoxes &p, cudaStream_t st);

// k_step_batch over a tile table, w threads per block
template <class L, int S>
int launch_step_batch(ilbm_ctx *ctx, const StepArgs *d_args, const StepTile *d_tiles, int ntiles, int V,
                      int w, int blocks, const int *steps, const int *limit, cudaStream_t st);

// resident blocks of w threads per SM of k_step_batch
template <class L, int S>
int occupancy_step_batch(const ilbm_ctx *ctx, int V, int w, int *per_sm);

}  // namespace ilbm
