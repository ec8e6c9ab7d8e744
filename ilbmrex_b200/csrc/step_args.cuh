// Kernel arguments of one box of a level step, shared by the level-step
// kernels (lbm_step.cu), the immersed boundary (ib.cu) and the batch engine
// (batch.cu), which keeps one StepArgs per case and buffer parity in device
// memory.
#pragma once

#include <stdint.h>

#include "ilbm_common.cuh"

namespace ilbm {

constexpr int kMaxLevelBoxes = 64;

// What becomes of populations that leave the box through a face
// (StepArgs::face_lo / face_hi): 0 is kept for "inside"
enum FaceState {
  FACE_WRAP = 1,       // periodic, self-filled: into the image cell
  FACE_REFLECT = 2,    // user_1: halfway bounce-back
  FACE_PHYS = 4,       // another physical face: ghost_push delivers what enters
  FACE_BOX = 8,        // another box of the level (or a coarse-fine face): as above
  FACE_PERIODIC = 16,  // periodic, caller-filled: as above
};

// division by a constant through a multiplication (fast_div)
struct DivMagic {
  uint32_t mul, shift;
};

struct StepArgs {
  // box valid region and allocated lower corners
  int lo[3], hi[3];
  int fgl[3];  // allocated lower corner of f arrays
  int mgl[3];  // allocated lower corner of macro / force arrays
  int64_t fs0, fs1, fs2;
  int64_t ms0, ms1, ms2;
  const void *f_in;
  void *f_out;
  const void *macro_in;
  const void *force;
  const void *force_prev;
  // level
  int dlo[3], dhi[3];
  int periodic[3];
  int bclo[3], bchi[3];
  double bvlo[3][4], bvhi[3][4];
  double tau;
  Tau64 tau64;
  int self_fill;
  int use_uniform;
  double uf[3];
  int flo[3], fhi[3];
  float f16_scale;
  float om32, omh32;  // 1/tau and 1 - 1/(2 tau) rounded to float, from the host
  // per-direction element offsets: q*fs2 (load) and c_q + q*fs2 (push target)
  int32_t loff[27], doff[27];
  // cells handled by this launch: [rlo, rhi], minus [slo, shi] when use_skip
  int rlo[3], rhi[3];
  int slo[3], shi[3];
  int use_skip;
  // the cells of this launch as a sequence of V-cell vectors: first column,
  // vectors per row, rows per k, vectors in all
  int vx0;
  uint32_t vpr, vny, nvec;
  DivMagic dvpr, dvny;
  int forced;  // a uniform force on every cell (no force arrays)
  // F16: per-direction storage factor w_q / scale and its inverse
  float sf[27], si[27];
  // blocks of the k_step grid that run ghost_push: one in ghost_every of the
  // leading ones, ghost_blocks in all
  uint32_t ghost_blocks, ghost_every;
  DivMagic dghost;
  // the ghost shell in one sequence: first index of each dimension's slab,
  // and the total (ghost_push)
  uint32_t goff[4];
  int face_lo[3], face_hi[3];  // what a face does with the populations that leave through it (FaceState)
  // boxes of the level (caller-filled ghosts): their number and the first one;
  // more come beside the arguments (LevelBoxes)
  int nlb;
  int lb0[6];
  // with use_mbox, macro_in holds stored values only on [mblo, mbhi]; cells
  // outside recover rho, u from f^n and F^{n-1}
  int use_mbox;
  int mblo[3], mbhi[3];
};

// the cell's rho, u come from macro_in (else from its populations)
__device__ __forceinline__ bool stored_macro_at(const StepArgs &a, int i, int j, int k) {
  if (!a.macro_in) return false;
  if (!a.use_mbox) return true;
  return i >= a.mblo[0] && i <= a.mbhi[0] && j >= a.mblo[1] && j <= a.mbhi[1] && k >= a.mblo[2] &&
         k <= a.mbhi[2];
}

// every box of a level (lo, hi), which decides whether a ghost cell is covered
struct LevelBoxes {
  int lb[kMaxLevelBoxes][6];
};

// The boxes of one launch of a level held in several boxes, passed by value
// (so a captured launch owns them): box n's blocks start at first[n].
constexpr int kMaxStepBoxes = 16;
struct StepBoxes {
  LevelBoxes lb;
  int nbox;
  uint32_t first[kMaxStepBoxes + 1];
  void *macro_out[kMaxStepBoxes];
  StepArgs a[kMaxStepBoxes];
};
static_assert(sizeof(StepBoxes) <= 32000, "kernel parameters hold at most 32,764 bytes");

// One work item of the batched level step (k_step_batch): blockDim.x vectors
// of case c from vector `first` on, or, with ghosts > 0, the ghost shell cells
// from `first` on in strides of `ghosts`; c = -1: a filler.
struct StepTile {
  int c;
  uint32_t first, ghosts;
};

// Work lists of the batched immersed-body stages: one entry per marker
// (case, marker) and tiles of kItemTile band cells of one case (case, first
// cell), so an item finds its case with one load.
struct ItemRef {
  int c, u;
};
constexpr int kItemTile = 256;

}  // namespace ilbm
