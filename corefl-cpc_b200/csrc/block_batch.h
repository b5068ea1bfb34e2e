// Batched closed blocks (block_batch.cu): the device records of one block and the launcher.
#pragma once
#include "common.cuh"
#include "launch.h"
#include "cb200_serve.h"

namespace cb2 {

// The phases of a step that run over every block's tiles or nodes in one launch each.
enum BatchPhase { kTilesX, kTilesY, kTilesZ, kNodes, kPadded, kFacesX, kFacesY, kFacesZ, kColumns, kBatchPhases };

struct BlockCase {
  Zone z;
  FaceBC pairs[3];   // the left face of each periodic direction, in face-list order
};

// What changes as a block runs.
struct BlockState {
  double time, t_end, dt_fixed, last_dt;
  unsigned long long dt_bits;  // this step's dt (the bits of a positive double, so that they order alike)
  int steps, status;
  int active, bad;             // takes this step; its CFL step is not a positive number
  unsigned flags;              // non-physical-state bits of this block's stage updates
};

// Device memory of one batch, kept by the context for its next calls (grown, never shrunk, freed
// with the context).
struct BatchStore {
  BlockCase *cases = nullptr;
  BlockState *state = nullptr;
  int *first = nullptr;   // [kBatchPhases][n + 1]: first tile of every block
  int *owner = nullptr;   // the block of every tile, phase after phase
  int *n_active = nullptr;
  int n_cap = 0;
  long long owner_cap = 0;
};

bool block_batch_supported(const Param &p);
// CTAs of every phase for blocks of these zones, as prefix sums [kBatchPhases][n + 1] (ni: y/z tile
// width); false if a phase has more than 2^31 - 1.
bool batch_layout(const std::vector<BlockCase> &cases, int ni, std::vector<int> &first);
// Fills store.owner from store.first.
int launch_batch_owners(const BatchStore &b, int n, const std::vector<int> &first, cudaStream_t s, int &n_launch);
// mode 0: up to max_steps steps of every block; mode 1: one residual (dq) of every block, for timing.
int launch_block_batch(const BatchStore &b, int n, const std::vector<int> &first, const Param &p, int max_steps,
                       int mode, int ni, cudaStream_t s, int &n_launch);

}  // namespace cb2
