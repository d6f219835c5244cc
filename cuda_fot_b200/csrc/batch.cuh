// Device views shared by the batched executors (batch.cu: hierarchical
// tiles; atomic_batch.cu: atomic tiles, compiled with multiply-add
// contraction like the other atomic units).
#pragma once

#include <cstdint>

#include "executors.cuh"

namespace fot {

struct BatchMesh {
  LoopData d;
  HierPlanDev P;
  int loop;
};

struct BatchDev {
  const BatchMesh *mesh;
  const uint32_t *tile_mesh;  // per tile of one iteration: mesh index
  const uint32_t *tile_block; // per tile: block of that mesh
  uint32_t tiles_per_iter;
  uint32_t total_tiles;
  uint32_t n_mesh;
  uint32_t tile_cells; // atomic plans: cells per tile
  unsigned int *done; // per mesh
  Ctl *ctl;           // ticket / exited / error
};

// Cells per tile of the atomic batch: the larger one spares look-ups, but a
// batch that has less than 2.5 such tiles for each CTA is over sooner with the
// smaller: AOS aggregated, one iteration, 1.3 tiles a CTA 16.0 us and 23.8 with
// the larger, 2.1 26.1 and 28.9, 2.8 38.7 and 35.4, 6.8 98.2 and 88.4.
constexpr uint32_t kAtomicTile = 1024, kAtomicTileSmall = 256;

// the atomic batch kernel for a set of loop kinds (atomic_batch.cu)
const void *batch_atomic_kernel_for(bool soa, bool agg, uint32_t loop_mask);

} // namespace fot
