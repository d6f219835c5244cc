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
// smaller: AOS aggregated, one iteration, 0.8 tiles a CTA 12.3 us and 13.1 with
// the larger, 1.5 18.6 and 19.9, 2.2 26.0 and 26.9, 3.5 53.2 and 51.1, 7.1 104.5
// and 98.7.  (Several iterations a call come to more tiles a CTA: with two, 0.8
// 10.2 and 10.8, 1.5 16.7 and 16.5, 2.2 25.1 and 23.5 an iteration.)
constexpr uint32_t kAtomicTile = 1024, kAtomicTileSmall = 256;

// the atomic batch kernel for a set of loop kinds (atomic_batch.cu)
const void *batch_atomic_kernel_for(bool soa, bool agg, uint32_t loop_mask);

} // namespace fot
