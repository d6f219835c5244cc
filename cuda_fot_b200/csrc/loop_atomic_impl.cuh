// Instantiates the atomic executor (a) for the loop selected by FOT_ADAPTER.
// Included once by each atomic_*.cu.  Those translation units are compiled
// WITH multiply-add contraction (the build compiles atomic_*.cu with
// -fmad=true, as the reference compiles its own device code): the atomic
// executor's results differ from the serial loop by summation order anyway
// (contract: normwise relative error <= 1e-12 FP64 / 1e-5 FP32), and the
// fused multiply-adds cut the instruction count of the heavy functors
// (mini_aero's Roe flux).  The coloured executors stay in the exact units
// (loop_*.cu, -fmad=false) where a run is bit-identical to its CPU replay.
#pragma once

#include <algorithm>

#define FOT_NS_SUFFIX _fma
#define FOT_CONTRACTED 1  // functors may take a form with fewer operations
#include "engine.hpp"
#include "loops.cuh"

namespace fot {
namespace {

using LA = FOT_LNS(FOT_ADAPTER_NS)::Loop;

// whether the loop has a form of its own for scattered rows
template <bool SOA> constexpr bool has_scattered() {
  return SOA && LA::kAtomicScatteredMinBlocks != LA::kAtomicMinBlocks;
}

// `iterations` iterations in one launch (more only where the grid would grow
// past 2^30 CTAs).
template <bool SOA, bool AGG, bool SCATTERED = false>
int launch_atomic(const LoopData &d, bool scattered, uint32_t resident, uint32_t iterations,
                  bool backwards, cudaStream_t st) {
  if constexpr (!SCATTERED && has_scattered<SOA>()) {
    if (scattered) return launch_atomic<SOA, AGG, true>(d, true, resident, iterations, backwards, st);
  }
  AtomicGrid g;
  g.flip = backwards;
  g.tiles = (d.n_cells + 255u) / 256u;
  g.resident = std::max(1u, std::min(g.tiles, resident));
  const uint32_t all = (g.tiles + g.resident - 1) / g.resident;
  constexpr uint32_t above = LA::kAtomicSplitAbove[2 * SOA + AGG];
  const uint32_t phases = above && all > above ? (all + LA::kAtomicRounds - 1) / LA::kAtomicRounds : 1;
  g.rounds = (all + phases - 1) / phases;
  g.ctas = phases * g.resident;
  const uint32_t most = std::max(1u, (1u << 30) / g.ctas);
  while (iterations) {
    const uint32_t now = std::min(iterations, most);
    Chained c(dim3(g.ctas * now), dim3(256), 0, st);
    FOT_CUDA(cudaLaunchKernelEx(&c.cfg, k_atomic<LA, SOA, AGG, SCATTERED>, d, g));
    iterations -= now;
    g.flip += now;
  }
  return FOT_OK;
}

template <bool SOA, bool AGG> const void *atomic_kernel(bool scattered) {
  if constexpr (has_scattered<SOA>()) {
    if (scattered) return reinterpret_cast<const void *>(&k_atomic<LA, SOA, AGG, true>);
  }
  return reinterpret_cast<const void *>(&k_atomic<LA, SOA, AGG, false>);
}

} // namespace

int FOT_CAT(atomic_run_, FOT_ADAPTER_NS)(const LoopData &d, bool soa, bool agg, bool scattered,
                                         uint32_t resident, uint32_t iterations, bool backwards,
                                         cudaStream_t st) {
  if (soa) return agg ? launch_atomic<true, true>(d, scattered, resident, iterations, backwards, st)
                      : launch_atomic<true, false>(d, scattered, resident, iterations, backwards, st);
  return agg ? launch_atomic<false, true>(d, scattered, resident, iterations, backwards, st)
             : launch_atomic<false, false>(d, scattered, resident, iterations, backwards, st);
}

int FOT_CAT(atomic_occupancy_, FOT_ADAPTER_NS)(bool soa, bool agg, bool scattered, int *per_sm) {
  const void *k = soa ? (agg ? atomic_kernel<true, true>(scattered) : atomic_kernel<true, false>(scattered))
                      : (agg ? atomic_kernel<false, true>(scattered) : atomic_kernel<false, false>(scattered));
  FOT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k, 256, 0));
  return FOT_OK;
}

} // namespace fot
