// Batched atomic executor: tiles of consecutive cells of every
// mesh and every iteration in one grid-stride launch (iterations need no
// ordering: the loops never read the dataset they increment).  Compiled with
// multiply-add contraction, like the single-mesh atomic units (see
// loop_atomic_impl.cuh); the functors are instantiated under res_calc_fma,
// ... to keep their symbols apart from the exact ones of batch.cu.
#define FOT_ADAPTER_ALL 1
#define FOT_NS_SUFFIX _fma
#define FOT_CONTRACTED 1  // functors may take a form with fewer operations
#include "batch.cuh"
#include "engine.hpp"
#include "loops.cuh"

namespace fot {

// Registers per thread: the most that a loop of the batch asks for in the tile
// kernels; one CTA an SM more (48 registers for res_calc with volna) spills the
// addresses.  An iteration of two, so and with one more: SOA without aggregation,
// 36 meshes of 2,500 to 70,000 cells 27.3 us and 34.1, 40 of 4,000 to 250,000 94.5
// and 98.9; AOS aggregated 25.1 and 26.8, 83.3 and 80.0 (98.7 and 87.8 alone).
template <class... Ls> constexpr int batch_min_blocks() {
  int m = 0;
  ((m = Ls::kRegCap > m ? Ls::kRegCap : m), ...);
  return 65536 / (256 * m) > 0 ? 65536 / (256 * m) : 1;
}

// The cells [start, start + cells) of one mesh.  Its addresses are
// copied first: read through the pointer, they would be read again after
// every reduction.
template <class L, bool SOA, bool AGG>
__device__ __forceinline__ void batch_atomic_tile(const BatchMesh &m, uint32_t start, uint32_t cells) {
  const LoopData d = m.d;
#pragma unroll 1
  for (uint32_t k = 0; k < cells; k += 256u) {
    CellMap<L> map;
    map.load(d, start + k + threadIdx.x);
    atomic_warp<L, SOA, AGG>(d, start + k + (threadIdx.x & ~31u), map);
  }
}

template <bool SOA, bool AGG, class... Ls>
__global__ void __launch_bounds__(256, batch_min_blocks<Ls...>()) k_batch_atomic(BatchDev B) {
  griddep_wait();
  for (uint32_t t = blockIdx.x; t < B.total_tiles; t += gridDim.x) {
    const uint32_t it = t / B.tiles_per_iter, i = t - it * B.tiles_per_iter;
    // iterations alternate in direction, see AtomicGrid
    const uint32_t r = (it & 1u) ? B.tiles_per_iter - 1u - i : i;
    const BatchMesh &m = B.mesh[__ldg(B.tile_mesh + r)];
    const uint32_t start = __ldg(B.tile_block + r);
    const int loop = m.loop;
    ((loop == Ls::kLoop ? (batch_atomic_tile<Ls, SOA, AGG>(m, start, B.tile_cells), 0) : 0), ...);
  }
}

template <bool SOA, bool AGG> const void *batch_atomic_kernel(uint32_t loop_mask) {
  using RC = res_calc_fma::Loop;
  using MA = mini_aero_fma::Loop;
  using LU = lulesh_fma::Loop;
  using VO = volna_fma::Loop;
  using GA = getacc_fma::Loop;
  switch (loop_mask) {
  case 1u << FOT_LOOP_RES_CALC: return (const void *)&k_batch_atomic<SOA, AGG, RC>;
  case 1u << FOT_LOOP_MINI_AERO: return (const void *)&k_batch_atomic<SOA, AGG, MA>;
  case 1u << FOT_LOOP_LULESH: return (const void *)&k_batch_atomic<SOA, AGG, LU>;
  case 1u << FOT_LOOP_VOLNA: return (const void *)&k_batch_atomic<SOA, AGG, VO>;
  case 1u << FOT_LOOP_GETACC: return (const void *)&k_batch_atomic<SOA, AGG, GA>;
  case (1u << FOT_LOOP_RES_CALC) | (1u << FOT_LOOP_VOLNA):
    return (const void *)&k_batch_atomic<SOA, AGG, RC, VO>;
  }
  return nullptr;
}

const void *batch_atomic_kernel_for(bool soa, bool agg, uint32_t loop_mask) {
  if (soa) return agg ? batch_atomic_kernel<true, true>(loop_mask) : batch_atomic_kernel<true, false>(loop_mask);
  return agg ? batch_atomic_kernel<false, true>(loop_mask) : batch_atomic_kernel<false, false>(loop_mask);
}

} // namespace fot
