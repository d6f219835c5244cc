// The split write-back hierarchical-colour kernel (variant kVariantSplit).
//
// The coloured replay of a plan (blocks in block-colour order; in a block,
// cells in thread-colour order accumulate into a zeroed per-block sum; then
// out[p] += sum for each written point) fixes, for every point p, the order
// out[p] = ((out[p] + S_b1) + S_b2) + ... over the blocks b1 < b2 < ... (plan
// order) that write p.  The kernel reproduces that order without making
// any tile wait for another:
//   * a point written by ONE block (private) gets out[p] += S_b as soon as
//     the block's sum is ready -- a fire-and-forget L2 reduction (RED.F64) for
//     FP64 data, whose single rounding equals the replay's add; FP32 data
//     (atomics there flush subnormals) take a load-add-store;
//   * a point written by several blocks (shared) gets S_b stored into the
//     point's slot for that block (plain stores, one buffer per iteration
//     parity); the NEXT launch -- the next iteration's, or the flush launch
//     that ends a run -- adds out[p] + S_b1 + S_b2 ... in plan order while its
//     own tiles fill the other buffer.  Private and shared points are
//     disjoint, so the combine never races with the tiles.
// Block colours therefore fix the summation order but never stall a tile.
// One launch runs ONE iteration; consecutive launches are chained with
// programmatic dependent launch: every CTA lets the next grid start at once
// (in a call's first grid: once what precedes the call is complete), and the
// next grid's tiles gather and compute (they only read datasets the loop never
// writes) before they wait (griddepcontrol.wait) for this grid to complete and
// only then write.  What a cell function writes to cell data is
// held in a register until then (an iteration of 10, waiting before it computes
// and so: LULESH 45^3 10.6 and 9.1 us, 30^3 8.1 and 6.0).
//
// One CTA runs one tile (k_hier_dsplit); extra CTAs at the end of the grid do
// the combine.  A warp-specialised persistent form that staged each tile's
// read rows in shared memory (a record warp, a staging warp, two tiles in
// flight) was slower on every loop, layout and partition once this one summed
// its contributions from lists, and is gone (when it went, parts of 256, AOS,
// staged and direct: res_calc 1000^2 60.0 and 54.7 us, 44.8 today; LULESH 96^3 113.9
// and 87.2, 83.0 today; miniAero 96^3 634 and 413).
#pragma once

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "hier_pipe.cuh"

namespace fot {

// A tile's write-back data (built by plan.cu): the written
// points, their slots (0xFFFFFFFF: private), and per point its contributions
// pc_idx[pc_off[j], pc_off[j + 1]) = slot * threads + cell, in thread-colour
// order.
struct DirectRecord {
  const uint32_t *pts, *wslot;
  const uint16_t *pc_off, *pc_idx;
  __host__ __device__ DirectRecord(const unsigned char *r, uint32_t n0)
      : pts(reinterpret_cast<const uint32_t *>(r)), wslot(pts + n0),
        pc_off(reinterpret_cast<const uint16_t *>(wslot + n0)), pc_idx(pc_off + n0 + 1) {}
  // bytes for n0 written points and E contributions, a multiple of 16
  __host__ __device__ static uint32_t bytes(uint32_t n0, uint32_t E) {
    return (8u * n0 + 2u * (n0 + 1 + E) + 15u) & ~15u;
  }
};

// Row r of K values (side by side) of L2-resident data, in 16-byte loads where
// rows are a multiple of 16 bytes.
template <int K, class T> __device__ __forceinline__ void load_row_cg(const T *base, size_t r, T (&v)[K]) {
  if constexpr (sizeof(T) == 4 && K == 4) {
    const float4 w = __ldcg(reinterpret_cast<const float4 *>(base) + r);
    v[0] = w.x;
    v[1] = w.y;
    v[2] = w.z;
    v[3] = w.w;
  } else if constexpr (sizeof(T) == 8 && K % 2 == 0) {
#pragma unroll
    for (int k = 0; k < K; k += 2) {
      const double2 w = __ldcg(reinterpret_cast<const double2 *>(base + r * K + k));
      v[k] = w.x;
      v[k + 1] = w.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = __ldcg(base + r * K + k);
  }
}
template <int K, class T> __device__ __forceinline__ void store_row_cg(T *base, size_t r, const T (&v)[K]) {
  if constexpr (sizeof(T) == 4 && K == 4) {
    __stcg(reinterpret_cast<float4 *>(base) + r, make_float4(v[0], v[1], v[2], v[3]));
  } else if constexpr (sizeof(T) == 8 && K % 2 == 0) {
#pragma unroll
    for (int k = 0; k < K; k += 2)
      __stcg(reinterpret_cast<double2 *>(base + r * K + k), make_double2(v[k], v[k + 1]));
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k) __stcg(base + r * K + k, v[k]);
  }
}

// Shared points [g0, g1) of the previous launch's buffer: out[p] plus the
// blocks' sums in plan order (thread t of nt, a point a thread: its K sums
// are independent chains).
template <class L, bool SOA>
__device__ __forceinline__ void combine_shared(const LoopData &d, const HierPlanDev &P, uint32_t g0,
                                               uint32_t g1, uint32_t t, uint32_t nt) {
  using out_t = typename L::out_t;
  constexpr int K = L::kOut;
  const out_t *part = static_cast<const out_t *>(P.partial) + (size_t)(P.put_buf ^ 1u) * P.n_slots * K;
  out_t *out = static_cast<out_t *>(d.out);
  for (uint32_t g = g0 + t; g < g1; g += nt) {
    const uint32_t p = __ldg(P.comb_point + g), e0 = __ldg(P.comb_base + g), e1 = __ldg(P.comb_base + g + 1);
    out_t o[K], v[K];
    if constexpr (SOA) {
#pragma unroll
      for (int k = 0; k < K; ++k) o[k] = __ldcg(out + out_index(true, d.n_points[0], p, K, k));
    } else {
      load_row_cg<K>(out, p, o);
    }
    for (uint32_t e = e0; e < e1; ++e) {
      load_row_cg<K>(part, e, v);
#pragma unroll
      for (int k = 0; k < K; ++k) o[k] += v[k];
    }
    if constexpr (SOA) {
#pragma unroll
      for (int k = 0; k < K; ++k) __stcg(out + out_index(true, d.n_points[0], p, K, k), o[k]);
    } else {
      store_row_cg<K>(out, p, o);
    }
  }
}

__device__ __forceinline__ void comb_chunk(uint32_t n, uint32_t c, uint32_t parts, uint32_t &g0,
                                           uint32_t &g1) {
  g0 = (uint32_t)((uint64_t)n * c / parts);
  g1 = (uint32_t)((uint64_t)n * (c + 1) / parts);
}

// How a tile's written points are shared out over its threads.
// Rows of doubles in AOS data: one (point, component) per thread, so that the
// K lanes of a point write whole 32-byte sectors (a reduction per sector
// instead of one per element, see add_rows_f64).  Otherwise one point per
// thread with its K sums in registers: neighbouring lanes then write
// neighbouring addresses of each component (SOA), or each a 16-byte row (FP32
// AOS), and a point's contribution list is walked once.  Direct form, parts of
// 256, an iteration of 10, by element and by point: res_calc 1000^2 AOS 44.8 and
// 62.1 us, getacc 1024^2 AOS 45.7 and 61.0; in SOA by point is the better one
// (res_calc 51 us and 63 by element, when both were last there).
template <class L, bool SOA> constexpr bool by_element() {
  return !SOA && sizeof(typename L::out_t) == 8;
}
template <class L, bool SOA> constexpr bool by_row4() {
  return !SOA && sizeof(typename L::out_t) == 4 && L::kOut == 4;
}

// The increments of a tile in shared memory: entry ie = slot * T + cell holds
// K values, side by side for AOS point data (a point's lanes, or its one
// 16-byte load, read one row), component by component for SOA.  Rows of 4
// doubles swap halves every 4 rows, so that the 16-byte stores of 8 lanes fall
// into 8 different bank groups (2-way conflicts otherwise: res_calc 1000^2, parts
// of 256, 47.7 us and 44.8 so, getacc 1024^2 47.5 and 45.7).
template <class L, bool SOA, int T>
__device__ __forceinline__ uint32_t inc_index(uint32_t ie, uint32_t k) {
  if constexpr (SOA) return k * (L::kDim * T) + ie;
  if constexpr (by_element<L, SOA>() && L::kOut == 4) return ie * 4u + (k ^ ((ie >> 1) & 2u));
  return ie * L::kOut + k;
}

template <class L, bool SOA, int T>
__device__ __forceinline__ void put_increments(typename L::out_t *inc,
                                               const typename L::out_t (&v)[L::kDim][L::kOut], uint32_t t) {
  constexpr int K = L::kOut;
#pragma unroll
  for (int q = 0; q < L::kDim; ++q) {
    if constexpr (by_element<L, SOA>() && K % 2 == 0) {
#pragma unroll
      for (int k = 0; k < K; k += 2)
        *reinterpret_cast<double2 *>(inc + inc_index<L, SOA, T>(q * T + t, k)) = make_double2(v[q][k], v[q][k + 1]);
    } else if constexpr (by_row4<L, SOA>()) {
      *reinterpret_cast<float4 *>(inc + (q * T + t) * 4) = make_float4(v[q][0], v[q][1], v[q][2], v[q][3]);
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) inc[inc_index<L, SOA, T>(q * T + t, k)] = v[q][k];
    }
  }
}

// All n0 written points of a tile (thread t of T): sum a point's
// contributions in thread-colour order from the increments in shared memory,
// then add the sum (private point: this block alone writes it in this
// iteration) or store it into its slot of this launch's buffer (shared).
template <class L, bool SOA, int T>
__device__ __forceinline__ void split_writeback(const LoopData &d, const HierPlanDev &P, uint32_t n0,
                                                const uint32_t *pts, const uint32_t *wslot,
                                                const uint16_t *pc_off, const uint16_t *pc_idx,
                                                const typename L::out_t *inc, uint32_t t) {
  using out_t = typename L::out_t;
  constexpr int K = L::kOut;
  out_t *out = static_cast<out_t *>(d.out);
  out_t *put = static_cast<out_t *>(P.partial) + (size_t)P.put_buf * P.n_slots * K;
  if constexpr (by_element<L, SOA>()) {
    for (uint32_t i = t; i < n0 * (uint32_t)K; i += T) {
      const uint32_t j = i / K, k = i % K;
      out_t acc = out_t(0);
      const uint32_t e1 = pc_off[j + 1];
      for (uint32_t e = pc_off[j]; e < e1; ++e) acc += inc[inc_index<L, SOA, T>(pc_idx[e], k)];
      const uint32_t ws = wslot[j];
      if (ws == 0xFFFFFFFFu) atomicAdd(out + (size_t)pts[j] * K + k, acc);
      else __stcg(put + (size_t)ws * K + k, acc);
    }
    return;
  }
  for (uint32_t j = t; j < n0; j += T) {
    out_t acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = out_t(0);
    const uint32_t e1 = pc_off[j + 1];
    for (uint32_t e = pc_off[j]; e < e1; ++e) {
      const uint32_t ie = pc_idx[e];
      if constexpr (by_row4<L, SOA>()) {
        const float4 v = *reinterpret_cast<const float4 *>(inc + ie * 4);
        acc[0] += v.x;
        acc[1] += v.y;
        acc[2] += v.z;
        acc[3] += v.w;
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] += inc[inc_index<L, SOA, T>(ie, k)];
      }
    }
    const uint32_t ws = wslot[j];
    if (ws != 0xFFFFFFFFu) {
      store_row_cg<K>(put, ws, acc);
      continue;
    }
    const uint32_t p = pts[j];
    if constexpr (by_row4<L, SOA>()) {
      out_t o[K];
      load_row_cg<K>(out, p, o);
#pragma unroll
      for (int k = 0; k < K; ++k) o[k] += acc[k];
      store_row_cg<K>(out, p, o);
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        out_t *o = out + out_index(SOA, d.n_points[0], p, K, k);
        if constexpr (sizeof(out_t) == 8) atomicAdd(o, acc[k]);
        else __stcg(o, __ldcg(o) + acc[k]);
      }
    }
  }
}

// CTAs [0, n_blocks) run one tile each, the comb_ctas after
// them combine the previous buffer (hardware CTA scheduling keeps several tiles per SM in
// different phases; a persistent form with one tile in flight per CTA and
// the next tile's plan data prefetched measured slower).  One thread per cell
// gathers its rows through the plan-ordered mapping straight from HBM/L2 and
// puts its increments into shared memory; after ONE barrier each written
// point's contributions are summed in thread-colour order (the replay's
// order, bit for bit) and go out (RED for private points, the slot for shared
// ones).  What the write-back needs -- points, slots, contribution lists -- is
// one record per tile (DirectRecord), bulk-copied while the cells compute; the
// tile header (start, cells | colours << 16, written points, record offset)
// is one 16-byte load.
// A cell function's value for cell data, where it writes one.
template <class L, bool = L::kWritesCell> struct HeldValue {};
template <class L> struct HeldValue<L, true> {
  typename L::written_t value;
};

// CAP: registers per thread (L::kDirectRegCap, or of plans with scattered
// blocks L::kScatteredRegCap).
constexpr int dsplit_min_blocks(int threads, int cap) {
  return 65536 / (threads * cap) > 0 ? 65536 / (threads * cap) : 1;
}

template <class L, bool SOA, int T, int CAP>
__global__ void __launch_bounds__(T, dsplit_min_blocks(T, CAP)) k_hier_dsplit(LoopData d, HierPlanDev P) {
  using out_t = typename L::out_t;
  constexpr int D = L::kDim, K = L::kOut;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_full;
  out_t *const inc = reinterpret_cast<out_t *>(smem + P.inc_off);
  const uint32_t tid = threadIdx.x;
  // The first grid of a call waits before it lets the next one start: what
  // precedes the call may write what tiles read, and the next grid's tiles
  // read before their own wait.  Triggering first, they could start while that
  // work still runs (a kernel that lets its dependents start early, or whose
  // writes are not flushed yet) and gather what it has not written.
  if (P.ordered) griddep_wait();
  // Where the next grid has tiles that can gather and compute meanwhile, let it
  // start (an iteration of 10 with and without: res_calc 1000^2 44.8 us and 46.3,
  // 200x210 3.8 and 4.5, LULESH 45^3 9.1 and 10.7); the flush can only wait and
  // gains nothing (one iteration, 200x210 7.4 us and 7.3 started early, LULESH
  // 30^3 9.9 and 9.8).
  if (P.more) griddep_launch_dependents();
  const uint32_t n_tiles = P.tiles_on ? P.n_blocks : 0u;
  if (blockIdx.x >= n_tiles) {
    // the combine CTAs come last, so that the tiles are scheduled first
    // (they gather and compute before their wait; these only wait)
    griddep_wait();
    uint32_t g0, g1;
    comb_chunk(P.n_shared, blockIdx.x - n_tiles, P.comb_ctas, g0, g1);
    combine_shared<L, SOA>(d, P, g0, g1, tid, T);
    return;
  }
  const uint4 h = __ldg(P.tile_hdr + (P.backwards ? n_tiles - 1u - blockIdx.x : blockIdx.x));
  const uint32_t start = h.x, ncell = h.y & 0xFFFFu, n0 = h.z;
  if (tid == 0) {
    const uint32_t bytes = DirectRecord::bytes(n0, D * ncell);
    mbar_init(&s_full, 1);
    mbar_fence_init();
    mbar_expect_tx(&s_full, bytes);
    bulk_copy_g2s(smem, P.rec + (size_t)h.w * 16, bytes, &s_full);
  }
  [[maybe_unused]] HeldValue<L> held;
  if (tid < ncell) {
    const uint32_t pos = start + tid;
    GlobalRows<L, SOA> rows;
    load_row<D>(d.map[0], pos, rows.p[0]);
    if constexpr (L::kHasClass1) load_row<D>(d.map[1], pos, rows.p[1]);
    rows.bind(d);
    out_t v[D][K];
    const Direct dir{d.cell, pos, d.n_cells};
    if constexpr (L::kWritesCell) L::cell(rows, HeldDirect(dir, &held.value), v);
    else L::cell(rows, dir, v);
    put_increments<L, SOA, T>(inc, v, tid);
  }
  __syncthreads();
  if (!mbar_wait(&s_full, 0)) {
    if (tid == 0) atomicOr(&P.ctl->error, kErrWaitLimit);
    griddep_wait();
    return;
  }
  griddep_wait();  // the previous iteration's writes are visible
  if constexpr (L::kWritesCell) {
    if (tid < ncell)
      *Direct{d.cell, start + tid, d.n_cells}.template wptr<typename L::written_t>(L::kWrittenSet) = held.value;
  }
  const DirectRecord m(smem, n0);
  split_writeback<L, SOA, T>(d, P, n0, m.pts, m.wslot, m.pc_off, m.pc_idx, inc, tid);
}

} // namespace fot
