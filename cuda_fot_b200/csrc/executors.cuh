// The two executors, templated on a loop adapter (loops.cuh).
//
// (a) Global atomics (FOT_EXEC_ATOMIC) -- replaces the reference's
//     global-colouring executor (problem.hpp:90-194, one launch and one
//     cudaDeviceSynchronize per colour).  One thread per cell, mapping rows
//     read as vectors, read sets gathered straight from HBM/L2, increments
//     added with native atomics (f64 RED, AOS rows laid end to end across the
//     warp first; one 16-byte f32x4 RED per row for the FP32 loop).  With warp aggregation, runs of neighbouring lanes whose
//     slot targets one point are summed in registers by a segmented shuffle
//     tree before the run's first lane issues the atomics.
//
// (b) Hierarchical colouring (FOT_EXEC_HIER / _HIER_LAUNCH) -- replaces
//     loopGPUHierarchical (problem.hpp:198-339) and its kernels
//     (e.g. res_calc.hpp:218-383).  A block of cells is one CTA tile.  The
//     CTA stages the read rows of the block's unique points into shared memory
//     with cp.async, computes every cell's increments, adds them into a
//     zeroed shared accumulator in thread-colour order (one __syncthreads per
//     thread colour) and finally adds the accumulator to point dataset 0 in
//     HBM.  Blocks of one block colour write disjoint points.  In the
//     persistent forms (FOT_EXEC_HIER) CTAs claim tiles from a queue stored
//     in block-colour order (and iteration after iteration); a tile computes
//     immediately -- the loops never read the dataset they increment -- and
//     only its write-back waits, with a bounded spin, until what it conflicts
//     with has been written back: every tile of the earlier colours for the
//     simple kernel (k_hier, hier.cuh), the conflicting blocks' completion
//     flags for the pipelined warp-specialised kernel (k_hier_pipe,
//     hier_pipe.cuh).  The split write-back kernel (k_hier_dsplit,
//     hier_split.cuh, the default) makes no tile wait: points written by one
//     block are added at once, points shared by several blocks through
//     per-block partial sums that the next launch (or a final combine-only
//     launch) adds in colour order.  The result is therefore deterministic
//     and equal to replaying the colours in order on the CPU.
#pragma once

#include <cstdint>

#include "common.cuh"

namespace fot {

// Device view of a problem's data for one run (current cell order).
struct LoopData {
  const uint32_t *map[2]; // class 0 = mapping 0; class 1 = a second distinct mapping
  const void *point[4];   // point datasets by set index
  void *out;              // point dataset 0
  void *cell[8];          // cell datasets (SOA, stride n_cells)
  uint32_t n_points[4];
  uint32_t n_cells;
  uint32_t n_cell_sets;
  uint32_t cell_dim[8];   // components of each cell dataset
  uint32_t cell_size[8];  // bytes of one component
};

// Device view of a hierarchical plan.
struct HierPlanDev {
  const uint32_t *block_start; // n_blocks+1 positions
  const uint32_t *block_wait;  // tiles of earlier colours (per block)
  const uint8_t *block_ntcol;  // thread colours per block
  const uint8_t *tcol;         // thread colour per position
  const uint32_t *pts_off[2];  // per class: n_blocks+1 offsets
  const uint32_t *pts[2];      // per class: unique points of each block
  const uint16_t *lidx[2];     // per class: kDim x n_cells local indices (SOA)
  uint32_t n_blocks;
  uint32_t total_tiles;        // iterations * n_blocks (persistent form)
  uint32_t read_off[4];        // shared-memory byte offset of each read set
  uint32_t acc_off;            // shared-memory byte offset of the accumulator
  uint32_t pts_smem_off;       // shared-memory byte offset of the tile's point lists
  Ctl *ctl;
  // pipelined kernel
  const unsigned char *rec;    // tile records
  const uint32_t *rec_off;     // n_blocks+1 byte offsets of the records
  uint32_t rec_slot;           // bytes of one tile-record slot (slots start at offset 0)
  uint32_t rows_off;           // first read-row slot (read_off[] are relative to a slot)
  uint32_t rows_bytes;         // bytes of one read-row slot
  uint32_t inc_off;            // per-slot increments
  uint32_t outbuf_off;         // first prefetched-output-row slot
  uint32_t outbuf_bytes;       // bytes of one output-row slot
  unsigned int *block_done;    // per block: completed iterations (relative to ctl->base)
  // split write-back kernel
  void *partial;               // 2 x n_slots partial-sum rows (AOS, point dataset 0's type)
  const uint32_t *comb_point;  // shared point g -> point number
  const uint32_t *comb_base;   // shared point g -> its slots [base[g], base[g+1])
  uint32_t n_slots, n_shared;
  const uint4 *tile_hdr;       // per tile (launch order): start, cells | colours << 16,
                               // written points, its record's offset in
                               // units of 16 bytes (DirectRecord)
  // per launch: tiles run (0: combine only), the buffer they fill, CTAs
  // combining the other buffer (previous iteration)
  uint32_t tiles_on, put_buf, comb_ctas;
  // the first launch of a call waits for what precedes it before it reads and
  // before it lets the next start; the next launch has tiles too; tiles last to
  // first (every other iteration)
  uint32_t ordered, more, backwards;
};

// Direct (cell) data of one cell: SOA with stride n_cells.
struct Direct {
  void *const *base;
  uint32_t idx;
  unsigned stride;
  template <class T> __device__ __forceinline__ const T *ptr(int j) const {
    return static_cast<const T *>(base[j]) + idx;
  }
  template <class T> __device__ __forceinline__ T *wptr(int j) const {
    return static_cast<T *>(base[j]) + idx;
  }
};

// Read rows straight from global memory (problem layout AOS or SOA).  AOS rows
// of a multiple of 4 doubles are fetched whole, one 32-byte load a sector,
// where a cell's fit into registers; the user function then reads those:
// coloured res_calc 1000^2, parts of 256, 44.8 us an iteration, 48.1 without (the
// atomic form 32.2 and 32.6).  miniAero's 56 values do not (96^3 AOS 187 us, 258
// fetched).
constexpr int kMostFetched = 16;
template <class L, bool SOA> struct GlobalRows {
  using T = typename L::read_t;
  __host__ __device__ static constexpr bool wide(int r) {
    return !SOA && sizeof(T) == 8 && L::read_dim(r) % 4 == 0;
  }
  // values of the wide sets before set r, over all slots
  __host__ __device__ static constexpr int values_before(int r) {
    int n = 0;
    for (int i = 0; i < r; ++i) n += wide(i) ? L::kDim * L::read_dim(i) : 0;
    return n;
  }
  static constexpr bool kFetch = values_before(L::kNumRead) > 0 && values_before(L::kNumRead) <= kMostFetched;
  const T *base[L::kNumRead > 0 ? L::kNumRead : 1];
  unsigned np[L::kNumRead > 0 ? L::kNumRead : 1];
  uint32_t p[2][L::kDim];
  T fetched[kFetch ? values_before(L::kNumRead) : 1];
  // takes the datasets; p[][] has been set
  __device__ __forceinline__ void bind(const LoopData &d);
  template <int R> __device__ __forceinline__ const T *ptr(int s) const {
    if constexpr (kFetch && wide(R)) return fetched + values_before(R) + s * L::read_dim(R);
    const uint32_t q = p[L::read_class(R)][s];
    const T *r = base[R] + (SOA ? (size_t)q : (size_t)q * L::read_dim(R));
    // AOS rows of a multiple of 16 bytes start 16-byte aligned: the compiler
    // may then merge neighbouring element loads into vector loads
    if constexpr (!SOA && (L::read_dim(R) * sizeof(T)) % 16 == 0)
      return static_cast<const T *>(__builtin_assume_aligned(r, 16));
    return r;
  }
  template <int R> __device__ __forceinline__ unsigned stride() const {
    return SOA ? np[R] : 1u;
  }
};

// Read rows staged in shared memory (AOS rows, stride 1).
template <class L> struct SmemRows {
  using T = typename L::read_t;
  const T *base[L::kNumRead > 0 ? L::kNumRead : 1];
  uint16_t l[2][L::kDim];
  template <int R> __device__ __forceinline__ const T *ptr(int s) const {
    const T *r = base[R] + (uint32_t)l[L::read_class(R)][s] * L::read_dim(R);
    if constexpr ((L::read_dim(R) * sizeof(T)) % 16 == 0)
      return static_cast<const T *>(__builtin_assume_aligned(r, 16));
    return r;
  }
  template <int R> __device__ __forceinline__ unsigned stride() const { return 1u; }
};

// Direct data whose written value is held back: the cell function's store to
// cell dataset j goes to *held, for the kernel to store later.
template <class T> struct HeldDirect : Direct {
  T *held;
  __device__ __forceinline__ HeldDirect(const Direct &d, T *h) : Direct(d), held(h) {}
  template <class U> __device__ __forceinline__ U *wptr(int) const { return held; }
};

template <class L, int I = 0, class F>
__device__ __forceinline__ void static_for_read(F &&f) {
  if constexpr (I < L::kNumRead) {
    f(std::integral_constant<int, I>{});
    static_for_read<L, I + 1>(f);
  }
}

// N values (a multiple of 4 doubles, 32-byte aligned as the rows of datasets are).
template <int N> __device__ __forceinline__ void load_wide(const double *p, double *v) {
#pragma unroll
  for (int k = 0; k < N; k += 4)
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[k]), "=d"(v[k + 1]), "=d"(v[k + 2]), "=d"(v[k + 3])
                 : "l"(p + k));
}

template <class L, bool SOA>
__device__ __forceinline__ void GlobalRows<L, SOA>::bind(const LoopData &d) {
  static_for_read<L>([&](auto r) {
    constexpr int R = decltype(r)::value;
    base[R] = static_cast<const T *>(d.point[L::read_set(R)]);
    np[R] = d.n_points[L::read_set(R)];
    if constexpr (kFetch && wide(R)) {
      constexpr int N = L::read_dim(R);
#pragma unroll
      for (int s = 0; s < L::kDim; ++s)
        load_wide<N>(base[R] + (size_t)p[L::read_class(R)][s] * N, fetched + values_before(R) + s * N);
    }
  });
}

__device__ __forceinline__ size_t out_index(bool soa, uint32_t np0, uint32_t p,
                                            int dim, int k) {
  return soa ? (size_t)k * np0 + p : (size_t)p * dim + k;
}

// Load mapping row `c` of a class into q[kDim] with vector loads.
template <int D>
__device__ __forceinline__ void load_row(const uint32_t *__restrict__ map, uint32_t c,
                                         uint32_t (&q)[D]) {
  if constexpr (D == 2) {
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(map) + c);
    q[0] = v.x;
    q[1] = v.y;
  } else if constexpr (D == 4) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(map) + c);
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
  } else if constexpr (D == 8) {
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(map) + 2 * (size_t)c);
    const uint4 b = __ldg(reinterpret_cast<const uint4 *>(map) + 2 * (size_t)c + 1);
    q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
    q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
  } else {
#pragma unroll
    for (int s = 0; s < D; ++s) q[s] = __ldg(map + (size_t)c * D + s);
  }
}

// ===========================================================================
// (a) atomic executor
// ===========================================================================

constexpr uint32_t kAtomicWarps = 8;  // warps per CTA of the atomic kernels

template <class T> __device__ __forceinline__ void atomic_add(T *a, T v) { atomicAdd(a, v); }

// Add the warp's 32 rows of K doubles (row of lane l: inc, for point key,
// kNoPoint: none) to AOS point data, through the warp's slice of shared
// memory: reduction instruction i then covers elements [32 i, 32 i + 32) of
// the rows laid end to end, so that neighbouring lanes fall into the same
// 32-byte sectors of `out` (K = 4: 8 whole sectors an instruction).  Lane by
// lane, component by component, each instruction would touch 32 sectors, and
// the L2's rate of atomic sectors bound the loop: one iteration of res_calc
// 1000^2 (4 doubles a row) after RCM 98.8 us so and 41.6 laid end to end (38.5 by
// quads, below); getacc 1024^2 97.8 and 50.4 us; LULESH 96^3 (3 doubles) 92.2 and
// 46.4 us.  FP32 rows of 4 are one 16-byte reduction and SOA data one run of
// addresses a component: neither needs it.
constexpr uint32_t kNoPoint = 0xFFFFFFFFu;
template <int K>
__device__ __forceinline__ void add_rows_f64(double *__restrict__ out, double *buf, uint32_t key,
                                             const double (&inc)[K]) {
  const uint32_t lane = threadIdx.x & 31u;
  __syncwarp();  // the previous slot's rows have been read
  if constexpr (K % 2 == 0) {
#pragma unroll
    for (int k = 0; k < K; k += 2)
      *reinterpret_cast<double2 *>(buf + lane * K + k) = make_double2(inc[k], inc[k + 1]);
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k) buf[lane * K + k] = inc[k];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const uint32_t e = i * 32u + lane, row = e / K;
    const uint32_t p = __shfl_sync(0xFFFFFFFFu, key, row);
    if (p != kNoPoint) atomic_add(out + (size_t)p * K + (e - row * K), buf[e]);
  }
}

// The same for rows of 4, without shared memory: the 4 lanes of a quad transpose
// their 4x4 values with two exchanges, after which lane q holds component q
// of the quad's 4 rows.  Neighbouring rows with one key are then neighbouring
// values of one lane: aggregation (AGG) sums those runs without a shuffle (runs
// across quads stay separate reductions).  It spares half of the shared-memory
// passes, and the L1's data path is what bounds loops that gather AOS rows:
// res_calc 1000^2, an iteration of 10 after RCM, 32.2 us so and 33.8 through
// shared memory, aggregated 26.9 and 33.9.  A loop that gathers none is better
// off with shared memory's fewer instructions: getacc 1024^2 44.6 us by quads
// and 38.5 (aggregated 44.9 and 39.6).
template <class L> constexpr bool by_quads() {
  return sizeof(typename L::out_t) == 8 && L::kOut == 4 && L::kNumRead > 0;
}
template <bool AGG>
__device__ __forceinline__ void add_rows4_f64(double *__restrict__ out, uint32_t key, double (&v)[4]) {
  const uint32_t q = threadIdx.x & 3u;
  const bool odd = q & 1u, high = q & 2u;
  // rows 2i, 2i + 1 (lanes q, q ^ 1): components 2i and 2i + 1 change places
  double a = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[0] : v[1], 1);
  double b = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[2] : v[3], 1);
  if (odd) {
    v[0] = a;
    v[2] = b;
  } else {
    v[1] = a;
    v[3] = b;
  }
  // halves (lanes q, q ^ 2)
  a = __shfl_xor_sync(0xFFFFFFFFu, high ? v[0] : v[2], 2);
  b = __shfl_xor_sync(0xFFFFFFFFu, high ? v[1] : v[3], 2);
  if (high) {
    v[0] = a;
    v[1] = b;
  } else {
    v[2] = a;
    v[3] = b;
  }
  uint32_t p[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) p[j] = __shfl_sync(0xFFFFFFFFu, key, (threadIdx.x & 28u) + j);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if constexpr (AGG) {
      if (j < 3 && p[j] == p[j + 1]) {
        v[j + 1] += v[j];
        continue;
      }
    }
    if (p[j] != kNoPoint) atomic_add(out + (size_t)p[j] * 4 + q, v[j]);
  }
}

// Warp aggregation: sum the rows of each run of neighbouring lanes with one
// key into the run's first lane (returns true there).  Orderings sort cells by
// their points, so that equal keys lie side by side (2 edges, 3 faces of a
// first cell); equal keys further apart stay separate reductions.  A warp
// without runs pays one shuffle and one vote.  Grouping every lane with
// __match_any_sync instead and gathering the group lane by lane costs more than
// the reductions it saves: one iteration of volna 1024^2 70.2 us, 42.6 us by runs;
// res_calc 1000^2 SOA 38.4 and 30.8 us; LULESH 96^3 SOA 73.8 and 44.7 us (after
// RCM).
template <int K, class T>
__device__ __forceinline__ bool sum_runs(uint32_t key, T (&inc)[K]) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, key, 1);
  const unsigned first = __ballot_sync(0xFFFFFFFFu, lane == 0 || before != key);
  // bit l: lane l + off lies in lane l's run (the same mask in every lane)
  unsigned inside = ~first >> 1;
  for (uint32_t off = 1; inside; inside &= inside >> off, off <<= 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const T v = __shfl_down_sync(0xFFFFFFFFu, inc[k], off);
      if ((inside >> lane) & 1u) inc[k] += v;
    }
  }
  return (first >> lane) & 1u;
}

// A cell's rows of the mappings (of a cell past n_cells: unchanged).
template <class L> struct CellMap {
  uint32_t p[2][L::kDim] = {};
  __device__ __forceinline__ void load(const LoopData &d, uint32_t c) {
    if (c >= d.n_cells) return;
    load_row<L::kDim>(d.map[0], c, p[0]);
    if constexpr (L::kHasClass1) load_row<L::kDim>(d.map[1], c, p[1]);
  }
};

// Cells [base, base + 32) of one mesh, one per lane of the calling warp
// (cells past n_cells are masked), whose mapping rows are given: compute,
// optionally sum the runs of lanes with one target point, add with atomics.
template <class L, bool SOA, bool AGG>
__device__ __forceinline__ void atomic_warp(const LoopData &d, uint32_t base, const CellMap<L> &map) {
  using out_t = typename L::out_t;
  constexpr int D = L::kDim, K = L::kOut;
  const uint32_t lane = threadIdx.x & 31u;
  out_t *__restrict__ out = static_cast<out_t *>(d.out);
  const uint32_t c = base + lane;
  const bool valid = c < d.n_cells;
  GlobalRows<L, SOA> rows;
  out_t inc[D][K];
#pragma unroll
  for (int s = 0; s < D; ++s) {
    rows.p[0][s] = map.p[0][s];
    rows.p[1][s] = map.p[1][s];
#pragma unroll
    for (int k = 0; k < K; ++k) inc[s][k] = out_t(0);
  }
  if (valid) {
    rows.bind(d);
    Direct dir{d.cell, c, d.n_cells};
    L::cell(rows, dir, inc);
  }
#pragma unroll
  for (int s = 0; s < D; ++s) {
    const uint32_t key = valid ? rows.p[0][s] : kNoPoint;
    if constexpr (!SOA && by_quads<L>()) {
      add_rows4_f64<AGG>(out, key, inc[s]);
      continue;
    }
    bool leader = valid;
    if constexpr (AGG) leader = sum_runs<K>(key, inc[s]) && valid;
    if constexpr (!SOA && sizeof(out_t) == 8) {
      __shared__ __align__(16) out_t s_rows[kAtomicWarps][32 * K];
      add_rows_f64<K>(out, s_rows[threadIdx.x >> 5], leader ? key : kNoPoint, inc[s]);
    } else if (leader) {
      if constexpr (!SOA && sizeof(out_t) == 4 && K == 4) {
        float4 v = make_float4(inc[s][0], inc[s][1], inc[s][2], inc[s][3]);
        atomicAdd(reinterpret_cast<float4 *>(out) + key, v);
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k)
          atomic_add(out + out_index(SOA, d.n_points[0], key, K, k), inc[s][k]);
      }
    }
  }
}

__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Prefetch cell c's mapping rows and direct data (every component of every
// cell dataset, SOA) into L2; one instruction per array covers a warp's 32
// consecutive cells.  Straight-line code: the loops over the loop's cell
// datasets and their (at most kMaxPrefetchDim) components are unrolled.
constexpr uint32_t kMaxPrefetchDim = 12;
template <class L> __device__ __forceinline__ void prefetch_cell(const LoopData &d, uint32_t c) {
  prefetch_l2(d.map[0] + (size_t)c * L::kDim);
  if constexpr (L::kHasClass1) prefetch_l2(d.map[1] + (size_t)c * L::kDim);
#pragma unroll
  for (int j = 0; j < L::kNumDirect; ++j) {
    const char *b = static_cast<const char *>(d.cell[j]) + (size_t)c * d.cell_size[j];
    const size_t stride = (size_t)d.n_cells * d.cell_size[j];
#pragma unroll
    for (uint32_t k = 0; k < kMaxPrefetchDim; ++k)
      if (k < d.cell_dim[j]) prefetch_l2(b + k * stride);
  }
}

// The launch of the atomic executor: tiles of 256 cells (32 per warp), taken
// in phases.  CTA c of a phase's `resident` CTAs takes tiles first + c,
// first + c + resident, ...: neighbouring CTAs run side by side through the
// mesh, so that a row one warp reads as a cell's first point is still in L2
// when another reads it as a second point.  A CTA that lags behind loses
// that, lags further, and the launch ends with idle SMs; at a phase's end the
// CTAs fall into step again (the next phase's CTA starts where one finished
// first), at the price of a CTA start per phase.  Which loops drift was
// measured, one iteration in phases of R rounds a CTA and in one phase for all:
// miniAero SOA 128^3 422 us (R = 4) and 582, 120^3 341 and 351, but 96^3 175 and 170
// (24 rounds in all: not split); getacc 1024^2 SOA 44.0 and 45.6 (R = 4; AOS 50 and
// 50); volna 1024^2 SOA 41.8 and 43.0 (R = 8; AOS 38 and 38); res_calc SOA without
// aggregation 1000^2 37.8 and 38.6, 1200^2 52.4 and 55.4, 2000^2 132 and 150 (R = 6),
// aggregated 1200^2 45.9 and 43.4, AOS 1000^2 39.4 and 38.7 (neither split); LULESH
// 96^3 45.6 and 44.4, miniAero AOS 128^3 486 and 452 (never split).
//
// The iterations of a call are one launch as well (no iteration reads what
// another writes), each running through the mesh in the direction opposite to
// the one before it, so that it starts on what is left in L2.  An iteration of
// 10, warm, as a launch of its own / in one launch in one direction / in
// alternating directions: res_calc 1000^2 SOA 34.6 / 31.6 / 29.7 us, LULESH 96^3 SOA
// 43.0 / 36.7 / 36.3, volna 1024^2 AOS 32.4 / 32.7 / 27.8, getacc 1024^2 AOS 41.4 /
// 43.7 / 38.5 (the launches of their own alternate too; miniAero 128^3, 1.29 GB,
// gains its launch gaps only).
//
// The grid starts while the one before it on the stream drains and waits for
// its end (griddep_wait) before it touches memory, which hides the launch:
// calls of one iteration one after the other, with and without, 64x48 res_calc
// 3.1 us (the host's rate) and 4.9, 200x210 3.5 and 6.2, volna 300^2 5.1 and 6.9,
// LULESH 30^3 7.0 and 8.3.  It does not let the next grid start before its own
// CTAs end (which all it could do is wait): with an early
// griddepcontrol.launch_dependents LULESH 30^3 takes 11.6 us, the others the same.
struct AtomicGrid {
  uint32_t tiles;     // of one iteration
  uint32_t resident;  // CTAs of a phase
  uint32_t rounds;    // tiles a CTA takes, at most
  uint32_t ctas;      // of one iteration: phases * resident
  uint32_t flip;      // iteration i runs last tile to first when i + flip is odd
};

// With L::kAtomicPrefetch, in the SOA form, each warp first prefetches the
// cells it will take next, so that their mapping rows and direct data come
// from L2 then; with L::atomic_carry it loads their mapping rows into
// registers, a memory latency ahead of the rows that they point to.
// SCATTERED: the form of problems whose rows are scattered (loops.cuh).
template <class L, bool SCATTERED> constexpr int atomic_min_blocks() {
  return SCATTERED ? L::kAtomicScatteredMinBlocks : L::kAtomicMinBlocks;
}
template <class L, bool SOA, bool AGG, bool SCATTERED>
__global__ void __launch_bounds__(256, (atomic_min_blocks<L, SCATTERED>())) k_atomic(LoopData d, AtomicGrid g) {
  const uint32_t in_tile = threadIdx.x & ~31u, lane = threadIdx.x & 31u;
  griddep_wait();
  const uint32_t it = blockIdx.x / g.ctas, b = blockIdx.x - it * g.ctas;
  const bool back = (it + g.flip) & 1u;
  const uint32_t phase = b / g.resident;
  uint32_t t = phase * g.rounds * g.resident + (b - phase * g.resident);
  constexpr bool kCarry = L::atomic_carry(SOA, AGG);
  CellMap<L> map;
  if (kCarry && t < g.tiles) map.load(d, (back ? g.tiles - 1u - t : t) * 256u + in_tile + lane);
  for (uint32_t r = 0; r < g.rounds && t < g.tiles; ++r, t += g.resident) {
    const uint32_t base = (back ? g.tiles - 1u - t : t) * 256u + in_tile;
    const uint32_t n = t + g.resident;
    const uint32_t next = (back ? g.tiles - 1u - n : n) * 256u + in_tile + lane;
    const bool more = r + 1 < g.rounds && n < g.tiles;
    if constexpr (L::kAtomicPrefetch && SOA && !SCATTERED) {
      if (more && next < d.n_cells) prefetch_cell<L>(d, next);
    }
    if constexpr (kCarry) {
      CellMap<L> ahead;
      if (more) ahead.load(d, next);
      atomic_warp<L, SOA, AGG>(d, base, map);
      map = ahead;
    } else {
      map.load(d, base + lane);
      atomic_warp<L, SOA, AGG>(d, base, map);
    }
  }
}

} // namespace fot

#include "hier.cuh"
#include "hier_pipe.cuh"
#include "hier_split.cuh"
