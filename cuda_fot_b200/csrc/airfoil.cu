// The Airfoil time step around the res_calc loop.
//
// The reference drives res_calc alone (res_calc.cu, Problem::loop*(num)).
// An Airfoil solver step also needs the loops on each side of it, which the
// reference does not contain; they restate the Airfoil finite-volume scheme
// (explicit two-stage update with local time steps, Roe-type edge fluxes
// with scalar dissipation) on the res_calc problem's own data:
//
//   per iteration:  save_soln  qold = q
//                   2 x { adt_calc   per cell: adt = sum over its 4 sides of
//                                    (|u dy - v dx| + c |side|), over cfl
//                         res_calc   per edge (the engine's plan: atomic or
//                                    coloured)
//                         bres_calc  per boundary edge: wall pressure, or the
//                                    res_calc flux against the free stream
//                         update     per cell: q = qold - res / adt, res = 0,
//                                    rms += |q change|^2 }
//                   rms = sqrt(rms / cells) of the second stage
//
// Data: the res_calc problem's point sets res (0), x (1, nodes), q (2),
// adt (3) in its current numbering and layout, plus the airfoil's own qold,
// cell -> 4 nodes, boundary edge -> 2 nodes / 1 cell / bound flag (given in
// the original numbering and renumbered here whenever the problem's
// numbering changes).  The per-cell loops run fused, each cell's values
// unchanged: bres_calc + update + the next stage's adt_calc in one pass (and
// between iterations + save_soln), whose last CTA sums the rms: an iteration
// is two res_calc runs and two cell passes.  bres_calc (4 edges of a cell at
// most, here) and the rms as launches of their own were 3 of 7 launches an
// iteration, each a few us of start and drain for next to no work: an
// iteration of 1000^2 was 185 us so (169 us as a graph) and 173 us (165) once
// fused; it is 141 us (141) now, 300^2 22.7 us.  Of that: each kernel started
// while the one before it drains (152 us without, 300^2 31.9), res_calc running
// against the cell passes' direction (it starts on the cells they left in L2:
// 150 us in their direction), a cell's corners asked for before anything is
// stored (163 us before that step).
// Every kernel is compiled without multiply-add
// contraction, and every sum has a fixed order: boundary edges are added per
// cell in increasing edge order (one thread per boundary cell), the rms is a
// fixed-shape tree.  With a coloured res_calc plan a step is therefore
// bit-identical to its CPU restatement replaying the same plan.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "engine.hpp"

namespace fot {
namespace {

constexpr double kGam = 1.4, kGm1 = 0.4, kEps = 0.05; // gm1 and eps as res_calc_func.hpp
constexpr uint32_t kThreads = 256;
#ifndef FOT_AIRFOIL_MAX_CTAS
#define FOT_AIRFOIL_MAX_CTAS 592
#endif
#ifndef FOT_CELLS_MINB
#define FOT_CELLS_MINB 4
#endif
// resident CTAs per SM of a cell pass (64 registers; 5 spill): 1000^2 an iteration
// 141 us, 148 with 3, 147 with 5
constexpr int kCellsMinCtas = FOT_CELLS_MINB;
// CTAs of a cell pass (grid-stride beyond): those a B200 holds at once, 148 SMs x 4
// (1000^2 141 us an iteration, 144 with twice as many).  Only speed and the order
// of the rms's sum follow it, which is one partial per CTA.
constexpr uint32_t kMaxUpdateCtas = FOT_AIRFOIL_MAX_CTAS;

struct AirfoilDev {
  const double *x;
  double *q, *qold, *adt, *res;
  uint32_t n_nodes, n_cells;
  int soa;
  const uint4 *cell_nodes;      // per cell: its 4 nodes, counter-clockwise
  // boundary cells: bit c & 31 of boundary[c / 32] is set, the cell's rank i
  // among them is before[c / 32] plus the set bits below
  const uint32_t *boundary, *before;
  const uint32_t *bcell_off;    // edges [off[i], off[i+1]) of boundary cell i in bedge order
  const uint2 *bedge_nodes;     // per boundary edge (grouped by cell): node 1, node 2
  const int *bedge_bound;       // 1: solid wall, else far field
  unsigned int *arrived;        // CTAs of a pass that wrote their partial sum
  double *rms;
  double qinf[4];
  double cfl;
};

__device__ __forceinline__ size_t at(int soa, uint32_t n, uint32_t i, int dim, int k) {
  return soa ? (size_t)k * n + i : (size_t)i * dim + k;
}

// The corners of a cell with nodes nd.
struct Corners {
  double px[4], py[4];
  __device__ __forceinline__ void load(const AirfoilDev &a, const uint4 &nd) {
    const uint32_t node[4] = {nd.x, nd.y, nd.z, nd.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (a.soa) {
        px[j] = a.x[node[j]];
        py[j] = a.x[(size_t)a.n_nodes + node[j]];
      } else {
        const double2 xy = *reinterpret_cast<const double2 *>(a.x + 2 * (size_t)node[j]);
        px[j] = xy.x;
        py[j] = xy.y;
      }
    }
  }
};

// adt_calc of a cell from its state q.
__device__ __forceinline__ double cell_adt(const AirfoilDev &a, const Corners &n, const double (&q)[4]) {
  const double ri = 1.0 / q[0];
  const double u = ri * q[1], v = ri * q[2];
  const double snd = sqrt(kGam * kGm1 * (ri * q[3] - 0.5 * (u * u + v * v)));
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double dx = n.px[(j + 1) & 3] - n.px[j];
    const double dy = n.py[(j + 1) & 3] - n.py[j];
    s += fabs(u * dy - v * dx) + snd * sqrt(dx * dx + dy * dy);
  }
  return s / a.cfl;
}

// bres_calc of boundary cell i (state q, time step adt1): its boundary edges
// added to its residual r in increasing edge order.
__device__ __forceinline__ void add_boundary(const AirfoilDev &a, uint32_t i, const double (&q)[4],
                                             double adt1, double (&r)[4]) {
  for (uint32_t e = a.bcell_off[i]; e < a.bcell_off[i + 1]; ++e) {
    const uint2 nd = a.bedge_nodes[e];
    const double dx = a.x[at(a.soa, a.n_nodes, nd.x, 2, 0)] - a.x[at(a.soa, a.n_nodes, nd.y, 2, 0)];
    const double dy = a.x[at(a.soa, a.n_nodes, nd.x, 2, 1)] - a.x[at(a.soa, a.n_nodes, nd.y, 2, 1)];
    const double ri = 1.0 / q[0];
    const double p1 = kGm1 * (q[3] - 0.5 * ri * (q[1] * q[1] + q[2] * q[2]));
    if (a.bedge_bound[e] == 1) {
      r[1] += p1 * dy;
      r[2] += -p1 * dx;
    } else {
      const double vol1 = ri * (q[1] * dy - q[2] * dx);
      const double *qi = a.qinf;
      const double ri2 = 1.0 / qi[0];
      const double p2 = kGm1 * (qi[3] - 0.5 * ri2 * (qi[1] * qi[1] + qi[2] * qi[2]));
      const double vol2 = ri2 * (qi[1] * dy - qi[2] * dx);
      const double mu = adt1 * kEps;
      r[0] += 0.5 * (vol1 * q[0] + vol2 * qi[0]) + mu * (q[0] - qi[0]);
      r[1] += 0.5 * (vol1 * q[1] + p1 * dy + vol2 * qi[1] + p2 * dy) + mu * (q[1] - qi[1]);
      r[2] += 0.5 * (vol1 * q[2] - p1 * dx + vol2 * qi[2] - p2 * dx) + mu * (q[2] - qi[2]);
      r[3] += 0.5 * (vol1 * (q[3] + p1) + vol2 * (qi[3] + p2)) + mu * (q[3] - qi[3]);
    }
  }
}

// Sum of the block's values in a fixed order (warp trees, then the warps'
// sums in warp order); the result is valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) s += smem[w];
  return s;
}

// The per-cell loops of the iteration, fused (each cell's values are the
// same as loop by loop): UPDATE (bres_calc where the cell has boundary edges,
// q = qold - res / adt, res = 0), with RMS the squared updates summed per CTA
// in a fixed order into partial[] and those by the last CTA to arrive, in CTA
// order; then SAVE (qold = q: save_soln of the next iteration) and ADT
// (adt_calc on the new q).
template <bool UPDATE, bool SAVE, bool ADT, bool RMS>
__global__ void __launch_bounds__(kThreads, kCellsMinCtas) k_cells(AirfoilDev a, double *partial) {
  __shared__ double smem[kThreads / 32];
  __shared__ bool s_last;
  griddep_wait();
  double sum = 0.0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < a.n_cells; c += stride) {
    double q[4];
    // a cell's nodes are asked for first and its corners before anything is
    // stored: after the stores their two dependent loads would wait for
    // everything before them (the compiler may not move loads up across
    // stores)
    uint4 nodes;
    Corners corners;
    if constexpr (ADT) nodes = __ldg(a.cell_nodes + c);
    if constexpr (UPDATE) {
      const double adt = a.adt[c];
      double r[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) r[k] = a.res[at(a.soa, a.n_cells, c, 4, k)];
      const uint32_t word = a.boundary[c >> 5], bit = 1u << (c & 31u);
      if (word & bit) {
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = a.q[at(a.soa, a.n_cells, c, 4, k)];
        add_boundary(a, a.before[c >> 5] + __popc(word & (bit - 1u)), q, adt, r);
      }
      double old[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) old[k] = a.qold[at(a.soa, a.n_cells, c, 4, k)];
      if constexpr (ADT) corners.load(a, nodes);
      const double adti = 1.0 / adt;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const size_t o = at(a.soa, a.n_cells, c, 4, k);
        const double del = adti * r[k];
        q[k] = old[k] - del;
        a.q[o] = q[k];
        a.res[o] = 0.0;
        if constexpr (RMS) sum += del * del;
      }
    } else {
      if constexpr (ADT) corners.load(a, nodes);
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = a.q[at(a.soa, a.n_cells, c, 4, k)];
    }
    if constexpr (SAVE) {
#pragma unroll
      for (int k = 0; k < 4; ++k) a.qold[at(a.soa, a.n_cells, c, 4, k)] = q[k];
    }
    if constexpr (ADT) a.adt[c] = cell_adt(a, corners, q);
  }
  if constexpr (RMS) {
    const double s = block_sum(sum, smem);
    if (threadIdx.x == 0) {
      partial[blockIdx.x] = s;
      __threadfence();
      s_last = atomicAdd(a.arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double v = 0.0;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += blockDim.x) v += __ldcg(partial + i);
    const double all = block_sum(v, smem);
    if (threadIdx.x == 0) {
      *a.rms = sqrt(all / (double)a.n_cells);
      *a.arrived = 0;
    }
  }
}

template <bool UPDATE, bool SAVE, bool ADT, bool RMS>
int launch_cells(const AirfoilDev &d, double *partial, uint32_t ctas, cudaStream_t st) {
  Chained c(dim3(ctas), dim3(kThreads), 0, st);
  FOT_CUDA(cudaLaunchKernelEx(&c.cfg, k_cells<UPDATE, SAVE, ADT, RMS>, d, partial));
  return FOT_OK;
}

uint32_t update_ctas(uint32_t n_cells) {
  return std::max<uint32_t>(1, std::min<uint32_t>((n_cells + kThreads - 1) / kThreads, kMaxUpdateCtas));
}

} // namespace
} // namespace fot

using namespace fot;

struct fot_airfoil {
  fot_problem *prob = nullptr;
  uint64_t version = 0; // problem numbering the device maps were built for
  uint32_t n_cells = 0, n_nodes = 0, n_bedges = 0;
  // original numbering (host)
  std::vector<uint32_t> cell_nodes, bedge_nodes, bedge_cell;
  std::vector<int32_t> bound;
  double qinf[4] = {0, 0, 0, 0};
  double cfl = 0.0;
  // device, current numbering
  DevBuf d_cell_nodes, d_boundary, d_before, d_bcell_off, d_bedge_nodes, d_bedge_bound;
  DevBuf qold, partial, rms, arrived;
};

namespace {

int upload(DevBuf &b, const void *host, size_t bytes) {
  FOT_TRY(b.alloc(bytes));
  if (bytes) FOT_CUDA(cudaMemcpy(b.ptr, host, bytes, cudaMemcpyHostToDevice));
  return FOT_OK;
}

// Copies from pageable memory and memsets may still be under way on the default
// stream when their calls return.  A run on a non-blocking stream does not wait
// for that stream, and a count of arrived CTAs cleared in the middle of a pass
// would never come to its end again: nothing is handed out before they are done.
int finish_uploads() {
  FOT_CUDA(cudaStreamSynchronize(nullptr));
  return FOT_OK;
}

// Rebuild the device maps for the problem's current numbering.
int airfoil_renumber(fot_airfoil *a) {
  fot_problem *p = a->prob;
  const std::vector<uint32_t> &cperm = p->point_perm[0], &nperm = p->point_perm[1];
  if (cperm.size() != a->n_cells || nperm.size() != a->n_nodes)
    return fail(FOT_ERR_STATE, "res_calc problem has no point permutation of the expected size");
  // cell -> nodes, rows moved to the cells' current numbers
  std::vector<uint32_t> cn((size_t)a->n_cells * 4);
  for (uint32_t c = 0; c < a->n_cells; ++c)
    for (int j = 0; j < 4; ++j) cn[(size_t)cperm[c] * 4 + j] = nperm[a->cell_nodes[(size_t)c * 4 + j]];
  // boundary edges grouped by (current) cell, increasing edge order inside a cell
  std::vector<uint32_t> idx(a->n_bedges);
  for (uint32_t e = 0; e < a->n_bedges; ++e) idx[e] = e;
  std::stable_sort(idx.begin(), idx.end(),
                   [&](uint32_t x, uint32_t y) { return cperm[a->bedge_cell[x]] < cperm[a->bedge_cell[y]]; });
  std::vector<uint32_t> bcell, boff, bnodes((size_t)a->n_bedges * 2);
  std::vector<int32_t> bb(a->n_bedges);
  for (uint32_t i = 0; i < a->n_bedges; ++i) {
    const uint32_t e = idx[i], c = cperm[a->bedge_cell[e]];
    if (bcell.empty() || bcell.back() != c) {
      bcell.push_back(c);
      boff.push_back(i);
    }
    bnodes[2 * (size_t)i] = nperm[a->bedge_nodes[2 * (size_t)e]];
    bnodes[2 * (size_t)i + 1] = nperm[a->bedge_nodes[2 * (size_t)e + 1]];
    bb[i] = a->bound[e];
  }
  boff.push_back(a->n_bedges);
  std::vector<uint32_t> boundary((a->n_cells + 31) / 32, 0), before(boundary.size(), 0);
  for (uint32_t c : bcell) boundary[c >> 5] |= 1u << (c & 31u);
  for (size_t w = 1; w < boundary.size(); ++w)
    before[w] = before[w - 1] + (uint32_t)__builtin_popcount(boundary[w - 1]);
  FOT_TRY(upload(a->d_cell_nodes, cn.data(), cn.size() * sizeof(uint32_t)));
  FOT_TRY(upload(a->d_boundary, boundary.data(), boundary.size() * sizeof(uint32_t)));
  FOT_TRY(upload(a->d_before, before.data(), before.size() * sizeof(uint32_t)));
  FOT_TRY(upload(a->d_bcell_off, boff.data(), boff.size() * sizeof(uint32_t)));
  FOT_TRY(upload(a->d_bedge_nodes, bnodes.data(), bnodes.size() * sizeof(uint32_t)));
  FOT_TRY(upload(a->d_bedge_bound, bb.data(), bb.size() * sizeof(int32_t)));
  FOT_TRY(finish_uploads());
  a->version = p->version;
  return FOT_OK;
}

} // namespace

void fot_airfoil_detach(fot_airfoil *a) {
  if (a) a->prob = nullptr;
}

extern "C" {

int fot_airfoil_create(fot_problem *p, const fot_airfoil_desc *desc, fot_airfoil **out) {
  if (!p || !desc || !out) return fail(FOT_ERR_ARG, "null argument");
  *out = nullptr;
  if (p->loop != FOT_LOOP_RES_CALC) return fail(FOT_ERR_ARG, "the Airfoil step runs on a res_calc problem");
  if (!desc->cell_to_node || (desc->n_bedges && (!desc->bedge_to_node || !desc->bedge_to_cell || !desc->bound)))
    return fail(FOT_ERR_ARG, "null mapping");
  if (!(desc->cfl > 0.0) || !(desc->qinf[0] > 0.0)) return fail(FOT_ERR_ARG, "cfl and qinf[0] must be positive");
  const uint32_t n_cells = p->n_points[0], n_nodes = p->n_points[1];
  for (size_t i = 0; i < (size_t)n_cells * 4; ++i)
    if (desc->cell_to_node[i] >= n_nodes) return fail(FOT_ERR_ARG, "cell_to_node[%zu] = %u out of range", i, desc->cell_to_node[i]);
  for (uint32_t e = 0; e < desc->n_bedges; ++e) {
    if (desc->bedge_to_cell[e] >= n_cells) return fail(FOT_ERR_ARG, "bedge_to_cell[%u] out of range", e);
    if (desc->bedge_to_node[2 * (size_t)e] >= n_nodes || desc->bedge_to_node[2 * (size_t)e + 1] >= n_nodes)
      return fail(FOT_ERR_ARG, "bedge_to_node[%u] out of range", e);
  }
  auto *a = new fot_airfoil;
  a->prob = p;
  a->n_cells = n_cells;
  a->n_nodes = n_nodes;
  a->n_bedges = desc->n_bedges;
  a->cell_nodes.assign(desc->cell_to_node, desc->cell_to_node + (size_t)n_cells * 4);
  a->bedge_nodes.assign(desc->bedge_to_node, desc->bedge_to_node + (size_t)desc->n_bedges * 2);
  a->bedge_cell.assign(desc->bedge_to_cell, desc->bedge_to_cell + desc->n_bedges);
  a->bound.assign(desc->bound, desc->bound + desc->n_bedges);
  std::memcpy(a->qinf, desc->qinf, sizeof(a->qinf));
  a->cfl = desc->cfl;
  int rc = airfoil_renumber(a);
  if (rc == FOT_OK) rc = a->qold.alloc((size_t)n_cells * 4 * sizeof(double));
  if (rc == FOT_OK) rc = a->partial.alloc(update_ctas(n_cells) * sizeof(double));
  if (rc == FOT_OK) rc = a->rms.alloc(sizeof(double));
  if (rc == FOT_OK) rc = a->arrived.alloc(sizeof(unsigned int));
  if (rc == FOT_OK && (cudaMemset(a->rms.ptr, 0, sizeof(double)) != cudaSuccess ||
                       cudaMemset(a->arrived.ptr, 0, sizeof(unsigned int)) != cudaSuccess))
    rc = fail(FOT_ERR_CUDA, "cudaMemset failed");
  if (rc == FOT_OK) rc = finish_uploads();
  if (rc != FOT_OK) {
    delete a;
    return rc;
  }
  p->airfoils.push_back(a);
  *out = a;
  return FOT_OK;
}

int fot_airfoil_destroy(fot_airfoil *a) {
  if (!a) return FOT_OK;
  if (a->prob) {
    auto &v = a->prob->airfoils;
    v.erase(std::remove(v.begin(), v.end(), a), v.end());
  }
  delete a;
  return FOT_OK;
}

} // extern "C"

namespace {

// Launch `iterations` solver iterations on st (no synchronisation).
int airfoil_enqueue(fot_airfoil *a, fot_plan *plan, uint32_t iterations, cudaStream_t st) {
  fot_problem *p = a->prob;
  AirfoilDev d{};
  d.x = static_cast<const double *>(p->point[1].ptr);
  d.q = static_cast<double *>(p->point[2].ptr);
  d.adt = static_cast<double *>(p->point[3].ptr);
  d.res = static_cast<double *>(p->point[0].ptr);
  d.qold = static_cast<double *>(a->qold.ptr);
  d.n_nodes = a->n_nodes;
  d.n_cells = a->n_cells;
  d.soa = p->layout == FOT_SOA;
  d.cell_nodes = a->d_cell_nodes.as<uint4>();
  d.boundary = a->d_boundary.as<uint32_t>();
  d.before = a->d_before.as<uint32_t>();
  d.bcell_off = a->d_bcell_off.as<uint32_t>();
  d.bedge_nodes = a->d_bedge_nodes.as<uint2>();
  d.bedge_bound = a->d_bedge_bound.as<int>();
  d.arrived = a->arrived.as<unsigned int>();
  d.rms = a->rms.as<double>();
  std::memcpy(d.qinf, a->qinf, sizeof(d.qinf));
  d.cfl = a->cfl;
  const uint32_t ctas = update_ctas(a->n_cells);
  double *part = a->partial.as<double>();
  // save_soln + adt_calc of the first stage; afterwards each update carries
  // the next stage's adt_calc (and, between iterations, save_soln)
  FOT_TRY((launch_cells<false, true, true, false>(d, part, ctas, st)));
  for (uint32_t it = 0; it < iterations; ++it) {
    for (int stage = 0; stage < 2; ++stage) {
      // backwards: from the cells that the pass before it left in L2, to those
      // that the pass after it starts with
      FOT_TRY(run_plan(p, plan, 1, true, st));
      if (stage == 0) FOT_TRY((launch_cells<true, false, true, false>(d, part, ctas, st)));
      else if (it + 1 < iterations) FOT_TRY((launch_cells<true, true, true, true>(d, part, ctas, st)));
      else FOT_TRY((launch_cells<true, false, false, true>(d, part, ctas, st)));
    }
  }
  return FOT_OK;
}

int airfoil_ready(fot_airfoil *a, fot_plan *plan) {
  if (!a || !plan) return fail(FOT_ERR_ARG, "null argument");
  if (!a->prob) return fail(FOT_ERR_STATE, "the airfoil's problem was destroyed");
  if (plan->prob != a->prob) return fail(FOT_ERR_STATE, "plan belongs to another (or a destroyed) problem");
  if (a->version != a->prob->version) FOT_TRY(airfoil_renumber(a));
  return FOT_OK;
}

} // namespace

extern "C" {

int fot_airfoil_run(fot_airfoil *a, fot_plan *plan, uint32_t iterations, double *rms, void *stream) {
  FOT_TRY(airfoil_ready(a, plan));
  if (iterations == 0) return FOT_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  FOT_TRY(airfoil_enqueue(a, plan, iterations, st));
  if (rms) {
    FOT_CUDA(cudaMemcpyAsync(rms, a->rms.ptr, sizeof(double), cudaMemcpyDeviceToHost, st));
    FOT_CUDA(cudaStreamSynchronize(st));
  }
  return FOT_OK;
}

int fot_airfoil_graph_create(fot_airfoil *a, fot_plan *plan, uint32_t iterations, void *stream,
                             fot_graph **out) {
  if (!out) return fail(FOT_ERR_ARG, "null argument");
  *out = nullptr;
  FOT_TRY(airfoil_ready(a, plan));
  if (iterations == 0) return fail(FOT_ERR_ARG, "a graph of zero iterations");
  struct Ctx {
    fot_airfoil *a;
    fot_plan *plan;
    uint32_t iterations;
  } ctx{a, plan, iterations};
  auto enqueue = [](void *c, cudaStream_t st) {
    const Ctx *x = static_cast<const Ctx *>(c);
    return airfoil_enqueue(x->a, x->plan, x->iterations, st);
  };
  FOT_TRY(capture_graph(static_cast<cudaStream_t>(stream), enqueue, &ctx, out));
  (*out)->prob = a->prob;
  (*out)->plan = plan;
  (*out)->ctl = plan->ctl.as<Ctl>();
  (*out)->version = a->prob->version;
  return FOT_OK;
}

int fot_airfoil_get_rms(fot_airfoil *a, double *rms, void *stream) {
  if (!a || !rms) return fail(FOT_ERR_ARG, "null argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  FOT_CUDA(cudaMemcpyAsync(rms, a->rms.ptr, sizeof(double), cudaMemcpyDeviceToHost, st));
  FOT_CUDA(cudaStreamSynchronize(st));
  return FOT_OK;
}

} // extern "C"
