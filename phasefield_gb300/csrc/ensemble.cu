// Batched ensemble of independent explicit Allen-Cahn simulations (block 1 of
// applications/allen_cahn/explicit) of uneven mesh size, degree (Q1/Q2) and parameters,
// advanced by ONE kernel launch per time step, the step loop captured in a CUDA graph.
//
// GB300 design:
//   * no grid-wide barrier: the state of each instance is kept as its un-normalised
//     accumulator; a step reads the accumulator of step k, forms n = invM (.) acc on the fly
//     in the gather (the same product the single-simulation finalize kernel computes), and
//     scatters the cell integrals of step k+1 into a second accumulator, while it zeroes a
//     third one (read one step earlier, so no block of this launch touches it). The three
//     accumulators rotate; a launch depends only on the previous launch having finished.
//   * one persistent launch for every instance and both degrees: a global list of cell tiles
//     (instance, first cell), the Q1 instances' first, of which each block takes a contiguous share,
//     with the instance's parameters (m_well, kappa) and its cell tables, built once
//     on the host with the engine's table builder for the instance's mesh spacing and copied into
//     shared memory where a block's share moves on to another instance;
//   * a tile is 32 cells on the lane kernel's layout and arithmetic (prismspf/gpu/cell_kernel_lanes.cuh:
//     a lane a cell, every contraction in exact 64-bit integers, the terms in registers), n warps a
//     tile and several tiles a block, so both degrees fill the same block of threads;
//   * the warps of a block and the grid size are chosen by a project-written autotuner that times
//     candidates on the ensemble itself.
// FP64 contractions (small ensembles, or PPF_FP64_CONTRACTIONS=1) run on one thread per point, tiles of
// up to 64 cells. Bound by instruction issue and the callback's FP64 operations (9 a point). 48 instances
// of 32 to 256 cells a side: 169 us a step (8 blocks of 6 warps an SM at 40 registers; 203 us with 2
// blocks of 18 warps at 56), against 273 us on one thread per point with the tables copied for each tile.
// Natural boundary conditions (the ensemble workload has no constraints).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ppf_gb300.h"
#include "graph_lengths.h"
#include "handle.h"
#include "models.cuh"

#include <prismspf/gpu/cell_kernel_lanes.cuh>

namespace ppf {
namespace {

struct EnsInstance {
  int degree;
  int nc[2];
  int nn[2];
  long long N;
  long long off;      // offset of the instance's vectors in the packed arrays
  long long tab_off;  // offset (bytes, 16-aligned) of its CellTables in the packed tables
  double h[2];
  double m_well, kappa;
};

struct EnsLaunch {
  const EnsInstance* inst;
  const int* tile_inst;         // instance of each tile
  const long long* tile_cell0;  // first cell of each tile
  long long ntiles;
  const double* invm;
  const double* acc_in;
  double* acc_out;
  double* acc_zero;
  long long total_len;
  double dt;
  const unsigned char* tables;  // per-instance CellTables<2, degree, double>
  long long ntiles1;            // tiles of Q1 instances (the first of the list)
};

template <int degree, int CPB>
__device__ void ens_tile(const EnsLaunch& P, const EnsInstance& I, long long cell0, double* smem) {
  constexpr int n = degree + 1, nq = n * n;
  using Tab = pg::CellTables<2, degree, double>;
  Tab* tab = reinterpret_cast<Tab*>(smem);
  double* vals = smem + pg::staged_table_room<2, degree, double>() / 8;
  double* outs = vals + CPB * nq;
  const int t = threadIdx.x;
  // stage the instance's tables (built on the host for its mesh spacing)
  {
    const unsigned int* src = reinterpret_cast<const unsigned int*>(P.tables + I.tab_off);
    unsigned int* dst = reinterpret_cast<unsigned int*>(tab);
    for (int k = t; k < (int)(pg::staged_table_bytes<2, degree, double>() / 4); k += blockDim.x) dst[k] = src[k];
  }
  const int lc = t / nq, q = t - lc * nq;
  const bool in_tile = lc < CPB;
  const long long cell = cell0 + lc;
  const long long ncells = (long long)I.nc[0] * I.nc[1];
  const bool active = in_tile && cell < ncells;
  const int qa = q % n, qb = q / n;
  long long node = 0;
  int cx = 0, cy = 0;
  if (active) {
    // instances hold fewer than 2^31 cells (int32 DoF indices): 32-bit division
    const unsigned int cl = (unsigned int)cell, n0 = (unsigned int)I.nc[0];
    cy = (int)(cl / n0);
    cx = (int)(cl - (unsigned int)cy * n0);
    node = (long long)(degree * cy + qb) * I.nn[0] + (degree * cx + qa);
    // gather: n = invM (.) acc of the previous step
    const double v = P.invm[I.off + node] * P.acc_in[I.off + node];
    vals[lc * nq + q] = v;
  }
  if (in_tile)
    for (int r = 0; r < 3; ++r) outs[r * CPB * nq + lc * nq + q] = 0.0;
  __syncthreads();
  pg::CellCtx<2, degree, double> ctx;
  ctx.tab = tab;
  ctx.vals = vals;
  ctx.outs = outs;
  ctx.stride = CPB * nq;
  ctx.lc = lc;
  ctx.q = q;
  ctx.cell[0] = cx;
  ctx.cell[1] = cy;
  ctx.cell[2] = 0;
  ctx.err = nullptr;
  ctx.submitted = 0;
  if (active) {
    AllenCahn<2, degree, double> pde{I.m_well, I.kappa};
    FieldContainer<2, degree, double> fc(ctx);
    pde.compute_rhs(fc, SimulationTimer(P.dt, 0.0), 1u);
  }
  __syncthreads();
  if (active) {
    double r = outs[lc * nq + q];
    {
      const double* g = outs + 1 * CPB * nq + lc * nq + (q - qa);
      const double* w = tab->jdt[0][q];
#pragma unroll
      for (int j = 0; j < n; ++j) r = fma(w[j], g[j], r);
    }
    {
      const double* g = outs + 2 * CPB * nq + lc * nq + (q - qb * n);
      const double* w = tab->jdt[1][q];
#pragma unroll
      for (int j = 0; j < n; ++j) r = fma(w[j], g[j * n], r);
    }
    atomicAdd(P.acc_out + I.off + node, r);
  }
  __syncthreads();
}

// The lane layout. Shared memory of one tile: its instance's tables, the nodal values (double and
// fixed-point), the gradient terms of the first direction, then the block exponents (two buffers of
// one value row and one component).
template <int degree>
constexpr size_t ens_lane_tile_bytes() {
  constexpr int nq = LaneShape<2, degree>::nq;
  return (sizeof(pg::CellTables<2, degree, double>) + 15) / 16 * 16 + 8 * LANE_CPT * 3 * nq + 4 * LANE_CPT * 4;
}

// tile groups of a degree: WARPS / n tiles, n warps each
template <int degree, int WARPS>
__host__ __device__ constexpr long long ens_groups(long long ntiles) {
  return (ntiles + WARPS / (degree + 1) - 1) / (WARPS / (degree + 1));
}

// this block's groups [first, last) of one degree (cell_kernel_lanes with one scalar row and one
// component). wait() comes before the first access to what earlier launches write.
template <int degree, int WARPS, class Wait>
__device__ void ens_lane_tiles(const EnsLaunch& P, unsigned char* smem, long long tile0, long long ntiles,
                               long long first, long long last, Wait&& wait) {
  using S = LaneShape<2, degree>;
  using Tab = pg::CellTables<2, degree, double>;
  namespace fx = pg::fx;
  constexpr int n = S::n, nq = S::nq, cols = S::cols, k = degree, CPT = LANE_CPT, per = WARPS / cols;
  constexpr int ROW = nq * CPT, JS = cols * CPT;
  constexpr int TOPT = n == 2 ? fx::LANE_TOP_INTEGRAL_Q1 : fx::LANE_TOP_INTEGRAL;
  constexpr unsigned int FLOOR = fx::EXP_FLOOR << 20;
  const int lc = threadIdx.x & 31;
  const int wi = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
  const int sub = wi / cols, w = wi - sub * cols;  // tile of the block's group, point of the first direction
  unsigned char* base = smem + (size_t)sub * ens_lane_tile_bytes<degree>();
  Tab* tab = reinterpret_cast<Tab*>(base);
  double* vals = reinterpret_cast<double*>(base + (sizeof(Tab) + 15) / 16 * 16);
  long long* vfx = reinterpret_cast<long long*>(vals + ROW);
  long long* outs = vfx + ROW;
  unsigned int* ex = reinterpret_cast<unsigned int*>(outs + ROW);  // [2][value row, component][cell]
  const int p0 = w * CPT + lc;
  const int step0 = w == k ? -CPT : CPT;
  if (first >= last) return;
  if (sub >= per) {  // a spare warp of a degree whose tiles do not fill the block: the barriers only
    __syncthreads();
    for (long long step = first; step < last; ++step)
      for (int b = 0; b < 4; ++b) __syncthreads();
    return;
  }
  // (the terms' floor is the instance's, below)
  for (int i = w * 32 + lc; i < 4 * CPT; i += cols * 32) ex[i] = (i / CPT) & 1 ? 0u : FLOOR;
  __syncthreads();
  int held = -1;  // the instance whose tables are in shared memory
  int par = 0;
  for (long long step = first; step < last; ++step, par ^= 1) {
    // spare tiles of the last group redo the last tile and scatter nothing
    const long long own = step * per + sub;
    const long long tile = tile0 + (own < ntiles ? own : ntiles - 1);
    const int inst = P.tile_inst[tile];
    const EnsInstance& I = P.inst[inst];
    if (inst != held) {  // (the tables were last read before the previous tile's last barrier)
      // (both 16-byte aligned and padded to whole 16 bytes)
      const uint4* src = reinterpret_cast<const uint4*>(P.tables + I.tab_off);
      uint4* dst = reinterpret_cast<uint4*>(tab);
#pragma unroll 4
      for (int i = w * 32 + lc; i < (int)((sizeof(Tab) + 15) / 16); i += cols * 32) dst[i] = __ldg(src + i);
      held = inst;
    }
    unsigned int* exi = ex + par * 2 * CPT;
    unsigned int* exo = exi + CPT;
    unsigned int* exn = ex + (par ^ 1) * 2 * CPT;
    const unsigned int ncells = (unsigned int)I.nc[0] * (unsigned int)I.nc[1];
    const unsigned int cell_t = (unsigned int)P.tile_cell0[tile] + lc;
    const bool active = own < ntiles && cell_t < ncells;
    const unsigned int cell = cell_t < ncells ? cell_t : ncells - 1;
    const unsigned int nn0 = (unsigned int)I.nn[0];
    const unsigned int cy = cell / (unsigned int)I.nc[0];
    const unsigned int cx = cell - cy * (unsigned int)I.nc[0];
    const long long node0 = I.off + (long long)(k * cy) * nn0 + (k * cx + w);
    wait();
    {
      // gather: n = invM (.) acc of the previous step
      double v[n];
#pragma unroll
      for (int j = 0; j < n; ++j) v[j] = P.invm[node0 + j * (long long)nn0] * P.acc_in[node0 + j * (long long)nn0];
      unsigned int m = 0;
#pragma unroll
      for (int j = 0; j < n; ++j) {
        vals[p0 + j * JS] = v[j];
        m = max(m, lane_abs_hi(v[j]));
      }
      atomicMax(&exi[lc], m);
    }
    __syncthreads();  // tables, nodal values and their block exponents complete
    {
      const unsigned int E = fx::high_exponent((int)(exi[lc] >> 20));
#pragma unroll
      for (int j = 0; j < n; ++j) vfx[p0 + j * JS] = fx::to_fixed_cut<fx::LANE_TOP_VALUES>(vals[p0 + j * JS], E);
      if (w == 0) exn[lc] = FLOOR;
      if (w == cols - 1) exn[CPT + lc] = 0u;
    }
    __syncthreads();  // fixed-point copies visible
    AllenCahn<2, degree, double> pde{I.m_well, I.kappa};
    const SimulationTimer timer(P.dt, 0.0);
    double term[n][3];
    unsigned int em[3] = {0, 0, 0};
#pragma unroll
    for (int j = 0; j < n; ++j) {
      pg::CellCtx<2, degree, double> ctx;
      ctx.tab = tab;
      ctx.vals = vals;
      ctx.outs = nullptr;
      ctx.stride = ROW;
      ctx.lc = lc;
      ctx.q = w + j * cols;
      ctx.cell[0] = (int)cx;
      ctx.cell[1] = (int)cy;
      ctx.cell[2] = 0;
      ctx.err = nullptr;
      ctx.submitted = 0;
      ctx.vals_fx = vfx;
      ctx.ex_in = reinterpret_cast<const int*>(exi);
      ctx.cpb = CPT;
      ctx.cpt = CPT;
      ctx.lean = 1;
      ctx.qi[0] = w;
      ctx.qi[1] = j;
      ctx.pe = p0 + j * JS;
      ctx.step[0] = step0;
      ctx.step[1] = j == k ? -JS : JS;
      ctx.nterm = 1;
#pragma unroll
      for (int i = 0; i < 3; ++i) ctx.term[i] = 0.0;
      FieldContainer<2, degree, double> fc(ctx);
      pde.compute_rhs(fc, timer, 1u);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        term[j][i] = ctx.term[i];
        em[i] = max(em[i], lane_abs_hi(ctx.term[i]));
      }
    }
    {
      const unsigned int raw = max(max(em[0], em[1]), em[2]);
      const unsigned int e = max(max(em[0] + tab->hadd, em[1] + tab->radd[0]), max(em[2] + tab->radd[1], tab->floor_out));
      atomicMax(&exo[lc], raw >= 0x7ff00000u ? 0xfff00000u : e);
    }
    __syncthreads();  // the terms' block exponents complete
    const int E = (int)(exo[lc] >> 20) - fx::EXP_BIAS;
    const unsigned long long isig = tab->isig[0];
    const int lsb = E - 1023 - TOPT + tab->ik[0];
    long long X[n], Gx[n], Gy[n];
#pragma unroll
    for (int j = 0; j < n; ++j) {
      X[j] = tab->hpow2 ? fx::to_fixed_cut<TOPT>(term[j][0], fx::high_exponent(E - tab->hk))
                        : fx::to_fixed_cut_scaled<TOPT>(term[j][0], fx::high_exponent(E), tab->hsig, tab->hk);
      Gx[j] = fx::to_fixed_cut<TOPT>(term[j][1], fx::high_exponent(E));
      Gy[j] = tab->rpow2[1] ? fx::to_fixed_cut<TOPT>(term[j][2], fx::high_exponent(E - tab->rk[1]))
                            : fx::to_fixed_cut_scaled<TOPT>(term[j][2], fx::high_exponent(E), tab->rsig[1], tab->rk[1]);
      outs[p0 + j * JS] = Gx[j];
    }
    __syncthreads();  // fixed-point terms visible
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const long long* g = outs + p0 + j * JS;
      if (n > 2 && w == 1) X[j] = lane_add_integral<n>(1, X[j], 0, g[-step0], g[step0]);
      else X[j] = lane_add_integral<n>(w, X[j], Gx[j], g[step0], n > 2 ? g[2 * step0] : 0ll);
    }
#pragma unroll
    for (int j = 0; j < n; ++j) {
      if (n > 2 && j == 1) X[j] = lane_add_integral<n>(1, X[j], 0, Gy[0], Gy[n - 1]);
      else X[j] = lane_add_integral<n>(j, X[j], Gy[j], Gy[j == 0 ? 1 : n - 2], Gy[j == 0 ? n - 1 : 0]);
      const int vw = (n > 2 && w == 1 ? 2 : 0) + (n > 2 && j == 1 ? 2 : 0);
      const double r = fx::to_double_cut(X[j], lsb + vw, isig, true, E >= fx::EXP_WIDE, E >= fx::EXP_NONFINITE);
      if (active) atomicAdd(P.acc_out + node0 + j * (long long)nn0, r);
    }
  }
}

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 48 / WARPS) ensemble_lane_kernel(const EnsLaunch P) {
  extern __shared__ __align__(16) unsigned char ens_lane_smem[];
  bool waited = false;
  auto wait = [&]() {
    if (waited) return;
    waited = true;
    chain_wait();
    chain_release();
    // zero the third accumulator (read one step earlier, untouched by this launch)
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P.total_len;
         i += (long long)gridDim.x * blockDim.x)
      P.acc_zero[i] = 0.0;
  };
  // an equal share of all the work, the Q1 groups first: a thread has 2 points of a Q1 group, 3 of a
  // Q2 group. Small ensembles have at most one group a block, where a share of either degree for every
  // block ran two, one after the other; their step is latency, so the tile's look-ups and tables,
  // which no launch writes, come before the wait for the previous step (100 steps of 8 instances of
  // 16 to 32 cells a side: 1.32 ms before, 0.87 ms).
  const long long g1 = ens_groups<1, WARPS>(P.ntiles1), g2 = ens_groups<2, WARPS>(P.ntiles - P.ntiles1);
  auto group = [&](long long b) {
    const long long u = (2 * g1 + 3 * g2) * b / gridDim.x;
    return u < 2 * g1 ? u / 2 : g1 + (u - 2 * g1) / 3;
  };
  const long long first = group(blockIdx.x), last = group(blockIdx.x + 1);
  ens_lane_tiles<1, WARPS>(P, ens_lane_smem, 0, P.ntiles1, first, last < g1 ? last : g1, wait);
  if (first < g1 && last > g1) __syncthreads();
  ens_lane_tiles<2, WARPS>(P, ens_lane_smem, P.ntiles1, P.ntiles - P.ntiles1, first > g1 ? first - g1 : 0, last - g1, wait);
  wait();
}

template <int WARPS>
constexpr size_t ens_lane_smem_bytes() {
  const size_t a = ens_lane_tile_bytes<1>() * (WARPS / 2), b = ens_lane_tile_bytes<2>() * (WARPS / 3);
  return a > b ? a : b;
}

template <int CPB1, int CPB2, int THREADS>
__global__ void __launch_bounds__(THREADS) ensemble_step_kernel(const EnsLaunch P) {
  extern __shared__ __align__(16) double ens_smem[];
  chain_wait();
  chain_release();
  // zero the third accumulator (read one step earlier, untouched by this launch)
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P.total_len;
       i += (long long)gridDim.x * blockDim.x)
    P.acc_zero[i] = 0.0;
  for (long long tile = blockIdx.x; tile < P.ntiles; tile += gridDim.x) {
    const EnsInstance I = P.inst[P.tile_inst[tile]];
    const long long cell0 = P.tile_cell0[tile];
    if (I.degree == 1) ens_tile<1, CPB1>(P, I, cell0, ens_smem);
    else ens_tile<2, CPB2>(P, I, cell0, ens_smem);
  }
}

template <int CPB1, int CPB2>
size_t ens_smem_bytes() {
  // tables, values and three output rows
  const size_t t1 = pg::staged_table_room<2, 1, double>() + 8 * 4 * CPB1 * 4;
  const size_t t2 = pg::staged_table_room<2, 2, double>() + 8 * 4 * CPB2 * 9;
  return std::max(t1, t2) + 64;
}

// extraction of the field values: n = invM (.) acc
__global__ void ensemble_extract_kernel(double* out, const double* invm, const double* acc, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = invm[i] * acc[i];
}

// tile-shape candidates: cells per tile for Q1 and for Q2, threads per block; on the lane layout
// (32 cells a tile) 6, 12 or 3 warps a block
struct Shape {
  int cpb1, cpb2, threads;
};
constexpr Shape SHAPES[] = {{64, 28, 256}, {32, 14, 128}, {16, 7, 64}};
constexpr Shape LANE_SHAPES[] = {{LANE_CPT, LANE_CPT, 192}, {LANE_CPT, LANE_CPT, 384}, {LANE_CPT, LANE_CPT, 96}};
constexpr int NSHAPES = 3;
// The default by tiles of 32 cells an SM. Up to 3 a step is the latency of one tile, shortest with one
// thread a point and FP64 sums, 128 threads a block (100 steps of 8 instances of 16 to 32 and 20 of
// 16 to 32 cells a side: 0.57 and 0.96 ms, lane layout 0.83 and 1.19 ms; 16 of 24 to 48, just above:
// 1.29 ms and 1.15 ms). Up to 32, blocks of 3 warps spread the tiles over the SMs (40 instances of 32
// to 64: 2.4 ms, 2.6 ms with 6 warps); from there on 6 warps.
constexpr long long POINT_TILES = 3, SPREAD_TILES = 32;
constexpr int POINT_SHAPE = 1, SPREAD_SHAPE = 2;
Shape shape_of(bool lanes, int s) { return lanes ? LANE_SHAPES[s] : SHAPES[s]; }

typedef void (*EnsKernel)(const EnsLaunch);
EnsKernel kernel_for(bool lanes, int s) {
  if (lanes) return s == 0 ? ensemble_lane_kernel<6> : (s == 1 ? ensemble_lane_kernel<12> : ensemble_lane_kernel<3>);
  switch (s) {
    case 0: return ensemble_step_kernel<64, 28, 256>;
    case 1: return ensemble_step_kernel<32, 14, 128>;
    default: return ensemble_step_kernel<16, 7, 64>;
  }
}
size_t smem_for(bool lanes, int s) {
  if (lanes) return s == 0 ? ens_lane_smem_bytes<6>() : (s == 1 ? ens_lane_smem_bytes<12>() : ens_lane_smem_bytes<3>());
  switch (s) {
    case 0: return ens_smem_bytes<64, 28>();
    case 1: return ens_smem_bytes<32, 14>();
    default: return ens_smem_bytes<16, 7>();
  }
}

}  // namespace
}  // namespace ppf

struct ppf_ensemble_s {
  int n = 0;
  std::vector<ppf::EnsInstance> h_inst;
  ppf::EnsInstance* d_inst = nullptr;
  long long total = 0;
  double* invm = nullptr;
  double* acc[3] = {nullptr, nullptr, nullptr};
  double* scratch = nullptr;
  int* tile_inst = nullptr;
  long long* tile_cell0 = nullptr;
  long long ntiles = 0, ntiles1 = 0;
  int shape = 0;
  int grid_mult = 4;
  int sms = 0;
  double dt = 0.0;
  long long step = 0;  // accumulator rotation counter
  cudaStream_t stream = nullptr;
  cudaStream_t own_stream = nullptr;
  // the captured steps, by the accumulator rotation's phase they start from: one rotation, and several
  struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    int rotations = 0;
    long long replayed = 0;  // rotations
  };
  StepGraph graph[3][2];
  int graph_shape = -1, graph_grid = -1;  // what they were captured with
  std::string err;
  double gl_w[2][3];
  double gl_D[2][3][3];
  unsigned char* d_tables = nullptr;  // per-instance CellTables, 16-byte aligned
  bool lanes = false;                 // every instance's tables allow the lane layout
};

namespace ppf {
namespace {

void drop_graphs(ppf_ensemble e) {
  for (auto& phase : e->graph)
    for (auto& g : phase) {
      if (g.exec) cudaGraphExecDestroy(g.exec);
      g = {};
    }
}

int efail(ppf_ensemble e, int code, const std::string& m) {
  if (e) e->err = m;
  return code;
}

#define ENS_CUDA(e, call)                                                                            \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess) return efail(e, PPF_ERR_CUDA, std::string(#call ": ") + cudaGetErrorString(e_)); \
  } while (0)

// tile list for the current shape
int build_tiles(ppf_ensemble e) {
  const Shape sh = shape_of(e->lanes, e->shape);
  std::vector<int> ti;
  std::vector<long long> tc;
  for (int i = 0; i < e->n; ++i) {
    const EnsInstance& I = e->h_inst[i];
    const long long nc = (long long)I.nc[0] * I.nc[1];
    const int cpb = I.degree == 1 ? sh.cpb1 : sh.cpb2;
    for (long long c = 0; c < nc; c += cpb) {
      ti.push_back(i);
      tc.push_back(c);
    }
  }
  // on the lane layout the Q1 instances' tiles first, each instance's together; else interleave
  // instances so consecutive tiles (and thus the blocks of one wave) mix instances of both degrees
  std::vector<size_t> order(ti.size());
  for (size_t k = 0; k < order.size(); ++k) order[k] = k;
  e->ntiles1 = 0;
  for (int i : ti) e->ntiles1 += e->h_inst[i].degree == 1;
  if (e->lanes)
    std::stable_sort(order.begin(), order.end(),
                     [&](size_t a, size_t b) { return e->h_inst[ti[a]].degree < e->h_inst[ti[b]].degree; });
  else
    std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) {
      const long long ra = tc[a] / (e->h_inst[ti[a]].degree == 1 ? sh.cpb1 : sh.cpb2);
      const long long rb = tc[b] / (e->h_inst[ti[b]].degree == 1 ? sh.cpb1 : sh.cpb2);
      return ra < rb;
    });
  std::vector<int> ti2(ti.size());
  std::vector<long long> tc2(tc.size());
  for (size_t k = 0; k < order.size(); ++k) {
    ti2[k] = ti[order[k]];
    tc2[k] = tc[order[k]];
  }
  drop_graphs(e);  // the captured steps point at the previous tile list
  cudaFree(e->tile_inst);
  cudaFree(e->tile_cell0);
  e->ntiles = (long long)ti2.size();
  ENS_CUDA(e, cudaMalloc(&e->tile_inst, sizeof(int) * e->ntiles));
  ENS_CUDA(e, cudaMalloc(&e->tile_cell0, sizeof(long long) * e->ntiles));
  ENS_CUDA(e, cudaMemcpy(e->tile_inst, ti2.data(), sizeof(int) * e->ntiles, cudaMemcpyHostToDevice));
  ENS_CUDA(e, cudaMemcpy(e->tile_cell0, tc2.data(), sizeof(long long) * e->ntiles, cudaMemcpyHostToDevice));
  return PPF_OK;
}

EnsLaunch make_launch(ppf_ensemble e, long long step) {
  EnsLaunch L;
  std::memset(&L, 0, sizeof(L));
  L.inst = e->d_inst;
  L.tile_inst = e->tile_inst;
  L.tile_cell0 = e->tile_cell0;
  L.ntiles = e->ntiles;
  L.invm = e->invm;
  L.acc_in = e->acc[step % 3];
  L.acc_out = e->acc[(step + 1) % 3];
  L.acc_zero = e->acc[(step + 2) % 3];
  L.total_len = e->total;
  L.dt = e->dt;
  L.tables = e->d_tables;
  L.ntiles1 = e->ntiles1;
  return L;
}

int launch_step(ppf_ensemble e, long long step, cudaStream_t s) {
  EnsKernel k = kernel_for(e->lanes, e->shape);
  const size_t smem = smem_for(e->lanes, e->shape);
  const Shape sh = shape_of(e->lanes, e->shape);
  long long grid = (long long)e->sms * e->grid_mult;
  long long work = e->ntiles;
  if (e->lanes) {
    const long long t1 = e->ntiles1, t2 = e->ntiles - t1;
    work = e->shape == 0 ? ens_groups<1, 6>(t1) + ens_groups<2, 6>(t2)
                         : (e->shape == 1 ? ens_groups<1, 12>(t1) + ens_groups<2, 12>(t2)
                                          : ens_groups<1, 3>(t1) + ens_groups<2, 3>(t2));
  }
  grid = std::max<long long>(1, std::min(grid, work));
  if (launch_chained(k, dim3((unsigned)grid), dim3(sh.threads), smem, s, make_launch(e, step)) != cudaSuccess)
    return efail(e, PPF_ERR_CUDA, "ensemble step launch failed");
  return PPF_OK;
}

}  // namespace
}  // namespace ppf

using namespace ppf;

extern "C" {

int ppf_ensemble_create(int n_instances, const ppf_mesh_desc* meshes, const double* m_well, const double* kappa,
                        double dt, ppf_ensemble* out) {
  if (!out || n_instances < 1 || !meshes || !m_well || !kappa) return PPF_ERR_ARG;
  *out = nullptr;
  auto* e = new ppf_ensemble_s();
  e->n = n_instances;
  e->dt = dt;
  for (int deg = 1; deg <= 2; ++deg) {
    GLRule g = gauss_lobatto(deg + 1);
    for (int i = 0; i <= deg; ++i) {
      e->gl_w[deg - 1][i] = g.w[i];
      for (int j = 0; j <= deg; ++j) e->gl_D[deg - 1][i][j] = g.D[i][j];
    }
  }
  long long off = 0;
  std::vector<double> invm;
  std::vector<unsigned char> tables;
  // the instance tables: block 1 of the Allen-Cahn application reads old n (value and gradient)
  // and submits n's value and gradient terms
  signed char slot_of[pg::MAX_FIELDS][pg::NAGE], slot_comp0[pg::MAX_SLOTS], out_of[pg::MAX_FIELDS],
      out_row0[pg::MAX_OUTS];
  std::memset(slot_of, -1, sizeof(slot_of));
  std::memset(slot_comp0, 0, sizeof(slot_comp0));
  std::memset(out_of, -1, sizeof(out_of));
  std::memset(out_row0, 0, sizeof(out_row0));
  slot_of[0][1] = 0;
  out_of[0] = 0;
  for (int i = 0; i < n_instances; ++i) {
    const ppf_mesh_desc& m = meshes[i];
    if (m.dim != 2 || m.degree < 1 || m.degree > 2 || m.periodic[0] || m.periodic[1]) {
      delete e;
      return PPF_ERR_UNSUPPORTED;
    }
    EnsInstance I{};
    I.degree = m.degree;
    for (int d = 0; d < 2; ++d) {
      I.nc[d] = m.subdivisions[d] << m.global_refinement;
      I.nn[d] = m.degree * I.nc[d] + 1;
      I.h[d] = m.size[d] / I.nc[d];
    }
    I.N = (long long)I.nn[0] * I.nn[1];
    I.off = off;
    {
      const double lo[3] = {0.0, 0.0, 0.0}, hh[3] = {I.h[0], I.h[1], 1.0};
      auto tb = build_cell_tables(2, I.degree, 0, lo, hh, slot_of, slot_comp0, out_of, out_row0, 1u);
      if (tb.empty()) {
        delete e;
        return PPF_ERR_UNSUPPORTED;
      }
      I.tab_off = (long long)tables.size();
      // (the lane body's value rows start from the floor of cells up to 2^32, EXP_FLOOR)
      e->lanes = (i == 0 || e->lanes) && tables_lanes(tb, 2, I.degree) != 0 && std::max(I.h[0], I.h[1]) <= 0x1p32;
      tables.insert(tables.end(), tb.begin(), tb.end());
      tables.resize((tables.size() + 15) / 16 * 16, 0);
    }
    I.m_well = m_well[i];
    I.kappa = kappa[i];
    off += I.N;
    e->h_inst.push_back(I);
    // lumped mass of the instance (natural boundaries)
    std::vector<double> m1[2];
    for (int d = 0; d < 2; ++d) {
      m1[d].assign(I.nn[d], 0.0);
      for (int c = 0; c < I.nc[d]; ++c)
        for (int a = 0; a <= I.degree; ++a) m1[d][I.degree * c + a] += e->gl_w[I.degree - 1][a] * I.h[d];
    }
    for (int J = 0; J < I.nn[1]; ++J)
      for (int K = 0; K < I.nn[0]; ++K) invm.push_back(1.0 / (m1[0][K] * m1[1][J]));
  }
  e->total = off;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, dev);
  auto bail = [&](int code) {
    ppf_ensemble_destroy(e);
    return code;
  };
  if (cudaStreamCreateWithFlags(&e->own_stream, cudaStreamNonBlocking) != cudaSuccess) return bail(PPF_ERR_CUDA);
  e->stream = e->own_stream;
  if (cudaMalloc(&e->d_inst, sizeof(EnsInstance) * n_instances) != cudaSuccess) return bail(PPF_ERR_CUDA);
  cudaMemcpy(e->d_inst, e->h_inst.data(), sizeof(EnsInstance) * n_instances, cudaMemcpyHostToDevice);
  if (cudaMalloc(&e->d_tables, tables.size()) != cudaSuccess) return bail(PPF_ERR_CUDA);
  cudaMemcpy(e->d_tables, tables.data(), tables.size(), cudaMemcpyHostToDevice);
  if (cudaMalloc(&e->invm, sizeof(double) * off) != cudaSuccess) return bail(PPF_ERR_CUDA);
  cudaMemcpy(e->invm, invm.data(), sizeof(double) * off, cudaMemcpyHostToDevice);
  for (int k = 0; k < 3; ++k) {
    if (cudaMalloc(&e->acc[k], sizeof(double) * off) != cudaSuccess) return bail(PPF_ERR_CUDA);
    cudaMemset(e->acc[k], 0, sizeof(double) * off);
  }
  if (cudaMalloc(&e->scratch, sizeof(double) * off) != cudaSuccess) return bail(PPF_ERR_CUDA);
  {
    long long tiles = 0;
    for (const EnsInstance& I : e->h_inst) tiles += ((long long)I.nc[0] * I.nc[1] + LANE_CPT - 1) / LANE_CPT;
    if (tiles <= POINT_TILES * e->sms) {
      e->lanes = false;
      e->shape = POINT_SHAPE;
    }
    if (e->lanes) {
      e->grid_mult = 8;  // 48 of an SM's warps with 6 a block
      if (tiles <= SPREAD_TILES * e->sms) e->shape = SPREAD_SHAPE;
    }
  }
  for (int s = 0; s < NSHAPES; ++s)
    cudaFuncSetAttribute(kernel_for(e->lanes, s), cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_for(e->lanes, s));
  if (build_tiles(e)) return bail(PPF_ERR_CUDA);
  *out = e;
  return PPF_OK;
}

void ppf_ensemble_destroy(ppf_ensemble e) {
  if (!e) return;
  if (e->stream) cudaStreamSynchronize(e->stream);
  drop_graphs(e);
  cudaFree(e->d_inst);
  cudaFree(e->d_tables);
  cudaFree(e->invm);
  for (int k = 0; k < 3; ++k) cudaFree(e->acc[k]);
  cudaFree(e->scratch);
  cudaFree(e->tile_inst);
  cudaFree(e->tile_cell0);
  if (e->own_stream) cudaStreamDestroy(e->own_stream);
  delete e;
}

const char* ppf_ensemble_last_error(ppf_ensemble e) { return e ? e->err.c_str() : "null ensemble"; }

long long ppf_ensemble_instance_length(ppf_ensemble e, int i) {
  if (!e || i < 0 || i >= e->n) return -1;
  return e->h_inst[i].N;
}

// upload instance i's field (lattice order): the accumulator holds mass (.) n
int ppf_ensemble_upload(ppf_ensemble e, int i, const double* host) {
  if (!e || !host || i < 0 || i >= e->n) return PPF_ERR_ARG;
  const EnsInstance& I = e->h_inst[i];
  std::vector<double> im(I.N), acc(I.N);
  ENS_CUDA(e, cudaMemcpy(im.data(), e->invm + I.off, sizeof(double) * I.N, cudaMemcpyDeviceToHost));
  for (long long k = 0; k < I.N; ++k) acc[k] = host[k] / im[k];
  ENS_CUDA(e, cudaMemcpy(e->acc[e->step % 3] + I.off, acc.data(), sizeof(double) * I.N, cudaMemcpyHostToDevice));
  return PPF_OK;
}

int ppf_ensemble_download(ppf_ensemble e, int i, double* host) {
  if (!e || !host || i < 0 || i >= e->n) return PPF_ERR_ARG;
  const EnsInstance& I = e->h_inst[i];
  ensemble_extract_kernel<<<grid_for(I.N), 256, 0, e->stream>>>(e->scratch + I.off, e->invm + I.off,
                                                                  e->acc[e->step % 3] + I.off, I.N);
  ENS_CUDA(e, cudaGetLastError());
  ENS_CUDA(e, cudaMemcpyAsync(host, e->scratch + I.off, sizeof(double) * I.N, cudaMemcpyDeviceToHost, e->stream));
  ENS_CUDA(e, cudaStreamSynchronize(e->stream));
  return PPF_OK;
}

namespace ppf {
namespace {

// captures `rotations` rotations of steps from the present phase into g
int capture_steps(ppf_ensemble e, ppf_ensemble_s::StepGraph& g, int rotations) {
  if (g.exec) cudaGraphExecDestroy(g.exec);
  g = {};
  cudaGraph_t graph = nullptr;
  ENS_CUDA(e, cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
  int rc = PPF_OK;
  for (int k = 0; k < 3 * rotations && !rc; ++k) rc = launch_step(e, e->step + k, e->stream);
  const cudaError_t end = cudaStreamEndCapture(e->stream, &graph);
  if (!rc && (end != cudaSuccess || cudaGraphInstantiate(&g.exec, graph, 0) != cudaSuccess))
    rc = efail(e, PPF_ERR_CUDA, "ensemble step capture failed");
  if (graph) cudaGraphDestroy(graph);
  g.rotations = rc ? 0 : rotations;
  return rc;
}

}  // namespace
}  // namespace ppf

// advance every instance by n_steps explicit steps: one launch per step; with use_graph whole
// accumulator rotations (three steps) are replayed from captured graphs, their lengths by
// graph_lengths.h
int ppf_ensemble_run(ppf_ensemble e, int n_steps, int use_graph) {
  if (!e || n_steps < 0) return PPF_ERR_ARG;
  int done = 0;
  if (use_graph && (e->graph_shape != e->shape || e->graph_grid != e->grid_mult)) {
    drop_graphs(e);
    e->graph_shape = e->shape;
    e->graph_grid = e->grid_mult;
  }
  while (use_graph && n_steps - done >= 3) {
    auto& held = e->graph[e->step % 3];
    const int rotations = (n_steps - done) / 3;
    const GraphChoice c = choose_graph(rotations, held[0].exec != nullptr, held[0].replayed, held[1].rotations);
    auto& g = held[c.replay > 1];
    if (c.capture)
      if (const int rc = capture_steps(e, g, c.capture)) return rc;
    for (int r = rotations / c.replay; r > 0; --r) {
      ENS_CUDA(e, cudaGraphLaunch(g.exec, e->stream));
      done += 3 * c.replay;
      e->step += 3 * c.replay;  // phase unchanged
      g.replayed += c.replay;
    }
  }
  for (; done < n_steps; ++done) {
    int rc = launch_step(e, e->step, e->stream);
    if (rc) return rc;
    e->step++;
  }
  return PPF_OK;
}

// autotuner: times each tile shape and grid size on `steps` steps of this ensemble (on a copy
// of the state, which is restored) and keeps the fastest; returns its time per step in ms
int ppf_ensemble_autotune(ppf_ensemble e, int steps, double* best_ms, int* best_shape, int* best_grid) {
  if (!e || steps < 1) return PPF_ERR_ARG;
  // save the state
  std::vector<double> save(e->total);
  ENS_CUDA(e, cudaStreamSynchronize(e->stream));
  ENS_CUDA(e, cudaMemcpy(save.data(), e->acc[e->step % 3], sizeof(double) * e->total, cudaMemcpyDeviceToHost));
  const long long step0 = e->step;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  double best = 1e300;
  int bs = e->shape, bg = e->grid_mult;
  const int grids[] = {1, 2, 4, 8};
  for (int s = 0; s < NSHAPES; ++s) {
    e->shape = s;
    if (build_tiles(e)) return PPF_ERR_CUDA;
    for (int gm : grids) {
      e->grid_mult = gm;
      launch_step(e, e->step, e->stream);  // warm-up
      e->step++;
      cudaEventRecord(a, e->stream);
      for (int k = 0; k < steps; ++k) {
        launch_step(e, e->step, e->stream);
        e->step++;
      }
      cudaEventRecord(b, e->stream);
      cudaEventSynchronize(b);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, a, b);
      if (ms / steps < best) {
        best = ms / steps;
        bs = s;
        bg = gm;
      }
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  e->shape = bs;
  e->grid_mult = bg;
  if (build_tiles(e)) return PPF_ERR_CUDA;
  // restore the state
  e->step = step0;
  for (int k = 0; k < 3; ++k) ENS_CUDA(e, cudaMemset(e->acc[k], 0, sizeof(double) * e->total));
  ENS_CUDA(e, cudaMemcpy(e->acc[e->step % 3], save.data(), sizeof(double) * e->total, cudaMemcpyHostToDevice));
  if (best_ms) *best_ms = best;
  if (best_shape) *best_shape = bs;
  if (best_grid) *best_grid = bg;
  return PPF_OK;
}

int ppf_ensemble_synchronize(ppf_ensemble e) {
  if (!e) return PPF_ERR_ARG;
  ENS_CUDA(e, cudaStreamSynchronize(e->stream));
  return PPF_OK;
}

int ppf_ensemble_set_stream(ppf_ensemble e, void* stream) {
  if (!e) return PPF_ERR_ARG;
  ENS_CUDA(e, cudaStreamSynchronize(e->stream));
  drop_graphs(e);
  e->stream = stream ? static_cast<cudaStream_t>(stream) : e->own_stream;
  return PPF_OK;
}

}  // extern "C"
