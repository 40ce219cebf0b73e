// Lane kernel: the cell loop of an FP64 Q1/Q2 operator with every contraction in exact 64-bit
// integers, laid out so that one lane of a warp is one cell.
//
// The same per-cell work as cell_kernel (MFOperator::compute_local_operator,
// src/solvers/mf_operator.cc:34-80, with FieldContainer::reinit_and_eval /
// integrate_and_distribute, include/prismspf/core/field_container.h:794-882): gather ->
// user callback per quadrature point -> integrate -> condensed scatter. The layout and the
// arithmetic differ:
//   * a thread block owns a tile of 32 cells; lane l of every warp is cell l of the tile. Warp w
//     takes the w-th point of the cell's first dim-1 directions and each of its threads the n
//     points above it along the last direction (a line of its cell): point (w, j) is
//     q = w + j * n^(dim-1) (Q2 3-D: 9 warps, 3 points a thread). Rows of shared memory are
//     [point][cell], so every access is a contiguous warp row, a point's position on its lines
//     is uniform across the warp, and the per-cell block exponents are shared-memory atomics on
//     32 distinct words, one per thread and row;
//   * derivatives: exact integer line sums of the nodal values' fixed-point copies, taken from the
//     point outwards and rounded once with 1/h_d folded in (FieldContainer::lane_deriv);
//   * integration: the submitted value term (as h_0 v) and gradient terms (as (h_0 / h_d) g_d) of a
//     cell and output component share one block exponent; with the integer quadrature weights
//     (1, 1 or 1, 4, 1 per direction) divided out of its node, an integral is the exact sum
//     x + sum_d L_d, L_d = +-(4 (own + m) - (own + f)) at the ends of a Q2 line and g_0 - g_2 in its
//     middle: no weight is multiplied in, 25 is the largest coefficient sum, and the terms keep 57
//     bits (59 on Q1 cells) below the cell's largest one. It is rounded once with the scale detJ / (h_0 W^dim) and
//     the node's weight as an exponent. No FP64 instruction outside the user's callback: on GB300
//     the FP64 pipe retires about two operations per SM per clock and every FP64 conversion runs
//     on it too, so the integer path (issue slots) replaces 9-10 FP64 operations per point;
//   * the terms a callback submits stay in registers: with one output component from the callback
//     through the exponent barrier to the integration (only the gradient rows other threads read
//     pass through shared memory), with several until they are stored;
//   * four block barriers per tile: nodal values and exponents, fixed-point copies, the terms'
//     exponents, their fixed-point copies. The exponents alternate between two buffers so that
//     resetting the next tile's needs no extra barrier;
//   * the cell tables and the flat row lists are kernel parameters (constant-bank loads), with the
//     slots by (field, age) so that a getter's look-up is one operand; every output component is
//     integrated (rows the callback leaves stay zero), so no branch depends on which terms were
//     submitted; lanes past the last cell recompute the last cell and skip its scatter.
// Accuracy: every derivative and every node's integral is one rounding of an exact sum of values
// cut to 2^-59 (derivatives) or 2^-57 (integration, 2^-59 on Q1 cells) of the largest magnitude of their cell and row.
//
// What bounds it: instruction issue (53-61 % of the slots at 32 warps an SM, the ALU pipe 42-49 %, the
// FP64 pipe 34-59 %; DRAM 3-5 %). Cahn-Hilliard 64^3 Q2, per launch of the c and the mu block: 130 and
// 157 us at 460 instructions a point, against 208 and 213 us at 690 with rounded instead of cut conversions,
// weights as 64-bit shifts and the terms through shared memory, and 243 and 293 us for cell_kernel.
// Stretched cells (64 x 60 x 52): 105 and 128 us against 188 and 226 us for cell_kernel.
#pragma once

#include <cuda_runtime.h>

#include <cstring>

#include <prismspf/gpu/cell_kernel.cuh>

#pragma push_macro("compute_rhs")
#pragma push_macro("compute_lhs")
#undef compute_rhs
#undef compute_lhs

namespace ppf {

// Q1/Q2 on a lane kernel tile: lane l of every warp is cell l of a 32-cell tile; warp w holds
// the w-th point of the cell's first dim-1 directions, and its thread the n points above it
// along the last direction (a line of the cell): point (w, j) is q = w + j * cols.
template <int dim, int degree>
struct LaneShape {
  static constexpr int n = degree + 1;
  static constexpr int nq = pg::ipow(n, dim);
  static constexpr int cols = nq / n;  // warps per block
  static constexpr int threads = 32 * cols;
};
constexpr int LANE_CPT = 32;  // cells per tile

// An operator may ask for a register budget (`cell_lane_min_blocks`, resident blocks per SM);
// the default aims at about 48 registers a thread (Cahn-Hilliard Q2 3-D, c block: 4 blocks of 288
// threads at 56 registers measured 130 us a launch against 143 us for 5 blocks and 146 us for 3)
template <class PDE, int threads, class = void>
struct CellLaneMinBlocks {
  static constexpr int value = 65536 / (threads * 48) > 0 ? (65536 / (threads * 48) < 32 ? 65536 / (threads * 48) : 32) : 1;
};
template <class PDE, int threads>
struct CellLaneMinBlocks<PDE, threads, std::void_t<decltype(PDE::cell_lane_min_blocks)>> {
  static constexpr int value = PDE::cell_lane_min_blocks;
};

// ... of a launch with NC output components: with several, shared memory admits fewer blocks than the
// register budget would (3 components on Q2 3-D: 104 KB, 2 blocks), and the registers they leave free
// go to the callback (the 48^3 Q2 elasticity product: 296 us at 56 registers, spilling, 248 us at 87)
template <class PDE, int dim, int degree, int NC>
constexpr int lane_min_blocks() {
  using S = LaneShape<dim, degree>;
  constexpr int regs = CellLaneMinBlocks<PDE, S::threads>::value;
  constexpr int smem = 232448 / (S::nq * LANE_CPT * 8 * (NC == 1 ? 1 : NC * (2 + dim)));
  return NC == 1 || regs < smem ? regs : (smem > 0 ? smem : 1);
}

// The output components (bit c: c components in a block) an operator's lane kernels are compiled
// for: `cell_lane_components`, by default 1 to 4
template <class PDE, class = void>
struct CellLaneComponents {
  static constexpr unsigned int value = 2u | 4u | 8u | 16u;
};
template <class PDE>
struct CellLaneComponents<PDE, std::void_t<decltype(PDE::cell_lane_components)>> {
  static constexpr unsigned int value = PDE::cell_lane_components;
};

// shared memory of a tile: the double copies of the nv value rows, the fixed-point copies of the
// ng gradient rows, the gradient terms of the nout components (one component keeps its value and
// last-direction terms in registers: dim - 1 rows; several keep 1 + dim rows each), then the block
// exponents of the gradient rows and of the components (two buffers each)
template <int dim, int degree>
__host__ __device__ constexpr size_t lane_smem_bytes(int nv, int ng, int nout) {
  using S = LaneShape<dim, degree>;
  return (size_t)S::nq * LANE_CPT * 8 * (size_t)(nv + ng + (nout == 1 ? dim - 1 : nout * (1 + dim))) +
         4 * (size_t)LANE_CPT * (size_t)(2 * ng + 2 * nout);
}

// t plus the line integral over its node's integer weight (1 at the ends, 4 in the middle of a Q2
// line), from the point's own term outwards: own, its neighbour m and the far end f for an end of
// the line, the line's first and last term as m and f for its middle
template <int n>
__device__ __forceinline__ long long lane_add_integral(int j, long long t, long long own, long long m, long long f) {
  if constexpr (n == 2) {
    return j == 0 ? t - own - m : t + own + m;
  } else {
    if (j == 1) return t + m - f;
    if (j == 0) return t - ((own + m) << 2) + own + f;
    return t + ((own + m) << 2) - own - f;
  }
}

// The rows of one launch as flat lists (built on the host from the launch record): input rows
// (one per component of each dependency slot) and output components (one per component of each
// block field).
constexpr int LANE_MAX_IN = 6;
constexpr int LANE_MAX_OUT = pg::LANE_MAX_OUT;
struct LaneRows {
  int nin;
  int nout;
  int nv;                                // input rows with a double copy (read as values or Hessians)
  int ng;                                // input rows with a fixed-point copy (read as gradients)
  unsigned int div_m[2], div_l[2];       // cell index -> (x, y, z): multiply-high divisors of nc[0], nc[1]
  const double* in_base[LANE_MAX_IN];    // vector of the row's slot
  const int* in_cmap[LANE_MAX_IN];       // constraint map for a constrained read, else null
  unsigned int in_off[LANE_MAX_IN];      // component offset c * N
  int in_v[LANE_MAX_IN], in_g[LANE_MAX_IN];  // the row's double and fixed-point copy, -1 without one
  double* out_acc[LANE_MAX_OUT];         // accumulator of the output's field
  const int* out_cmap[LANE_MAX_OUT];     // condensation map, else null
  unsigned int out_off[LANE_MAX_OUT];    // component offset c * N
  int out_row[LANE_MAX_OUT];             // value row of the component (dim gradient rows follow)
};

// the high word of |v|, whose bits above 20 are the biased exponent: ordered like |v|
__device__ __forceinline__ unsigned int lane_abs_hi(double v) { return (unsigned int)__double2hiint(v) & 0x7fffffffu; }

// NC: output components of the launch. One component keeps the terms of the thread's n points in
// registers between the callback and the integration; several pass them through shared memory.
template <class PDE, int dim, int degree, int MODE, int NC, int MINB>
__global__ void __launch_bounds__(LaneShape<dim, degree>::threads, MINB)
    cell_kernel_lanes(const __grid_constant__ CellLaunch P, const __grid_constant__ PDE pde,
                      const __grid_constant__ pg::CellTables<dim, degree, double> T,
                      const __grid_constant__ LaneRows R) {
  static_assert(degree <= 2 && MODE != MODE_DIAG, "the lane kernel covers FP64 Q1/Q2 RHS and LHS launches");
  using S = LaneShape<dim, degree>;
  using Tab = pg::CellTables<dim, degree, double>;
  namespace fx = pg::fx;
  constexpr int n = S::n, nq = S::nq, cols = S::cols, k = degree, CPT = LANE_CPT;
  constexpr int ROW = nq * CPT;   // entries of one row
  constexpr int JS = cols * CPT;  // entry stride between a thread's points
  constexpr int TOPT = n == 2 ? fx::LANE_TOP_INTEGRAL_Q1 : fx::LANE_TOP_INTEGRAL;
  constexpr int TC = 1 + dim;     // terms of a component
  constexpr bool REGS = NC == 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // the tables are a kernel parameter: read-only constant-bank loads, uniform where their index is
  const Tab* tab = &T;
  double* vals = reinterpret_cast<double*>(smem_raw);               // [nv][q][cell]
  long long* vfx = reinterpret_cast<long long*>(vals + R.nv * ROW);  // [ng][q][cell]
  long long* outs = vfx + R.ng * ROW;                               // terms [row][q][cell]
  // block exponents of the gradient rows and (EXP_BIAS more) of the components, as high words
  unsigned int* ex_in = reinterpret_cast<unsigned int*>(outs + (REGS ? dim - 1 : NC * TC) * ROW);  // [2][ng][cell]
  unsigned int* ex_out = ex_in + 2 * R.ng * CPT;                    // [2][NC][cell]

  const int t = threadIdx.x;
  const int lc = t & 31;
  const int w = __shfl_sync(0xffffffffu, t >> 5, 0);  // point of the first dim-1 directions (uniform)
  const int p0 = w * CPT + lc;   // entry of the thread's first point; point j at p0 + j * JS
  const int qa = w % n;
  const int qb = dim > 2 ? w / n : 0;
  // entry steps from the thread's points along the first directions (back from a line's last point)
  const int step0 = qa == k ? -CPT : CPT;
  const int step1 = qb == k ? -n * CPT : n * CPT;
  const int hpow2 = tab->hpow2, hk = tab->hk;
  const unsigned long long hsig = tab->hsig;
  const unsigned int floor_in = tab->floor_in, floor_out = tab->floor_out;  // (read once: 1 % of a launch)
  for (int i = t; i < 2 * (R.ng + NC) * CPT; i += S::threads) ex_in[i] = i < 2 * R.ng * CPT ? floor_in : floor_out;
  const unsigned int nn0 = (unsigned int)P.nn[0], nn1 = (unsigned int)P.nn[1];
  const unsigned int lstride = dim > 2 ? nn0 * nn1 : nn0;  // lattice stride of the last direction
  const unsigned int ncells = (unsigned int)P.ncells;
  const unsigned int ntiles = (ncells + CPT - 1) / CPT;
  chain_wait();
  chain_release();
  __syncthreads();  // exponent buffers set

  int par = 0;
  for (unsigned int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, par ^= 1) {
    unsigned int* exi = ex_in + par * R.ng * CPT;
    unsigned int* exn = ex_in + (par ^ 1) * R.ng * CPT;
    unsigned int* exo = ex_out + par * NC * CPT;
    unsigned int* exon = ex_out + (par ^ 1) * NC * CPT;
    // lanes past the last cell redo the last cell and skip its scatter
    const unsigned int cell_t = tile * CPT + lc;
    const bool active = cell_t < ncells;
    const unsigned int cell = active ? cell_t : ncells - 1;
    int cx, cy = 0, cz = 0;
    {
      const unsigned int q0 = (__umulhi(cell, R.div_m[0]) + cell) >> R.div_l[0];
      cx = (int)(cell - q0 * (unsigned int)P.nc[0]);
      if (dim == 2) cy = (int)q0;
      if (dim > 2) {
        const unsigned int q1 = (__umulhi(q0, R.div_m[1]) + q0) >> R.div_l[1];
        cy = (int)(q0 - q1 * (unsigned int)P.nc[1]);
        cz = (int)q1;
      }
    }
    // lattice node of the thread's first point (last-direction index 0)
    const unsigned int node0 = dim > 2 ? ((unsigned int)(k * cz) * nn1 + (unsigned int)(k * cy + qb)) * nn0 + (unsigned int)(k * cx + qa)
                                       : (unsigned int)(k * cy) * nn0 + (unsigned int)(k * cx + qa);

    // gather (read_dof_values_plain, or read_dof_values for a constrained src) and the block
    // exponents of the rows read as gradients
#pragma unroll
    for (int r = 0; r < LANE_MAX_IN; ++r) {
      if (r < R.nin) {
        const double* base = global_ptr(R.in_base[r] + R.in_off[r]);
        double v[n];
        if (R.in_cmap[r]) {
          const int* cm = R.in_cmap[r] + R.in_off[r];
#pragma unroll
          for (int j = 0; j < n; ++j) {
            const unsigned int idx = node0 + (unsigned int)j * lstride;
            const int m = __ldg(cm + idx);
            const double own = base[idx];
            v[j] = m == (int)(idx + R.in_off[r]) ? own : (m >= 0 ? global_ptr(R.in_base[r] + m)[0] : 0.0);
          }
        } else {
#pragma unroll
          for (int j = 0; j < n; ++j) v[j] = base[node0 + (unsigned int)j * lstride];
        }
        const int vs = R.in_v[r], gs = R.in_g[r];
        if (vs >= 0) {
#pragma unroll
          for (int j = 0; j < n; ++j) vals[vs * ROW + p0 + j * JS] = v[j];
        }
        if (gs >= 0) {
          unsigned int m = 0;
#pragma unroll
          for (int j = 0; j < n; ++j) {
            // a gradient row's double stays in its fixed-point slot until converted in place
            vfx[gs * ROW + p0 + j * JS] = __double_as_longlong(v[j]);
            m = max(m, lane_abs_hi(v[j]));
          }
          atomicMax(&exi[gs * CPT + lc], m);
        }
      }
    }
    __syncthreads();  // nodal values and their block exponents complete

    // fixed-point copies; reset the next tile's exponents
#pragma unroll
    for (int g = 0; g < LANE_MAX_IN; ++g) {
      if (g < R.ng) {
        // (a cell holding a non-finite value gets meaningless copies: every result read from them
        // is replaced by NaN)
        const unsigned int E = fx::high_exponent((int)(exi[g * CPT + lc] >> 20));
        long long* x = vfx + g * ROW + p0;
#pragma unroll
        for (int j = 0; j < n; ++j) x[j * JS] = fx::to_fixed_cut<fx::LANE_TOP_VALUES>(__longlong_as_double(x[j * JS]), E);
      }
    }
    for (int g = w; g < R.ng; g += cols) exn[g * CPT + lc] = floor_in;
    for (int o = w; o < NC; o += cols) exon[o * CPT + lc] = floor_out;
    __syncthreads();  // fixed-point copies visible

    // the user callback at each of the thread's points
    const SimulationTimer& timer = P.timer_dev ? *P.timer_dev : P.timer;
    double term[REGS ? n * TC : 1];
    unsigned int em[NC * TC];  // largest magnitude of each term over the thread's points
#pragma unroll
    for (int i = 0; i < NC * TC; ++i) em[i] = 0;
    auto point = [&](int j, double* keep) {
      pg::CellCtx<dim, degree, double> ctx;
      ctx.tab = tab;
      ctx.vals = vals;
      ctx.outs = nullptr;
      ctx.stride = ROW;
      ctx.lc = lc;
      ctx.q = w + j * cols;
      ctx.cell[0] = cx;
      ctx.cell[1] = cy;
      ctx.cell[2] = cz;
      ctx.err = P.err;
      ctx.submitted = 0;
      ctx.vals_fx = vfx;
      ctx.ex_in = reinterpret_cast<const int*>(exi);
      ctx.cpb = CPT;
      ctx.cpt = CPT;
      ctx.lean = 1;
      ctx.qi[0] = qa;
      ctx.qi[1] = dim > 2 ? qb : j;
      ctx.qi[2] = dim > 2 ? j : 0;
      ctx.pe = p0 + j * JS;
      ctx.step[0] = step0;
      ctx.step[1] = dim > 2 ? step1 : (j == k ? -JS : JS);
      ctx.step[2] = dim > 2 ? (j == k ? -JS : JS) : 0;
      ctx.nterm = NC;
#pragma unroll
      for (int i = 0; i < NC * TC; ++i) ctx.term[i] = 0.0;
      FieldContainer<dim, degree, double> fc(ctx);
      if constexpr (MODE == MODE_LHS) pde.compute_lhs(fc, timer, P.block_id);
      else pde.compute_rhs(fc, timer, P.block_id);
#pragma unroll
      for (int i = 0; i < NC * TC; ++i) em[i] = max(em[i], lane_abs_hi(ctx.term[i]));
      if constexpr (REGS) {
#pragma unroll
        for (int i = 0; i < TC; ++i) keep[i] = ctx.term[i];
      } else {
#pragma unroll
        for (int i = 0; i < NC * TC; ++i) outs[i * ROW + p0 + j * JS] = __double_as_longlong(ctx.term[i]);
      }
    };
    if constexpr (REGS) {
#pragma unroll
      for (int j = 0; j < n; ++j) point(j, term + j * TC);
    } else {
      // (one copy of the callback's code)
#pragma unroll 1
      for (int j = 0; j < n; ++j) point(j, nullptr);
    }
    // block exponents of every output component's terms (those the callback left are zero): the
    // value term enters as h v, the gradient terms as (h_0 / h_d) g
#pragma unroll
    for (int o = 0; o < NC; ++o) {
      unsigned int e = em[o * TC] + tab->hadd, raw = em[o * TC];
#pragma unroll
      for (int d = 0; d < dim; ++d) {
        e = max(e, em[o * TC + 1 + d] + tab->radd[d]);
        raw = max(raw, em[o * TC + 1 + d]);
      }
      atomicMax(&exo[o * CPT + lc], raw >= 0x7ff00000u ? 0xfff00000u : e);
    }
    __syncthreads();  // submitted terms and their block exponents complete

    // the submitted terms to fixed point (with a non-finite term the copies are meaningless and the
    // integral is replaced by NaN)
    auto fixed_value = [&](double v, int E) {
      return hpow2 ? fx::to_fixed_cut<TOPT>(v, fx::high_exponent(E - hk))
                   : fx::to_fixed_cut_scaled<TOPT>(v, fx::high_exponent(E), hsig, hk);
    };
    auto fixed_gradient = [&](double g, int d, int E) {
      if (d == 0) return fx::to_fixed_cut<TOPT>(g, fx::high_exponent(E));
      return tab->rpow2[d] ? fx::to_fixed_cut<TOPT>(g, fx::high_exponent(E - tab->rk[d]))
                           : fx::to_fixed_cut_scaled<TOPT>(g, fx::high_exponent(E), tab->rsig[d], tab->rk[d]);
    };
    // one node's integral from its component's value term x and line integrals, and its scatter
    // (distribute_local_to_global through the constraint map)
    const int sab = (n > 2 && qa == 1 ? 2 : 0) + (n > 2 && qb == 1 ? 2 : 0);
    auto scatter = [&](int o, int j, int E, long long Tx) {
      const int vw = sab + (n > 2 && j == 1 ? 2 : 0);
      const double r = fx::to_double_cut(Tx, E - 1023 - TOPT + tab->ik[0] + vw, tab->isig[0], true,
                                         E >= fx::EXP_WIDE, E >= fx::EXP_NONFINITE);
      const unsigned int idx = node0 + (unsigned int)j * lstride + R.out_off[o];
      const int target = R.out_cmap[o] ? __ldg(R.out_cmap[o] + idx) : (int)idx;
      if (active && target >= 0) atomicAdd(global_ptr(R.out_acc[o] + target), r);
    };
    if constexpr (REGS) {
      const int E = (int)(exo[lc] >> 20) - fx::EXP_BIAS;
      long long X[n], G[dim][n];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        X[j] = fixed_value(term[j * TC], E);
#pragma unroll
        for (int d = 0; d < dim; ++d) {
          G[d][j] = fixed_gradient(term[j * TC + 1 + d], d, E);
          if (d < dim - 1) outs[d * ROW + p0 + j * JS] = G[d][j];
        }
      }
      __syncthreads();  // fixed-point terms visible
      // the first directions' lines, the position on them uniform across the warp
#pragma unroll
      for (int d = 0; d < dim - 1; ++d) {
        const long long* g = outs + d * ROW + p0;
        const int st = d == 0 ? step0 : step1, id = d == 0 ? qa : qb;
        if (n > 2 && id == 1) {
#pragma unroll
          for (int j = 0; j < n; ++j) X[j] = lane_add_integral<n>(1, X[j], 0, g[j * JS - st], g[j * JS + st]);
        } else if (id == 0) {
#pragma unroll
          for (int j = 0; j < n; ++j)
            X[j] = lane_add_integral<n>(0, X[j], G[d][j], g[j * JS + st], n > 2 ? g[j * JS + 2 * st] : 0ll);
        } else {
#pragma unroll
          for (int j = 0; j < n; ++j)
            X[j] = lane_add_integral<n>(k, X[j], G[d][j], g[j * JS + st], n > 2 ? g[j * JS + 2 * st] : 0ll);
        }
      }
      // the last direction's line is the thread's own points
      const long long* z = G[dim - 1];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        if (n > 2 && j == 1) X[j] = lane_add_integral<n>(1, X[j], 0, z[0], z[n - 1]);
        else X[j] = lane_add_integral<n>(j, X[j], z[j], z[j == 0 ? 1 : n - 2], z[j == 0 ? n - 1 : 0]);
        scatter(0, j, E, X[j]);
      }
    } else {
#pragma unroll
      for (int o = 0; o < NC; ++o) {
        const int E = (int)(exo[o * CPT + lc] >> 20) - fx::EXP_BIAS;
#pragma unroll
        for (int i = 0; i < TC; ++i) {
          long long* x = outs + (o * TC + i) * ROW + p0;
#pragma unroll
          for (int j = 0; j < n; ++j) {
            const double v = __longlong_as_double(x[j * JS]);
            x[j * JS] = i == 0 ? fixed_value(v, E) : fixed_gradient(v, i - 1, E);
          }
        }
      }
      __syncthreads();  // fixed-point terms visible
#pragma unroll
      for (int o = 0; o < NC; ++o) {
        const int E = (int)(exo[o * CPT + lc] >> 20) - fx::EXP_BIAS;
        const long long* x = outs + o * TC * ROW + p0;
        const long long* z = x + dim * ROW;  // the last direction's line is the thread's own points
        const long long z0 = z[0], z1 = z[JS], z2 = n > 2 ? z[2 * JS] : 0ll;
#pragma unroll
        for (int j = 0; j < n; ++j) {
          long long Tx = x[j * JS];
#pragma unroll
          for (int d = 0; d < dim - 1; ++d) {
            const long long* g = x + (1 + d) * ROW + j * JS;
            const int st = d == 0 ? step0 : step1, id = d == 0 ? qa : qb;
            if (n > 2 && id == 1) Tx = lane_add_integral<n>(1, Tx, 0, g[-st], g[st]);
            else Tx = lane_add_integral<n>(id, Tx, g[0], g[st], n > 2 ? g[2 * st] : 0ll);
          }
          if (n > 2 && j == 1) Tx = lane_add_integral<n>(1, Tx, 0, z0, z2);
          else Tx = lane_add_integral<n>(j, Tx, j == 0 ? z0 : (n > 2 ? z2 : z1), j == 0 || n > 2 ? z1 : z0, j == 0 ? z2 : z0);
          scatter(o, j, E, Tx);
        }
      }
    }
  }
}

// FP32 operators (the smoothing levels of a mixed-precision V-cycle) on the same layout: 32 cells
// a tile, a line of each cell per thread, plain FP32 contractions (derivatives from the nodal
// values, integration with the tables' jdt weights), so a tile needs two barriers (nodal values;
// submitted terms). Any cell shape. (Keeping the terms of a thread's line in registers, 36 instead of
// 84 shared accesses a point, is no faster: 143 against 134 us for the 64^3 Q2 elasticity product.)
template <int dim, int degree>
__host__ __device__ constexpr size_t lane_f32_smem_bytes(int nrows_in, int nrows_out) {
  using S = LaneShape<dim, degree>;
  return (size_t)S::nq * LANE_CPT * 4 * (size_t)(nrows_in + nrows_out);
}

template <class PDE, int dim, int degree, int MODE, int MINB>
__global__ void __launch_bounds__(LaneShape<dim, degree>::threads, MINB)
    cell_kernel_lanes_f32(const __grid_constant__ CellLaunch P, const __grid_constant__ PDE pde,
                          const __grid_constant__ pg::CellTables<dim, degree, float> T,
                          const __grid_constant__ LaneRows R) {
  static_assert(degree <= 2 && MODE == MODE_LHS, "the FP32 lane kernel covers Q1/Q2 LHS launches");
  using S = LaneShape<dim, degree>;
  using Tab = pg::CellTables<dim, degree, float>;
  constexpr int n = S::n, nq = S::nq, cols = S::cols, k = degree, CPT = LANE_CPT;
  constexpr int ROW = nq * CPT;
  constexpr int JS = cols * CPT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Tab* tab = &T;
  float* vals = reinterpret_cast<float*>(smem_raw);  // [nin][q][cell]
  float* outs = vals + R.nin * ROW;                  // [out rows][q][cell]
  const int t = threadIdx.x;
  const int lc = t & 31;
  const int w = t >> 5;
  const int p0 = w * CPT + lc;
  const int qa = w % n;
  const int qb = dim > 2 ? w / n : 0;
  const unsigned int nn0 = (unsigned int)P.nn[0], nn1 = (unsigned int)P.nn[1];
  const unsigned int lstride = dim > 2 ? nn0 * nn1 : nn0;
  const unsigned int ncells = (unsigned int)P.ncells;
  const unsigned int ntiles = (ncells + CPT - 1) / CPT;
  chain_wait();
  chain_release();

  for (unsigned int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const unsigned int cell_t = tile * CPT + lc;
    const bool active = cell_t < ncells;
    const unsigned int cell = active ? cell_t : ncells - 1;
    int cx, cy = 0, cz = 0;
    {
      const unsigned int q0 = (__umulhi(cell, R.div_m[0]) + cell) >> R.div_l[0];
      cx = (int)(cell - q0 * (unsigned int)P.nc[0]);
      if (dim == 2) cy = (int)q0;
      if (dim > 2) {
        const unsigned int q1 = (__umulhi(q0, R.div_m[1]) + q0) >> R.div_l[1];
        cy = (int)(q0 - q1 * (unsigned int)P.nc[1]);
        cz = (int)q1;
      }
    }
    const unsigned int node0 = dim > 2 ? ((unsigned int)(k * cz) * nn1 + (unsigned int)(k * cy + qb)) * nn0 + (unsigned int)(k * cx + qa)
                                       : (unsigned int)(k * cy) * nn0 + (unsigned int)(k * cx + qa);
    // the previous tile's integration read the submitted terms and values: done by all threads
    __syncthreads();
#pragma unroll
    for (int r = 0; r < LANE_MAX_IN; ++r) {
      if (r < R.nin) {
        const float* base = global_ptr(reinterpret_cast<const float*>(R.in_base[r]));
#pragma unroll
        for (int j = 0; j < n; ++j) {
          const unsigned int idx = node0 + (unsigned int)j * lstride + R.in_off[r];
          float v;
          if (R.in_cmap[r]) {
            const int m = __ldg(R.in_cmap[r] + idx);
            const float own = base[idx];
            v = m == (int)idx ? own : (m >= 0 ? base[m] : 0.f);
          } else {
            v = base[idx];
          }
          vals[r * ROW + p0 + j * JS] = v;
        }
      }
    }
#pragma unroll
    for (int o = 0; o < LANE_MAX_OUT; ++o)
      if (o < R.nout)
#pragma unroll
        for (int i = 0; i <= dim; ++i)
#pragma unroll
          for (int j = 0; j < n; ++j) outs[(R.out_row[o] + i) * ROW + p0 + j * JS] = 0.f;
    __syncthreads();  // nodal values visible

    const SimulationTimer& timer = P.timer_dev ? *P.timer_dev : P.timer;
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      pg::CellCtx<dim, degree, float> ctx;
      ctx.tab = tab;
      ctx.vals = vals;
      ctx.outs = outs;
      ctx.stride = ROW;
      ctx.lc = lc;
      ctx.q = w + j * cols;
      ctx.cell[0] = cx;
      ctx.cell[1] = cy;
      ctx.cell[2] = cz;
      ctx.err = P.err;
      ctx.submitted = 0;
      ctx.cpt = CPT;
      FieldContainer<dim, degree, float> fc(ctx);
      pde.compute_lhs(fc, timer, P.block_id);
    }
    __syncthreads();  // submitted terms visible

    // integrate (the tables' jdt weights) and scatter
#pragma unroll
    for (int o = 0; o < LANE_MAX_OUT; ++o) {
      if (o < R.nout) {
        const int rv = R.out_row[o];
#pragma unroll
        for (int j = 0; j < n; ++j) {
          const int q = w + j * cols;
          const int qi[3] = {qa, dim > 2 ? qb : j, dim > 2 ? j : 0};
          float r = outs[rv * ROW + p0 + j * JS];
#pragma unroll
          for (int d = 0; d < dim; ++d) {
            const int sd = d == 0 ? 1 : (d == 1 ? n : n * n);
            const float* g = outs + (rv + 1 + d) * ROW + (q - qi[d] * sd) * CPT + lc;
            const float* wt = tab->jdt[d][q];
#pragma unroll
            for (int m = 0; m < n; ++m) r = fmaf(wt[m], g[m * sd * CPT], r);
          }
          const unsigned int idx = node0 + (unsigned int)j * lstride + R.out_off[o];
          const int target = R.out_cmap[o] ? __ldg(R.out_cmap[o] + idx) : (int)idx;
          if (active && target >= 0) atomicAdd(global_ptr(reinterpret_cast<float*>(R.out_acc[o]) + target), r);
        }
      }
    }
  }
}

// the flat row lists of a launch record; false when they exceed the lane kernel's limits
inline bool lane_rows(const CellLaunch& P, int dim, LaneRows* R) {
  std::memset(R, 0, sizeof(*R));
  int r = 0;
  for (int s = 0; s < P.nslots; ++s) {
    const SlotDesc& sd = P.slots[s];
    for (int c = 0; c < sd.ncomp; ++c, ++r) {
      if (r >= LANE_MAX_IN) return false;
      R->in_base[r] = static_cast<const double*>(sd.ptr);
      R->in_cmap[r] = sd.constrained_read ? sd.cmap : nullptr;
      R->in_off[r] = (unsigned int)(c * P.N);
    }
  }
  R->nin = r;
  if (r != P.nrows_in) return false;
  int o = 0, row = 0;
  for (int i = 0; i < P.nout; ++i) {
    const OutDesc& od = P.outs[i];
    for (int c = 0; c < od.ncomp; ++c, ++o) {
      if (o >= LANE_MAX_OUT) return false;
      R->out_acc[o] = static_cast<double*>(od.acc);
      R->out_cmap[o] = od.cmap;
      R->out_off[o] = (unsigned int)(c * P.N);
      R->out_row[o] = row;
      row += 1 + dim;
    }
  }
  R->nout = o;
  for (int d = 0; d < 2; ++d) {
    pg::fx::FastDiv f;
    f.init((unsigned int)P.nc[d]);
    R->div_m[d] = f.m;
    R->div_l[d] = f.l;
  }
  return row == P.nrows_out;
}

template <class PDE, int dim, int degree, int mode, int NC, int MINB>
cudaError_t launch_lanes(const CellLaunch& P, const LaneRows& R, const void* obj, cudaStream_t s) {
  using S = LaneShape<dim, degree>;
  auto kern = cell_kernel_lanes<PDE, dim, degree, mode, NC, MINB>;
  const size_t smem = lane_smem_bytes<dim, degree>(R.nv, R.ng, NC);
  constexpr int MAX_DEVICES = 64;
  static size_t attr_smem_of[MAX_DEVICES] = {};
  static int occ_of[MAX_DEVICES] = {};
  static int sms_of[MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
  size_t& attr_smem = attr_smem_of[dev];
  int& occ = occ_of[dev];
  int& sms = sms_of[dev];
  if (smem > attr_smem) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_smem = smem;
    occ = 0;
  }
  if (occ == 0) {
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, S::threads, smem);
    if (e != cudaSuccess) return e;
    if (occ < 1) occ = 1;
  }
  const long long ntiles = (P.ncells + LANE_CPT - 1) / LANE_CPT;
  long long grid = (long long)sms * occ;
  if (grid > ntiles) grid = ntiles;
  if (grid < 1) grid = 1;
  return launch_chained(kern, dim3((unsigned)grid), dim3(S::threads), smem, s, P, *reinterpret_cast<const PDE*>(obj),
                        *reinterpret_cast<const pg::CellTables<dim, degree, double>*>(P.tables_host), R);
}

template <class PDE, int dim, int degree, int MINB>
cudaError_t launch_lanes_f32(const CellLaunch& P, const LaneRows& R, const void* obj, cudaStream_t s) {
  using S = LaneShape<dim, degree>;
  auto kern = cell_kernel_lanes_f32<PDE, dim, degree, MODE_LHS, MINB>;
  const size_t smem = lane_f32_smem_bytes<dim, degree>(R.nin, P.nrows_out);
  constexpr int MAX_DEVICES = 64;
  static size_t attr_smem_of[MAX_DEVICES] = {};
  static int occ_of[MAX_DEVICES] = {};
  static int sms_of[MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
  size_t& attr_smem = attr_smem_of[dev];
  int& occ = occ_of[dev];
  int& sms = sms_of[dev];
  if (smem > attr_smem) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_smem = smem;
    occ = 0;
  }
  if (occ == 0) {
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, S::threads, smem);
    if (e != cudaSuccess) return e;
    if (occ < 1) occ = 1;
  }
  const long long ntiles = (P.ncells + LANE_CPT - 1) / LANE_CPT;
  long long grid = (long long)sms * occ;
  if (grid > ntiles) grid = ntiles;
  if (grid < 1) grid = 1;
  return launch_chained(kern, dim3((unsigned)grid), dim3(S::threads), smem, s, P, *reinterpret_cast<const PDE*>(obj),
                        *reinterpret_cast<const pg::CellTables<dim, degree, float>*>(P.tables_host), R);
}

// the FP32 lane kernel for an FP32 Q1/Q2 left-hand side, or cudaErrorNotSupported
template <class PDE, int dim, int degree>
cudaError_t launch_cell_kernel_lanes_f32_impl(const CellLaunch& P, const void* obj, cudaStream_t s) {
  constexpr int MINB = CellLaneMinBlocks<PDE, LaneShape<dim, degree>::threads>::value;
  LaneRows R;
  if (!P.tables_host || !lane_rows(P, dim, &R)) return cudaErrorNotSupported;
  if (lane_f32_smem_bytes<dim, degree>(R.nin, P.nrows_out) > 232448) return cudaErrorNotSupported;
  return launch_lanes_f32<PDE, dim, degree, MINB>(P, R, obj, s);
}

// launches the lane kernel, or returns cudaErrorNotSupported when the launch's rows exceed its
// limits (the caller then takes the thread-block kernel)
template <class PDE, int dim, int degree, int mode>
cudaError_t launch_cell_kernel_lanes_impl(const CellLaunch& P, const void* obj, cudaStream_t s) {
  LaneRows R;
  if (!P.tables_host || !lane_rows(P, dim, &R)) return cudaErrorNotSupported;
  const auto* tab = static_cast<const pg::CellTables<dim, degree, double>*>(P.tables_host);
  const unsigned int mask = (1u << R.nin) - 1u;
  R.nv = __builtin_popcount(tab->val_rows & mask);
  R.ng = __builtin_popcount(tab->fx_rows & mask);
  for (int r = 0; r < R.nin; ++r) {
    R.in_v[r] = tab->lane_vslot[r];
    R.in_g[r] = tab->lane_gslot[r];
  }
  if (lane_smem_bytes<dim, degree>(R.nv, R.ng, R.nout) > 232448) return cudaErrorNotSupported;
  constexpr unsigned int C = CellLaneComponents<PDE>::value;
  if constexpr (C & 2u)
    if (R.nout == 1) return launch_lanes<PDE, dim, degree, mode, 1, lane_min_blocks<PDE, dim, degree, 1>()>(P, R, obj, s);
  if constexpr (C & 4u)
    if (R.nout == 2) return launch_lanes<PDE, dim, degree, mode, 2, lane_min_blocks<PDE, dim, degree, 2>()>(P, R, obj, s);
  if constexpr (C & 8u)
    if (R.nout == 3) return launch_lanes<PDE, dim, degree, mode, 3, lane_min_blocks<PDE, dim, degree, 3>()>(P, R, obj, s);
  if constexpr (C & 16u)
    if (R.nout == 4) return launch_lanes<PDE, dim, degree, mode, 4, lane_min_blocks<PDE, dim, degree, 4>()>(P, R, obj, s);
  return cudaErrorNotSupported;
}

}  // namespace ppf

#pragma pop_macro("compute_lhs")
#pragma pop_macro("compute_rhs")
