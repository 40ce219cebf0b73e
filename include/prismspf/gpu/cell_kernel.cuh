// Matrix-free cell kernel: gather -> evaluate -> user callback per quadrature point ->
// integrate -> condensed scatter, for one solve block on a uniform hyper-rectangle mesh.
//
// Restates the per-cell work of MFOperator::compute_local_operator
// (src/solvers/mf_operator.cc:34-80) with FieldContainer::reinit_and_eval /
// integrate_and_distribute (include/prismspf/core/field_container.h:794-882) as one GPU
// kernel:
//   * DoF vectors are stored in lattice order (x fastest) with periodic images kept, so the
//     nodes of cell (cx,cy,cz) are a dense (k+1)^dim box of the lattice: the gather needs no
//     index map. Constraint maps are int32 arrays over the same index space:
//     cmap[i] = i (free), = master (periodic image), = -1-j (Dirichlet row j).
//   * one thread per (cell, quadrature point); cells_per_block cells per thread block; the
//     block walks cell tiles in a grid-stride loop so the per-launch tables are staged into
//     shared memory once per resident block;
//   * with Gauss-Lobatto collocation, values at quadrature points are the nodal values and
//     gradients are 1-D contractions (FieldContainer::deriv);
//   * integration is the transposed contraction over the pre-weighted submitted terms;
//   * distribute_local_to_global: rows constrained to a master add into the master,
//     Dirichlet rows are dropped; contributions of neighbouring cells meet through
//     atomicAdd into a zeroed accumulator (the finalize kernels apply invM and constraints).
//   * MODE_DIAG is the diagonal probe's own kernel (prismspf/gpu/cell_diagonal.cuh).
//   * FP64 Q1/Q2 launches contract exactly in 64-bit integers (prismspf/gpu/fixed_point.cuh):
//     rows read as gradients get a fixed-point copy with a per-cell block exponent, the
//     derivatives are integer line sums rounded once, and with fx_int the submitted gradient
//     terms are integrated the same way (else in FP64 with jdt); the launch record selects the
//     split, which the engine times per operator.
// `number` is the arithmetic type (double for the drop-in, float for mixed-precision
// multigrid smoothing).
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include <prismspf/core/field_container.h>

// prismspf/core/pde_operator_base.h re-declares the callback names as macros for user
// classes; the kernel calls them by their plain names.
#pragma push_macro("compute_rhs")
#pragma push_macro("compute_lhs")
#undef compute_rhs
#undef compute_lhs

// minimum resident blocks per SM the cell kernels are compiled for (register budget)
#ifndef PPF_CELL_MIN_BLOCKS
#define PPF_CELL_MIN_BLOCKS 1
#endif

namespace ppf {

// An operator may ask for a register budget through `static constexpr int cell_min_blocks`
// (resident blocks per SM); otherwise the kernels are compiled for PPF_CELL_MIN_BLOCKS.
template <class PDE, class = void>
struct CellMinBlocks {
  static constexpr int value = PPF_CELL_MIN_BLOCKS;
};
template <class PDE>
struct CellMinBlocks<PDE, std::void_t<decltype(PDE::cell_min_blocks)>> {
  static constexpr int value = PDE::cell_min_blocks;
};

using prismspf::FieldContainer;
using prismspf::SimulationTimer;
namespace pg = prismspf::gpu;

// Programmatic dependent launch (launch_chained): a kernel launched
// this way may start while the kernel before it on its stream still runs. chain_wait returns
// when that kernel has completed and its writes are visible; nothing another kernel writes may be
// touched before it. chain_release, called after it, lets the next kernel of the chain start (it waits
// in its own chain_wait; released before the wait, launches pile up behind one another: 7.4 instead of
// 8.3 us an increment of 48^2 Q1 cells this way round); every kernel of a chain waits, so completion is transitive along the stream. Both
// do nothing in a kernel that was launched plainly.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A pointer out of a launch record, told to be one to global memory: its plain loads may then move
// across shared-memory stores, as __ldg's do.
template <class T>
__device__ __forceinline__ T* global_ptr(T* p) {
  __builtin_assume(__isGlobal(p));
  return p;
}

// launches a kernel that begins with chain_wait as a dependent of the one before it on the stream
template <class... K, class... A>
cudaError_t launch_chained(void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<K>(args)...);
}

enum CellMode { MODE_RHS = 0, MODE_LHS = 1, MODE_DIAG = 2 };

struct SlotDesc {
  const void* ptr;    // component-major vector (ncomp * N) of the kernel's number type
  const int* cmap;    // constraint map, used when constrained_read
  int ncomp;
  int constrained_read;  // homogeneous constrained read (FEEvaluation::read_dof_values)
  int is_src;            // the SRC dependency of a block field (probed in MODE_DIAG)
  int out_index;         // block output the SRC slot belongs to (MODE_DIAG)
};

struct OutDesc {
  void* acc;         // accumulator (ncomp * N), zeroed before the launch
  const int* cmap;   // destination constraint map (condensation)
  int ncomp;
};

struct CellLaunch {
  int nc[3];
  int nn[3];
  long long N;       // lattice nodes per component
  long long ncells;
  int nslots;
  SlotDesc slots[pg::MAX_SLOTS];
  int nout;
  OutDesc outs[pg::MAX_OUTS];
  int nrows_in;      // sum of slot components
  int nrows_out;     // sum over outputs of ncomp * (1 + dim)
  const void* tables;  // device copy of CellTables<dim,degree,number>
  SimulationTimer timer;
  const SimulationTimer* timer_dev;  // when set (graph replays), the timer is read from here
  unsigned int block_id;
  int* err;
  // with integer contractions on in the tables: fx_deriv takes the derivatives in fixed point
  // (else FP64 from the nodal values), fx_int integrates in fixed point (else FP64 with jdt)
  int fx_deriv;
  int fx_int;
  // the lane kernel (prismspf/gpu/cell_kernel_lanes.cuh): all-integer contractions of an FP64
  // Q1/Q2 operator, when the tables allow it (fx_lanes); it takes the host copy of `tables`
  // (tables_host) as a kernel parameter
  int fx_lanes;
  const void* tables_host;
  // cell index -> coordinates: multiply-high divisors of nc[0] and nc[1] (filled by the launchers: a
  // thread that makes its own spends two 64-bit divisions before its first load)
  unsigned int div_m[2], div_l[2];
  int cells_per_tile;  // cells a block takes at a time (filled by the launchers)
  __device__ __forceinline__ unsigned int div(unsigned int v, int d) const {
    return (__umulhi(v, div_m[d]) + v) >> div_l[d];
  }
};

inline CellLaunch with_divisors(const CellLaunch& L) {
  CellLaunch P = L;
  for (int d = 0; d < 2; ++d) {
    pg::fx::FastDiv f;
    f.init((unsigned int)P.nc[d]);
    P.div_m[d] = f.m;
    P.div_l[d] = f.l;
  }
  return P;
}

template <int dim, int degree>
struct CellShape {
  static constexpr int n = degree + 1;
  static constexpr int nq = pg::ipow(n, dim);
  static constexpr int cpb = (256 / nq) > 0 ? (256 / nq) : 1;  // cells per thread block
  static constexpr int threads = cpb * nq;
};

// Cells a thread block takes at a time: a full block's, or on a mesh that gives an SM fewer than four
// blocks' cells an even share of them, so that small meshes use every SM and none waits for another's
// extra tile (the FP64 work of a point holds its SM's pipe; 64^2 Q1 cells are 64 full blocks on 152 SMs)
template <int dim, int degree>
inline int cells_per_tile(long long ncells, int sms) {
  using S = CellShape<dim, degree>;
  const long long share = (ncells + sms - 1) / sms;
  if (share >= 4 * S::cpb) return S::cpb;
  const long long tiles = (share + S::cpb - 1) / S::cpb;
  const long long cells = (share + tiles - 1) / tiles, least = (32 + S::nq - 1) / S::nq;
  return (int)(cells < least ? (least < S::cpb ? least : S::cpb) : cells);
}

// FP64 Q1/Q2 kernels contract in 64-bit fixed point (prismspf/gpu/fixed_point.cuh) when the
// launch's tables enable it; their shared memory then also holds the fixed-point nodal values
// and the per-cell block exponents of the value rows and of the output components.
template <int dim, int degree, typename number>
__host__ __device__ constexpr bool cell_fx_capable() {
  return std::is_same<number, double>::value && degree <= 2;
}

// Shape of the warp-resident alternative kernel (prismspf/gpu/cell_kernel_warp.cuh): whole
// cells per warp, 8 warps per thread block.
template <int dim, int degree>
struct WarpShape {
  static constexpr int n = degree + 1;
  static constexpr int nq = pg::ipow(n, dim);
  static constexpr int cpw = 32 / nq;       // cells per warp
  static constexpr int lanes = cpw * nq;    // lanes holding a (cell, quadrature point)
  static constexpr int warps = 8;           // warps per thread block
  static constexpr int threads = 32 * warps;
};

// bytes of one warp's region: nodal values, their fixed-point copies and the submitted terms
// (32 lanes each), then the block exponents of the value rows and output components per cell
template <int dim, int degree>
__host__ __device__ constexpr size_t warp_region_bytes(int nrows_in, int nrows_out) {
  using W = WarpShape<dim, degree>;
  return (8 * 32 * (size_t)(2 * nrows_in + nrows_out) + 4 * (size_t)W::cpw * (size_t)(nrows_in + nrows_out) + 15) /
         16 * 16;
}

template <int dim, int degree>
__host__ __device__ constexpr size_t cell_warp_smem_bytes(int nrows_in, int nrows_out) {
  using W = WarpShape<dim, degree>;
  return pg::staged_table_room<dim, degree, double>() +
         W::warps * warp_region_bytes<dim, degree>(nrows_in, nrows_out);
}

// Dynamic shared memory of a launch: enough for cell_kernel and, for FP64 Q1/Q2, for the
// warp-resident kernel as well (the launcher picks either).
template <int dim, int degree, typename number>
__host__ __device__ inline size_t cell_smem_bytes(int nrows_in, int nrows_out) {
  using S = CellShape<dim, degree>;
  const size_t tab = pg::staged_table_room<dim, degree, number>();
  size_t b = tab + sizeof(number) * (size_t)(nrows_in + nrows_out) * S::threads + 16;
  if (cell_fx_capable<dim, degree, number>()) {
    b += sizeof(long long) * (size_t)nrows_in * S::threads + sizeof(int) * (size_t)(nrows_in + nrows_out) * S::cpb;
    const size_t w = cell_warp_smem_bytes<dim, degree>(nrows_in, nrows_out);
    if (w > b) b = w;
  }
  return b;
}

template <int dim, int degree, typename number>
__device__ __forceinline__ number integrate_row(const pg::CellTables<dim, degree, number>* tab, const number* outs,
                                                int rv, bool has_v, bool has_g, int t, int lc, int q, int qa, int qb,
                                                int qc) {
  using S = CellShape<dim, degree>;
  constexpr int n = S::n, nq = S::nq;
  number r = has_v ? outs[rv * S::threads + t] : number(0);
  if (has_g) {
#pragma unroll
    for (int d = 0; d < dim; ++d) {
      const int sd = d == 0 ? 1 : (d == 1 ? n : n * n);
      const int id = d == 0 ? qa : (d == 1 ? qb : qc);
      const number* g = outs + (rv + 1 + d) * S::threads + lc * nq + (q - id * sd);
      const number* w = tab->jdt[d][q];
#pragma unroll
      for (int j = 0; j < n; ++j) r = fma(w[j], g[j * sd], r);
    }
  }
  return r;
}

// integrate_row with the submitted gradient terms already converted in place to fixed point
// (block exponent E of the output component): per direction the exact integer line sum with
// the weights iint, times the other directions' weights (a shift), rounded once with the
// scale c_d = JxW / (h_d w_int...) of the integer weights.
template <int dim, int degree>
__device__ __forceinline__ double integrate_row_fx(const pg::CellTables<dim, degree, double>* tab, const double* outs,
                                                   int rv, bool has_v, bool has_g, int t, int lc, int q, int qa, int qb,
                                                   int qc, int E) {
  using S = CellShape<dim, degree>;
  constexpr int n = S::n, nq = S::nq;
  namespace fx = pg::fx;
  double r = has_v ? outs[rv * S::threads + t] : 0.0;
  if (has_g) {
    if (E == fx::EXP_NONFINITE) return fx::quiet_nan();
    const long long* gx = reinterpret_cast<const long long*>(outs);
    const int lsb = E - 1023 - fx::TOP_TERMS;
    long long sum = 0;
    double rg = 0.0;
#pragma unroll
    for (int d = 0; d < dim; ++d) {
      const int sd = d == 0 ? 1 : (d == 1 ? n : n * n);
      const int id = d == 0 ? qa : (d == 1 ? qb : qc);
      const long long* g = gx + (rv + 1 + d) * S::threads + lc * nq + (q - id * sd);
      long long p = fx::line_integral<n>(id, g[0], g[sd], n > 2 ? g[2 * sd] : 0ll);
      p = (long long)((unsigned long long)p << tab->wo_sh[d][q]);
      if (tab->fx_cubic) sum += p;
      else rg += fx::to_double(p, lsb + tab->ik[d], tab->isig[d]);
    }
    if (tab->fx_cubic) rg = fx::to_double(sum, lsb + tab->ik[0], tab->isig[0]);
    r += rg;
  }
  return r;
}

// FXINT: compile the fixed-point integration path (modes 2 and 3); the mode-1 instantiation
// leaves it out, which keeps its register budget for the derivative path
template <class PDE, int dim, int degree, int MODE, typename number, bool FXINT = false>
__global__ void __launch_bounds__(CellShape<dim, degree>::threads, CellMinBlocks<PDE>::value)
    cell_kernel(const __grid_constant__ CellLaunch P, const __grid_constant__ PDE pde) {
  using S = CellShape<dim, degree>;
  using Tab = pg::CellTables<dim, degree, number>;
  constexpr int n = S::n, nq = S::nq, cpb = S::cpb, k = degree;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tab* tab = reinterpret_cast<Tab*>(smem_raw);
  number* vals = reinterpret_cast<number*>(smem_raw + pg::staged_table_room<dim, degree, number>());
  number* outs = vals + P.nrows_in * S::threads;
  __shared__ int sflags;
  // integer contractions: enabled by the launch's tables, and only with the shared memory for them
  constexpr bool FXC = cell_fx_capable<dim, degree, number>();
  long long* vals_fx = reinterpret_cast<long long*>(outs + P.nrows_out * S::threads);
  int* ex_in = reinterpret_cast<int*>(vals_fx + P.nrows_in * S::threads);
  int* ex_out = ex_in + P.nrows_in * cpb;
  bool fx_on = false, fx_int = false;  // fx_on: fixed-point derivatives
  unsigned int tab_fx_rows = 0;
  chain_wait();  // (the allocation-free step's tables come from the kernel before)
  chain_release();
  if constexpr (FXC) {
    unsigned int dyn;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    const Tab* gtab = reinterpret_cast<const Tab*>(P.tables);
    const bool fx_ok =
        gtab->fx != 0 && dyn >= (unsigned int)cell_smem_bytes<dim, degree, number>(P.nrows_in, P.nrows_out);
    tab_fx_rows = gtab->fx_rows;
    fx_on = fx_ok && P.fx_deriv != 0;
    if constexpr (FXINT) fx_int = fx_ok && P.fx_int != 0;
  }

  // stage the tables once per resident block
  {
    const int nwords = (int)(pg::staged_table_bytes<dim, degree, number>() / 4);
    const unsigned int* src = reinterpret_cast<const unsigned int*>(P.tables);
    unsigned int* dst = reinterpret_cast<unsigned int*>(tab);
    for (int i = threadIdx.x; i < nwords; i += blockDim.x) dst[i] = src[i];
  }

  const int t = threadIdx.x;
  const int lc = t / nq;
  const int q = t - lc * nq;
  const int qa = q % n;
  const int qb = dim > 1 ? (q / n) % n : 0;
  const int qc = dim > 2 ? q / (n * n) : 0;
  const int cpt = P.cells_per_tile;
  const long long ntiles = (P.ncells + cpt - 1) / cpt;

  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long cell = tile * cpt + lc;
    const bool active = cell < P.ncells;
    int cx = 0, cy = 0, cz = 0;
    long long node = 0;
    if (active) {
      const unsigned int cl = (unsigned int)cell;
      // (multiply-high division: cell indices stay below 2^31, DoF indices being int)
      const unsigned int q0 = P.div(cl, 0);
      cx = (int)(cl - q0 * (unsigned int)P.nc[0]);
      if (dim == 2) cy = (int)q0;
      if (dim > 2) {
        const unsigned int q1 = P.div(q0, 1);
        cy = (int)(q0 - q1 * (unsigned int)P.nc[1]);
        cz = (int)q1;
      }
      node = ((long long)(k * cz + qc) * P.nn[1] + (k * cy + qb)) * P.nn[0] + (k * cx + qa);
    }
    if constexpr (FXC) {
      // the value-row exponents were last read by the previous tile's callbacks; rows without a
      // fixed-point copy keep -1
      if (fx_on)
        for (int i = t; i < P.nrows_in * cpb; i += blockDim.x) ex_in[i] = ((tab_fx_rows >> (i / cpb)) & 1u) ? 0 : -1;
    }
    __syncthreads();  // tables staged; previous tile finished with vals/outs/sflags

    // gather (read_dof_values_plain, or read_dof_values for constrained src)
    {
      int row = 0;
#pragma unroll
      for (int s = 0; s < pg::MAX_SLOTS; ++s) {
        if (s < P.nslots) {
          const SlotDesc& sd = P.slots[s];
          {
            const number* ptr = global_ptr(static_cast<const number*>(sd.ptr));
            for (int c = 0; c < sd.ncomp; ++c) {
              number v = number(0);
              if (active) {
                const long long idx = node + c * P.N;
                if (sd.constrained_read) {
                  // the value load issues with the map load: almost every entry is free, so
                  // the dependent second load is only paid on constrained entries
                  const int m = __ldg(sd.cmap + idx);
                  const number own = ptr[idx];
                  v = m == (int)idx ? own : (m >= 0 ? ptr[m] : number(0));
                } else {
                  v = ptr[idx];
                }
              }
              vals[(row + c) * S::threads + t] = v;
              if constexpr (FXC) {
                if (fx_on && ((tab_fx_rows >> (row + c)) & 1u)) atomicMax(&ex_in[(row + c) * cpb + lc], pg::fx::exponent(v));
              }
            }
          }
          row += sd.ncomp;
        }
      }
    }

    {
      if constexpr (FXC) {
        if (fx_on) {
          __syncthreads();  // block exponents of the value rows complete
          for (int r = 0; r < P.nrows_in; ++r) {
            const int E = ex_in[r * cpb + lc];
            if (E >= 0 && E != pg::fx::EXP_NONFINITE)
              vals_fx[r * S::threads + t] = pg::fx::to_fixed(vals[r * S::threads + t], E, pg::fx::TOP_VALUES);
          }
        }
        if (fx_int)
          for (int i = t; i < P.nrows_out * cpb; i += blockDim.x) ex_out[i] = 0;
      }
      if (t == 0) sflags = 0;
      for (int r = 0; r < P.nrows_out; ++r) outs[r * S::threads + t] = number(0);
      __syncthreads();

      pg::CellCtx<dim, degree, number> ctx;
      ctx.tab = tab;
      ctx.vals = vals;
      ctx.outs = outs;
      ctx.stride = S::threads;
      ctx.lc = lc;
      ctx.q = q;
      ctx.cell[0] = cx;
      ctx.cell[1] = cy;
      ctx.cell[2] = cz;
      ctx.err = P.err;
      ctx.submitted = 0;
      if constexpr (FXC) {
        if (fx_on) {
          ctx.vals_fx = vals_fx;
          ctx.ex_in = ex_in;
          ctx.cpb = cpb;
        }
      }
      if (active) {
        FieldContainer<dim, degree, number> fc(ctx);
        const SimulationTimer timer = P.timer_dev ? *P.timer_dev : P.timer;
        if constexpr (MODE == MODE_LHS) pde.compute_lhs(fc, timer, P.block_id);
        else pde.compute_rhs(fc, timer, P.block_id);
        if (ctx.submitted) atomicOr(&sflags, ctx.submitted);
      }
      __syncthreads();
      const int flags = sflags;

      if constexpr (FXC) {
        if (fx_int) {
          // submitted gradient terms -> fixed point in place, one block exponent per cell and
          // output component (rows of component c of output o: value, then dim gradient rows)
          for (int o = 0; o < P.nout; ++o)
            if (flags & (2 << (2 * o)))
              for (int c = 0; c < P.outs[o].ncomp; ++c) {
                const int rv = tab->out_row0[o] + c * (1 + dim);
                int e = 0;
#pragma unroll
                for (int d = 0; d < dim; ++d) e = max(e, pg::fx::exponent(outs[(rv + 1 + d) * S::threads + t]));
                atomicMax(&ex_out[rv * cpb + lc], e);
              }
          __syncthreads();
          for (int o = 0; o < P.nout; ++o)
            if (flags & (2 << (2 * o)))
              for (int c = 0; c < P.outs[o].ncomp; ++c) {
                const int rv = tab->out_row0[o] + c * (1 + dim);
                const int E = ex_out[rv * cpb + lc];
#pragma unroll
                for (int d = 0; d < dim; ++d) {
                  double* gp = outs + (rv + 1 + d) * S::threads + t;
                  const long long x = E == pg::fx::EXP_NONFINITE ? 0 : pg::fx::to_fixed(*gp, E, pg::fx::TOP_TERMS);
                  *reinterpret_cast<long long*>(gp) = x;
                }
              }
          __syncthreads();
        }
      }

      if (active) {
#pragma unroll
        for (int o = 0; o < pg::MAX_OUTS; ++o) {
          if (o < P.nout) {
            const OutDesc& od = P.outs[o];
            const bool has_v = flags & (1 << (2 * o));
            const bool has_g = flags & (2 << (2 * o));
            const int row0 = tab->out_row0[o];
            for (int c = 0; c < od.ncomp; ++c) {
              number r;
              if constexpr (FXC) {
                const int rv = row0 + c * (1 + dim);
                if (fx_int)
                  r = integrate_row_fx<dim, degree>(tab, outs, rv, has_v, has_g, t, lc, q, qa, qb, qc,
                                                    ex_out[rv * cpb + lc]);
                else
                  r = integrate_row<dim, degree, number>(tab, outs, rv, has_v, has_g, t, lc, q, qa, qb, qc);
              } else {
                r = integrate_row<dim, degree, number>(tab, outs, row0 + c * (1 + dim), has_v, has_g, t, lc, q, qa,
                                                       qb, qc);
              }
              if (has_v || has_g) {
                const long long idx = node + c * P.N;
                const int target = od.cmap ? od.cmap[idx] : (int)idx;
                if (target >= 0) atomicAdd(static_cast<number*>(od.acc) + target, r);
              }
            }
          }
        }
      }
    }
  }
}

}  // namespace ppf

#pragma pop_macro("compute_lhs")
#pragma pop_macro("compute_rhs")
