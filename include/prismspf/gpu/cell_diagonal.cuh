// Diagonal of a left-hand side by unit probes: MFOperator::compute_local_field_diagonal
// (src/solvers/mf_operator.cc:147-218), which sets one cell node at a time to one (identity in every
// component, as the reference submits identity<Rank>()), evaluates the cell and keeps the integrated
// entry at the probed node.
//
// One thread per (cell, node i). A unit value at node i has derivatives only on the three node lines
// through i, and only the terms submitted on those lines enter node i's integral, so a probe
// evaluates the callback at 1 + dim (n - 1) points (Q2 3-D: 7 of 27), the probed dependency read in
// closed form (FieldContainer with CellCtx::probe) and the terms kept in registers: no nodal values
// of the probe, no barrier between probes, and bound by the callback's FP64 operations. (Evaluating
// every point for every node between two barriers, the six levels of a 32^3 Q2 elasticity hierarchy
// took 4.4 ms in FP64.)
// Other dependencies (a Newton block's current solution) are gathered once per tile.
#pragma once

#include <cuda_runtime.h>

#include <prismspf/gpu/cell_kernel.cuh>

#pragma push_macro("compute_lhs")
#undef compute_lhs

namespace ppf {

// shared memory: the tables, then the nodal values of the rows that are not probed
template <int dim, int degree, typename number>
__host__ __device__ constexpr size_t cell_diagonal_smem_bytes(int nrows_in) {
  using S = CellShape<dim, degree>;
  return pg::staged_table_room<dim, degree, number>() + sizeof(number) * (size_t)nrows_in * S::threads;
}

// NC: components of the block's one field
template <class PDE, int dim, int degree, typename number, int NC>
__global__ void __launch_bounds__(CellShape<dim, degree>::threads)
    cell_diagonal_kernel(const __grid_constant__ CellLaunch P, const __grid_constant__ PDE pde) {
  using S = CellShape<dim, degree>;
  using Tab = pg::CellTables<dim, degree, number>;
  constexpr int n = S::n, nq = S::nq, cpb = S::cpb, k = degree, TC = 1 + dim;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tab* tab = reinterpret_cast<Tab*>(smem_raw);
  number* vals = reinterpret_cast<number*>(smem_raw + pg::staged_table_room<dim, degree, number>());
  chain_wait();
  chain_release();
  {
    const unsigned int* src = reinterpret_cast<const unsigned int*>(P.tables);
    unsigned int* dst = reinterpret_cast<unsigned int*>(tab);
    for (int i = threadIdx.x; i < (int)(pg::staged_table_bytes<dim, degree, number>() / 4); i += blockDim.x) dst[i] = src[i];
  }
  unsigned int probe_rows = 0;
  {
    int row = 0;
    for (int s = 0; s < P.nslots; ++s) {
      if (P.slots[s].is_src) probe_rows |= ((1u << P.slots[s].ncomp) - 1u) << row;
      row += P.slots[s].ncomp;
    }
  }
  const int t = threadIdx.x;
  const int lc = t / nq;
  const int i = t - lc * nq;  // the probed node
  const int id[3] = {i % n, dim > 1 ? (i / n) % n : 0, dim > 2 ? i / (n * n) : 0};
  const long long ntiles = (P.ncells + cpb - 1) / cpb;
  const SimulationTimer timer = P.timer_dev ? *P.timer_dev : P.timer;

  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long cell = tile * cpb + lc;
    const bool active = cell < P.ncells;
    int c3[3] = {0, 0, 0};
    long long node = 0;
    if (active) {
      const unsigned int cl = (unsigned int)cell;
      const unsigned int q0 = P.div(cl, 0);
      c3[0] = (int)(cl - q0 * (unsigned int)P.nc[0]);
      if (dim == 2) c3[1] = (int)q0;
      if (dim > 2) {
        const unsigned int q1 = P.div(q0, 1);
        c3[1] = (int)(q0 - q1 * (unsigned int)P.nc[1]);
        c3[2] = (int)q1;
      }
      node = ((long long)(k * c3[2] + id[2]) * P.nn[1] + (k * c3[1] + id[1])) * P.nn[0] + (k * c3[0] + id[0]);
    }
    __syncthreads();  // tables staged; the previous tile has read vals
    {
      int row = 0;
      for (int s = 0; s < P.nslots; ++s) {
        const SlotDesc& sd = P.slots[s];
        const number* ptr = global_ptr(static_cast<const number*>(sd.ptr));
        if (!sd.is_src)
          for (int c = 0; c < sd.ncomp; ++c) vals[(row + c) * S::threads + t] = active ? ptr[node + c * P.N] : number(0);
        row += sd.ncomp;
      }
    }
    __syncthreads();
    if (!active) continue;

    number r[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) r[c] = number(0);
#pragma unroll 1
    for (int p = 0; p < 1 + dim * (n - 1); ++p) {
      // point p: the node itself, then the others of its line along each direction
      const int pd = p == 0 ? -1 : (p - 1) / (n - 1);
      int j = p == 0 ? 0 : (p - 1) % (n - 1);
      const int own = pd <= 0 ? id[0] : (pd == 1 ? id[1] : id[2]);
      if (j >= own) ++j;
      const int sd = pd <= 0 ? 1 : (pd == 1 ? n : n * n);
      pg::CellCtx<dim, degree, number> ctx;
      ctx.tab = tab;
      ctx.vals = vals;
      ctx.outs = nullptr;
      ctx.stride = S::threads;
      ctx.lc = lc;
      ctx.q = p == 0 ? i : i + (j - own) * sd;
      ctx.cell[0] = c3[0];
      ctx.cell[1] = c3[1];
      ctx.cell[2] = c3[2];
      ctx.err = P.err;
      ctx.submitted = 0;
      ctx.probe = i;
      ctx.probe_rows = probe_rows;
      ctx.nterm = NC;
#pragma unroll
      for (int e = 0; e < NC * TC; ++e) ctx.term[e] = number(0);
      FieldContainer<dim, degree, number> fc(ctx);
      pde.compute_lhs(fc, timer, P.block_id);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (p == 0) r[c] += ctx.term[c * TC] * tab->jxw[i];
#pragma unroll
        for (int d = 0; d < dim; ++d)
          if (p == 0 || d == pd) r[c] = fma(tab->jdt[d][i][p == 0 ? id[d] : j], ctx.term[c * TC + 1 + d], r[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const long long idx = node + c * P.N;
      const int target = P.outs[0].cmap ? P.outs[0].cmap[idx] : (int)idx;
      if (target >= 0) atomicAdd(static_cast<number*>(P.outs[0].acc) + target, r[c]);
    }
  }
}

template <class PDE, int dim, int degree, typename number, int NC>
cudaError_t launch_cell_diagonal_nc(const CellLaunch& P, const void* obj, cudaStream_t s) {
  using S = CellShape<dim, degree>;
  auto kern = cell_diagonal_kernel<PDE, dim, degree, number, NC>;
  const size_t smem = cell_diagonal_smem_bytes<dim, degree, number>(P.nrows_in);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const long long ntiles = (P.ncells + S::cpb - 1) / S::cpb;
  const long long grid = std::max<long long>(1, std::min<long long>(ntiles, (long long)sms * 8));
  return launch_chained(kern, dim3((unsigned)grid), dim3(S::threads), smem, s, P, *reinterpret_cast<const PDE*>(obj));
}

// the diagonal of a block with one field (scalar or vector)
template <class PDE, int dim, int degree, typename number>
cudaError_t launch_cell_diagonal(const CellLaunch& L, const void* obj, cudaStream_t s) {
  const CellLaunch P = with_divisors(L);
  if (P.nout != 1) return cudaErrorNotSupported;
  if (P.outs[0].ncomp == 1) return launch_cell_diagonal_nc<PDE, dim, degree, number, 1>(P, obj, s);
  if (P.outs[0].ncomp == dim) return launch_cell_diagonal_nc<PDE, dim, degree, number, dim>(P, obj, s);
  return cudaErrorNotSupported;
}

}  // namespace ppf

#pragma pop_macro("compute_lhs")
