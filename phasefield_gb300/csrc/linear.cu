// Linear solves of a single-field Linear block: CG preconditioned by nothing, by Chebyshev on
// the fine operator, or by a geometric-multigrid V-cycle (LinearSolver + MGContext,
// include/prismspf/solvers/linear_solver.h:47-553).
//
//   * operator: the LHS cell kernel (MODE_LHS) on each level, src read with the level's
//     homogeneous constraints, output zero on constrained rows, scaled by invM^1/2 unless the
//     tolerance type is AbsoluteResidual (MFOperator::compute_operator, mf_operator.cc:17-32);
//   * diagonal: unit probes (prismspf/gpu/cell_diagonal.cuh), same scaling, zero entries set to one, inverted
//     (MFOperator::compute_diagonal + eval_matrix_diagonal, mf_operator.cc:82-255);
//   * Chebyshev smoother of the first kind on [lambda_max/range, lambda_max] with
//     lambda_max = 1.2 x the largest eigenvalue of the Lanczos matrix of eig_cg_iterations
//     CG steps (Jacobi-preconditioned) on the pattern (i mod 11) minus its mean;
//   * transfers: the Gauss-Lobatto nodal interpolation from a level to the next finer one
//     (prolongation; in one pass by closed forms for degrees 1 and 2, axis by axis for 3 and 4) and
//     its transpose (restriction); images of periodic nodes are condensed onto their masters and
//     constrained rows zeroed;
//   * V-cycle: pre-smooth from zero (vmult), residual, restrict, recurse, prolongate-add,
//     post-smooth (step); the coarsest level applies the smoother (MGCoarseGridApplySmoother);
//   * mixed precision: all levels but the coarsest in FP32 (smoother, level operators,
//     transfers); the coarsest level, the outer CG and its residuals and inner products FP64;
//   * solve: LinearSolver::solve_impl (linear_solver.h:305-345): rhs = S b_rhs - S A g with
//     g the Dirichlet values (plain read), CG from the previous homogeneous solution,
//     x = x_hom + g, constraints distributed.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <cstdlib>
#include <string>
#include <vector>

#include "handle.h"

namespace ppf {

// ------------------------------------------------------------------------------------------
// vector kernels
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void axpby_kernel(long long n, double a, const T* __restrict__ x, double b, T* __restrict__ y) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = T(a * double(x[i]) + b * double(y[i]));
}

template <typename Tin, typename Tout>
__global__ void convert_kernel(long long n, const Tin* __restrict__ x, Tout* __restrict__ y) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = Tout(x[i]);
}

// Sum of one double per thread over the grid: per-block tree sums, summed in block order by the
// block that finishes last (the same sum whichever that is), so a reduction is part of the launch
// that makes its terms. True in the last block's thread 0, with the sum in *total.
__device__ bool grid_sum(double v, double* partial, unsigned int* counter, double* total) {
  __shared__ double s[256];
  __shared__ bool last;
  const unsigned nb = gridDim.x * gridDim.y, b = blockIdx.y * gridDim.x + blockIdx.x;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[b] = s[0];
    __threadfence();
    last = atomicAdd(counter, 1u) == nb - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double acc = 0.0;
  for (unsigned i = threadIdx.x; i < nb; i += blockDim.x) acc += __ldcg(partial + i);
  __syncthreads();
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x != 0) return false;
  *total = s[0];
  *counter = 0;
  return true;
}

// out = x.y in FP64
template <typename T>
__global__ void __launch_bounds__(256) dot_kernel(long long n, const T* x, const T* y, double* partial,
                                                  unsigned int* counter, double* out) {
  chain_wait();
  chain_release();
  double acc = 0.0, total;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    acc += double(x[i]) * double(y[i]);
  if (grid_sum(acc, partial, counter, &total)) *out = total;
}

// The kernels below read a product's accumulator and clear the level's other one (`clear`) for the
// next product. The scatter adds nothing to constrained rows (images are condensed onto their
// masters, Dirichlet rows dropped), so a product's constrained rows are zero without a look-up in the
// constraint map. (Clearing the same accumulator in place needs no second one, but storing to the rows
// the cells' atomic adds have just left took five times as long: 73 instead of 13 us on 48^3 Q2
// vectors.)

// dst = scale (.) acc (per node scale, component blocks); with `out` also out = w.dst
template <typename T>
__global__ void __launch_bounds__(256) level_finalize_kernel(T* dst, const T* acc, T* clear, const T* __restrict__ scale,
                                                             long long N, const T* w,
                                                             double* partial, unsigned int* counter, double* out) {
  chain_wait();
  chain_release();
  const long long base = blockIdx.y * N;
  double sum = 0.0, total;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const long long gi = base + i;
    const T v = scale ? acc[gi] * scale[i] : acc[gi];
    if (clear) clear[gi] = T(0);
    dst[gi] = v;
    if (out) sum += double(w[gi]) * double(v);
  }
  if (out && grid_sum(sum, partial, counter, &total)) *out = total;
}

// inverse diagonal: d = scale (.) acc, zero entries -> 1, inverted
template <typename T>
__global__ void inv_diag_kernel(T* inv, const T* acc, T* clear, const T* __restrict__ scale, long long N) {
  chain_wait();
  chain_release();
  const long long base = blockIdx.y * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const long long gi = base + i;
    T d = scale ? acc[gi] * scale[i] : acc[gi];
    clear[gi] = T(0);
    if (d == T(0)) d = T(1);
    inv[gi] = T(1) / d;
  }
}

// A transfer between two levels
struct Transfer {
  int nout[3], nin[3];   // lattice extents of the output and the input level
  int periodic[3];
  int dim;
  long long Nout, Nin;
  pg::fx::FastDiv fd[2];  // multiply-high divisors of nout[0] and nout[1]
  // the lattice indices of an output node
  __device__ __forceinline__ void indices(unsigned node, int* i) const {
    const unsigned r = fd[0].div(node), z = fd[1].div(r);
    i[0] = (int)(node - r * (unsigned)nout[0]);
    i[1] = (int)(r - z * (unsigned)nout[1]);
    i[2] = (int)z;
  }
};

// Degrees 1 and 2, whose nodes nest, in closed form. A fine row of an axis is its coarse node, or
// Q1 {1/2, 1/2}, Q2 {3/8, 3/4, -1/8} and its mirror image on the coarse cell's nodes; a coarse row
// of the transpose Q1 {1/2, 1, 1/2}, Q2 {3/4, 1, 3/4} at a cell's middle node and
// {-1/8, 0, 3/8, 1, 3/8, 0, -1/8} at a vertex, on the fine nodes around it.
struct FineTaps {
  int c0, n;  // first coarse node and number of taps
  float w[3];
};
template <int degree>
__device__ __forceinline__ FineTaps fine_taps(int i) {
  FineTaps t;
  t.n = 1;
  t.w[0] = 1.f;
  t.w[1] = t.w[2] = 0.f;
  t.c0 = i >> 1;
  if constexpr (degree == 1) {
    if (i & 1) {
      t.n = 2;
      t.w[0] = t.w[1] = 0.5f;
    }
  } else {
    if (i & 1) {
      const bool first = (i & 3) == 1;
      t.n = 3;
      t.c0 = (i >> 2) * 2;
      t.w[0] = first ? 0.375f : -0.125f;
      t.w[1] = 0.75f;
      t.w[2] = first ? -0.125f : 0.375f;
    }
  }
  return t;
}
// weight of fine node 2 i + o in coarse row i (o from -3 to 3)
template <int degree>
__device__ __forceinline__ float coarse_weight(int i, int o) {
  const int a = o < 0 ? -o : o;
  if (a == 0) return 1.f;
  if (degree == 1) return a == 1 ? 0.5f : 0.f;
  if (i & 1) return a == 1 ? 0.75f : 0.f;
  return a == 1 ? 0.375f : (a == 3 ? -0.125f : 0.f);
}

// the row (i0, i1, i2) of the prolongation applied to e
template <typename T, typename Tc, int degree>
__device__ __forceinline__ T prolong_row(const Transfer& A, const Tc* e, int i0, int i1, int i2) {
  const FineTaps t0 = fine_taps<degree>(i0), t1 = fine_taps<degree>(i1), t2 = fine_taps<degree>(i2);
  T s2 = T(0);
  for (int k2 = 0; k2 < t2.n; ++k2) {
    T s1 = T(0);
    for (int k1 = 0; k1 < t1.n; ++k1) {
      const Tc* row = e + ((long long)(t2.c0 + k2) * A.nin[1] + (t1.c0 + k1)) * A.nin[0] + t0.c0;
      T s0 = T(t0.w[0]) * T(row[0]);
      if (t0.n > 1) s0 += T(t0.w[1]) * T(row[1]);
      if (t0.n > 2) s0 += T(t0.w[2]) * T(row[2]);
      s1 += T(k1 == 0 ? t1.w[0] : (k1 == 1 ? t1.w[1] : t1.w[2])) * s0;
    }
    s2 += T(k2 == 0 ? t2.w[0] : (k2 == 1 ? t2.w[1] : t2.w[2])) * s1;
  }
  return s2;
}

// the coarse row (i0, i1, i2) of the restriction applied to r
template <typename T, int degree>
__device__ __forceinline__ T restrict_row(const Transfer& A, const T* r, int i0, int i1, int i2) {
  constexpr int H = degree == 1 ? 1 : 3;
  const int h0 = degree == 2 && (i0 & 1) ? 1 : H, h1 = degree == 2 && (i1 & 1) ? 1 : H;
  const int h2 = A.dim < 3 ? 0 : (degree == 2 && (i2 & 1) ? 1 : H);
  T s2 = T(0);
  for (int o2 = -h2; o2 <= h2; ++o2) {
    const T w2 = T(coarse_weight<degree>(i2, o2));
    const int f2 = 2 * i2 + o2;
    if (w2 == T(0) || f2 < 0 || f2 >= A.nin[2]) continue;
    T s1 = T(0);
    for (int o1 = -h1; o1 <= h1; ++o1) {
      const T w1 = T(coarse_weight<degree>(i1, o1));
      const int f1 = 2 * i1 + o1;
      if (w1 == T(0) || f1 < 0 || f1 >= A.nin[1]) continue;
      const T* row = r + ((long long)f2 * A.nin[1] + f1) * A.nin[0] + 2 * i0;
      T s0 = row[0];
      const T e1 = T(coarse_weight<degree>(i0, 1));
      if (i0 > 0) s0 += e1 * row[-1];
      if (2 * i0 + 1 < A.nin[0]) s0 += e1 * row[1];
      if (h0 == 3) {
        const T e3 = T(coarse_weight<degree>(i0, 3));
        if (i0 > 1) s0 += e3 * row[-3];
        if (2 * i0 + 3 < A.nin[0]) s0 += e3 * row[3];
      }
      s1 += w1 * s0;
    }
    s2 += w2 * s1;
  }
  return s2;
}

// Degrees 3 and 4 go axis by axis. A coarse row of degree 4 has up to 17 entries an axis, a fine one 5:
// all axes in one pass are 4,913 and 125 multiplications a row where three passes take 51 and 15.
// (V-cycle-preconditioned CG on 8^3 cells, three levels: degree 3 65 ms and degree 4 385 ms in one pass,
// 57 and 276 ms with a launch per axis and component, 42 and 227 ms this way.)
template <typename T>
struct AxisPass {
  const int* ptr;  // CSR rows of the axis: output index -> input entries
  const int* col;
  const T* val;
  int axis, nin;   // and the input's extent along it; the others are the output's
  Transfer g;      // the pass's output (nout, Nout, and the input's Nin)
};

template <typename T, typename Ti>
__device__ __forceinline__ T axis_row(const AxisPass<T>& A, const Ti* in, const int* i) {
  const int row = A.axis == 0 ? i[0] : (A.axis == 1 ? i[1] : i[2]);
  const long long d0 = A.axis == 0 ? A.nin : A.g.nout[0], d1 = A.axis == 1 ? A.nin : A.g.nout[1];
  const long long step = A.axis == 0 ? 1 : (A.axis == 1 ? d0 : d0 * d1);
  const Ti* line = in + ((A.axis == 2 ? 0 : i[2]) * d1 + (A.axis == 1 ? 0 : i[1])) * d0 + (A.axis == 0 ? 0 : i[0]);
  T s = T(0);
  for (int k = A.ptr[row]; k < A.ptr[row + 1]; ++k) s += A.val[k] * T(line[A.col[k] * step]);
  return s;
}

// one axis of a transfer before the last
template <typename T, typename Ti>
__global__ void __launch_bounds__(256) transfer_axis_kernel(const __grid_constant__ AxisPass<T> A, T* out, const Ti* in) {
  chain_wait();
  chain_release();
  const long long N = A.g.Nout;
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < N; n += (long long)gridDim.x * blockDim.x) {
    int i[3];
    A.g.indices((unsigned)n, i);
    out[blockIdx.y * N + n] = axis_row<T, Ti>(A, in + blockIdx.y * A.g.Nin, i);
  }
}

// x += P e: with `row` the prolongation's row at a lattice node; images take their master's row,
// Dirichlet rows nothing
template <typename T, class Row>
__device__ __forceinline__ void prolongate_add(const Transfer& A, T* x, const int* __restrict__ cmap, Row&& row) {
  const long long base = blockIdx.y * A.Nout;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < A.Nout; i += (long long)gridDim.x * blockDim.x) {
    const int m = cmap ? cmap[base + i] : (int)(base + i);
    if (m < 0) continue;
    int k[3];
    A.indices((unsigned)(m - base), k);
    x[base + i] += row(k);
  }
}

// b = P^T r on the coarse level: with `row` the restriction's row at a lattice node; a periodic node
// sums its images' rows as well, constrained rows are zero
template <typename T, typename Tc, class Row>
__device__ __forceinline__ void restrict_to(const Transfer& A, Tc* b, const int* __restrict__ cmap, Row&& row) {
  const long long base = blockIdx.y * A.Nout;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < A.Nout; i += (long long)gridDim.x * blockDim.x) {
    T s = T(0);
    if (!cmap || cmap[base + i] == (int)(base + i)) {
      int k[3];
      A.indices((unsigned)i, k);
      const int m0 = A.periodic[0] && k[0] == 0, m1 = A.periodic[1] && k[1] == 0, m2 = A.periodic[2] && k[2] == 0;
      for (int e2 = 0; e2 <= m2; ++e2)
        for (int e1 = 0; e1 <= m1; ++e1)
          for (int e0 = 0; e0 <= m0; ++e0) {
            const int image[3] = {e0 ? A.nout[0] - 1 : k[0], e1 ? A.nout[1] - 1 : k[1], e2 ? A.nout[2] - 1 : k[2]};
            s += row(image);
          }
    }
    b[base + i] = Tc(s);
  }
}

// Degrees 1 and 2: all axes in one pass (at most 27 entries a row, 8 on average for Q2 3-D, read from
// L1/L2), where one launch per component and axis went through fine-sized work vectors
template <typename T, typename Tc, int degree>
__global__ void __launch_bounds__(256) prolongate_add_kernel(const __grid_constant__ Transfer A, T* x, const Tc* e,
                                                             const int* __restrict__ cmap) {
  chain_wait();
  chain_release();
  const Tc* in = e + blockIdx.y * A.Nin;
  prolongate_add(A, x, cmap, [&](const int* k) { return prolong_row<T, Tc, degree>(A, in, k[0], k[1], k[2]); });
}
template <typename T, typename Tc, int degree>
__global__ void __launch_bounds__(256) restrict_kernel(const __grid_constant__ Transfer A, Tc* b, const T* r,
                                                       const int* __restrict__ cmap) {
  chain_wait();
  chain_release();
  const T* in = r + blockIdx.y * A.Nin;
  restrict_to<T>(A, b, cmap, [&](const int* k) { return restrict_row<T, degree>(A, in, k[0], k[1], k[2]); });
}
// the last axis of the others
template <typename T>
__global__ void __launch_bounds__(256) prolongate_add_axis_kernel(const __grid_constant__ AxisPass<T> A, T* x, const T* e,
                                                                  const int* __restrict__ cmap) {
  chain_wait();
  chain_release();
  const T* in = e + blockIdx.y * A.g.Nin;
  prolongate_add(A.g, x, cmap, [&](const int* k) { return axis_row<T, T>(A, in, k); });
}
template <typename T, typename Tc>
__global__ void __launch_bounds__(256) restrict_axis_kernel(const __grid_constant__ AxisPass<T> A, Tc* b, const T* r,
                                                            const int* __restrict__ cmap) {
  chain_wait();
  chain_release();
  const T* in = r + blockIdx.y * A.g.Nin;
  restrict_to<T>(A.g, b, cmap, [&](const int* k) { return axis_row<T, T>(A, in, k); });
}

// First Chebyshev step from x = 0: x = u = c2 P b
template <typename T>
__global__ void __launch_bounds__(256) cheb_start_kernel(long long n, T* x, T* u, const T* b,
                                                         const T* pinv, double c2) {
  chain_wait();
  chain_release();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const T ui = T(c2) * pinv[i] * b[i];
    u[i] = ui;
    x[i] = ui;
  }
}

// A Chebyshev step from the raw product: Ax = scale (.) acc; u = c1 u + c2 P (b - Ax);
// x += u (one pass instead of a memset, a finalize and an update launch with Ax in between: 20 % of
// the mixed-precision iterations' kernel time)
template <typename T>
__global__ void __launch_bounds__(256) cheb_step_kernel(T* x, T* u, const T* b, const T* acc, T* clear,
                                                        const T* __restrict__ scale, const T* pinv, double c1,
                                                        double c2, long long N) {
  chain_wait();
  chain_release();
  const long long base = blockIdx.y * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const long long gi = base + i;
    const T Ax = scale ? acc[gi] * scale[i] : acc[gi];
    clear[gi] = T(0);
    const T r = b[gi] - Ax;
    const T ui = c1 == 0.0 ? T(c2) * pinv[gi] * r : T(c1) * u[gi] + T(c2) * pinv[gi] * r;
    u[gi] = ui;
    x[gi] += ui;
  }
}

// r = b - scale (.) acc
template <typename T>
__global__ void __launch_bounds__(256) residual_kernel(T* r, const T* b, const T* acc, T* clear,
                                                       const T* __restrict__ scale, long long N) {
  chain_wait();
  chain_release();
  const long long base = blockIdx.y * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const long long gi = base + i;
    const T Ax = scale ? acc[gi] * scale[i] : acc[gi];
    clear[gi] = T(0);
    r[gi] = b[gi] - Ax;
  }
}

// Krylov scalars on the device (LinearState::scal), so that an iteration needs no value on the host
// but the residual norm its caller tests
enum Scalar { SC_RZ = 0 /* two, alternating */, SC_PQ = 2, SC_RR = 3, SC_DONE = 4, SC_TMP = 5, SC_EIG = 8 };

// CG: x += alpha p, r -= alpha q with alpha = rz / pq, and rr = r.r; sc[SC_DONE] is set once
// sqrt(rr) < tol, after which the kernel does nothing (iterations queued past convergence)
__global__ void __launch_bounds__(256) cg_update_kernel(long long n, double* sc, int rz, const double* p, const double* q,
                                                        double* x, double* r, double tol, double* partial,
                                                        unsigned int* counter) {
  chain_wait();
  chain_release();
  if (sc[SC_DONE] != 0.0) return;
  const double alpha = sc[SC_RZ + rz] / sc[SC_PQ];
  double acc = 0.0, total;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    x[i] += alpha * p[i];
    const double ri = r[i] - alpha * q[i];
    r[i] = ri;
    acc += ri * ri;
  }
  if (grid_sum(acc, partial, counter, &total)) {
    sc[SC_RR] = total;
    if (sqrt(total) < tol) sc[SC_DONE] = 1.0;
  }
}

// p = z + beta p with beta = rz_new / rz (first: p = z)
__global__ void __launch_bounds__(256) cg_direction_kernel(long long n, const double* sc, int rz, int first,
                                                           const double* z, double* p) {
  chain_wait();
  chain_release();
  const double beta = first ? 0.0 : sc[SC_RZ + rz] / sc[SC_RZ + 1 - rz];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = first ? z[i] : z[i] + beta * p[i];
}

// The eigenvalue estimate's CG: r -= alpha q, z = P r with the sums r.r and r.z of step `it`
// (start: z = P r, p = z and the sums of r alone); e holds per step pq, rr, rz
template <typename T>
__global__ void __launch_bounds__(256) eig_update_kernel(long long n, double* e, int it, const T* q, T* r, T* z, T* p,
                                                         const T* pinv, double* partial, unsigned int* counter) {
  chain_wait();
  chain_release();
  const bool start = it < 0;
  const double alpha = start ? 0.0 : e[3 * it + 2] / e[3 * it + 3];
  double rr = 0.0, rz = 0.0, total;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const T ri = start ? r[i] : T(-alpha * double(q[i]) + double(r[i]));
    const T zi = pinv[i] * ri;
    r[i] = ri;
    z[i] = zi;
    if (start) p[i] = zi;
    rr += double(ri) * double(ri);
    rz += double(ri) * double(zi);
  }
  // e: rr_0, rz_0 at 1, 2; step it: pq at 3 it + 3, rr at 3 it + 4, rz at 3 it + 5
  if (grid_sum(rr, partial, counter, &total)) e[3 * it + 4] = total;
  __syncthreads();
  if (grid_sum(rz, partial + 1024, counter + 1, &total)) e[3 * it + 5] = total;
}
template <typename T>
__global__ void __launch_bounds__(256) eig_direction_kernel(long long n, const double* e, int it, const T* z, T* p) {
  chain_wait();
  chain_release();
  const double beta = e[3 * it + 5] / e[3 * it + 2];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = T(double(z[i]) + beta * double(p[i]));
}

// the Dirichlet values of the constrained rows, zero elsewhere (the inhomogeneous lift's vector)
__global__ void lift_values_kernel(double* g, const int* __restrict__ cmap, const double* dvals, long long len) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    const int m = cmap[i];
    g[i] = m < 0 ? dvals[-1 - m] : 0.0;
  }
}

// ------------------------------------------------------------------------------------------
// helpers
// ------------------------------------------------------------------------------------------
static size_t esize(int precision) { return precision ? sizeof(float) : sizeof(double); }

// blocks of a reduction over n entries (at most 1024 partial sums)
static unsigned dot_blocks(long long n) { return (unsigned)std::max<long long>(1, std::min<long long>(1024, (n + 255) / 256)); }

static unsigned int* counters(LinearState& L) { return reinterpret_cast<unsigned int*>(L.partial + 2048); }

// work space of the reductions and the Krylov scalars, on the device and in pinned host memory (zeroed
// on the handle's stream, ahead of the kernels that count on it: its own stream does not wait for the
// default one)
static int ensure_scalars(ppf_handle h, LinearState& L) {
  const size_t len = SC_EIG + 8 + 3 * (size_t)L.params.eig_cg_iterations;
  if (L.scal && len > L.scal_len) {  // (parameters set again before a block's first linear solve)
    PPF_CUDA(h, cudaFree(L.scal));
    L.scal = nullptr;
  }
  if (!L.scal) {
    PPF_CUDA(h, cudaMalloc(&L.scal, sizeof(double) * len));
    PPF_CUDA(h, cudaMemsetAsync(L.scal, 0, sizeof(double) * len, h->stream));
    L.scal_len = len;
  }
  if (L.partial) return PPF_OK;
  PPF_CUDA(h, cudaMalloc(&L.partial, sizeof(double) * 2056));
  PPF_CUDA(h, cudaMemsetAsync(L.partial, 0, sizeof(double) * 2056, h->stream));
  PPF_CUDA(h, cudaMallocHost(&L.h_scal, sizeof(double) * 4));
  for (auto& ev : L.scal_ev) PPF_CUDA(h, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  return PPF_OK;
}

// sc = x.y on the device
template <typename T>
static int dot_device(ppf_handle h, LinearState& L, long long n, const T* x, const T* y, double* out) {
  PPF_CUDA(h, launch_chained(dot_kernel<T>, dim3(dot_blocks(n)), dim3(256), 0, h->stream, n, x, y, L.partial, counters(L), out));
  h->all_launches++;
  return PPF_OK;
}

// x.y on the host (waits for the stream)
static int dot(ppf_handle h, LinearState& L, int, long long n, const void* x, const void* y, double* out) {
  int rc = ensure_scalars(h, L);
  if (!rc) rc = dot_device<double>(h, L, n, (const double*)x, (const double*)y, L.scal + SC_TMP);
  if (rc) return rc;
  PPF_CUDA(h, cudaMemcpyAsync(out, L.scal + SC_TMP, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  return PPF_OK;
}

static void axpby(ppf_handle h, int precision, long long n, double a, const void* x, double b, void* y) {
  if (precision) axpby_kernel<float><<<grid_for(n), 256, 0, h->stream>>>(n, a, (const float*)x, b, (float*)y);
  else axpby_kernel<double><<<grid_for(n), 256, 0, h->stream>>>(n, a, (const double*)x, b, (double*)y);
  h->all_launches++;
}

static void convert(ppf_handle h, int pin, int pout, long long n, const void* x, void* y) {
  if (pin == pout) {
    cudaMemcpyAsync(y, x, n * esize(pin), cudaMemcpyDeviceToDevice, h->stream);
    return;
  }
  if (pin == 0) convert_kernel<double, float><<<grid_for(n), 256, 0, h->stream>>>(n, (const double*)x, (float*)y);
  else convert_kernel<float, double><<<grid_for(n), 256, 0, h->stream>>>(n, (const float*)x, (double*)y);
  h->all_launches++;
}

// lumped mass on a lattice of nc cells per axis (periodic images condensed), inverted sqrt
// ------------------------------------------------------------------------------------------
// level set-up on the device (constraint map, inverse mass root, eigenvalue-estimate pattern)
// ------------------------------------------------------------------------------------------
struct LevelGeom {
  int nn[3];
  int periodic[3];
  int dim;
  long long N;
};

// pass 1: periodic images fold onto the lower face; free nodes on a Dirichlet face of their
// component (bit b of dmask[c]) become Dirichlet rows (-1)
__global__ void level_cmap_kernel(int* __restrict__ cm, LevelGeom g, int ncomp, unsigned dm0, unsigned dm1,
                                  unsigned dm2) {
  const long long len = ncomp * g.N;
  for (long long gi = blockIdx.x * (long long)blockDim.x + threadIdx.x; gi < len;
       gi += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(gi / g.N);
    const long long i = gi - c * g.N;
    long long I[3] = {i % g.nn[0], (i / g.nn[0]) % g.nn[1], i / ((long long)g.nn[0] * g.nn[1])};
    long long F[3] = {I[0], I[1], I[2]};
    for (int d = 0; d < g.dim; ++d)
      if (g.periodic[d] && F[d] == g.nn[d] - 1) F[d] = 0;
    const long long m = c * g.N + (F[2] * g.nn[1] + F[1]) * g.nn[0] + F[0];
    int v = (int)m;
    if (m == gi) {
      const unsigned dm = c == 0 ? dm0 : (c == 1 ? dm1 : dm2);
      for (int b = 0; b < 2 * g.dim; ++b)
        if ((dm >> b) & 1u) {
          const int d = b / 2;
          if ((b % 2 == 0 && I[d] == 0) || (b % 2 == 1 && I[d] == g.nn[d] - 1)) v = -1;
        }
    }
    cm[gi] = v;
  }
}

// pass 2: an image whose master is a Dirichlet row becomes a Dirichlet row
__global__ void level_cmap_close_kernel(int* __restrict__ cm, long long len) {
  for (long long gi = blockIdx.x * (long long)blockDim.x + threadIdx.x; gi < len;
       gi += (long long)gridDim.x * blockDim.x) {
    const int m = cm[gi];
    if (m >= 0 && m != (int)gi && cm[m] < 0) cm[gi] = -1;
  }
}

// invM^1/2 per node from the separable 1-D lumped masses m1 (axis d at m1 + off[d])
template <typename T>
__global__ void level_invm_sqrt_kernel(T* __restrict__ out, const double* __restrict__ m1, LevelGeom g, int off1,
                                       int off2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < g.N; i += (long long)gridDim.x * blockDim.x) {
    const long long I = i % g.nn[0], J = (i / g.nn[0]) % g.nn[1], K = i / ((long long)g.nn[0] * g.nn[1]);
    double m = m1[I];
    if (g.dim > 1) m *= m1[off1 + J];
    if (g.dim > 2) m *= m1[off2 + K];
    out[i] = m == 0.0 ? T(0) : T(sqrt(1.0 / m));
  }
}

// sum of (i mod 11) over free entries and their count (integers: exact in any order)
__global__ void pattern_sum_kernel(const int* __restrict__ cm, long long len, unsigned long long* sums) {
  unsigned long long s = 0, n = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    if (cm[i] == (int)i) {
      s += (unsigned long long)(i % 11);
      n += 1;
    }
  atomicAdd(sums, s);
  atomicAdd(sums + 1, n);
}

// the estimate's start vector: (i mod 11) - mean on free entries, zero on constrained ones
template <typename T>
__global__ void pattern_kernel(T* __restrict__ out, const int* __restrict__ cm, long long len, double mean) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    out[i] = cm[i] == (int)i ? T(double(i % 11) - mean) : T(0);
}

// 1-D prolongation from a coarse axis with ncc cells to the fine axis with 2 ncc cells
static void prolongation_1d(const GLRule& g, int k, int ncc, std::vector<int>& ptr, std::vector<int>& col,
                            std::vector<double>& val) {
  const int n = k + 1;
  const int nf = k * 2 * ncc + 1;
  ptr.assign(nf + 1, 0);
  col.clear();
  val.clear();
  for (int I = 0; I < nf; ++I) {
    const int cf = std::min(I / k, 2 * ncc - 1);
    const double xf = g.x[I - k * cf];
    const int cc = cf / 2;
    const double xc = ((cf % 2) + xf) * 0.5;
    for (int j = 0; j < n; ++j) {
      double L = 1.0;
      for (int m = 0; m < n; ++m)
        if (m != j) L *= (xc - g.x[m]) / (g.x[j] - g.x[m]);
      if (std::fabs(L) > 1e-14) {
        col.push_back(k * cc + j);
        val.push_back(L);
      }
    }
    ptr[I + 1] = (int)col.size();
  }
}

static void transpose_csr(int nrows, int ncols, const std::vector<int>& ptr, const std::vector<int>& col,
                          const std::vector<double>& val, std::vector<int>& tptr, std::vector<int>& tcol,
                          std::vector<double>& tval) {
  tptr.assign(ncols + 1, 0);
  for (int c : col) tptr[c + 1]++;
  for (int i = 0; i < ncols; ++i) tptr[i + 1] += tptr[i];
  tcol.assign(col.size(), 0);
  tval.assign(col.size(), 0.0);
  std::vector<int> pos(tptr.begin(), tptr.end() - 1);
  for (int r = 0; r < nrows; ++r)
    for (int q = ptr[r]; q < ptr[r + 1]; ++q) {
      const int p = pos[col[q]]++;
      tcol[p] = r;
      tval[p] = val[q];
    }
}

template <typename T>
static int upload_vec(ppf_handle h, void** dst, const std::vector<T>& v) {
  PPF_CUDA(h, cudaMalloc(dst, sizeof(T) * std::max<size_t>(1, v.size())));
  PPF_CUDA(h, cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return PPF_OK;
}

static int upload_real(ppf_handle h, void** dst, const std::vector<double>& v, int precision) {
  if (!precision) return upload_vec<double>(h, dst, v);
  std::vector<float> f(v.begin(), v.end());
  return upload_vec<float>(h, dst, f);
}

// ------------------------------------------------------------------------------------------
// level operators
// ------------------------------------------------------------------------------------------
// Contraction mode of the multigrid operators (levels and the outer FP64 operator):
// PPF_CONTRACTION_MODE if set, else the LHS plan's timed choice if a plain launch made one,
// else integer derivatives with FP64 integration.
static int multigrid_fx_mode(const BlockPlan& P, int lanes) {
  if (const int m = env_fx_mode(lanes)) return m;
  return P.fx_mode > 0 && (P.fx_mode < 4 || P.fx_mode == lanes) ? P.fx_mode : 1;
}

// Online choice of a contraction mode: the first 2 nm plain launches of an operator run modes
// 1 to 3 and its lane kernel mode (nm = 3, or 4 with one) twice under CUDA events (real work: the
// modes agree to rounding), then the fastest stays in `state`. begin returns the mode of this
// launch and the event slot (-1: not timed); end records the closing event and decides after
// the last timed launch.
static int online_mode_begin(ppf_handle h, int& state, int timed, cudaEvent_t* ev, int fallback, int* slot,
                             int lanes) {
  *slot = -1;
  if (state > 0) return state;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->stream, &cs) != cudaSuccess || h->capturing || cs != cudaStreamCaptureStatusNone) {
    state = fallback;  // no timing (nor event waits) inside a graph capture
    return state;
  }
  *slot = timed;
  for (int i = 2 * timed; i < 2 * timed + 2; ++i)
    if (!ev[i] && cudaEventCreate(&ev[i]) != cudaSuccess) {
      *slot = -1;
      state = fallback;
      return state;
    }
  cudaEventRecord(ev[2 * timed], h->stream);
  return timed_fx_mode(timed % (lanes ? 4 : 3), lanes);
}

static int online_mode_end(ppf_handle h, int& state, int& timed, cudaEvent_t* ev, int slot, int lanes) {
  if (slot < 0) return PPF_OK;
  const int nm = lanes ? 4 : 3;
  PPF_CUDA(h, cudaEventRecord(ev[2 * slot + 1], h->stream));
  if (++timed < 2 * nm) return PPF_OK;
  PPF_CUDA(h, cudaEventSynchronize(ev[4 * nm - 1]));
  float best[4] = {1e30f, 1e30f, 1e30f, 1e30f};
  for (int k = 0; k < 2 * nm; ++k) {
    float t = 0.f;
    PPF_CUDA(h, cudaEventElapsedTime(&t, ev[2 * k], ev[2 * k + 1]));
    best[k % nm] = std::min(best[k % nm], t);
  }
  int b = 0;
  for (int k = 1; k < nm; ++k)
    if (best[k] < best[b]) b = k;
  state = timed_fx_mode(b, lanes);
  for (int i = 0; i < 16; ++i) {
    if (ev[i]) cudaEventDestroy(ev[i]);
    ev[i] = nullptr;
  }
  return PPF_OK;
}

// what follows a launch that read the level's accumulator and cleared the other one
static void level_took(MGLevel& lv) {
  std::swap(lv.acc, lv.acc2);
  lv.acc_clean = true;
}

static int level_cell_launch(ppf_handle h, BlockState& B, MGLevel& lv, int mode, const void* src, bool plain_read) {
  const int f = B.desc.field_indices[0];
  FieldState& F = h->fields[f];
  CellLaunch L;
  std::memset(&L, 0, sizeof(L));
  for (int d = 0; d < 3; ++d) {
    L.nc[d] = lv.nc[d];
    L.nn[d] = lv.nn[d];
  }
  L.N = lv.N;
  L.ncells = lv.ncells;
  const BlockPlan& P = B.plan[1];
  L.nslots = P.nslots;
  for (int s = 0; s < P.nslots; ++s) {
    SlotDesc& sd = L.slots[s];
    sd.ncomp = h->fields[P.slot_field[s]].ncomp;
    if (P.slot_age[s] == 5) {
      sd.ptr = src;
      sd.is_src = 1;
      sd.out_index = 0;
      sd.constrained_read = plain_read ? 0 : (lv.constrained ? 1 : 0);
      sd.cmap = lv.cmap;
    } else {
      // other dependencies exist on the problem lattice only (FP64 single-level solves)
      sd.ptr = state_ptr(h, P.slot_field[s], P.slot_age[s]);
    }
  }
  L.nout = 1;
  L.outs[0].acc = lv.acc;
  L.outs[0].cmap = lv.constrained ? lv.cmap : nullptr;
  L.outs[0].ncomp = F.ncomp;
  L.nrows_in = P.nrows_in;
  L.nrows_out = P.nrows_out;
  L.tables = lv.tables;
  L.tables_host = lv.h_tables.data();
  L.timer = h->timer;
  L.block_id = (unsigned)B.desc.id;
  L.err = h->d_err;
  // integer contractions where the level's tables allow them (FP64 Q1/Q2); the mode is timed
  // online over the level's first plain LHS launches, so choosing costs no extra launches
  int slot = -1;
  int m = multigrid_fx_mode(P, lv.fx_lanes);
  const bool fixed = env_fx_mode(lv.fx_lanes) != 0;
  if (P.fx && lv.precision == 0 && mode == MODE_LHS && !fixed)
    m = online_mode_begin(h, lv.fx_mode, lv.fx_timed, lv.fx_ev, 1, &slot, lv.fx_lanes);
  set_fx_mode(L, m);
  // FP32 levels (mixed precision) run the FP32 lane kernel unless PPF_CONTRACTION_MODE fixes one
  // of the thread-block modes 1-3
  if (lv.precision == 1) {
    const int e = env_fx_mode(4);
    L.fx_lanes = e == 0 || e == 4 || env_fx_mode(5) == 5;
  }
  const size_t smem = cell_smem(h->dim, h->k, lv.precision, P.nrows_in, P.nrows_out);
  const void* obj = lv.precision ? h->model_obj_f32.data() : h->model_obj.data();
  // the level's accumulator is all zero where the kernel that read the other one cleared it, that is
  // unless a launch in between failed
  if (!lv.acc_clean) PPF_CUDA(h, cudaMemsetAsync(lv.acc, 0, lv.len * esize(lv.precision), h->stream));
  lv.acc_clean = false;
  const int rc = timed_cell_launch(h, lv.precision, mode, L, obj, smem);
  if (rc) return rc;
  return online_mode_end(h, lv.fx_mode, lv.fx_timed, lv.fx_ev, slot, lv.fx_lanes);
}

static bool scaled(const LinearState& L) { return L.params.tolerance_type != 0; }

template <typename T>
static const T* level_scale(const LinearState& L, const MGLevel& lv) {
  return scaled(L) ? (const T*)lv.invm_sqrt : nullptr;
}
static const int* level_map(const MGLevel& lv) { return lv.constrained ? lv.cmap : nullptr; }
static dim3 level_grid(ppf_handle h, const BlockState& B, const MGLevel& lv) {
  return dim3(grid_for(lv.N), h->fields[B.desc.field_indices[0]].ncomp);
}

// dst = S A src on level lv (S = invM^1/2 or identity); with `out` also out = src.dst
template <typename T>
static int level_apply(ppf_handle h, BlockState& B, MGLevel& lv, const T* src, T* dst, double* out = nullptr) {
  int rc = level_cell_launch(h, B, lv, MODE_LHS, src, false);
  if (rc) return rc;
  dim3 grid = level_grid(h, B, lv);
  if (out) grid.x = std::min(grid.x, 1024u / grid.y);
  PPF_CUDA(h, launch_chained(level_finalize_kernel<T>, grid, dim3(256), 0, h->stream, dst, (const T*)lv.acc, (T*)lv.acc2,
                             level_scale<T>(B.lin, lv), lv.N, src, B.lin.partial, counters(B.lin), out));
  level_took(lv);
  h->all_launches++;
  return PPF_OK;
}

template <typename T>
static int level_diagonal_t(ppf_handle h, BlockState& B, MGLevel& lv) {
  int rc = level_cell_launch(h, B, lv, MODE_DIAG, lv.x, false);
  if (rc) return rc;
  PPF_CUDA(h, launch_chained(inv_diag_kernel<T>, level_grid(h, B, lv), dim3(256), 0, h->stream, (T*)lv.inv_diag,
                             (const T*)lv.acc, (T*)lv.acc2, level_scale<T>(B.lin, lv), lv.N));
  level_took(lv);
  h->all_launches++;
  return PPF_OK;
}
static int level_diagonal(ppf_handle h, BlockState& B, MGLevel& lv) {
  return lv.precision ? level_diagonal_t<float>(h, B, lv) : level_diagonal_t<double>(h, B, lv);
}

// largest eigenvalue of the symmetric tridiagonal (diag a, off-diagonal b) by bisection
static double tridiag_max_eig(const std::vector<double>& a, const std::vector<double>& b) {
  const int m = (int)a.size();
  if (m == 0) return 1.0;
  double lo = a[0], hi = a[0];
  for (int i = 0; i < m; ++i) {
    const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i + 1 < m ? std::fabs(b[i]) : 0.0);
    lo = std::min(lo, a[i] - r);
    hi = std::max(hi, a[i] + r);
  }
  auto count_below = [&](double x) {  // Sturm count of eigenvalues < x
    int cnt = 0;
    double q = a[0] - x;
    if (q < 0) cnt++;
    for (int i = 1; i < m; ++i) {
      const double qq = q == 0.0 ? 1e-300 : q;
      q = a[i] - x - b[i - 1] * b[i - 1] / qq;
      if (q < 0) cnt++;
    }
    return cnt;
  };
  for (int it = 0; it < 200; ++it) {
    const double mid = 0.5 * (lo + hi);
    if (count_below(mid) >= m) hi = mid;
    else lo = mid;
    if (hi - lo <= 1e-14 * std::max(1.0, std::fabs(hi))) break;
  }
  return hi;
}

// Lanczos estimate of the largest eigenvalue of P A (P = inverse diagonal) on level lv:
// eig_cg_iterations CG steps on A x = pattern from x = 0 (uses lv.b, lv.r, lv.w0, lv.w1). The steps
// are queued without waiting for their scalars, which come to the host once at the end.
template <typename T>
static int estimate_eigenvalues(ppf_handle h, BlockState& B, MGLevel& lv) {
  LinearState& L = B.lin;
  const long long n = lv.len;
  int rc = ensure_scalars(h, L);
  if (rc) return rc;
  if (!(lv.pattern_mean >= 0.0)) {
    unsigned long long* d_sums = reinterpret_cast<unsigned long long*>(L.partial);
    PPF_CUDA(h, cudaMemsetAsync(d_sums, 0, 2 * sizeof(unsigned long long), h->stream));
    pattern_sum_kernel<<<grid_for(lv.len), 256, 0, h->stream>>>(lv.cmap, lv.len, d_sums);
    unsigned long long sums[2];
    PPF_CUDA(h, cudaMemcpyAsync(sums, d_sums, sizeof(sums), cudaMemcpyDeviceToHost, h->stream));
    PPF_CUDA(h, cudaStreamSynchronize(h->stream));
    lv.pattern_mean = double(sums[0]) / double(std::max<unsigned long long>(1, sums[1]));
    h->all_launches++;
  }
  T* r = (T*)lv.r;
  T* z = (T*)lv.w0;
  T* p = (T*)lv.w1;
  T* q = (T*)lv.b;
  double* e = L.scal + SC_EIG;
  pattern_kernel<T><<<grid_for(n), 256, 0, h->stream>>>(r, lv.cmap, n, lv.pattern_mean);
  PPF_CUDA(h, cudaGetLastError());
  PPF_CUDA(h, launch_chained(eig_update_kernel<T>, dim3(dot_blocks(n)), dim3(256), 0, h->stream, n, e, -1, q, r, z, p,
                             (const T*)lv.inv_diag, L.partial, counters(L)));
  h->all_launches += 2;
  const int steps = L.params.eig_cg_iterations;
  for (int it = 0; it < steps; ++it) {
    rc = level_apply<T>(h, B, lv, p, q, e + 3 * it + 3);
    if (rc) return rc;
    PPF_CUDA(h, launch_chained(eig_update_kernel<T>, dim3(dot_blocks(n)), dim3(256), 0, h->stream, n, e, it, q, r, z, p,
                               (const T*)lv.inv_diag, L.partial, counters(L)));
    PPF_CUDA(h, launch_chained(eig_direction_kernel<T>, dim3(grid_for(n)), dim3(256), 0, h->stream, n, e, it, z, p));
    h->all_launches += 2;
  }
  std::vector<double> he(3 * steps + 6);
  PPF_CUDA(h, cudaMemcpyAsync(he.data(), e, sizeof(double) * (3 * steps + 3), cudaMemcpyDeviceToHost, h->stream));
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  const double r0 = he[1];
  double rz = he[2];
  std::vector<double> alphas, betas;
  for (int it = 0; it < steps; ++it) {
    const double pq = he[3 * it + 3], rr = he[3 * it + 4], rz_new = he[3 * it + 5];
    if (pq <= 0.0 || !std::isfinite(pq)) break;
    alphas.push_back(rz / pq);
    if (std::sqrt(rr) < 1e-10 * std::sqrt(r0)) break;
    betas.push_back(rz_new / rz);
    rz = rz_new;
  }
  // Lanczos matrix of the CG coefficients
  const int m = (int)alphas.size();
  std::vector<double> a(m), b(m > 0 ? m - 1 : 0);
  for (int i = 0; i < m; ++i) {
    a[i] = 1.0 / alphas[i] + (i > 0 ? betas[i - 1] / alphas[i - 1] : 0.0);
    if (i + 1 < m) b[i] = std::sqrt(std::max(0.0, betas[i])) / alphas[i];
  }
  const double est = tridiag_max_eig(a, b);
  lv.lambda_max = 1.2 * est;
  lv.lambda_min = lv.lambda_max / L.params.smoothing_range;
  lv.eig_done = true;
  return PPF_OK;
}

// Chebyshev smoother on level lv: x <- x + p(P A)(P (b - A x)); zero_start: from x = 0
template <typename T>
static int chebyshev(ppf_handle h, BlockState& B, MGLevel& lv, bool zero_start, const T* b, T* x) {
  const double theta = 0.5 * (lv.lambda_max + lv.lambda_min);
  const double delta = 0.5 * (lv.lambda_max - lv.lambda_min);
  const double sigma = theta / delta;
  T* u = (T*)lv.w0;
  double rho_prev = 1.0 / sigma;
  for (int k = 0; k < B.lin.params.smoother_degree; ++k) {
    double c1, c2;
    if (k == 0) {
      c1 = 0.0;
      c2 = 1.0 / theta;
    } else {
      const double rho = 1.0 / (2.0 * sigma - rho_prev);
      c1 = rho * rho_prev;
      c2 = 2.0 * rho / delta;
      rho_prev = rho;
    }
    if (zero_start && k == 0) {
      PPF_CUDA(h, launch_chained(cheb_start_kernel<T>, dim3(grid_for(lv.len)), dim3(256), 0, h->stream, lv.len, x, u, b,
                                 (const T*)lv.inv_diag, c2));
    } else {
      int rc = level_cell_launch(h, B, lv, MODE_LHS, x, false);
      if (rc) return rc;
      PPF_CUDA(h, launch_chained(cheb_step_kernel<T>, level_grid(h, B, lv), dim3(256), 0, h->stream, x, u, b,
                                 (const T*)lv.acc, (T*)lv.acc2, level_scale<T>(B.lin, lv),
                                 (const T*)lv.inv_diag, c1, c2, lv.N));
      level_took(lv);
    }
    h->all_launches++;
  }
  return PPF_OK;
}

// the transfer between lattices of extents nin and nout
static Transfer transfer(ppf_handle h, const int* nout, const int* nin) {
  Transfer A;
  std::memset(&A, 0, sizeof(A));
  A.dim = h->dim;
  A.Nout = A.Nin = 1;
  for (int d = 0; d < 3; ++d) {
    A.nout[d] = nout[d];
    A.nin[d] = nin[d];
    A.periodic[d] = d < h->dim ? h->mesh.periodic[d] : 0;
    A.Nout *= nout[d];
    A.Nin *= nin[d];
  }
  for (int d = 0; d < 2; ++d) A.fd[d].init((unsigned)nout[d]);
  return A;
}

// The passes of a transfer of degree 3 or 4 between level c and the next finer one f, the last axis
// left to `last(pass, in)`; the levels' work vectors of a smoothing step hold what lies in between
template <typename T, typename Ti, class Last>
static int transfer_axes(ppf_handle h, const BlockState& B, const MGLevel& c, const MGLevel& f, bool prolongate,
                         const Ti* in, Last&& last) {
  const int ncomp = h->fields[B.desc.field_indices[0]].ncomp;
  int n[3] = {1, 1, 1};
  for (int d = 0; d < 3; ++d) n[d] = prolongate ? c.nn[d] : f.nn[d];
  const T* from = nullptr;
  for (int d = 0; d < h->dim; ++d) {
    AxisPass<T> A;
    A.ptr = prolongate ? c.p_ptr[d] : c.r_ptr[d];
    A.col = prolongate ? c.p_col[d] : c.r_col[d];
    A.val = (const T*)(prolongate ? c.p_val[d] : c.r_val[d]);
    A.axis = d;
    A.nin = n[d];
    int out[3] = {n[0], n[1], n[2]};
    out[d] = prolongate ? f.nn[d] : c.nn[d];
    A.g = transfer(h, out, n);
    if (d == h->dim - 1) return last(A, from);
    T* to = (T*)(d == 0 ? f.w1 : f.w0);
    const dim3 grid(grid_for(A.g.Nout), ncomp);
    if (d == 0) PPF_CUDA(h, launch_chained(transfer_axis_kernel<T, Ti>, grid, dim3(256), 0, h->stream, A, to, in));
    else PPF_CUDA(h, launch_chained(transfer_axis_kernel<T, T>, grid, dim3(256), 0, h->stream, A, to, from));
    h->all_launches++;
    from = to;
    n[d] = out[d];
  }
  return PPF_OK;
}

// c.b = P^T f.r
template <typename T, typename Tc>
static int restrict_residual(ppf_handle h, const BlockState& B, MGLevel& c, const MGLevel& f) {
  const dim3 grid = level_grid(h, B, c);
  h->all_launches++;
  if (h->k > 2)
    return transfer_axes<T, T>(h, B, c, f, false, (const T*)f.r, [&](const AxisPass<T>& A, const T* in) -> int {
      PPF_CUDA(h, launch_chained(restrict_axis_kernel<T, Tc>, grid, dim3(256), 0, h->stream, A, (Tc*)c.b, in, level_map(c)));
      return PPF_OK;
    });
  PPF_CUDA(h, launch_chained(h->k == 1 ? restrict_kernel<T, Tc, 1> : restrict_kernel<T, Tc, 2>, grid, dim3(256), 0,
                             h->stream, transfer(h, c.nn, f.nn), (Tc*)c.b, (const T*)f.r, level_map(c)));
  return PPF_OK;
}

// x += P c.x on level f
template <typename T, typename Tc>
static int prolongate_correction(ppf_handle h, const BlockState& B, const MGLevel& c, const MGLevel& f, T* x) {
  const dim3 grid = level_grid(h, B, f);
  h->all_launches++;
  if (h->k > 2)
    return transfer_axes<T, Tc>(h, B, c, f, true, (const Tc*)c.x, [&](const AxisPass<T>& A, const T* in) -> int {
      PPF_CUDA(h, launch_chained(prolongate_add_axis_kernel<T>, grid, dim3(256), 0, h->stream, A, x, in, level_map(f)));
      return PPF_OK;
    });
  PPF_CUDA(h, launch_chained(h->k == 1 ? prolongate_add_kernel<T, Tc, 1> : prolongate_add_kernel<T, Tc, 2>, grid,
                             dim3(256), 0, h->stream, transfer(h, f.nn, c.nn), x, (const Tc*)c.x, level_map(f)));
  return PPF_OK;
}

static int vcycle(ppf_handle h, BlockState& B, int l, const void* b, void* x);

// V-cycle on level l (entries T) with the defect b; x receives the correction. Tc: the entries of
// the next coarser level.
template <typename T, typename Tc>
static int vcycle_level(ppf_handle h, BlockState& B, int l, const T* b, T* x) {
  auto& lvs = B.lin.levels;
  MGLevel& lv = lvs[l];
  int rc = chebyshev<T>(h, B, lv, true, b, x);
  if (rc || l == 0) return rc;  // coarse: the smoother as coarse solver
  MGLevel& cl = lvs[l - 1];
  rc = level_cell_launch(h, B, lv, MODE_LHS, x, false);
  if (rc) return rc;
  PPF_CUDA(h, launch_chained(residual_kernel<T>, level_grid(h, B, lv), dim3(256), 0, h->stream, (T*)lv.r, b,
                             (const T*)lv.acc, (T*)lv.acc2, level_scale<T>(B.lin, lv), lv.N));
  level_took(lv);
  h->all_launches++;
  if ((rc = restrict_residual<T, Tc>(h, B, cl, lv))) return rc;
  if ((rc = vcycle(h, B, l - 1, cl.b, cl.x))) return rc;
  if ((rc = prolongate_correction<T, Tc>(h, B, cl, lv, x))) return rc;
  return chebyshev<T>(h, B, lv, false, b, x);
}

static int vcycle(ppf_handle h, BlockState& B, int l, const void* b, void* x) {
  const int prec = B.lin.levels[l].precision;
  const int coarse = l > 0 ? B.lin.levels[l - 1].precision : prec;
  if (prec && coarse) return vcycle_level<float, float>(h, B, l, (const float*)b, (float*)x);
  if (prec) return vcycle_level<float, double>(h, B, l, (const float*)b, (float*)x);
  return vcycle_level<double, double>(h, B, l, (const double*)b, (double*)x);
}

// ------------------------------------------------------------------------------------------
// set-up
// ------------------------------------------------------------------------------------------
static int alloc_real(ppf_handle h, void** p, long long n, int precision) {
  PPF_CUDA(h, cudaMalloc(p, std::max<long long>(1, n) * esize(precision)));
  PPF_CUDA(h, cudaMemset(*p, 0, std::max<long long>(1, n) * esize(precision)));
  return PPF_OK;
}

static int init_linear(ppf_handle h, int b) {
  BlockState& B = h->blocks[b];
  LinearState& L = B.lin;
  if (!L.params_set) {
    ppf_default_linear_params(&L.params);
    L.params_set = true;
  }
  if (B.desc.n_fields != 1) return fail(h, PPF_ERR_UNSUPPORTED, "linear blocks with more than one field");
  if (!B.plan[1].valid) return fail(h, PPF_ERR_ARG, "linear block has no LHS dependencies or no compiled LHS");
  for (int s = 0; s < B.plan[1].nslots; ++s)
    if (B.plan[1].slot_age[s] != 5 && L.params.preconditioner == 2)
      return fail(h, PPF_ERR_UNSUPPORTED, "GMG: the LHS may only depend on src in this build");
  const int f = B.desc.field_indices[0];
  FieldState& F = h->fields[f];
  const long long len = F.len;
  PPF_CUDA(h, cudaMalloc(&L.rhs, sizeof(double) * len));
  PPF_CUDA(h, cudaMalloc(&L.g, sizeof(double) * len));
  PPF_CUDA(h, cudaMalloc(&L.x_hom, sizeof(double) * len));
  PPF_CUDA(h, cudaMemset(L.x_hom, 0, sizeof(double) * len));
  PPF_CUDA(h, cudaMalloc(&L.r, sizeof(double) * len));
  PPF_CUDA(h, cudaMalloc(&L.p, sizeof(double) * len));
  PPF_CUDA(h, cudaMalloc(&L.q, sizeof(double) * len));
  PPF_CUDA(h, cudaMalloc(&L.z, sizeof(double) * len));
  if (const int rc = ensure_scalars(h, L)) return rc;
  // levels: coarsest refinement R - depth + 1 .. R (depth 1 = the fine level only)
  const int R = h->mesh.global_refinement;
  int depth = L.params.preconditioner == 2 ? std::max(1, L.params.mg_depth) : 1;
  depth = std::min(depth, R + 1);
  L.levels.resize(depth);
  const GLRule g = gauss_lobatto(h->n);
  for (int l = 0; l < depth; ++l) {
    MGLevel& lv = L.levels[l];
    lv.refine = R - depth + 1 + l;
    lv.N = 1;
    lv.ncells = 1;
    for (int d = 0; d < 3; ++d) {
      if (d < h->dim) {
        lv.nc[d] = h->mesh.subdivisions[d] << lv.refine;
        lv.nn[d] = h->k * lv.nc[d] + 1;
        lv.h[d] = h->mesh.size[d] / lv.nc[d];
      } else {
        lv.nc[d] = lv.nn[d] = 1;
        lv.h[d] = 1.0;
      }
      lv.N *= lv.nn[d];
      lv.ncells *= lv.nc[d];
    }
    lv.len = F.ncomp * lv.N;
    const bool is_fine = l == depth - 1;
    lv.precision = (L.params.preconditioner == 2 && L.params.mixed_precision && l > 0) ? 1 : 0;
    // constraint map and invM^1/2 of the level, built on the device
    LevelGeom geom;
    geom.dim = h->dim;
    geom.N = lv.N;
    unsigned dmask[3] = {0u, 0u, 0u};
    bool any_constraint = false;
    for (int d = 0; d < 3; ++d) {
      geom.nn[d] = lv.nn[d];
      geom.periodic[d] = d < h->dim ? h->mesh.periodic[d] : 0;
      any_constraint |= geom.periodic[d] != 0;
    }
    for (int c = 0; c < F.ncomp; ++c)
      for (int bid = 0; bid < 2 * h->dim; ++bid)
        if (F.desc.dirichlet[c][bid]) {
          dmask[c] |= 1u << bid;
          any_constraint = true;
        }
    lv.constrained = any_constraint;
    PPF_CUDA(h, cudaMalloc(&lv.cmap, sizeof(int) * std::max<long long>(1, lv.len)));
    level_cmap_kernel<<<grid_for(lv.len), 256, 0, h->stream>>>(lv.cmap, geom, F.ncomp, dmask[0], dmask[1], dmask[2]);
    level_cmap_close_kernel<<<grid_for(lv.len), 256, 0, h->stream>>>(lv.cmap, lv.len);
    {
      std::vector<double> m1;
      int offs[3] = {0, 0, 0};
      for (int d = 0; d < h->dim; ++d) {
        offs[d] = (int)m1.size();
        std::vector<double> a(lv.nn[d], 0.0);
        for (int cc = 0; cc < lv.nc[d]; ++cc)
          for (int q = 0; q < h->n; ++q) a[h->k * cc + q] += g.w[q] * lv.h[d];
        if (h->mesh.periodic[d]) {
          a[0] += a[lv.nn[d] - 1];
          a[lv.nn[d] - 1] = 0.0;
        }
        m1.insert(m1.end(), a.begin(), a.end());
      }
      void* d_m1 = nullptr;
      int rc = upload_vec<double>(h, &d_m1, m1);
      if (rc) return rc;
      PPF_CUDA(h, cudaMalloc(&lv.invm_sqrt, esize(lv.precision) * std::max<long long>(1, lv.N)));
      if (lv.precision)
        level_invm_sqrt_kernel<float><<<grid_for(lv.N), 256, 0, h->stream>>>((float*)lv.invm_sqrt, (const double*)d_m1,
                                                                             geom, offs[1], offs[2]);
      else
        level_invm_sqrt_kernel<double><<<grid_for(lv.N), 256, 0, h->stream>>>((double*)lv.invm_sqrt,
                                                                              (const double*)d_m1, geom, offs[1], offs[2]);
      PPF_CUDA(h, cudaGetLastError());
      PPF_CUDA(h, cudaStreamSynchronize(h->stream));
      cudaFree(d_m1);
    }
    int rc = PPF_OK;
    // LHS tables of this level (the block's LHS dependency slots)
    signed char slot_of[pg::MAX_FIELDS][pg::NAGE];
    signed char slot_comp0[pg::MAX_SLOTS] = {};
    signed char out_of[pg::MAX_FIELDS];
    signed char out_row0[pg::MAX_OUTS] = {};
    std::memset(slot_of, -1, sizeof(slot_of));
    std::memset(out_of, -1, sizeof(out_of));
    int row = 0;
    for (int s = 0; s < B.plan[1].nslots; ++s) {
      slot_of[B.plan[1].slot_field[s]][B.plan[1].slot_age[s]] = (signed char)s;
      slot_comp0[s] = (signed char)row;
      row += h->fields[B.plan[1].slot_field[s]].ncomp;
    }
    out_of[f] = 0;
    double lo[3] = {h->mesh.lower[0], h->mesh.lower[1], h->mesh.lower[2]};
    auto tab = build_cell_tables(h->dim, h->k, lv.precision, lo, lv.h, slot_of, slot_comp0, out_of, out_row0,
                                 B.plan[1].fx_rows, B.plan[1].val_rows);
    PPF_CUDA(h, cudaMalloc(&lv.tables, tab.size()));
    PPF_CUDA(h, cudaMemcpy(lv.tables, tab.data(), tab.size(), cudaMemcpyHostToDevice));
    lv.fx_lanes = lv.precision == 0 ? tables_lanes(tab, h->dim, h->k) : 0;
    lv.h_tables = std::move(tab);
    for (void** p : {&lv.inv_diag, &lv.acc, &lv.acc2, &lv.x, &lv.b, &lv.r, &lv.w0, &lv.w1}) {
      rc = alloc_real(h, p, lv.len, lv.precision);
      if (rc) return rc;
    }
    lv.acc_clean = true;
    (void)is_fine;
  }
  // transfers between consecutive levels as rows of each axis (stored on the coarse level; degrees 1
  // and 2 have closed forms)
  for (int l = 0; l + 1 < depth && h->k > 2; ++l) {
    MGLevel& cl = L.levels[l];
    MGLevel& fl = L.levels[l + 1];
    const int tp = fl.precision;  // transfers run in the fine level's precision
    for (int d = 0; d < h->dim; ++d) {
      std::vector<int> ptr, col, tptr, tcol;
      std::vector<double> val, tval;
      prolongation_1d(g, h->k, cl.nc[d], ptr, col, val);
      transpose_csr(fl.nn[d], cl.nn[d], ptr, col, val, tptr, tcol, tval);
      int rc = upload_vec<int>(h, (void**)&cl.p_ptr[d], ptr);
      if (!rc) rc = upload_vec<int>(h, (void**)&cl.p_col[d], col);
      if (!rc) rc = upload_real(h, &cl.p_val[d], val, tp);
      if (!rc) rc = upload_vec<int>(h, (void**)&cl.r_ptr[d], tptr);
      if (!rc) rc = upload_vec<int>(h, (void**)&cl.r_col[d], tcol);
      if (!rc) rc = upload_real(h, &cl.r_val[d], tval, tp);
      if (rc) return rc;
    }
  }
  PPF_CUDA(h, cudaDeviceSynchronize());
  L.initialized = true;
  return PPF_OK;
}

// LinearSolver::normalization_value (linear_solver.h:414-427)
static double normalization(ppf_handle h, const LinearState& L, int n_fields = 1) {
  double v = 1.0;
  const int t = L.params.tolerance_type;
  if (t == 1 || t == 3) {
    double vol = 1.0;
    for (int d = 0; d < h->dim; ++d) vol *= h->mesh.size[d];
    v *= std::sqrt(vol);
  }
  if (t == 1 || t == 2) v *= std::sqrt((double)n_fields);
  return v;
}

// preconditioner application z = M^-1 r (FP64 fine vectors)
static int precondition(ppf_handle h, BlockState& B, const double* r, double* z) {
  LinearState& L = B.lin;
  const long long n = h->fields[B.desc.field_indices[0]].len;
  if (L.params.preconditioner == 0) {
    PPF_CUDA(h, cudaMemcpyAsync(z, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
    return PPF_OK;
  }
  MGLevel& fine = L.levels.back();
  const int top = (int)L.levels.size() - 1;
  if (!fine.precision)
    return L.params.preconditioner == 1 ? chebyshev<double>(h, B, fine, true, r, z) : vcycle(h, B, top, r, z);
  // an FP32 fine level's own vectors carry the V-cycle
  convert(h, 0, 1, n, r, fine.b);
  int rc = L.params.preconditioner == 1 ? chebyshev<float>(h, B, fine, true, (const float*)fine.b, (float*)fine.x)
                                        : vcycle(h, B, top, fine.b, fine.x);
  if (rc) return rc;
  convert(h, 1, 0, n, fine.x, z);
  return PPF_OK;
}

// precondition() through a CUDA graph: the first application of a solve runs as plain
// launches (every kernel is configured then), the second is captured and every later one
// replays the graph: a V-cycle is a few hundred small launches on the coarse levels, whose
// launch overhead the graph removes. The graph holds the solve's simulation time and level
// state, so it is rebuilt for each solve.
static void drop_pc_graph(LinearState& L) {
  if (L.pc_graph) cudaGraphExecDestroy(L.pc_graph);
  L.pc_graph = nullptr;
  L.pc_calls = 0;
}

static int precondition_graphed(ppf_handle h, BlockState& B, const double* r, double* z) {
  LinearState& L = B.lin;
  if (L.params.preconditioner == 0 || h->timing || !h->use_graph || L.pc_nograph) return precondition(h, B, r, z);
  if (L.pc_graph && L.pc_in == r && L.pc_out == z) {
    PPF_CUDA(h, cudaGraphLaunch(L.pc_graph, h->stream));
    h->all_launches++;
    return PPF_OK;
  }
  if (L.pc_calls++ == 0) return precondition(h, B, r, z);
  drop_pc_graph(L);
  L.pc_calls = 2;
  if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    L.pc_nograph = true;
    return precondition(h, B, r, z);
  }
  std::vector<void*> acc0;
  for (auto& lv : L.levels) acc0.push_back(lv.acc);
  int rc = precondition(h, B, r, z);
  // a replay starts where the capture did: a level left on its other accumulator (an odd number of
  // products, the coarsest level's) clears the first one and returns to it
  for (size_t l = 0; l < L.levels.size() && !rc; ++l) {
    MGLevel& lv = L.levels[l];
    if (lv.acc == acc0[l]) continue;
    std::swap(lv.acc, lv.acc2);
    if (cudaMemsetAsync(lv.acc, 0, lv.len * esize(lv.precision), h->stream) != cudaSuccess)
      rc = fail(h, PPF_ERR_CUDA, "preconditioner capture");
  }
  cudaGraph_t graph = nullptr;
  const cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
  if (!rc && e != cudaSuccess) rc = fail(h, PPF_ERR_CUDA, std::string("preconditioner capture: ") + cudaGetErrorString(e));
  if (!rc) {
    const cudaError_t ie = cudaGraphInstantiate(&L.pc_graph, graph, 0);
    if (ie != cudaSuccess) rc = fail(h, PPF_ERR_CUDA, std::string("preconditioner graph: ") + cudaGetErrorString(ie));
  }
  if (graph) cudaGraphDestroy(graph);
  if (rc) {
    // nothing that was recorded has run
    for (size_t l = 0; l < L.levels.size(); ++l) {
      MGLevel& lv = L.levels[l];
      if (lv.acc != acc0[l]) std::swap(lv.acc, lv.acc2);
      lv.acc_clean = false;
    }
    return rc;
  }
  L.pc_in = r;
  L.pc_out = z;
  PPF_CUDA(h, cudaGraphLaunch(L.pc_graph, h->stream));
  h->all_launches++;
  return PPF_OK;
}

// CG on A x = b from the residual r of the iterate x (SolverCG): M(r, z) applies the preconditioner,
// A(p, q, pq) the operator with pq = p.q on the device. alpha, beta and the convergence test stay on
// the device; the host reads each residual norm, one iteration behind the work it has queued where
// the preconditioner is cheap, so that it never waits with an empty stream (a V-cycle is longer than
// that wait, and queueing one past convergence would cost more). What runs past convergence changes
// neither x nor r.
template <class Mf, class Af>
static int conjugate_gradients(ppf_handle h, LinearState& L, long long n, double* x, double* r, double* z, double* p,
                               double* q, double tol, Mf&& M, Af&& A, int* its, double* res, bool* converged) {
  const int lag = L.params.preconditioner == 2 ? 0 : 1;
  const bool plain = L.params.preconditioner == 0;  // z is r itself
  double* sc = L.scal;
  int rc = PPF_OK;
  PPF_CUDA(h, cudaMemsetAsync(sc, 0, sizeof(double) * SC_EIG, h->stream));
  const int max_it = L.params.max_iterations;
  for (int it = 0;; ++it) {
    // it: iterations queued so far; `seen` is the newest whose residual the host reads now
    const int seen = it == max_it ? it : it - lag;
    for (int s = it == max_it ? std::max(1, it - lag) : seen; s >= 1 && s <= seen; ++s) {
      PPF_CUDA(h, cudaEventSynchronize(L.scal_ev[s & 3]));
      *res = std::sqrt(L.h_scal[s & 3]);
      *its = s;
      if (!std::isfinite(*res)) return fail(h, PPF_ERR_NAN, "non-finite residual in the linear solve");
      if (*res < tol) {
        *converged = true;
        return PPF_OK;
      }
    }
    if (it == max_it) return PPF_OK;
    const int rz = it & 1;
    const double* zz = plain ? r : z;
    if (!plain && (rc = M(r, z))) return rc;
    if ((rc = dot_device<double>(h, L, n, r, zz, sc + SC_RZ + rz))) return rc;
    PPF_CUDA(h, launch_chained(cg_direction_kernel, dim3(grid_for(n)), dim3(256), 0, h->stream, n, (const double*)sc, rz,
                               it == 0 ? 1 : 0, zz, p));
    if ((rc = A(p, q, sc + SC_PQ))) return rc;
    PPF_CUDA(h, launch_chained(cg_update_kernel, dim3(dot_blocks(n)), dim3(256), 0, h->stream, n, sc, rz,
                               (const double*)p, (const double*)q, x, r, tol, L.partial, counters(L)));
    h->all_launches += 2;
    const int s = it + 1;
    PPF_CUDA(h, cudaMemcpyAsync(L.h_scal + (s & 3), sc + SC_RR, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    PPF_CUDA(h, cudaEventRecord(L.scal_ev[s & 3], h->stream));
  }
}

int linear_solve(ppf_handle h, int b) {
  BlockState& B = h->blocks[b];
  LinearState& L = B.lin;
  L.last_init_ms = 0.0;
  if (h->amr) {
    // adaptive meshes: CG without a preconditioner on the current mesh's vectors, which are
    // re-made (warm start from zero) whenever the mesh changes
    if (!L.params_set) {
      ppf_default_linear_params(&L.params);
      L.params_set = true;
    }
    if (L.params.preconditioner != 0)
      return fail(h, PPF_ERR_UNSUPPORTED, "adaptive meshes: linear solves run without a preconditioner");
    if (B.desc.n_fields != 1) return fail(h, PPF_ERR_UNSUPPORTED, "linear blocks with more than one field");
    if (!B.plan[1].valid) return fail(h, PPF_ERR_ARG, "linear block has no LHS dependencies or no compiled LHS");
    if (L.mesh_version != h->mesh_version || !L.initialized) {
      const long long len = h->fields[B.desc.field_indices[0]].len;
      double** vecs[] = {&L.rhs, &L.g, &L.x_hom, &L.r, &L.p, &L.q, &L.z};
      for (double** v : vecs) {
        cudaFree(*v);
        *v = nullptr;
        PPF_CUDA(h, cudaMalloc(v, sizeof(double) * len));
      }
      PPF_CUDA(h, cudaMemsetAsync(L.x_hom, 0, sizeof(double) * len, h->stream));
      if (const int rc = ensure_scalars(h, L)) return rc;
      L.mesh_version = h->mesh_version;
      L.initialized = true;
    }
  } else if (!L.initialized) {
    const auto t0 = std::chrono::steady_clock::now();
    int rc = init_linear(h, b);
    if (rc) return rc;
    L.last_init_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  }
  const int f = B.desc.field_indices[0];
  FieldState& F = h->fields[f];
  const long long n = F.len;
  // FP64 outer operator on the problem lattice (the handle's FP64 LHS plan), also when the
  // fine multigrid level runs in FP32
  // (with `out` also out = src.dst)
  auto finalize = [&](double* dst, const double* w, double* out) -> int {
    dim3 grid(grid_for(h->N), F.ncomp);
    if (out) grid.x = std::min(grid.x, 1024u / grid.y);
    if (const int rc = ensure_acc2(h, F)) return rc;
    PPF_CUDA(h, launch_chained(level_finalize_kernel<double>, grid, dim3(256), 0, h->stream, dst, (const double*)F.acc,
                               F.acc2, scaled(L) ? h->d_invm_sqrt : nullptr, h->N, w,
                               L.partial, counters(L), out));
    h->all_launches++;
    std::swap(F.acc, F.acc2);
    F.acc_clean = true;
    return PPF_OK;
  };
  auto outer_apply = [&](const double* src, double* dst, bool plain, double* out) -> int {
    const double* srcs[PPF_MAX_FIELDS] = {src};
    int rc = clear_acc(h, F);
    if (rc) return rc;
    F.acc_clean = false;
    if (h->amr) {
      rc = launch_cell(h, b, 1, srcs, plain);
      return rc ? rc : finalize(dst, src, out);
    }
    CellLaunch Lc;
    std::memset(&Lc, 0, sizeof(Lc));
    for (int d = 0; d < 3; ++d) {
      Lc.nc[d] = h->nc[d];
      Lc.nn[d] = h->nn[d];
    }
    Lc.N = h->N;
    Lc.ncells = h->ncells;
    BlockPlan& P = B.plan[1];
    Lc.nslots = P.nslots;
    for (int s = 0; s < P.nslots; ++s) {
      SlotDesc& sd = Lc.slots[s];
      const int sf = P.slot_field[s];
      sd.ncomp = h->fields[sf].ncomp;
      if (P.slot_age[s] == 5) {
        sd.ptr = srcs[0];
        sd.constrained_read = plain ? 0 : (F.constrained ? 1 : 0);
        sd.cmap = F.cmap;
        sd.is_src = 1;
      } else {
        sd.ptr = state_ptr(h, sf, P.slot_age[s]);
      }
    }
    Lc.nout = 1;
    Lc.outs[0].acc = F.acc;
    Lc.outs[0].cmap = F.constrained ? F.cmap : nullptr;
    Lc.outs[0].ncomp = F.ncomp;
    Lc.nrows_in = P.nrows_in;
    Lc.nrows_out = P.nrows_out;
    Lc.tables = P.d_tables;
    Lc.tables_host = P.h_tables.data();
    Lc.timer = h->timer;
    Lc.block_id = (unsigned)B.desc.id;
    Lc.err = h->d_err;
    // the finest level is this operator on the same mesh: its timed mode if it has one; else
    // (an FP32 finest level) the plan's own mode, timed online over its first outer launches
    int slot = -1;
    {
      const int lm = L.levels.empty() ? -1 : L.levels.back().fx_mode;
      const bool fixed = env_fx_mode(P.fx_lanes) != 0;
      int m = multigrid_fx_mode(P, P.fx_lanes);
      if (!fixed && lm > 0 && (lm < 4 || lm == P.fx_lanes)) m = lm;
      else if (!fixed && P.fx) m = online_mode_begin(h, P.fx_mode, P.fx_timed, P.fx_ev, 1, &slot, P.fx_lanes);
      set_fx_mode(Lc, m);
    }
    const size_t smem = cell_smem(h->dim, h->k, 0, P.nrows_in, P.nrows_out);
    rc = timed_cell_launch(h, 0, MODE_LHS, Lc, h->model_obj.data(), smem);
    if (rc) return rc;
    rc = online_mode_end(h, P.fx_mode, P.fx_timed, P.fx_ev, slot, P.fx_lanes);
    return rc ? rc : finalize(dst, src, out);
  };
  // phase timers (host wall clock; each phase ends on a stream synchronisation)
  auto now = [] { return std::chrono::steady_clock::now(); };
  auto ms = [](std::chrono::steady_clock::time_point a, std::chrono::steady_clock::time_point b) {
    return std::chrono::duration<double, std::milli>(b - a).count();
  };
  drop_pc_graph(L);
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  const auto t_start = now();
  // diagonals of every level (recomputed for each solve, as the reference does)
  if (L.params.preconditioner != 0) {
    for (auto& lv : L.levels) {
      int rc = level_diagonal(h, B, lv);
      if (rc) return rc;
      if (!lv.eig_done) {
        rc = lv.precision ? estimate_eigenvalues<float>(h, B, lv) : estimate_eigenvalues<double>(h, B, lv);
        if (rc) return rc;
      }
    }
  }
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  const auto t_setup = now();
  // rhs = S * compute_rhs
  {
    int rc = clear_acc(h, F);
    if (rc) return rc;
    F.acc_clean = false;
    if (B.plan[0].valid && B.plan[0].nslots >= 0) {
      rc = launch_cell(h, b, 0, nullptr);
      if (rc) return rc;
    }
    rc = finalize(L.rhs, nullptr, nullptr);
    if (rc) return rc;
  }
  // inhomogeneous Dirichlet values g and rhs -= S A_plain g
  bool has_inhom = false;
  for (double v : F.h_dvals) has_inhom |= v != 0.0;
  if (has_inhom) {
    if (h->amr) {
      std::vector<double> gh(n, 0.0);
      for (long long i = 0; i < n; ++i)
        if (F.h_cmap[i] < 0) gh[i] = F.h_dvals[-1 - F.h_cmap[i]];
      amr_fill_hanging(h, F.ncomp, gh.data());  // hanging nodes on Dirichlet faces
      PPF_CUDA(h, cudaMemcpyAsync(L.g, gh.data(), sizeof(double) * n, cudaMemcpyHostToDevice, h->stream));
      PPF_CUDA(h, cudaStreamSynchronize(h->stream));
    } else {
      lift_values_kernel<<<grid_for(n), 256, 0, h->stream>>>(L.g, F.cmap, F.dvals, n);
      PPF_CUDA(h, cudaGetLastError());
      h->all_launches++;
    }
    int rc = outer_apply(L.g, L.q, true, nullptr);
    if (rc) return rc;
    axpby(h, 0, n, -1.0, L.q, 1.0, L.rhs);
  }
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  const auto t_rhs = now();
  // CG on S A x = rhs from the previous homogeneous solution (SolverCG)
  double* x = L.x_hom;
  const double tol = L.params.tolerance * normalization(h, L);
  int rc = outer_apply(x, L.q, false, nullptr);
  if (rc) return rc;
  PPF_CUDA(h, cudaMemcpyAsync(L.r, L.rhs, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
  axpby(h, 0, n, -1.0, L.q, 1.0, L.r);
  double rr;
  rc = dot(h, L, 0, n, L.r, L.r, &rr);
  if (rc) return rc;
  double res = std::sqrt(rr);
  int it = 0;
  bool converged = res < tol;
  if (!converged) {
    rc = conjugate_gradients(
        h, L, n, x, L.r, L.z, L.p, L.q, tol, [&](const double* in, double* out) { return precondition_graphed(h, B, in, out); },
        [&](const double* in, double* out, double* pq) { return outer_apply(in, out, false, pq); }, &it, &res, &converged);
    if (rc) return rc;
  }
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  const auto t_end = now();
  L.last_setup_ms = ms(t_start, t_setup);
  L.last_rhs_ms = ms(t_setup, t_rhs);
  L.last_iterate_ms = ms(t_rhs, t_end);
  L.last_iterations = it;
  L.last_residual = res / normalization(h, L);
  double bb;
  rc = dot(h, L, 0, n, L.rhs, L.rhs, &bb);
  if (rc) return rc;
  L.last_rhs_norm = std::sqrt(bb);
  // solution = x_hom + g, then constraints
  PPF_CUDA(h, cudaMemcpyAsync(F.cur, x, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
  if (has_inhom) axpby(h, 0, n, 1.0, L.g, 1.0, F.cur);
  rc = ppf_apply_constraints(h, f);
  if (rc) return rc;
  rc = check_err(h);
  if (rc) return rc;
  if (!converged) return fail(h, PPF_ERR_NOCONV, "linear solver did not converge before max iterations");
  return PPF_OK;
}

// ------------------------------------------------------------------------------------------
// Newton solves over all fields of a block (NewtonSolver::solve_impl, newton_solver.h:73-156,
// with LinearSolver::do_linear_solve, linear_solver.h:348-402). Block vectors concatenate the
// block's fields in block order on the device.
// ------------------------------------------------------------------------------------------
// dst = S op(src) on the block (which 0: compute_rhs, 1: compute_lhs with src read through
// the homogeneous constraints); constrained rows zero
static int block_op(ppf_handle h, int b, int which, const double* src, double* dst) {
  return ppf_apply_device(h, b, which, src, dst, scaled(h->blocks[b].lin) ? 2 : 0);
}

// Krylov solve of S A x = rhs from the initial guess in x (SolverCG or SolverBicgstab);
// preconditioner: identity, or the fine-level Chebyshev smoother for a single-field block
static int block_krylov(ppf_handle h, int b, const double* rhs, double* x, double tol, int* its, bool* conv) {
  BlockState& B = h->blocks[b];
  LinearState& L = B.lin;
  const long long n = L.block_len;
  double** v = L.kv;
  auto A = [&](const double* in, double* out) { return block_op(h, b, 1, in, out); };
  auto M = [&](const double* in, double* out) -> int {
    if (L.params.preconditioner == 0) {
      PPF_CUDA(h, cudaMemcpyAsync(out, in, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
      return PPF_OK;
    }
    return precondition(h, B, in, out);
  };
  double* r = v[0];
  double* q = v[1];
  int rc = A(x, q);
  if (rc) return rc;
  PPF_CUDA(h, cudaMemcpyAsync(r, rhs, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
  axpby(h, 0, n, -1.0, q, 1.0, r);
  double rr;
  rc = dot(h, L, 0, n, r, r, &rr);
  if (rc) return rc;
  double res = std::sqrt(rr);
  int it = 0;
  *conv = res < tol;
  if (!*conv && L.params.solver_type == 0) {
    rc = conjugate_gradients(
        h, L, n, x, r, v[2], v[3], q, tol, M,
        [&](const double* in, double* out, double* pq) -> int {
          const int e = A(in, out);
          return e ? e : dot_device<double>(h, L, n, in, out, pq);
        },
        &it, &res, conv);
    if (rc) return rc;
  } else if (!*conv) {
    // BiCGStab (van der Vorst), right-preconditioned, with the half-step convergence check
    double* rbar = v[2];
    double* p = v[3];
    double* vv = v[4];
    double* y = v[5];
    double* sv = v[6];
    double* t = v[7];
    double* zz = q;  // q is free from here on
    PPF_CUDA(h, cudaMemcpyAsync(rbar, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
    PPF_CUDA(h, cudaMemsetAsync(p, 0, sizeof(double) * n, h->stream));
    PPF_CUDA(h, cudaMemsetAsync(vv, 0, sizeof(double) * n, h->stream));
    double rho = 1.0, alpha = 1.0, omega = 1.0;
    int restarts = 0;
    // a breakdown (rho or omega zero, or |alpha| > 1e10) restarts from the current iterate with
    // the exact residual, as deal.II's SolverBicgstab does (at most 10 times)
    auto restart = [&]() -> int {
      if ((rc = A(x, q))) return rc;
      PPF_CUDA(h, cudaMemcpyAsync(r, rhs, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
      axpby(h, 0, n, -1.0, q, 1.0, r);
      PPF_CUDA(h, cudaMemcpyAsync(rbar, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
      PPF_CUDA(h, cudaMemsetAsync(p, 0, sizeof(double) * n, h->stream));
      PPF_CUDA(h, cudaMemsetAsync(vv, 0, sizeof(double) * n, h->stream));
      rho = alpha = omega = 1.0;
      return dot(h, L, 0, n, r, r, &rr);
    };
    // a breakdown right at convergence: the exact residual of the restart meets the tolerance
    auto restarted_converged = [&]() -> bool {
      res = std::sqrt(rr);
      return res < tol;
    };
    while (it < L.params.max_iterations) {
      double rho_new;
      if ((rc = dot(h, L, 0, n, rbar, r, &rho_new))) return rc;
      if (rho_new == 0.0 || omega == 0.0) {  // breakdown
        if (++restarts > 10) break;
        if ((rc = restart())) return rc;
        if (restarted_converged()) { *conv = true; break; }
        continue;
      }
      const double beta = (rho_new / rho) * (alpha / omega);
      rho = rho_new;
      axpby(h, 0, n, -omega, vv, 1.0, p);  // p = p - omega v
      axpby(h, 0, n, 1.0, r, beta, p);     // p = r + beta p
      if ((rc = M(p, y))) return rc;
      if ((rc = A(y, vv))) return rc;
      double sigma;
      if ((rc = dot(h, L, 0, n, rbar, vv, &sigma))) return rc;
      if (sigma == 0.0 || !(std::fabs(rho / sigma) <= 1e10)) {  // breakdown
        if (++restarts > 10) break;
        if ((rc = restart())) return rc;
        if (restarted_converged()) { *conv = true; break; }
        continue;
      }
      alpha = rho / sigma;
      PPF_CUDA(h, cudaMemcpyAsync(sv, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
      axpby(h, 0, n, -alpha, vv, 1.0, sv);  // s = r - alpha v
      ++it;
      double ss;
      if ((rc = dot(h, L, 0, n, sv, sv, &ss))) return rc;
      if (!std::isfinite(ss)) return fail(h, PPF_ERR_NAN, "non-finite residual in the linear solve");
      if (std::sqrt(ss) < tol) {
        axpby(h, 0, n, alpha, y, 1.0, x);
        res = std::sqrt(ss);
        *conv = true;
        break;
      }
      if ((rc = M(sv, zz))) return rc;
      if ((rc = A(zz, t))) return rc;
      double tt, ts;
      if ((rc = dot(h, L, 0, n, t, t, &tt))) return rc;
      if ((rc = dot(h, L, 0, n, t, sv, &ts))) return rc;
      omega = tt > 0.0 ? ts / tt : 0.0;
      axpby(h, 0, n, alpha, y, 1.0, x);
      axpby(h, 0, n, omega, zz, 1.0, x);
      PPF_CUDA(h, cudaMemcpyAsync(r, sv, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream));
      axpby(h, 0, n, -omega, t, 1.0, r);  // r = s - omega t
      if ((rc = dot(h, L, 0, n, r, r, &rr))) return rc;
      res = std::sqrt(rr);
      if (res < tol) {
        *conv = true;
        break;
      }
    }
  }
  *its = it;
  return PPF_OK;
}

int newton_solve(ppf_handle h, int b) {
  BlockState& B = h->blocks[b];
  LinearState& L = B.lin;
  if (!L.params_set) {
    ppf_default_linear_params(&L.params);
    L.params_set = true;
  }
  const int nbf = B.desc.n_fields;
  if (!B.plan[0].valid || !B.plan[1].valid)
    return fail(h, PPF_ERR_ARG, "Newton block needs compute_rhs and compute_lhs dependencies");
  if (L.params.preconditioner == 2)
    return fail(h, PPF_ERR_UNSUPPORTED, "Newton blocks: GMG levels would need the current solution on every level");
  if (h->amr && L.params.preconditioner != 0)
    return fail(h, PPF_ERR_UNSUPPORTED, "adaptive meshes: Newton blocks run without a preconditioner");
  if (L.params.preconditioner == 1 && nbf != 1)
    return fail(h, PPF_ERR_UNSUPPORTED, "Newton blocks: the Chebyshev preconditioner needs a single-field block");
  if (L.params.preconditioner == 1 && !L.initialized) {
    int rc = init_linear(h, b);
    if (rc) return rc;
  }
  long long off[PPF_MAX_FIELDS + 1] = {0};
  for (int i = 0; i < nbf; ++i) off[i + 1] = off[i] + h->fields[B.desc.field_indices[i]].len;
  const long long n = off[nbf];
  if (L.block_len != n || L.mesh_version != h->mesh_version) {
    L.mesh_version = h->mesh_version;
    cudaFree(L.newton_update);
    for (double*& p : L.kv) cudaFree(p);
    PPF_CUDA(h, cudaMalloc(&L.newton_update, sizeof(double) * n));
    PPF_CUDA(h, cudaMemsetAsync(L.newton_update, 0, sizeof(double) * n, h->stream));
    for (double*& p : L.kv) PPF_CUDA(h, cudaMalloc(&p, sizeof(double) * n));
    cudaFree(L.rhs);  // a Newton block's rhs vector holds its block residual
    PPF_CUDA(h, cudaMalloc(&L.rhs, sizeof(double) * n));
    if (const int rc = ensure_scalars(h, L)) return rc;
    L.block_len = n;
  }
  double* R = L.rhs;
  // start from the previous solution (old_1 where the field keeps one)
  for (int i = 0; i < nbf; ++i) {
    FieldState& F = h->fields[B.desc.field_indices[i]];
    if (F.n_old > 0)
      PPF_CUDA(h, cudaMemcpyAsync(F.cur, F.old[0], sizeof(double) * F.len, cudaMemcpyDeviceToDevice, h->stream));
  }
  const double norm = normalization(h, L, nbf);
  const double tol = L.newton_tolerance * norm;
  const double lin_tol = L.params.tolerance * norm;
  double l2 = -1.0;
  int iter = 0, lin_total = 0;
  while (iter < L.newton_max_iterations) {
    for (int i = 0; i < nbf; ++i) {
      int rc = ppf_apply_constraints(h, B.desc.field_indices[i]);
      if (rc) return rc;
    }
    int rc = block_op(h, b, 0, nullptr, R);
    if (rc) return rc;
    double rr;
    if ((rc = dot(h, L, 0, n, R, R, &rr))) return rc;
    l2 = std::sqrt(rr);
    if (!std::isfinite(l2)) return fail(h, PPF_ERR_NAN, "non-finite Newton residual");
    if (!(l2 > tol)) break;
    if (L.params.preconditioner == 1) {  // fine-level diagonal of the current Jacobian
      MGLevel& fine = L.levels.back();
      if ((rc = level_diagonal(h, B, fine))) return rc;
      fine.eig_done = false;
      if ((rc = estimate_eigenvalues<double>(h, B, fine))) return rc;
    }
    int its = 0;
    bool conv = false;
    if ((rc = block_krylov(h, b, R, L.newton_update, lin_tol, &its, &conv))) return rc;
    lin_total += its;
    for (int i = 0; i < nbf; ++i) {
      FieldState& F = h->fields[B.desc.field_indices[i]];
      axpby(h, 0, F.len, L.newton_step, L.newton_update + off[i], 1.0, F.cur);
    }
    ++iter;
  }
  L.last_newton_iterations = iter;
  L.last_newton_linear_iterations = lin_total;
  L.last_newton_residual = l2 / norm;
  int rc = check_err(h);
  if (rc) return rc;
  if (iter >= L.newton_max_iterations) return fail(h, PPF_ERR_NOCONV, "Newton solver did not converge");
  return PPF_OK;
}

void free_linear(LinearState& L) {
  drop_pc_graph(L);
  for (double* p : {L.rhs, L.g, L.x_hom, L.r, L.p, L.q, L.z, L.inv_diag, L.partial, L.scal, L.newton_update}) cudaFree(p);
  cudaFreeHost(L.h_scal);
  for (auto& ev : L.scal_ev)
    if (ev) cudaEventDestroy(ev);
  for (double*& p : L.kv) {
    cudaFree(p);
    p = nullptr;
  }
  L.newton_update = nullptr;
  L.block_len = 0;
  for (auto& lv : L.levels) {
    for (auto& ev : lv.fx_ev)
      if (ev) cudaEventDestroy(ev);
    cudaFree(lv.cmap);
    for (void* p : {lv.invm_sqrt, lv.inv_diag, lv.tables, lv.acc, lv.acc2, lv.x, lv.b, lv.r, lv.w0, lv.w1})
      cudaFree(p);
    for (int d = 0; d < 3; ++d) {
      cudaFree(lv.p_ptr[d]);
      cudaFree(lv.p_col[d]);
      cudaFree(lv.p_val[d]);
      cudaFree(lv.r_ptr[d]);
      cudaFree(lv.r_col[d]);
      cudaFree(lv.r_val[d]);
    }
  }
  L.levels.clear();
  L.initialized = false;
}

}  // namespace ppf

using namespace ppf;

extern "C" {

int ppf_default_linear_params(ppf_linear_params* p) {
  if (!p) return PPF_ERR_ARG;
  p->tolerance_type = 0;
  p->tolerance = 1e-10;
  p->max_iterations = 100;
  p->preconditioner = 0;
  p->mg_depth = 1;
  p->smoother_degree = 5;
  p->smoothing_range = 15.0;
  p->eig_cg_iterations = 10;
  p->mixed_precision = 0;
  p->solver_type = 0;
  return PPF_OK;
}

int ppf_set_linear_params(ppf_handle h, int b, const ppf_linear_params* p) {
  if (!h || !p || b < 0 || b >= (int)h->blocks.size()) return PPF_ERR_ARG;
  if (p->preconditioner < 0 || p->preconditioner > 2 || p->smoother_degree < 1 || p->mg_depth < 1 ||
      p->max_iterations < 1 || p->eig_cg_iterations < 1 || p->smoothing_range <= 1.0 || p->solver_type < 0 ||
      p->solver_type > 1)
    return fail(h, PPF_ERR_ARG, "invalid linear solver parameters");
  LinearState& L = h->blocks[b].lin;
  if (L.initialized) return fail(h, PPF_ERR_ARG, "linear parameters are fixed after the first solve");
  if (p->mixed_precision && h->model_obj_f32.empty())
    return fail(h, PPF_ERR_UNSUPPORTED, "mixed precision needs an FP32 instance of the operator");
  L.params = *p;
  L.params_set = true;
  return PPF_OK;
}

int ppf_linear_stats(ppf_handle h, int b, double* init_ms, double* setup_ms, double* rhs_ms, double* iterate_ms) {
  if (!h || b < 0 || b >= (int)h->blocks.size()) return PPF_ERR_ARG;
  const LinearState& L = h->blocks[b].lin;
  if (init_ms) *init_ms = L.last_init_ms;
  if (setup_ms) *setup_ms = L.last_setup_ms;
  if (rhs_ms) *rhs_ms = L.last_rhs_ms;
  if (iterate_ms) *iterate_ms = L.last_iterate_ms;
  return PPF_OK;
}

int ppf_set_newton_params(ppf_handle h, int b, int max_iterations, double tolerance, double step_length) {
  if (!h || b < 0 || b >= (int)h->blocks.size() || max_iterations < 1 || !(tolerance >= 0.0) || !(step_length > 0.0))
    return PPF_ERR_ARG;
  LinearState& L = h->blocks[b].lin;
  L.newton_max_iterations = max_iterations;
  L.newton_tolerance = tolerance;
  L.newton_step = step_length;
  return PPF_OK;
}

int ppf_newton_solve(ppf_handle h, int b, int* newton_iterations, int* linear_iterations, double* residual) {
  if (!h || b < 0 || b >= (int)h->blocks.size()) return PPF_ERR_ARG;
  if (h->blocks[b].desc.solve_type != PPF_NEWTON) return fail(h, PPF_ERR_ARG, "block is not Newton");
  const int rc = newton_solve(h, b);
  const LinearState& L = h->blocks[b].lin;
  if (newton_iterations) *newton_iterations = L.last_newton_iterations;
  if (linear_iterations) *linear_iterations = L.last_newton_linear_iterations;
  if (residual) *residual = L.last_newton_residual;
  return rc;
}

int ppf_linear_solve(ppf_handle h, int b, int* iterations, double* residual) {
  if (!h || b < 0 || b >= (int)h->blocks.size()) return PPF_ERR_ARG;
  if (h->blocks[b].desc.solve_type != PPF_LINEAR) return fail(h, PPF_ERR_ARG, "block is not Linear");
  const int rc = linear_solve(h, b);
  if (iterations) *iterations = h->blocks[b].lin.last_iterations;
  if (residual) *residual = h->blocks[b].lin.last_residual;
  return rc;
}

int ppf_lhs_diagonal(ppf_handle h, int b, double* out) {
  if (!h || !out || b < 0 || b >= (int)h->blocks.size()) return PPF_ERR_ARG;
  BlockState& B = h->blocks[b];
  if (!B.lin.initialized) {
    int rc = init_linear(h, b);
    if (rc) return rc;
  }
  MGLevel& fine = B.lin.levels.back();
  if (fine.precision) return fail(h, PPF_ERR_ARG, "diagonal export needs an FP64 fine level");
  int rc = level_diagonal(h, B, fine);
  if (rc) return rc;
  std::vector<double> inv(fine.len);
  PPF_CUDA(h, cudaMemcpyAsync(inv.data(), fine.inv_diag, sizeof(double) * fine.len, cudaMemcpyDeviceToHost, h->stream));
  PPF_CUDA(h, cudaStreamSynchronize(h->stream));
  for (long long i = 0; i < fine.len; ++i) out[i] = 1.0 / inv[i];
  return check_err(h);
}

}  // extern "C"
