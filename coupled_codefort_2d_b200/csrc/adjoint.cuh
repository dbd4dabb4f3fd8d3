// adjoint.cuh -- the transpose of the coupled operator (extension, no
// counterpart in the reference): the stencil of the linear map the Krylov
// solvers see, x_owned -> (A . BC(x))_owned (matvec_coupled,
// mod_operators.f90:341-443, after apply_velocity_bcs, :254-333), is measured
// by probing it with coloured unit vectors, then applied transposed by a
// gather kernel (a fixed summation order, no atomics).
//
// Every entry of a row couples unknowns at most 2 cells away in i and j
// (the 11-point coupling plus ghost values that mirror or wrap interior
// values); unit vectors of one colour are at least 5 cells apart (or the
// period divides the periodic extent), so each probe result entry belongs to
// exactly one column.  A probe entry that no column within reach can explain
// is counted as an error instead of being stored.
//
// Stencil storage: val[((cr * 3 + cc) * 25 + (di + 2) * 5 + (dj + 2)) * n + at(i, j)]
// = A[(cr, i, j), (cc, i + di, j + dj)] with component indices 0 = u, 1 = v,
// 2 = p and the column index wrapped in periodic directions.
#pragma once

#include "kernels.cuh"

namespace fugu {

constexpr int ADJ_SLOTS = 225;  // 3 row components x 3 column components x 5 x 5 offsets

// owned unknowns of a component (the coupled_dot index set)
__device__ __forceinline__ bool adj_owned(const Geo& g, int comp, int i, int j) {
  const int i1 = comp == 0 ? g.imax() : g.nx;
  const int j1 = comp == 1 ? g.jmax() : g.ny;
  return i >= 1 && i <= i1 && j >= 1 && j <= j1;
}
__device__ __forceinline__ int adj_wrap(int i, int len, int periodic) {
  if (!periodic) return i;
  return ((i - 1) % len + len) % len + 1;
}

// unit entries of component cc at owned (i, j) with colour ((i-1) % qx, (j-1) % qy) == (a, b)
__global__ void k_adj_probe_set(Geo g, double* X, long n, int cc, int qx, int qy, int a, int b) {
  FUGU_BOX_IJ
  if (adj_owned(g, cc, i, j) && (i - 1) % qx == a && (j - 1) % qy == b) X[cc * n + g.at(i, j)] = 1.0;
}

// store the probe result Y of colour (cc, a, b) into the stencil; grid z: the
// row component.  The column that explains an entry is the one of the colour's
// lattice within 2 cells, found per direction.
__global__ void k_adj_probe_collect(Geo g, const double* Y, long n, int cc, int qx, int qy, int a, int b,
                                    double* val, unsigned int* err) {
  FUGU_BOX_IJ
  const int cr = blockIdx.z;
  if (!adj_owned(g, cr, i, j)) return;
  const double y = Y[cr * n + k];
  // the colour's period is at least 5, so at most one offset per direction fits
  int di = 3, dj = 3;
#pragma unroll
  for (int d = -2; d <= 2; ++d) {
    const int ic = adj_wrap(i + d, g.nx, g.px), jc = adj_wrap(j + d, g.ny, g.py);
    const int i1 = cc == 0 ? g.imax() : g.nx, j1 = cc == 1 ? g.jmax() : g.ny;
    if (di == 3 && ic >= 1 && ic <= i1 && (ic - 1) % qx == a) di = d;
    if (dj == 3 && jc >= 1 && jc <= j1 && (jc - 1) % qy == b) dj = d;
  }
  if (di < 3 && dj < 3) val[(long)((cr * 3 + cc) * 25 + (di + 2) * 5 + (dj + 2)) * n + k] = y;
  else if (y != 0.0) atomicAdd(err, 1u);
}

// y = S A^T S x over the owned unknowns (S = diag(1, 1, sp): sp = -1 flips the
// pressure block, 1 gives plain A^T); every other entry of y is set to zero.
// Grid z: the component of y.  An entry is 75 products of a stencil value read
// once and a neighbour's x: the stencil (225 values per point) is what has to
// come from L2 or HBM, and a thread's loads of one row component (25 pairs) are
// issued together; one thread for the three components with a load per round
// took 50 us at 80 x 160.  The products are added in one fixed order.
__global__ void __launch_bounds__(256) k_adj_apply_t(Geo g, long n, const double* __restrict__ val, const double* __restrict__ x,
                                                     double* __restrict__ y, double sp, const int* active,
                                                     unsigned long long* matvecs) {
  if (active && !*active) return;
  FUGU_BOX_IJ
  const int cc = blockIdx.z;
  if (matvecs && blockIdx.x == 0 && blockIdx.y == 0 && cc == 0 && threadIdx.x == 0 && threadIdx.y == 0) ++*matvecs;
  const long e = cc * n + k;
  if (!adj_owned(g, cc, i, j)) {
    y[e] = 0.0;
    return;
  }
  int ir[5], jr[5];
#pragma unroll
  for (int d = 0; d < 5; ++d) {
    ir[d] = adj_wrap(i - (d - 2), g.nx, g.px);
    jr[d] = adj_wrap(j - (d - 2), g.ny, g.py);
  }
  double s = 0.0;
#pragma unroll
  for (int cr = 0; cr < 3; ++cr) {
    const double sr = cr == 2 ? sp : 1.0;
    const double* v = val + (long)(cr * 3 + cc) * 25 * n;
    double a[25], b[25];
#pragma unroll
    for (int q = 0; q < 25; ++q) {
      const bool on = adj_owned(g, cr, ir[q / 5], jr[q % 5]);
      const long p = on ? g.at(ir[q / 5], jr[q % 5]) : k;
      a[q] = on ? v[(long)q * n + p] : 0.0;
      b[q] = on ? x[cr * n + p] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 25; ++q)
      if (adj_owned(g, cr, ir[q / 5], jr[q % 5])) s += a[q] * (sr * b[q]);
  }
  y[e] = (cc == 2 ? sp : 1.0) * s;
}

// negate the pressure block of a triple (applies S)
__global__ void k_adj_flip_p(long n, double* x) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
    x[2 * n + q] = -x[2 * n + q];
}

}  // namespace fugu
