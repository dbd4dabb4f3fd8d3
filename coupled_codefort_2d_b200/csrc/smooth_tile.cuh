// smooth_tile.cuh -- several sweeps of the PCD's velocity smoother
// (solve_helmholtz_{u,v}, mod_subsolvers.f90:252-372: damped Jacobi; or the
// red-black SOR extension) of one component of a wall-bounded case per launch.
//
// A pass (a sweep of Jacobi, a colour of SOR) is a few hundred cycles; a launch
// per sweep is bound by launch latency and by reading six fields again.  A CTA
// takes a region of ST_SX columns and rows, keeps a ring of RING faces around
// its tile, and runs up to RING passes on it: the outermost faces become
// invalid one by one, the tile does not.  A thread owns a column strip of RPT
// rows whose values, couplings, diagonals and right-hand sides stay in
// registers (all loads issued together); shared memory holds only u, for the
// east, west and strip-end neighbours.  Every thread runs the same
// straight-line passes: what lies outside the valid part is computed and not
// used.  Odd columns start one row higher, so that row r of every strip has
// one colour and a pass of SOR updates static registers.
// Each update is jacobi_u_vals / jacobi_v_vals's formula with its operand order
// on the same neighbours, the division as the exact quotient from the
// diagonal's reciprocal (pcg_exchange.cuh), so the bits are those of one sweep
// per launch.  Periodic cases refresh their halo between passes and keep the
// one-sweep launches.
// Bound by its passes' serial chain (one stencil and one quotient per face and a
// barrier, about 0.25 us FP32) and, from 512^2 up, by L2.  B200, us, six sweeps
// of one component, a launch per sweep (SOR) or the staged six-sweep tiles
// (Jacobi) before / now:
//   SOR     128^2 FP32 33.3 / 7.8   256^2 33.4 / 10.2   320x640 38.3 / 15.4   2048^2 390 / 173
//           128^2 FP64 34.4 / 11.2  256^2 34.3 / 14.7   320x640 42.2 / 26.1   2048^2 581 / 375
//   Jacobi  128^2 FP32 13.6 / 7.6   256^2 13.8 / 7.9    320x640 18.1 / 11.6   2048^2 142 / 132
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "pcg_exchange.cuh"

namespace fugu {

enum { SMOOTH_JACOBI = 0, SMOOTH_RBSOR = 1 };
constexpr int ST_SX = 64, ST_TY = 8, ST_RPT = 4, ST_TPB = ST_SX * ST_TY;  // region columns, strips per column, their rows
// the tile inside the region (even sizes and offsets, so that colours line up)
__host__ __device__ constexpr int st_tx(int ring) { return ST_SX - 2 * ring; }
__host__ __device__ constexpr int st_ty(int ring) { return ST_TY * ST_RPT - 2 * ring - 2; }

// the exact quotient in FP32 (as quotient() in FP64)
__device__ __forceinline__ float quotient(float a, float b, float y) {
  const float q = a * y;
  return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}
// Whether quotient(a, b, 1 / b) may be taken for a / b, its remainder exact
// and nothing over- or underflowing: b within smooth_b, a +0 or |a| in
// [2^-80, 2^80) (FP32), [2^-480, 2^480) (FP64); not for infinities, NaN and -0
// (its quotient would be +0).
__device__ __forceinline__ bool smooth_a(float a) {
  const unsigned u = __float_as_uint(a), w = u * 2u;
  return w - (47u << 24) < (160u << 24) || u == 0u;
}
__device__ __forceinline__ bool smooth_a(double a) {
  const unsigned hi = (unsigned)__double2hiint(a), w = hi * 2u;
  return w - (543u << 21) < (960u << 21) || (hi | (unsigned)__double2loint(a)) == 0u;
}
template <typename T>
__device__ __forceinline__ bool smooth_b(T b) { return b >= T(0x1p-40) && b <= T(0x1p40); }

template <typename T>
struct SmoothArgs {
  Geo g;
  int passes;    // <= RING
  const T* uin;  // null: zero everywhere
  T* uout;       // the whole box
  const T *rhs, *rho, *kap, *zeta, *eta, *pen;
  T dt, om;
  const int* active;
};

// COMP: 0 u, 1 v
template <typename T, int MODE, int COMP, int RING>
__global__ void __launch_bounds__(ST_TPB) k_smooth_tile(SmoothArgs<T> a) {
  if (a.active && !*a.active) return;
  constexpr int RPT = ST_RPT;
  static_assert(RPT % 2 == 0 && RING % 2 == 0, "colours line up");
  constexpr bool SOR = MODE == SMOOTH_RBSOR;
  constexpr int W = ST_SX + 2, H = ST_TY * RPT + 3;  // one slot of padding around
  __shared__ T S[SOR ? 1 : 2][H * W];
  const Geo g = a.g;
  const int nx = g.nx, ny = g.ny, t = threadIdx.x, tx = t % ST_SX;
  const int ii = (int)blockIdx.x * st_tx(RING) - RING + tx, i = ii - 2;
  const int row0 = (t / ST_SX) * RPT + (tx & 1);  // region row of the strip's first face
  const int jj0 = (int)blockIdx.y * st_ty(RING) - (RING + 2) + row0, j0 = jj0 - 2;
  const T ix2 = T(g.idx2), iy2 = T(g.idy2), om = a.om;
  for (int q = t; q < H * W; q += ST_TPB) {
    S[0][q] = T(0);
    if constexpr (!SOR) S[1][q] = T(0);
  }
  // ---- the strip's faces
  T u[RPT], rh[RPT], cE[RPT], cW[RPT], cN[RPT], cS0 = T(0), dg[RPT], rc[RPT];
  unsigned k1 = 0u, k2 = 0u, k3 = 0u;  // owned faces, wall faces, faces that take the division
  const bool in_x = ii >= 0 && ii < g.P;
  auto inbox = [&](int r) { return in_x && jj0 + r >= 0 && jj0 + r < g.R; };
  auto owned = [&](int r) {
    const int j = j0 + r;
    return COMP == 0 ? (j >= 1 && j <= ny && i >= 1 && i <= nx - 1) : (i >= 1 && i <= nx && j >= 1 && j <= ny - 1);
  };
  {
    T kp[RPT + 1], kx[RPT], z0[RPT + 1], e0[RPT + 1], z1[RPT], e1[RPT], rho[RPT], pn[RPT];
    // comp 0: kap at (i, j), (i + 1, j); zeta, eta at (i, j - 1), (i, j)
    // comp 1: kap at (i, j), (i, j + 1); zeta, eta at (i, j), (i - 1, j)
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int k = ii + (jj0 + r) * g.P;
      const bool b = inbox(r), o = b && owned(r);
      u[r] = b && a.uin ? a.uin[k] : T(0);
      rh[r] = b ? a.rhs[k] : T(0);
      rho[r] = o ? a.rho[k] : T(1);
      pn[r] = o && a.pen ? a.pen[k] : T(0);
      kp[r] = o ? a.kap[k] : T(0);
      kx[r] = o ? (COMP == 0 ? a.kap[k + 1] : a.kap[k + g.P]) : T(0);
      z0[r] = o ? a.zeta[k] : T(0);
      e0[r] = o ? a.eta[k] : T(0);
      z1[r] = o ? (COMP == 0 ? a.zeta[k - g.P] : a.zeta[k - 1]) : T(0);
      e1[r] = o ? (COMP == 0 ? a.eta[k - g.P] : a.eta[k - 1]) : T(0);
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const T near = (z0[r] - e0[r]) * (COMP == 0 ? iy2 : ix2), far = (z1[r] - e1[r]) * (COMP == 0 ? iy2 : ix2);
      const T ka = kp[r] * (COMP == 0 ? ix2 : iy2), kb = kx[r] * (COMP == 0 ? ix2 : iy2);
      cE[r] = COMP == 0 ? kb : near;
      cW[r] = COMP == 0 ? ka : far;
      cN[r] = COMP == 0 ? near : kb;
      const T cS = COMP == 0 ? far : ka;
      if (r == 0) cS0 = cS;
      // (inside the strip cS of a face is cN of the face below when both are owned)
      T d = (rho[r] / a.dt) + cE[r] + cW[r] + cN[r] + cS;
      if (a.pen) d = d + pn[r];
      dg[r] = d;
      if (inbox(r) && owned(r)) {
        if (d > T(1.0e-15)) k1 |= 1u << r;
        if (!smooth_b(d)) k3 |= 1u << r;
      } else {
        dg[r] = T(1);
        const int j = j0 + r;
        if (inbox(r) && (COMP == 0 ? (j >= 1 && j <= ny && (i == 0 || i == nx)) : (i >= 1 && i <= nx && (j == 0 || j == ny))))
          k2 |= 1u << r;
        // an unowned face still carries the coupling its upper neighbour reads
        if (r + 1 < RPT && inbox(r + 1) && owned(r + 1))
          cN[r] = COMP == 0 ? (z1[r + 1] - e1[r + 1]) * iy2 : kp[r + 1] * iy2;
      }
      rc[r] = T(1) / dg[r];
    }
  }
  const int at = (row0 + 1) * W + tx + 1;  // slot of the strip's first face
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RPT; ++r) S[0][at + r * W] = u[r];
  __syncthreads();
  int cur = 0;
  for (int s = 0; s < a.passes; ++s) {
    const T* P = S[SOR ? 0 : cur];
    T* Nx = S[SOR ? 0 : cur ^ 1];
    const T below = P[at - W], above = P[at + RPT * W];
    // numerators of the pass's faces, their quotients, then the new values
    constexpr int N = SOR ? RPT / 2 : RPT;
    const int r0 = SOR ? s & 1 : 0;
    T num[N], quo[N];
    auto pass = [&](auto odd) {
      constexpr int R0 = decltype(odd)::value, DR = SOR ? 2 : 1;
      bool div = false;
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int r = R0 + DR * e, c = at + r * W;
        const T nn = r + 1 < RPT ? u[r + 1 < RPT ? r + 1 : r] : above, so = r ? u[r ? r - 1 : 0] : below;
        const T cS = r ? cN[r ? r - 1 : 0] : cS0;
        num[e] = rh[r] + madd(cS, so, madd(cN[r], nn, madd(cW[r], P[c - 1], cE[r] * P[c + 1])));
        quo[e] = quotient(num[e], dg[r], rc[r]);
        div |= !smooth_a(num[e]) || ((k3 >> r) & 1u);
      }
      if (div) {
#pragma unroll 1
        for (int e = 0; e < N; ++e) {
          T a = T(0), d = T(1);
#pragma unroll
          for (int f = 0; f < N; ++f)
            if (f == e) {
              a = num[f];
              d = dg[R0 + DR * f];
            }
          a = a / d;
#pragma unroll
          for (int f = 0; f < N; ++f)
            if (f == e) quo[f] = a;
        }
      }
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int r = R0 + DR * e;
        const T val = madd(T(1) - om, u[r], om * quo[e]);
        u[r] = (k1 >> r) & 1u ? val : (k2 >> r) & 1u ? rh[r] : u[r];
        Nx[at + r * W] = u[r];
      }
    };
    if (r0 == 0) pass(std::integral_constant<int, 0>{});
    else if constexpr (SOR) pass(std::integral_constant<int, 1>{});
    if constexpr (!SOR) cur ^= 1;
    __syncthreads();
  }
  // the tile, every element of it
  if (!in_x || tx < RING || tx >= ST_SX - RING) return;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int q = row0 + r;
    if (q >= RING + 2 && q < RING + 2 + st_ty(RING) && jj0 + r < g.R) a.uout[ii + (jj0 + r) * g.P] = u[r];
  }
}
inline dim3 smooth_grid(const Geo& g, int ring) {
  return dim3((g.P + st_tx(ring) - 1) / st_tx(ring), (g.R + st_ty(ring) - 1) / st_ty(ring));
}
inline int smooth_ctas(const Geo& g, int ring) {
  const dim3 d = smooth_grid(g, ring);
  return (int)(d.x * d.y);
}
template <typename T, int MODE, int COMP>
const void* smooth_ring_fn(int ring) {
  return ring == 2   ? (const void*)k_smooth_tile<T, MODE, COMP, 2>
         : ring == 4 ? (const void*)k_smooth_tile<T, MODE, COMP, 4>
         : ring == 6 ? (const void*)k_smooth_tile<T, MODE, COMP, 6>
                     : (const void*)k_smooth_tile<T, MODE, COMP, 12>;
}
template <typename T>
const void* smooth_fn(int mode, int comp, int ring) {
  if (mode == SMOOTH_JACOBI)
    return comp == 0 ? smooth_ring_fn<T, SMOOTH_JACOBI, 0>(ring) : smooth_ring_fn<T, SMOOTH_JACOBI, 1>(ring);
  return comp == 0 ? smooth_ring_fn<T, SMOOTH_RBSOR, 0>(ring) : smooth_ring_fn<T, SMOOTH_RBSOR, 1>(ring);
}

}  // namespace fugu
