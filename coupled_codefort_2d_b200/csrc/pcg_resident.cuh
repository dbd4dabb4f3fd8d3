// pcg_resident.cuh -- the PCG pressure Poisson solve (solve_poisson_pressure,
// mod_subsolvers.f90:32-246) with the whole problem resident on chip: CTA b
// owns the cell rows [b rows_per, (b + 1) rows_per), every vector lives in
// registers and the stencil's vector in shared memory.
//
// What bounds a PCG iteration here is latency, not bytes: the dependent chain
// is sums -> scalars -> update -> stencil -> sums, and most of it is the
// exchange of the sums between the CTAs.  So
//   - a thread owns segments of W = 16 / sizeof(T) consecutive cells of a row:
//     shared memory is read with 16-byte loads, a CTA needs few warps, and
//     the sums need few shuffles;
//   - one all-reduce carries the sums and the boundary rows together and
//     needs no barrier, only the arrival of the data (pcg_exchange.cuh);
//   - the reciprocals of the next scalars are formed while it is in flight.
// A neighbour's row needs one vector per iteration only: the rest of a halo
// row's recurrence is repeated locally from it with the owner's expressions,
// which gives the owner's bits.
//
// FP64 keeps the reference's recurrence (two all-reduces per iteration), in a
// thread-block cluster or over the whole device; its element-wise
// expressions and error-free sums give the oracle's bits whatever the
// partition.  FP32 over the whole device is k_pcg1's single-reduction
// iteration with its expressions and error-free sums, for the grids that do
// not fit a cluster, so that a case has the same states alone (here) and in a
// batch (k_pcg1).  FP32 in a cluster sums in plain double, where the order
// matters, and has its own kernel (pcg_cluster.cuh).
//
// Measured on a B200, us per iteration before (cluster barriers, k_pcg / k_pcg1's grid
// barriers) and now:
//   FP64 cluster  64 x 64 3.73 -> 2.14, 128 x 128 4.15 -> 2.82, 203 x 125 4.98 -> 4.01
//   FP64 grid     256 x 256 7.79 -> 4.39, 320 x 640 12.5 -> 6.05, 512 x 512 13.7 -> 6.17
//   FP32 grid     320 x 640 8.44 -> 3.68, 512 x 512 9.29 -> 3.70,
//                 768 x 768 12.8 -> 7.83, 1024 x 1024 17.0 -> 12.0
#pragma once

#include <type_traits>

#include "pcg_exchange.cuh"
#include "persistent.cuh"

namespace fugu {

template <typename T>
struct PcgResArgs {
  Geo g;
  const T* rhs;
  const T* cx;
  const T* cy;
  const T* dinv;
  T* phi;
  PcgOut* out;
  const int* active;
  double tol;
  int max_iter;
  int phi_zero;
  int timed;
  int rows_per;
  // grid exchange only
  Exchange x;
  int* err;                 // the launch's error flag (GridSync::error)
  unsigned int spin_limit;  // 0: FUGU_SPIN_LIMIT / 16 (a poll is a global round trip)
  int extra_arrivals;       // failure-detection test: wait for a slot nobody writes
  CxLimit wait;             // cluster exchange only
};

// Kernel shapes: segments per thread and largest block, by the segments of
// a CTA.  More segments per thread mean fewer warps to reduce over but a
// longer serial part; compared on a B200 (us per iteration, with a slower merge
// of the received sums than now): FP64 in 16 CTAs,
// 128 x 128 (512 segments) 2 x 256 2.81, 1 x 512 2.93; 128 x 256 (1024)
// 4 x 256 3.96, 2 x 512 4.01; FP32 over 128 CTAs, 320 x 640 (400) 2 x 256
// 4.22, 1 x 512 4.93; 768 x 768 (1152) 3 x 512 8.5, 4 x 512 10.5.
// PCGR_TALL is for narrow boxes in a cluster only (FP64, 4,096 cells per CTA and
// nx odd or 4): their half-empty last segments need a fifth one per thread and
// their rows packed coefficients.
constexpr int PCGR_SHAPES = 5, PCGR_TALL = 5;
struct PcgrShape {
  int seg, tpb;
};
__host__ __device__ constexpr PcgrShape pcgr_shape(int s) {
  return s == 0   ? PcgrShape{1, 256}
         : s == 1 ? PcgrShape{2, 256}
         : s == 2 ? PcgrShape{4, 256}
         : s == 3 ? PcgrShape{3, 512}
         : s == 4 ? PcgrShape{4, 512}
                  : PcgrShape{5, 512};
}

// coefficients in registers where they fit beside the vectors
template <typename T>
__host__ __device__ constexpr bool pcgr_reg_coefs(int seg, int tpb) {
  return seg * tpb <= 1024;
}
// row pitch in shared memory: a vector of padding either side holds the
// ghost columns
template <typename T>
__host__ __device__ inline int pcgr_pitch(int nx) {
  const int W = 16 / (int)sizeof(T);
  return ((nx + W - 1) / W + 2) * W;
}
// pitch of the coefficients' rows there: padded like the vector's, or (five
// segments per thread) packed, with one vector of padding for cx's column 0
template <typename T>
__host__ __device__ constexpr int pcgr_pad(int seg, bool is_cx) {
  const int W = 16 / (int)sizeof(T);
  return seg < pcgr_shape(PCGR_TALL).seg ? 2 * W : is_cx ? W : 0;
}
// shared memory (elements of T): the stencil's vector with its two halo
// rows, the received halo rows (two parities), their recurrence in the
// single-reduction form (s, r and the inverse diagonal), and the
// coefficients when they are not in registers
template <typename T>
__host__ __device__ inline long pcgr_smem_elems(int nx, int rows_per, int seg, int tpb) {
  const int W = 16 / (int)sizeof(T);
  const long p = pcgr_pitch<T>(nx), px = p - 2 * W + pcgr_pad<T>(seg, true), py = p - 2 * W + pcgr_pad<T>(seg, false);
  long n = (rows_per + 2) * p + 4 * p;
  if (sizeof(T) == 4) n += 6 * p;
  if (!pcgr_reg_coefs<T>(seg, tpb)) n += rows_per * px + (2 * rows_per + 1) * py;
  return n;
}

// running error-free sum of a thread's terms
struct RSum {
  DD v{0.0, 0.0};
  __device__ __forceinline__ void add(double x) { dd_add(v, x); }
};

// The solve of one case by the CTAs rank 0 .. G - 1 of a cluster (CL) or a
// cooperative grid.  SEG segments per thread, TPB threads at most.
template <typename T, int SEG, int TPB, bool CL>
__device__ __forceinline__ void pcgr_body(const PcgResArgs<T>& a, const int rank, const int G) {
  constexpr int W = VecW<T>::value;
  constexpr bool RC = pcgr_reg_coefs<T>(SEG, TPB);
  constexpr bool ONE = sizeof(T) == 4;  // the single-reduction iteration
  static_assert(!(ONE && CL), "FP32 in a cluster: pcg_cluster.cuh");
  const Geo g = a.g;
  const int nx = g.nx, ny = g.ny, rp = a.rows_per;
  const int j0 = 1 + rank * rp, R = min(rp, ny - rank * rp);
  const int nseg = (nx + W - 1) / W, P = (nseg + 2) * W;
  const bool closed = !g.px && !g.py;
  const bool has_bot = rank > 0 || g.py, has_top = rank < G - 1 || g.py;
  const int below = rank > 0 ? rank - 1 : G - 1, above = rank < G - 1 ? rank + 1 : 0;
  const int tid = threadIdx.x, tpb = blockDim.x;

  extern __shared__ __align__(16) unsigned char pcgr_smem[];
  T* us = reinterpret_cast<T*>(pcgr_smem);  // row 0: below the CTA, 1..R own, R + 1 above
  T* hw = us + (rp + 2) * P;                // received halo rows [parity][bottom, top]
  T* hs = hw + 4 * P;                       // single reduction: s, r and dinv of the halo rows
  T* hr = hs + 2 * P;
  T* hd = hr + 2 * P;
  T* cxs = ONE ? hd + 2 * P : hs;           // (only without RC) cx, cy (rows j0 - 1 ..), dinv
  // their pitches and the slot of column 1
  constexpr bool PACK = pcgr_pad<T>(SEG, false) == 0;
  const int PX = PACK ? P - W : P, PY = PACK ? P - 2 * W : P;
  constexpr int Y1 = PACK ? 0 : W;
  T* cys = cxs + rp * PX;
  T* dis = cys + (rp + 1) * PY;
  __shared__ std::conditional_t<CL, ClusterXSmem<TPB>, GridXSmem<TPB>> xs;
  auto x = [&] {
    if constexpr (CL) return ClusterX<TPB, true>(xs, rank, G, a.wait);
    else return GridX<TPB>(xs, a.x, rank, G, a.extra_arrivals, a.spin_limit, a.err);
  }();

  // ---- the thread's segments
  int row[SEG], i0[SEG], nv[SEG];
#pragma unroll
  for (int k = 0; k < SEG; ++k) {
    const int q = tid + k * tpb;
    const bool on = q < R * nseg;
    row[k] = on ? q / nseg : 0;
    i0[k] = on ? (q % nseg) * W + 1 : 1;
    nv[k] = on ? min(W, nx - i0[k] + 1) : 0;
  }
#define PCGR_SEGS _Pragma("unroll") for (int k = 0; k < SEG; ++k)
#define PCGR_E _Pragma("unroll") for (int e = 0; e < W; ++e)
  // index of column i0[k] in row lr of a pitched array
  auto sx = [&](int k, int lr) { return lr * P + W + i0[k] - 1; };

  // ---- coefficients
  T cE[RC ? SEG : 1][W], cN[RC ? SEG : 1][W], cS[RC ? SEG : 1][W], dg[RC ? SEG : 1][W], di[RC ? SEG : 1][W],
      cW0[RC ? SEG : 1];
  if constexpr (RC) {
    PCGR_SEGS {
      const int j = j0 + row[k];
      cW0[k] = nv[k] ? a.cx[g.at(i0[k] - 1, j)] : T(0);
      PCGR_E {
        const bool on = e < nv[k];
        const int c = on ? g.at(i0[k] + e, j) : g.P;
        cE[k][e] = on ? a.cx[c] : T(0);
        cN[k][e] = on ? a.cy[c] : T(0);
        cS[k][e] = on ? a.cy[c - g.P] : T(0);
        di[k][e] = on ? a.dinv[c] : T(0);
      }
      PCGR_E dg[k][e] = cE[k][e] + (e ? cE[k][e ? e - 1 : 0] : cW0[k]) + cN[k][e] + cS[k][e];
    }
  } else {
    for (int q = tid; q < R * PX; q += tpb) {
      const int lr = q / PX, i = q % PX - W + 1;
      cxs[q] = (i >= 0 && i <= nx) ? a.cx[g.at(i, j0 + lr)] : T(0);
      if constexpr (!PACK) dis[q] = (i >= 1 && i <= nx) ? a.dinv[g.at(i, j0 + lr)] : T(0);
    }
    for (int q = tid; q < (R + 1) * PY; q += tpb) {
      const int lf = q / PY - 1, i = q % PY - Y1 + 1;
      cys[q] = (i >= 1 && i <= nx) ? a.cy[g.at(i, j0 + lf)] : T(0);
      if constexpr (PACK)
        if (lf >= 0) dis[q - PY] = i <= nx ? a.dinv[g.at(i, j0 + lf)] : T(0);
    }
  }
  // every slot of the stencil's vector is finite (padding is read, times a
  // zero coefficient)
  for (int q = tid; q < (R + 2) * P; q += tpb) us[q] = T(0);
  if constexpr (ONE) {
    for (int q = tid; q < 2 * P; q += tpb) {
      const int side = q / P, i = q % P - W + 1;
      const int jb = side == 0 ? (j0 - 1 >= 1 ? j0 - 1 : ny) : (j0 + R <= ny ? j0 + R : 1);
      const bool on = i >= 1 && i <= nx && (side == 0 ? has_bot : has_top);
      hd[q] = on ? a.dinv[g.at(i, jb)] : T(0);
      hs[q] = T(0);
      hr[q] = T(0);
    }
  }
  x.start();

  // send segment k's values v to the neighbours of its row, if there are any
  auto push = [&](int k, const T* v) {
    if (!nv[k]) return;
    if constexpr (CL) {
      const unsigned at = smem_u32(hw + x.parity() * 2 * P + W + i0[k] - 1);
      // my first row is the row above the CTA below; my last row the row below the CTA above
      if (row[k] == 0 && has_bot) push16(mapa(at + (unsigned)(P * sizeof(T)), below), x.bar(below), v);
      if (row[k] == R - 1 && has_top) push16(mapa(at, above), x.bar(above), v);
    } else {
      if (row[k] == 0 && has_bot) gx_put_seg(x.outbox(rank, 0) + (i0[k] - 1) / W * 4, v, x.ep);
      if (row[k] == R - 1 && has_top) gx_put_seg(x.outbox(rank, 1) + (i0[k] - 1) / W * 4, v, x.ep);
    }
  };
  // sum NV values and, with HALO, receive the halo rows into hwc; false when
  // a wait gave up
  const T* hwc = hw;
  auto allreduce = [&](auto nvc, auto haloc, const DD* v, double* out, auto between) -> bool {
    constexpr int NV = decltype(nvc)::value;
    constexpr bool HALO = decltype(haloc)::value;
    T* to = hw + x.parity() * 2 * P;
    if constexpr (HALO) hwc = to;
    if constexpr (CL) {
      return x.template allreduce<NV>(v, out, HALO ? (unsigned)(((int)has_bot + (int)has_top) * nseg * 16) : 0u, between);
    } else {
      return x.template allreduce<NV>(
          v, out,
          [&](GxWait& gw) {
            if constexpr (HALO) {
              for (int c = tid; c < 2 * nseg; c += tpb) {
                const int side = c >= nseg ? 1 : 0, seg = c - side * nseg;
                if (!(side == 0 ? has_bot : has_top)) continue;
                const unsigned long long* hp = x.outbox(side == 0 ? below : above, 1 - side) + 4L * seg;
                GxSeg sg;
                sg.load(hp);
                while (!sg.ready(x.ep)) {
                  if (!gw.again()) return false;
                  sg.load(hp);
                }
                T hv[W];
                sg.get(hv);
                stv(to + side * P + W + seg * W, hv);
              }
            }
            return true;
          },
          between);
    }
  };
  auto nothing = [] {};
  auto leave = [&]() {
    if constexpr (CL) x.leave();
  };
  auto gave_up = [&]() {
    if (tid == 0) a.out->status = 1;
    if constexpr (CL) x.abandon();
  };
  using IC1 = std::integral_constant<int, 1>;
  using IC2 = std::integral_constant<int, 2>;
  using IC3 = std::integral_constant<int, 3>;
  using YES = std::true_type;
  using NO = std::false_type;

  T phi[SEG][W], r[SEG][W];
  double red[3];
  // ---- zero-mean projection and rhs norm (mod_subsolvers.f90:89-121)
  double mean = 0.0;
  if (closed) {
    RSum s;
    PCGR_SEGS PCGR_E if (e < nv[k]) s.add(double(a.rhs[g.at(i0[k] + e, j0 + row[k])]));
    if (!allreduce(IC1{}, NO{}, &s.v, red, nothing)) return gave_up();
    mean = red[0] / (double)(nx * ny);
  }
  {
    RSum ss;
    PCGR_SEGS PCGR_E {
      T rw = T(0);
      if (e < nv[k]) {
        const T b = a.rhs[g.at(i0[k] + e, j0 + row[k])];
        rw = closed ? T(double(b) - mean) : b;
        ss.add(double(rw) * double(rw));
      }
      r[k][e] = rw;
      phi[k][e] = T(0);
    }
    if (!a.phi_zero) {
      // ghosts of phi (halo exchange + Neumann), then r = rhs_work - A phi
      const long tot = g.n();
      for (long q = rank * (long)tpb + tid; q < tot; q += (long)G * tpb) {
        const int gi = (int)(q % g.P) - 2, gj = (int)(q / g.P) - 2;
        if (gi < -1 || gj < -1 || gi > nx + 2 || gj > ny + 2) continue;
        if (gi >= 1 && gi <= nx && gj >= 1 && gj <= ny) continue;
        const int mi = (gi >= 1 && gi <= nx) ? gi : (g.px ? (gi < 1 ? gi + nx : gi - nx) : (gi < 1 ? 1 - gi : 2 * nx + 1 - gi));
        const int mj = (gj >= 1 && gj <= ny) ? gj : (g.py ? (gj < 1 ? gj + ny : gj - ny) : (gj < 1 ? 1 - gj : 2 * ny + 1 - gj));
        a.phi[q] = a.phi[g.at(mi, mj)];
      }
      PCGR_SEGS PCGR_E if (e < nv[k]) {
        const T* gp = a.phi;
        const int i = i0[k] + e, j = j0 + row[k];
        phi[k][e] = gp[g.at(i, j)];
        r[k][e] = r[k][e] - poisson_ap<T>(g, a.cx, a.cy, i, j, [&](int x, int y) { return gp[g.at(x, y)]; });
      }
    }
    if constexpr (ONE) PCGR_SEGS push(k, r[k]);
    if (!allreduce(IC1{}, std::integral_constant<bool, ONE>{}, &ss.v, red, nothing)) return gave_up();
  }
  const double rhs_norm = sqrt(red[0]);
  if (rhs_norm < 1.0e-14) {
    const long tot = g.n();
    for (long q = rank * (long)tpb + tid; q < tot; q += (long)G * tpb) a.phi[q] = T(0);
    if (rank == 0 && tid == 0) {
      a.out->iters = 0;
      a.out->res = 0.0;
      a.out->calls += 1;
      if constexpr (!CL) x.finish();
    }
    return leave();
  }
  // the stopping test |r| / |rhs| < tol is evaluated as it stands, but only
  // when rr is within rounding of passing it (a square root and a division
  // off the critical path of every other iteration)
  const double thr = a.tol * rhs_norm;
  const double rr_maybe = thr * thr * (1.0 + 1.0e-12) + 1.0e-300;

  // the segment's values into the stencil's vector, with the ghost columns
  // (a wall repeats the edge cell, as the reference's index clamps do)
  auto put = [&](int k, const T* v) {
    if (!nv[k]) return;
    T* d = us + sx(k, row[k] + 1);
    if (nv[k] == W) stv(d, v);
    else {
      PCGR_E if (e < nv[k]) d[e] = v[e];
    }
    T* rowp = us + (row[k] + 1) * P + W - 1;  // column 0
    if (i0[k] == 1) rowp[g.px ? nx + 1 : 0] = v[0];
    if (i0[k] + nv[k] - 1 == nx) {
      T last = v[0];
      PCGR_E if (e == nv[k] - 1) last = v[e];
      rowp[g.px ? 0 : nx + 1] = last;
    }
  };
  // A v of segment k (own values in v, neighbours in shared memory)
  auto apply = [&](int k, const T* v, T* o) {
    const int lr = row[k], j = j0 + lr;
    const int c = sx(k, lr + 1);
    T n[W], s[W];
    ldv(us + c + P, n);
    ldv(us + c - P, s);
    const T wv = us[c - 1], ev = us[c + nv[k]];
    T xE[W], xN[W], xS[W], xW0;
    if constexpr (!RC) {
      const int q = lr * PX + W + i0[k] - 1, qy = lr * PY + Y1 + i0[k] - 1;
      ldv(cxs + q, xE);
      xW0 = cxs[q - 1];
      ldv(cys + qy + PY, xN);
      ldv(cys + qy, xS);
    }
    PCGR_E {
      const T fE = RC ? cE[RC ? k : 0][e] : xE[e];
      const T fW = e ? (RC ? cE[RC ? k : 0][e ? e - 1 : 0] : xE[e ? e - 1 : 0]) : (RC ? cW0[RC ? k : 0] : xW0);
      const T fN = RC ? cN[RC ? k : 0][e] : xN[e], fS = RC ? cS[RC ? k : 0][e] : xS[e];
      const T fd = RC ? dg[RC ? k : 0][e] : fE + fW + fN + fS;
      const T vE = (e + 1 < nv[k]) ? v[e + 1 < W ? e + 1 : e] : ev;
      const T vW = e ? v[e ? e - 1 : 0] : wv;
      const T vN = (j == ny && !g.py) ? v[e] : n[e];
      const T vS = (j == 1 && !g.py) ? v[e] : s[e];
      o[e] = fd * v[e] - (fE * vE + fW * vW + fN * vN + fS * vS);
    }
  };
  auto dinv_of = [&](int k, T* d) {
    if constexpr (RC) {
      PCGR_E d[e] = di[k][e];
    } else {
      ldv(dis + row[k] * PY + Y1 + i0[k] - 1, d);
    }
  };
  // the halo rows' segments: f(side, index of the segment in a halo array,
  // the row's segment in the stencil's vector)
  auto halo_rows = [&](auto f) {
    for (int q = tid; q < 2 * nseg; q += tpb) {
      const int side = q >= nseg ? 1 : 0, c = W + (q - side * nseg) * W;
      if (side == 0 ? has_bot : has_top) f(side * P + c, us + (side == 0 ? 0 : R + 1) * P + c);
    }
  };

  double rr = 0.0;
  int iter;
  if constexpr (ONE) {
    T w[SEG][W], p[SEG][W], s[SEG][W], u[RC ? SEG : 1][W];
    auto u_of = [&](int k, T* o) {
      if constexpr (RC) {
        PCGR_E o[e] = u[k][e];
      } else {
        ldv(us + sx(k, row[k] + 1), o);
      }
    };
    // u0 = dinv r0 and its halo rows, w0 = A u0
    PCGR_SEGS {
      T d[W], uu[W];
      dinv_of(k, d);
      PCGR_E {
        uu[e] = d[e] * r[k][e];
        p[k][e] = T(0);
        s[k][e] = T(0);
        if constexpr (RC) u[k][e] = uu[e];
      }
      put(k, uu);
    }
    halo_rows([&](int c, T* to) {
      T rv[W], d[W], uv[W];
      ldv(hwc + c, rv);
      ldv(hd + c, d);
      PCGR_E uv[e] = d[e] * rv[e];
      stv(hr + c, rv);
      stv(to, uv);
    });
    __syncthreads();
    double gam = 0.0, gam_old = 0.0, del = 0.0, alpha = 0.0, ialpha = 0.0, igam = 0.0;
    auto stencil_and_sums = [&]() -> bool {
      RSum x0, x1, x2;
      PCGR_SEGS {
        T uu[W];
        u_of(k, uu);
        apply(k, uu, w[k]);
        push(k, w[k]);
        PCGR_E if (e < nv[k]) {
          x0.add(double(r[k][e]) * double(uu[e]));
          x1.add(double(w[k][e]) * double(uu[e]));
          x2.add(double(r[k][e]) * double(r[k][e]));
        }
      }
      const DD v[3] = {x0.v, x1.v, x2.v};
      return allreduce(IC3{}, YES{}, v, red, [&] {
        igam = 1.0 / gam;  // of the sums before these
        ialpha = 1.0 / alpha;
        // formed here, not where they are used (two divisions less on the
        // chain from the sums to the update)
        asm volatile("" : "+d"(igam), "+d"(ialpha));
      });
    };
    if (!stencil_and_sums()) return gave_up();
    gam = red[0];
    del = red[1];
    rr = red[2];
    for (iter = 1; iter <= a.max_iter; ++iter) {
      double beta = 0.0, den = del;
      if (iter > 1) {
        beta = quotient(gam, gam_old, igam);
        den = del - quotient(beta * gam, alpha, ialpha);
      }
      if (fabs(den) < 1.0e-30) break;
      alpha = gam / den;
      const T tb = T(beta), ta = T(alpha);
      PCGR_SEGS {
        T d[W], uu[W];
        dinv_of(k, d);
        u_of(k, uu);
        PCGR_E {
          p[k][e] = madd(tb, p[k][e], uu[e]);
          s[k][e] = madd(tb, s[k][e], w[k][e]);
          r[k][e] = madd(-ta, s[k][e], r[k][e]);
          uu[e] = d[e] * r[k][e];
          if constexpr (RC) u[k][e] = uu[e];
        }
        put(k, uu);
        PCGR_E phi[k][e] = madd(ta, p[k][e], phi[k][e]);
      }
      halo_rows([&](int c, T* to) {
        T wv[W], sv[W], rv[W], d[W], uv[W];
        ldv(hwc + c, wv);
        ldv(hs + c, sv);
        ldv(hr + c, rv);
        ldv(hd + c, d);
        PCGR_E {
          sv[e] = madd(tb, sv[e], wv[e]);
          rv[e] = madd(-ta, sv[e], rv[e]);
          uv[e] = d[e] * rv[e];
        }
        stv(to, uv);
        stv(hs + c, sv);
        stv(hr + c, rv);
      });
      __syncthreads();
      if (!stencil_and_sums()) return gave_up();
      gam_old = gam;
      gam = red[0];
      del = red[1];
      rr = red[2];
      if (rr < rr_maybe && sqrt(rr) / rhs_norm < a.tol) break;
    }
  } else {
    T ap[SEG][W];
    T z[RC ? SEG : 1][W], p[RC ? SEG : 1][W];
    auto p_of = [&](int k, T* o) {
      if constexpr (RC) {
        PCGR_E o[e] = p[k][e];
      } else {
        ldv(us + sx(k, row[k] + 1), o);
      }
    };
    auto z_of = [&](int k, T* o) {
      T d[W];
      dinv_of(k, d);
      PCGR_E o[e] = d[e] * r[k][e];
    };
    {
      RSum rz;
      PCGR_SEGS {
        T zz[W];
        z_of(k, zz);
        PCGR_E {
          if constexpr (RC) z[k][e] = zz[e];
          if (e < nv[k]) rz.add(double(r[k][e]) * double(zz[e]));
        }
        push(k, zz);
      }
      if (!allreduce(IC1{}, YES{}, &rz.v, red, nothing)) return gave_up();
    }
    double rz_old = red[0], beta = 0.0, irz = 0.0;
    for (iter = 1; iter <= a.max_iter; ++iter) {
      const T tb = T(beta);
      // p_k of the own cells and of the halo rows
      PCGR_SEGS {
        T zz[W], pp[W];
        if constexpr (RC) {
          PCGR_E zz[e] = z[k][e];
        } else {
          z_of(k, zz);
        }
        if (iter == 1) {
          PCGR_E pp[e] = zz[e];
        } else {
          p_of(k, pp);
          PCGR_E pp[e] = madd(tb, pp[e], zz[e]);
        }
        if constexpr (RC) PCGR_E p[k][e] = pp[e];
        put(k, pp);
      }
      halo_rows([&](int c, T* to) {
        T zv[W], pv[W];
        ldv(hwc + c, zv);
        ldv(to, pv);
        PCGR_E pv[e] = iter == 1 ? zv[e] : madd(tb, pv[e], zv[e]);
        stv(to, pv);
      });
      __syncthreads();
      RSum papd;
      PCGR_SEGS {
        T pp[W];
        p_of(k, pp);
        apply(k, pp, ap[k]);
        PCGR_E if (e < nv[k]) papd.add(double(pp[e]) * double(ap[k][e]));
      }
      if (!allreduce(IC1{}, NO{}, &papd.v, red, [&] {
            irz = 1.0 / rz_old;  // for beta, off the chain from the next sums to the update
            asm volatile("" : "+d"(irz));
          }))
        return gave_up();
      const double pap = red[0];
      if (fabs(pap) < 1.0e-30) break;
      const double alpha = rz_old / pap;
      const T ta = T(alpha);
      RSum rrd, rzd;
      PCGR_SEGS {
        T d[W], zz[W], pp[W];
        dinv_of(k, d);
        p_of(k, pp);
        PCGR_E {
          r[k][e] = madd(-ta, ap[k][e], r[k][e]);
          zz[e] = d[e] * r[k][e];
          if constexpr (RC) z[k][e] = zz[e];
        }
        push(k, zz);
        PCGR_E {
          phi[k][e] = madd(ta, pp[e], phi[k][e]);
          if (e < nv[k]) {
            rrd.add(double(r[k][e]) * double(r[k][e]));
            rzd.add(double(r[k][e]) * double(zz[e]));
          }
        }
      }
      const DD v2[2] = {rrd.v, rzd.v};
      if (!allreduce(IC2{}, YES{}, v2, red, nothing)) return gave_up();
      rr = red[0];
      if (rr < rr_maybe && sqrt(rr) / rhs_norm < a.tol) break;
      beta = quotient(red[1], rz_old, irz);
      rz_old = red[1];
    }
  }
  if (closed) {
    RSum s;
    PCGR_SEGS PCGR_E if (e < nv[k]) s.add(double(phi[k][e]));
    if (!allreduce(IC1{}, NO{}, &s.v, red, nothing)) return gave_up();
    const double m = red[0] / (double)(nx * ny);
    PCGR_SEGS PCGR_E phi[k][e] = T(double(phi[k][e]) - m);
  }
  PCGR_SEGS PCGR_E if (e < nv[k]) a.phi[g.at(i0[k] + e, j0 + row[k])] = phi[k][e];
  if (rank == 0 && tid == 0) {
    const int it = iter < a.max_iter ? iter : a.max_iter;
    a.out->iters = it;
    a.out->res = sqrt(rr) / rhs_norm;
    a.out->total_iters += (unsigned long long)it;
    if (a.timed) a.out->timed_iters += (unsigned long long)it;
    a.out->calls += 1;
    if constexpr (!CL) x.finish();
  }
  leave();
#undef PCGR_SEGS
#undef PCGR_E
}

template <typename T, int SHAPE, bool CL>
__global__ void __launch_bounds__(pcgr_shape(SHAPE).tpb, 1) k_pcg_resident(PcgResArgs<T> a) {
  if (a.active && !*a.active) return;
  constexpr PcgrShape sh = pcgr_shape(SHAPE);
  if constexpr (CL) {
    cgc::cluster_group cl = cgc::this_cluster();
    pcgr_body<T, sh.seg, sh.tpb, true>(a, (int)cl.block_rank(), (int)cl.num_blocks());
  } else {
    pcgr_body<T, sh.seg, sh.tpb, false>(a, blockIdx.x, gridDim.x);
  }
}
template <typename T, bool CL>
const void* pcgr_fn(int shape) {
  switch (shape) {
    case 0: return (const void*)k_pcg_resident<T, 0, CL>;
    case 1: return (const void*)k_pcg_resident<T, 1, CL>;
    case 2: return (const void*)k_pcg_resident<T, 2, CL>;
    case 3: return (const void*)k_pcg_resident<T, 3, CL>;
    case 4: return (const void*)k_pcg_resident<T, 4, CL>;
    case PCGR_TALL:
      if constexpr (CL) return (const void*)k_pcg_resident<T, PCGR_TALL, CL>;
      break;
  }
  return nullptr;
}

// the launch of a resident solve: G CTAs of tpb threads and rows_per rows
struct PcgrPlan {
  bool ok = false;
  int G = 0, rows_per = 0, shape = 0, tpb = 0;
  size_t smem = 0;
};
// the plan for want_G CTAs (or fewer, when ny does not divide) with the first
// of the shapes [s0, s1) that holds a CTA's rows; not ok when none does
template <typename T>
PcgrPlan pcgr_plan(int nx, int ny, int want_G, int s0 = 0, int s1 = PCGR_SHAPES) {
  PcgrPlan p;
  const int W = 16 / (int)sizeof(T), nseg = (nx + W - 1) / W;
  p.rows_per = (ny + want_G - 1) / want_G;
  p.G = (ny + p.rows_per - 1) / p.rows_per;
  const long segs = (long)p.rows_per * nseg;
  for (int s = s0; s < s1 && !p.ok; ++s) {
    const PcgrShape sh = pcgr_shape(s);
    if (segs > (long)sh.seg * sh.tpb) continue;
    p.shape = s;
    p.tpb = 32;
    while ((long)p.tpb * sh.seg < segs) p.tpb *= 2;
    p.smem = sizeof(T) * (size_t)pcgr_smem_elems<T>(nx, p.rows_per, sh.seg, sh.tpb);
    p.ok = true;
  }
  return p;
}

}  // namespace fugu
