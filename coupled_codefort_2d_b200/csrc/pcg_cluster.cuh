// pcg_cluster.cuh -- the FP32 PCG pressure Poisson solve of the mixed form
// (solve_poisson_pressure, mod_subsolvers.f90:32-246) resident in one
// thread-block cluster of up to 16 CTAs.
//
// The FP32 inner solve sums its exact float products in plain double, so the
// states depend on the order of the sums: thread t of CTA r owns column
// t % nx + 1 and a strip of up to CPT consecutive rows of the CTA's rows, its
// terms are added from the strip's first row to its last, and the threads,
// warps and CTAs are merged by trees over 16, 8, 4, 2, 1.  The same holds for
// a case alone and in a batch with the same number of CTAs.
//
// Two kernels:
//   k_pcg_column        strips of up to 16 cells.  One all-reduce per
//     iteration (the Chronopoulos-Gear arrangement of preconditioned CG):
//     with u = M^-1 r, w = A u and s = A p carried as vectors, the dot
//     products (r, u), (w, u) and (r, r) are formed in one pass:
//       beta = gamma / gamma_old,  alpha = gamma / (delta - beta gamma / alpha_old)
//       p = u + beta p,  s = w + beta s,  phi += alpha p,  r -= alpha s,
//       u = M^-1 r,  w = A u
//     The vectors live in registers, u of the CTA's cells in shared memory
//     (the east, west and strip-end neighbours).  The rows just outside the
//     CTA belong to single columns of its edge threads: each receives w of its
//     halo cell with the sums and repeats the cell's s, r and u itself.
//   k_pcg_cluster_lean  strips of 17 to 32 cells, alone or in a batch, such as
//     320 x 384, 400 x 400 or 200 x 600, with the reference's recurrence: five
//     register arrays of 32 cells do not fit, so z is recomputed from r and p_k
//     lives in shared memory.  Halo rows of z and p are pushed into the
//     neighbouring CTAs and the CTAs meet at hardware cluster barriers.  15.2 us
//     per iteration at 320 x 384 on a B200.
//
// k_pcg_column is bound by the latency chain of its iteration and, at 4,096
// cells per CTA, by the conversions to double of the three products per cell
// (16 per cycle and SM).  us per iteration on a B200, with cluster barriers
// and pulled sums before, and now with pushed data and the mbarrier
// (pcg_exchange.cuh), reciprocals formed in flight and coefficients in
// registers:
//   64 x 64 1.93 -> 1.28, 128 x 128 2.20 -> 1.49, 203 x 125 2.56 -> 1.79,
//   256 x 256 3.55 -> 2.43, 192 x 384 7.25 -> 3.70, 256 x 512 8.52 -> 4.04
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "fugu_internal.cuh"
#include "pcg_exchange.cuh"
#include "persistent.cuh"

namespace fugu {

constexpr int PCGC_TPB = 512;

struct PcgClusterArgs {
  Geo g;
  const float* rhs;
  const float* cx;
  const float* cy;
  const float* dinv;
  float* phi;
  PcgOut* out;
  const int* active;
  double tol;
  int max_iter;
  int phi_zero;
  int rows_per;  // rows of every CTA but possibly the last
  int timed;     // the launch is timed: add its iterations to out->timed_iters
  CxLimit wait;  // k_pcg_column's waits
};

// ------------------------------------------------------------ column strips
constexpr int PCGC_COL_CPT = 16;  // cells of a thread's strip
// coefficients in registers beside the six vectors up to this strip
constexpr int PCGC_COL_REG = 8;
// shared memory in floats: u of the CTA's cells, the received halo rows
// [parity][bottom, top], and for long strips cx, cy, dinv and phi
__host__ __device__ inline long pcgcol_smem_elems(int nx, int rows_per, int cpt) {
  long n = (long)rows_per * nx + 4L * nx;
  if (cpt > PCGC_COL_REG) n += (long)rows_per * (nx + 1) + (long)(rows_per + 1) * nx + 2L * rows_per * nx;
  return n;
}

template <int CPT>
__device__ __forceinline__ void pcg_column_body(const PcgClusterArgs& a, const int rank, const int C) {
  using T = float;
  constexpr bool RC = CPT <= PCGC_COL_REG;  // coefficients and phi in registers
  const Geo g = a.g;
  const int nx = g.nx, ny = g.ny, rp = a.rows_per;
  const int j0 = 1 + rank * rp;
  const int R = min(rp, ny - rank * rp);
  const bool closed = !g.px && !g.py;
  const int S = (R + CPT - 1) / CPT;  // strips per column
  const int t = threadIdx.x;
  const bool act = t < nx * S;
  const int i = act ? t % nx + 1 : 1;
  const int lr0 = act ? (t / nx) * CPT : 0;
  const int nr = act ? min(CPT, R - lr0) : 0;
  const int ie = (i < nx) ? i + 1 : (g.px ? 1 : nx);
  const int iw = (i > 1) ? i - 1 : (g.px ? nx : 1);
  const bool has_bot = rank > 0 || g.py, has_top = rank < C - 1 || g.py;
  const int below = rank > 0 ? rank - 1 : C - 1, above = rank < C - 1 ? rank + 1 : 0;
  // the thread's cells at the CTA's edges: it sends their w to the neighbour
  // and keeps the neighbour's cell across the edge
  const bool edge_b = act && lr0 == 0 && has_bot, edge_t = act && lr0 + nr == R && has_top;

  extern __shared__ __align__(16) unsigned char pcgcol_smem[];
  T* uc = reinterpret_cast<T*>(pcgcol_smem);  // u of own cells, rp x nx
  T* hw = uc + rp * nx;                          // received halo rows [parity][bottom, top]
  T* cxs = hw + 4 * nx;                          // (without RC) cx rp x (nx + 1), cy (rp + 1) x nx, dinv, phi
  T* cys = cxs + rp * (nx + 1);
  T* dis = cys + (rp + 1) * nx;
  T* phs = dis + rp * nx;
  __shared__ ClusterXSmem<PCGC_TPB> xs;
  ClusterX<PCGC_TPB, false> x(xs, rank, C, a.wait);

#define COL_CELLS _Pragma("unroll") for (int c = 0; c < CPT; ++c) if (c < nr)
  T phi_r[RC ? CPT : 1], r_r[CPT], u_r[RC ? CPT : 1], w_r[CPT], p_r[CPT], s_r[CPT];
  T cE[RC ? CPT : 1], cW[RC ? CPT : 1], cN[RC ? CPT : 1], di[RC ? CPT : 1], cS0 = T(0);
  if constexpr (RC) {
    COL_CELLS {
      const int k = g.at(i, j0 + lr0 + c);
      cE[c] = a.cx[k];
      cW[c] = a.cx[k - 1];
      cN[c] = a.cy[k];
      di[c] = a.dinv[k];
      if (c == 0) cS0 = a.cy[k - g.P];
    }
  } else {
    for (int q = t; q < R * (nx + 1); q += blockDim.x) cxs[q] = a.cx[g.at(q % (nx + 1), j0 + q / (nx + 1))];
    for (int q = t; q < (R + 1) * nx; q += blockDim.x) cys[q] = a.cy[g.at(q % nx + 1, j0 - 1 + q / nx)];
    for (int q = t; q < R * nx; q += blockDim.x) dis[q] = a.dinv[g.at(q % nx + 1, j0 + q / nx)];
  }
  // the halo cells' inverse diagonal, s and r
  const T hdb = edge_b ? a.dinv[g.at(i, j0 > 1 ? j0 - 1 : ny)] : T(0);
  const T hdt = edge_t ? a.dinv[g.at(i, j0 + R <= ny ? j0 + R : 1)] : T(0);
  T hsb = T(0), hst = T(0), hrb = T(0), hrt = T(0);
  x.start();

  auto push = [&](T first, T last) {
    const unsigned at = smem_u32(hw + x.parity() * 2 * nx + i - 1);
    if (edge_b) push4(mapa(at + (unsigned)(nx * sizeof(T)), below), x.bar(below), first);
    if (edge_t) push4(mapa(at, above), x.bar(above), last);
  };
  const unsigned halo_bytes = (unsigned)(((int)has_bot + (int)has_top) * nx * (int)sizeof(T));
  const T* hwc = hw;  // the halo rows received last
  auto nothing = [] {};
  auto gave_up = [&]() {
    if (t == 0) a.out->status = 1;
    x.abandon();
  };
  double red[3];

  double mean = 0.0;
  if (closed) {
    DD s{0.0, 0.0};
    COL_CELLS s.hi += double(a.rhs[g.at(i, j0 + lr0 + c)]);
    if (!x.template allreduce<1>(&s, red, 0u, nothing)) return gave_up();
    mean = red[0] / (double)(nx * ny);
  }
  {
    DD ss{0.0, 0.0};
    COL_CELLS {
      const T b = a.rhs[g.at(i, j0 + lr0 + c)];
      const T rw = closed ? T(double(b) - mean) : b;
      r_r[c] = rw;
      ss.hi = __fma_rn(double(rw), double(rw), ss.hi);
    }
    if (!a.phi_zero) {
      // ghosts of phi (halo exchange + Neumann); r0 = rhs_work - A phi0
      const long tot = g.n();
      for (long q = rank * (long)blockDim.x + t; q < tot; q += (long)C * blockDim.x) {
        const int gi = (int)(q % g.P) - 2, gj = (int)(q / g.P) - 2;
        if (gi < -1 || gj < -1 || gi > nx + 2 || gj > ny + 2) continue;
        if (gi >= 1 && gi <= nx && gj >= 1 && gj <= ny) continue;
        const int mi = (gi >= 1 && gi <= nx) ? gi : (g.px ? (gi < 1 ? gi + nx : gi - nx) : (gi < 1 ? 1 - gi : 2 * nx + 1 - gi));
        const int mj = (gj >= 1 && gj <= ny) ? gj : (g.py ? (gj < 1 ? gj + ny : gj - ny) : (gj < 1 ? 1 - gj : 2 * ny + 1 - gj));
        a.phi[q] = a.phi[g.at(mi, mj)];
      }
      COL_CELLS {
        const int j = j0 + lr0 + c;
        const T* gp = a.phi;
        r_r[c] = r_r[c] - poisson_ap<T>(g, a.cx, a.cy, i, j, [&](int xx, int yy) { return gp[g.at(xx, yy)]; });
      }
    }
    COL_CELLS {
      const T ph = a.phi_zero ? T(0) : a.phi[g.at(i, j0 + lr0 + c)];
      if constexpr (RC) phi_r[c] = ph;
      else phs[(lr0 + c) * nx + i - 1] = ph;
    }
    T last = T(0);
    COL_CELLS if (c == nr - 1) last = r_r[c];
    push(r_r[0], last);
    hwc = hw + x.parity() * 2 * nx;
    if (!x.template allreduce<1>(&ss, red, halo_bytes, nothing)) return gave_up();
  }
  const double rhs_norm = sqrt(red[0]);
  if (rhs_norm < 1.0e-14) {
    const long tot = g.n();
    for (long q = rank * (long)blockDim.x + t; q < tot; q += (long)C * blockDim.x) a.phi[q] = T(0);
    if (rank == 0 && t == 0) {
      a.out->iters = 0;
      a.out->res = 0.0;
      a.out->calls += 1;
    }
    return x.leave();
  }
  // |r| / |rhs| < tol is evaluated as it stands, but only when rr is within
  // rounding of passing it
  const double thr = a.tol * rhs_norm;
  const double rr_maybe = thr * thr * (1.0 + 1.0e-12) + 1.0e-300;

  T hub = T(0), hut = T(0);  // u of the halo cells
  COL_CELLS {
    const int q = (lr0 + c) * nx + i - 1;
    const T uu = (RC ? di[RC ? c : 0] : dis[q]) * r_r[c];
    if constexpr (RC) u_r[c] = uu;
    uc[q] = uu;
    p_r[c] = T(0);
    s_r[c] = T(0);
  }
  if (edge_b) {
    hrb = hwc[i - 1];
    hub = hdb * hrb;
  }
  if (edge_t) {
    hrt = hwc[nx + i - 1];
    hut = hdt * hrt;
  }
  __syncthreads();
  double gam = 0.0, gam_old = 0.0, del = 0.0, rr = 0.0, alpha = 0.0, ialpha = 0.0, igam = 0.0;
  // w = A u, the three sums and their exchange.  At a wall the coefficient is
  // zero, so the value across it does not matter (it is zero too).
  auto cells = [&](auto fullc, DD* v, T& last) {
    constexpr bool FULL = decltype(fullc)::value;  // the strip has all CPT cells
    const T utop = act ? (lr0 + nr < R ? uc[(lr0 + nr) * nx + i - 1] : hut) : T(0);
    const T ubot = lr0 > 0 ? uc[(lr0 - 1) * nx + i - 1] : hub;
    T below_u = ubot;  // u of the cell below
#pragma unroll
    for (int c = 0; c < CPT; ++c)
      if (FULL || c < nr) {
        const int lr = lr0 + c, q = lr * nx + i - 1;
        const T uk = RC ? u_r[RC ? c : 0] : uc[q];
        const T uE = uc[lr * nx + (ie - 1)], uW = uc[lr * nx + (iw - 1)];
        T un;
        if (FULL ? c + 1 < CPT : c + 1 < nr) un = RC ? u_r[RC ? (c + 1 < CPT ? c + 1 : c) : 0] : uc[q + nx];
        else un = utop;
        T fE, fW, fN, fS;
        if constexpr (RC) {
          fE = cE[c]; fW = cW[c]; fN = cN[c]; fS = c ? cN[c ? c - 1 : 0] : cS0;
        } else {
          fE = cxs[lr * (nx + 1) + i]; fW = cxs[lr * (nx + 1) + i - 1];
          fN = cys[q + nx]; fS = cys[q];
        }
        const T off = madd(fS, below_u, madd(fN, un, madd(fW, uW, fE * uE)));
        const T wv = madd(fE + fW + fN + fS, uk, -off);
        below_u = uk;
        w_r[c] = wv;
        last = wv;
        // exact products: one rounding per term either way
        v[0].hi = __fma_rn(double(r_r[c]), double(uk), v[0].hi);
        v[1].hi = __fma_rn(double(wv), double(uk), v[1].hi);
        v[2].hi = __fma_rn(double(r_r[c]), double(r_r[c]), v[2].hi);
      }
  };
  auto stencil_and_sums = [&]() -> bool {
    DD v[3] = {DD{0.0, 0.0}, DD{0.0, 0.0}, DD{0.0, 0.0}};
    T last = T(0);
    if (nr == CPT) cells(std::true_type{}, v, last);
    else cells(std::false_type{}, v, last);
    push(w_r[0], last);
    hwc = hw + x.parity() * 2 * nx;
    return x.template allreduce<3>(v, red, halo_bytes, [&] {
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
  int iter;
  for (iter = 1; iter <= a.max_iter; ++iter) {
    double beta = 0.0, den = del;
    if (iter > 1) {
      beta = quotient(gam, gam_old, igam);
      den = del - quotient(beta * gam, alpha, ialpha);
    }
    if (fabs(den) < 1.0e-30) break;
    alpha = gam / den;
    const T tb = T(beta), ta = T(alpha);
    auto update = [&](auto fullc) {
      constexpr bool FULL = decltype(fullc)::value;
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        if (FULL || c < nr) {
          const int q = (lr0 + c) * nx + i - 1;
          const T uk = RC ? u_r[RC ? c : 0] : uc[q];
          p_r[c] = madd(tb, p_r[c], uk);
          s_r[c] = madd(tb, s_r[c], w_r[c]);
          r_r[c] = madd(-ta, s_r[c], r_r[c]);
          const T uu = (RC ? di[RC ? c : 0] : dis[q]) * r_r[c];
          uc[q] = uu;
          if constexpr (RC) {
            u_r[c] = uu;
            phi_r[c] = madd(ta, p_r[c], phi_r[c]);
          } else {
            phs[q] = madd(ta, p_r[c], phs[q]);
          }
        }
    };
    if (nr == CPT) update(std::true_type{});
    else update(std::false_type{});
    // the halo cells' recurrence, with their owners' expressions
    if (edge_b) {
      hsb = madd(tb, hsb, hwc[i - 1]);
      hrb = madd(-ta, hsb, hrb);
      hub = hdb * hrb;
    }
    if (edge_t) {
      hst = madd(tb, hst, hwc[nx + i - 1]);
      hrt = madd(-ta, hst, hrt);
      hut = hdt * hrt;
    }
    __syncthreads();
    if (!stencil_and_sums()) return gave_up();
    gam_old = gam;
    gam = red[0];
    del = red[1];
    rr = red[2];
    if (rr < rr_maybe && sqrt(rr) / rhs_norm < a.tol) break;
  }
  double m = 0.0;
  if (closed) {
    DD s{0.0, 0.0};
    COL_CELLS s.hi += double(RC ? phi_r[RC ? c : 0] : phs[(lr0 + c) * nx + i - 1]);
    if (!x.template allreduce<1>(&s, red, 0u, nothing)) return gave_up();
    m = red[0] / (double)(nx * ny);
  }
  COL_CELLS {
    const T ph = RC ? phi_r[RC ? c : 0] : phs[(lr0 + c) * nx + i - 1];
    a.phi[g.at(i, j0 + lr0 + c)] = closed ? T(double(ph) - m) : ph;
  }
  if (rank == 0 && t == 0) {
    const int it = iter < a.max_iter ? iter : a.max_iter;
    a.out->iters = it;
    a.out->res = sqrt(rr) / rhs_norm;
    a.out->total_iters += (unsigned long long)it;
    if (a.timed) a.out->timed_iters += (unsigned long long)it;
    a.out->calls += 1;
  }
  x.leave();
#undef COL_CELLS
}
template <int CPT>
__global__ void __launch_bounds__(PCGC_TPB, 1) k_pcg_column(PcgClusterArgs a) {
  if (a.active && !*a.active) return;
  cgc::cluster_group cl = cgc::this_cluster();
  pcg_column_body<CPT>(a, (int)cl.block_rank(), (int)cl.num_blocks());
}
inline const void* pcg_column_fn(int cpt) {
  switch (cpt) {
    case 1: return (const void*)k_pcg_column<1>;
    case 2: return (const void*)k_pcg_column<2>;
    case 4: return (const void*)k_pcg_column<4>;
    case 8: return (const void*)k_pcg_column<8>;
    case 16: return (const void*)k_pcg_column<16>;
  }
  return nullptr;
}
// threads of a launch: every strip's, to a power of two (the sums' trees)
inline int pcg_column_tpb(int nx, int rows_per, int cpt) {
  int tpb = 32;
  while (tpb < nx * ((rows_per + cpt - 1) / cpt)) tpb *= 2;
  return tpb;
}

// ------------------------------------------------------------- lean variant
constexpr int PCGC_LEAN_CPT = 32;  // cells of a thread's strip
// shared-memory footprint in floats for rows_per rows of nx cells: p_k of the
// CTA's cells, 4 halo rows, cx, cy and dinv
__host__ __device__ inline long pcgc_smem_elems(int nx, int rows_per) {
  return (long)rows_per * nx + 4L * nx + (long)rows_per * (nx + 1) + (long)(rows_per + 1) * nx + (long)rows_per * nx;
}

__device__ __forceinline__ void pcg_cluster_lean_body(const PcgClusterArgs& a) {
  using T = float;
  constexpr int CPT = PCGC_LEAN_CPT;
  cgc::cluster_group cl = cgc::this_cluster();
  const int C = (int)cl.num_blocks();
  const int rank = (int)cl.block_rank();
  const Geo g = a.g;
  const int nx = g.nx, ny = g.ny, rp = a.rows_per;
  const int j0 = 1 + rank * rp;
  const int R = min(rp, ny - rank * rp);  // rows of this CTA (>= 1)
  const bool closed = !g.px && !g.py;
  const int S = (R + CPT - 1) / CPT;       // strips per column
  const int t = threadIdx.x;
  const bool act = t < nx * S;
  const int i = act ? t % nx + 1 : 1;
  const int lr0 = act ? (t / nx) * CPT : 0;
  const int nr = act ? min(CPT, R - lr0) : 0;
  const int ie = (i < nx) ? i + 1 : (g.px ? 1 : nx);
  const int iw = (i > 1) ? i - 1 : (g.px ? nx : 1);

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* pcs = reinterpret_cast<T*>(smem_raw);  // p_k of the CTA's cells, rp x nx
  T* zt = pcs + rp * nx;                     // z of the row above the CTA
  T* zb = zt + nx;                           // z of the row below
  T* pt = zb + nx;                           // p of the row above
  T* pb = pt + nx;                           // p of the row below
  T* cxs = pb + nx;
  T* cys = cxs + rp * (nx + 1);
  T* dis = cys + (rp + 1) * nx;
  __shared__ double sh[32];
  __shared__ double red[6];  // 0 pAp, 1 rr, 2 rz, 3 sum / mean, 4 rhs norm, 5 initial rz

  // cluster sum: block sum -> own slot -> barrier -> every CTA merges the C
  // slots in rank order (identical everywhere).  The float products are exact
  // in double and summed in a fixed order.
  __shared__ double sh2[32];
  auto bsum2 = [&](double v, double u, double& dv, double& du) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
      v += __shfl_down_sync(0xffffffffu, v, o);
      u += __shfl_down_sync(0xffffffffu, u, o);
    }
    __syncthreads();
    if (l == 0) {
      sh[w] = v;
      sh2[w] = u;
    }
    __syncthreads();
    if (w == 0) {
      v = l < nw ? sh[l] : 0.0;
      u = l < nw ? sh2[l] : 0.0;
      for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_down_sync(0xffffffffu, v, o);
        u += __shfl_down_sync(0xffffffffu, u, o);
      }
      if (l == 0) {
        dv = v;
        du = u;
      }
    }
  };
  // merge the C slots after a cluster barrier: lane r of warp 0 loads rank
  // r's slot (one DSMEM round trip for all ranks), a fixed shuffle tree sums
  // them, and the result is broadcast through shared memory.  Two slots can
  // be merged in the same pass (slot2 < 0: one).
  __shared__ double bcast[2];
  auto merge2 = [&](int slot, int slot2) {
    if (threadIdx.x < 32) {
      const int l = threadIdx.x;
      double a0 = 0.0, a1 = 0.0;
      if (l < C) {
        a0 = *cl.map_shared_rank(&red[slot], l);
        if (slot2 >= 0) a1 = *cl.map_shared_rank(&red[slot2], l);
      }
      for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_down_sync(0xffffffffu, a0, o);
        a1 += __shfl_down_sync(0xffffffffu, a1, o);
      }
      if (l == 0) {
        bcast[0] = a0;
        bcast[1] = a1;
      }
    }
    __syncthreads();
  };
  auto csum = [&](double acc, int slot) -> double {
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) red[slot] = acc;
    cl.sync();
    merge2(slot, -1);
    return bcast[0];
  };
  // owners of the CTA's first / last row publish z and p into the halo rows
  // of the neighbouring CTAs (the row above CTA r-1 is my first row, the row
  // below CTA r+1 is my last row)
  auto push = [&](int c, T zv, T pv) {
    const int lr = lr0 + c;
    if (lr == 0 && (rank > 0 || g.py)) {
      const int dst = (rank - 1 + C) % C;
      cl.map_shared_rank(zt, dst)[i - 1] = zv;
      cl.map_shared_rank(pt, dst)[i - 1] = pv;
    }
    if (lr == R - 1 && (rank < C - 1 || g.py)) {
      const int dst = (rank + 1) % C;
      cl.map_shared_rank(zb, dst)[i - 1] = zv;
      cl.map_shared_rank(pb, dst)[i - 1] = pv;
    }
  };

  // ---- coefficients of the own rows
  for (int q = threadIdx.x; q < R * (nx + 1); q += blockDim.x) {
    const int lr = q / (nx + 1), ii = q % (nx + 1);
    cxs[lr * (nx + 1) + ii] = a.cx[g.at(ii, j0 + lr)];
  }
  for (int q = threadIdx.x; q < (R + 1) * nx; q += blockDim.x) {
    const int lf = q / nx - 1, ii = q % nx + 1;  // face rows j0-1 .. j0+R-1
    cys[(lf + 1) * nx + (ii - 1)] = a.cy[g.at(ii, j0 + lf)];
  }
  for (int q = threadIdx.x; q < R * nx; q += blockDim.x) dis[q] = a.dinv[g.at(q % nx + 1, j0 + q / nx)];

  T phi_r[CPT], r_r[CPT], ap_r[CPT];
  // z and p_k of the own cell in local row lr
#define PCGC_Z(c, lr) (dis[(lr) * nx + (i - 1)] * r_r[c])
#define PCGC_P(c, lr) pcs[(lr) * nx + (i - 1)]
#define PCGC_CELLS _Pragma("unroll") for (int c = 0; c < CPT; ++c)
#define PCGC_CELL             \
  if (c >= nr) continue;      \
  const int lr = lr0 + c;     \
  const int j = j0 + lr;      \
  (void)j;

  // ---- (b) zero-mean projection and rhs norm
  double mean = 0.0;
  if (closed) {
    double s = 0.0;
    PCGC_CELLS { PCGC_CELL s += double(a.rhs[g.at(i, j)]); }
    mean = csum(s, 3) / (double)(nx * ny);
  }
  double ss = 0.0;
  PCGC_CELLS {
    PCGC_CELL
    const T rw = closed ? T(double(a.rhs[g.at(i, j)]) - mean) : a.rhs[g.at(i, j)];
    r_r[c] = rw;
    ss += double(rw) * double(rw);
  }
  const double rhs_norm = sqrt(csum(ss, 4));
  if (rhs_norm < 1.0e-14) {
    const long tot = g.n();
    for (long q = rank * (long)blockDim.x + threadIdx.x; q < tot; q += (long)C * blockDim.x) a.phi[q] = T(0);
    if (rank == 0 && threadIdx.x == 0) {
      a.out->iters = 0;
      a.out->res = 0.0;
      a.out->calls += 1;
    }
    cl.sync();
    return;
  }

  // ---- (c) phi ghosts (halo + Neumann), initial residual, z, p_1 = z
  if (!a.phi_zero) {
    const long tot = g.n();
    for (long q = rank * (long)blockDim.x + threadIdx.x; q < tot; q += (long)C * blockDim.x) {
      const int gi = (int)(q % g.P) - 2, gj = (int)(q / g.P) - 2;
      if (gi < -1 || gj < -1 || gi > nx + 2 || gj > ny + 2) continue;
      if (gi >= 1 && gi <= nx && gj >= 1 && gj <= ny) continue;
      const int mi = (gi >= 1 && gi <= nx) ? gi : (g.px ? (gi < 1 ? gi + nx : gi - nx) : (gi < 1 ? 1 - gi : 2 * nx + 1 - gi));
      const int mj = (gj >= 1 && gj <= ny) ? gj : (g.py ? (gj < 1 ? gj + ny : gj - ny) : (gj < 1 ? 1 - gj : 2 * ny + 1 - gj));
      a.phi[q] = a.phi[g.at(mi, mj)];
    }
  }
  __syncthreads();  // coefficients in shared memory
  double rz = 0.0;
  PCGC_CELLS {
    PCGC_CELL
    T rr = r_r[c];
    T ph = T(0);
    if (!a.phi_zero) {
      const T* gp = a.phi;
      ph = gp[g.at(i, j)];
      const T apv = poisson_ap<T>(g, a.cx, a.cy, i, j, [&](int x, int y) { return gp[g.at(x, y)]; });
      rr = rr - apv;
    }
    const T zz = dis[lr * nx + (i - 1)] * rr;
    phi_r[c] = ph;
    r_r[c] = rr;
    push(c, zz, zz);
    rz += double(rr) * double(zz);
  }
  double rz_old = csum(rz, 5);  // its barrier also publishes the halos

  double res_norm = 0.0, beta = 0.0;
  int iter;
  for (iter = 1; iter <= a.max_iter; ++iter) {
    const T tb = T(beta);
    // phase A: p_k of the own cells, then A p_k
    PCGC_CELLS {
      PCGC_CELL
      const T zk = PCGC_Z(c, lr);
      const T pk = (iter == 1) ? zk : madd(tb, PCGC_P(c, lr), zk);
      pcs[lr * nx + (i - 1)] = pk;
    }
    __syncthreads();
    double papd = 0.0;
    PCGC_CELLS {
      PCGC_CELL
      const T pk = PCGC_P(c, lr);
      const T cE = cxs[lr * (nx + 1) + i], cW = cxs[lr * (nx + 1) + i - 1];
      const T cN = cys[(lr + 1) * nx + (i - 1)], cS = cys[lr * nx + (i - 1)];
      const T pE = pcs[lr * nx + (ie - 1)], pW = pcs[lr * nx + (iw - 1)];
      T pN, pS;
      if (j == ny && !g.py) pN = pk;
      else if (c + 1 < nr) pN = PCGC_P(c + 1, lr + 1);
      else if (lr + 1 < R) pN = pcs[(lr + 1) * nx + (i - 1)];
      else pN = (iter == 1) ? zt[i - 1] : madd(tb, pt[i - 1], zt[i - 1]);
      if (j == 1 && !g.py) pS = pk;
      else if (c > 0) pS = PCGC_P(c - 1, lr - 1);
      else if (lr > 0) pS = pcs[(lr - 1) * nx + (i - 1)];
      else pS = (iter == 1) ? zb[i - 1] : madd(tb, pb[i - 1], zb[i - 1]);
      // (cE + cW + cN + cS) pk - (((cE pE + cW pW) + cN pN) + cS pS)
      const T off = madd(cS, pS, madd(cN, pN, madd(cW, pW, cE * pE)));
      const T apv = madd(cE + cW + cN + cS, pk, -off);
      ap_r[c] = apv;
      papd += double(pk) * double(apv);
    }
    const double pap = csum(papd, 0);  // barrier: every CTA is done reading pcs / halos
    if (fabs(pap) < 1.0e-30) break;
    const double alpha = rz_old / pap;
    const T ta = T(alpha);
    // phase B: phi, r, z updates; publish the boundary rows' z and p_k
    double rrd = 0.0, rzd = 0.0;
    PCGC_CELLS {
      PCGC_CELL
      const T rv = madd(-ta, ap_r[c], r_r[c]);
      const T zv = dis[lr * nx + (i - 1)] * rv;
      const T pk = PCGC_P(c, lr);
      phi_r[c] = madd(ta, pk, phi_r[c]);
      r_r[c] = rv;
      push(c, zv, pk);
      rrd += double(rv) * double(rv);
      rzd += double(rv) * double(zv);
    }
    bsum2(rrd, rzd, red[1], red[2]);
    cl.sync();
    merge2(1, 2);
    res_norm = sqrt(bcast[0]);
    if (res_norm / rhs_norm < a.tol) break;
    const double rz_new = bcast[1];
    beta = rz_new / rz_old;
    rz_old = rz_new;
  }
  if (closed) {
    double s = 0.0;
    PCGC_CELLS { PCGC_CELL s += double(phi_r[c]); }
    const double m = csum(s, 3) / (double)(nx * ny);
    PCGC_CELLS { PCGC_CELL phi_r[c] = T(double(phi_r[c]) - m); }
  }
  PCGC_CELLS { PCGC_CELL a.phi[g.at(i, j)] = phi_r[c]; }
  if (rank == 0 && threadIdx.x == 0) {
    const int it = iter < a.max_iter ? iter : a.max_iter;
    a.out->iters = it;
    a.out->res = res_norm / rhs_norm;
    a.out->total_iters += (unsigned long long)it;
    if (a.timed) a.out->timed_iters += (unsigned long long)it;
    a.out->calls += 1;
  }
  cl.sync();  // no CTA leaves while another may still read its shared memory
#undef PCGC_CELLS
#undef PCGC_CELL
#undef PCGC_Z
#undef PCGC_P
}
__global__ void __launch_bounds__(PCGC_TPB, 1) k_pcg_cluster_lean(PcgClusterArgs a) {
  if (a.active && !*a.active) return;
  pcg_cluster_lean_body(a);
}

}  // namespace fugu
