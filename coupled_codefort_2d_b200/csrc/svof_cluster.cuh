// svof_cluster.cuh -- the SVOF Helmholtz filter (svof_helmholtz_filter,
// mod_vof.f90:145-194) resident in one thread-block cluster, several Jacobi
// sweeps per exchange.
//
// The grid-wide kernel (k_svof, persistent.cuh) pays a grid barrier and a pass
// over L2 per sweep, 2.6 us at 256 x 256.  Here CTA r owns rows of cells,
// thread t a column strip of them in registers (east, west and strip-end
// neighbours through two alternating shared-memory buffers), and every
// SVOF_T sweeps the CTAs exchange SVOF_T boundary rows: a CTA keeps that many
// rows of its neighbours and sweeps them too, one row less each time, with
// their owners' expressions.  The stopping test (largest change < tol) is a
// bit per sweep, or-ed over the cluster with the rows.  A filter that stops
// inside a group of sweeps goes back to the group's start (kept in the work
// buffer and the received rows) and repeats the sweeps up to the stop, so the
// result and the sweep count are those of one test per sweep.  The division
// by the constant diagonal is the exact quotient (pcg_exchange.cuh), and a
// division where that is not exact (svofc_exact).  A sweep is straight-line code: every thread sweeps CPT
// rows, whether they are the CTA's own, kept or padding, and a row whose
// neighbour is not there repeats itself (at a wall that is the mirror; beyond
// the kept rows the value is not used again before it is received anew).
// What bounds it: the FP64 operations of the rows of a SM (11 per cell and
// sweep at 64 per cycle) and the barrier between sweeps.
// us on a B200 before and now (sweeps to the step's tolerance): 64 x 128 (71)
// 238 -> 43, 128 x 256 (73) 249 -> 85, 256 x 256 (115) 392 -> 240, 192 x 384
// (73) 249 -> 177; a batch's cases, which ran the grid-wide kernel on 8 CTAs,
// gain more.  256 x 512 needs 24 rows per thread, which spill (528 against
// 319), so it and wider grids keep the grid-wide kernel.
#pragma once

#include "pcg_exchange.cuh"
#include "persistent.cuh"

namespace fugu {

constexpr int SVOFC_TPB = 512;
constexpr int SVOF_T = 4;  // sweeps per exchange

struct SvofClusterArgs {
  SvofArgs a;
  int rows_per;  // rows of every CTA but possibly the last (at least SVOF_T each)
  CxLimit wait;
};
// shared memory in doubles: two buffers of every thread's rows, and the
// received rows [parity][bottom, top][SVOF_T]
inline long svofc_smem_elems(int nx, int cpt) { return 2L * (SVOFC_TPB / nx) * cpt * nx + 4L * SVOF_T * nx; }

// Whether quotient(num, diag, 1 / diag) is num / diag for a diag within
// [1, 2^100]: +0 or |num| in [2^-900, 2^900), where the remainder is exact.  Not
// for infinities, NaN, -0 and values whose remainder would underflow.  Of the
// filter's time the test takes 4 us at 64 x 128 and 28 us at 256 x 256 (212 us
// without it), 9-13 %.
__device__ __forceinline__ bool svofc_exact(double num) {
  const unsigned hi = (unsigned)__double2hiint(num), w = hi * 2u;
  return w - (123u << 21) < (1800u << 21) || (hi | (unsigned)__double2loint(num)) == 0u;
}

template <int CPT>
__global__ void __launch_bounds__(SVOFC_TPB, 1) k_svof_cluster(SvofClusterArgs p) {
  cgc::cluster_group cl = cgc::this_cluster();
  const SvofArgs& a = p.a;
  const Geo g = a.g;
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int nx = g.nx, ny = g.ny, rp = p.rows_per;
  const int j0 = 1 + rank * rp, R = min(rp, ny - rank * rp);
  const bool has_bot = rank > 0 || g.py, has_top = rank < C - 1 || g.py;
  const int below = rank > 0 ? rank - 1 : C - 1, above = rank < C - 1 ? rank + 1 : 0;
  const int hb = has_bot ? SVOF_T : 0, RR = R + hb + (has_top ? SVOF_T : 0);  // rows with the kept ones
  const int strips = SVOFC_TPB / nx, t = threadIdx.x;
  const bool act = t < strips * nx;
  const int strip = act ? t / nx : 0, col = act ? t % nx : 0;
  const int q0 = strip * CPT;
  const int de = col + 1 < nx ? 1 : (g.px ? 1 - nx : 0), dw = col > 0 ? -1 : (g.px ? nx - 1 : 0);

  extern __shared__ __align__(16) double svofc_smem[];
  double* S0 = svofc_smem;  // two buffers, strips * CPT rows of nx
  const int ss = strips * CPT * nx;  // buffer stride
  double* hw = S0 + 2 * ss;
  const int at = q0 * nx + col;  // the thread's first cell in a buffer
  __shared__ unsigned mask[2], rcv[2][CX_MAXC];
  __shared__ __align__(8) unsigned long long mbar[2];
  __shared__ int s_fail;
  if (t == 0) {
    mask[0] = mask[1] = 0u;
    s_fail = 0;
    for (int b = 0; b < 2; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the thread's own rows, as bits, and the cells it takes over on each change
  unsigned own = 0u;
#pragma unroll
  for (int c = 0; c < CPT; ++c)
    if (act && q0 + c >= hb && q0 + c < hb + R) own |= 1u << c;
  const int ctop = RR - 1 - q0;  // the strip's row without a row above (if in 0..CPT-1)
  double v[CPT], cr[CPT];
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    int j = j0 + min(q0 + c, RR - 1) - hb;  // a kept row's row in the grid (periodic y wraps)
    j = j < 1 ? j + ny : j > ny ? j - ny : j;
    cr[c] = a.craw[g.at(col + 1, j)];
    v[c] = cr[c];
    if (act) S0[at + c * nx] = v[c];
  }
  cl.sync();  // the mbarriers are initialised before any push
  const double diag = a.diag, idiag = 1.0 / diag;
  const bool usual = diag >= 1.0 && diag <= 0x1p100;
  int cur = 0;
  // one sweep; true when a cell of the thread's own rows changed by tol or more
  auto sweep = [&]() -> bool {
    if (!act) return false;
    const double* S = S0 + cur * ss + at;
    double* D = S0 + (cur ^ 1) * ss + at;
    double so = strip > 0 ? S[-nx] : v[0];  // the old value below
    const double nend = strip + 1 < strips ? S[CPT * nx] : v[CPT - 1];
    unsigned big = 0u, odd = 0u;
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const double old = v[c];
      const double e = S[c * nx + de], w = S[c * nx + dw];
      double nn = c + 1 < CPT ? v[c + 1 < CPT ? c + 1 : c] : nend;
      if (c == ctop) nn = old;
      const double num = cr[c] + a.cx * (e + w) + a.cy * (nn + so);
      const double val = quotient(num, diag, idiag);
      const bool exact = usual && svofc_exact(num);
      if (!exact) odd |= 1u << c;
      v[c] = val;
      D[c * nx] = exact ? val : num;
      if (fabs(val - old) >= a.tol) big |= 1u << c;
      so = old;
    }
    if (odd) {  // rarely: divide what the quotient is not exact for
#pragma unroll 1
      for (int c = 0; c < CPT; ++c)
        if ((odd >> c) & 1u) D[c * nx] = D[c * nx] / diag;
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        if ((odd >> c) & 1u) {
          v[c] = D[c * nx];
          big = fabs(v[c] - S[c * nx]) >= a.tol ? big | 1u << c : big & ~(1u << c);
        }
    }
    return (big & own) != 0u;
  };
  // the kept rows of a group's start: received, or at the first group the input's
  auto take_kept = [&](const double* h, bool first, bool own_too) {
    if (!act) return;
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const int q = q0 + c;
      if (q >= RR) continue;
      if ((own >> c) & 1u) {
        if (!own_too) continue;
        v[c] = a.work[g.at(col + 1, j0 + q - hb)];
      } else {
        v[c] = first ? cr[c] : q < hb ? h[q * nx + col] : h[(SVOF_T + q - hb - R) * nx + col];
      }
      S0[cur * ss + at + c * nx] = v[c];
    }
  };
  const bool tests = a.tol > 0.0;
  unsigned ep = 0;
  int done = 0, used = 0;
  bool failed = false;
  while (done < a.max_iter) {
    const int T = min(SVOF_T, a.max_iter - done);
    if (done > 0) {  // the rows received with the last exchange
      take_kept(hw + ((ep - 1) & 1u) * 2 * SVOF_T * nx, false, false);
      __syncthreads();
    }
    if (tests && T > 1) {  // the group's start, in case it stops inside
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        if ((own >> c) & 1u) a.work[g.at(col + 1, j0 + q0 + c - hb)] = v[c];
    }
    unsigned bits = 0u;
    for (int s = 1; s <= T; ++s) {
      if (sweep()) bits |= 1u << (s - 1);
      cur ^= 1;
      __syncthreads();
    }
    const bool last = done + T >= a.max_iter;
    const unsigned par = ep & 1u, mb = smem_u32(&mbar[par]);
    if (t == 0)
      asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(mb),
                   "r"((unsigned)(4 * C) + p.wait.extra_bytes + (last ? 0u : (unsigned)(((int)has_bot + (int)has_top) * SVOF_T * nx * 8)))
                   : "memory");
    if (!last) {
      const unsigned hp = smem_u32(hw + par * 2 * SVOF_T * nx);
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        if ((own >> c) & 1u) {
          const int lr = q0 + c - hb;
          // my first rows are the top kept rows of the CTA below, my last rows the bottom ones of the CTA above
          if (lr < SVOF_T && has_bot)
            push8(mapa(hp + (unsigned)(((SVOF_T + lr) * nx + col) * 8), below), mapa(mb, below), v[c]);
          if (lr >= R - SVOF_T && has_top)
            push8(mapa(hp + (unsigned)(((lr - R + SVOF_T) * nx + col) * 8), above), mapa(mb, above), v[c]);
        }
    }
    bits = __reduce_or_sync(0xffffffffu, bits);
    if ((t & 31) == 0 && bits) atomicOr(&mask[par], bits);
    __syncthreads();
    if (t < C) {
      const unsigned dst = mapa(smem_u32(&rcv[par][rank]), t);
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
                   "r"(mask[par]), "r"(mapa(mb, t))
                   : "memory");
    }
    if (t < 32) {
      unsigned spins = 0;
      bool ok = true;
      while (!mbar_test(mb, (ep >> 1) & 1u))
        if (++spins > p.wait.polls()) {
          ok = false;
          break;
        }
      const unsigned m = __reduce_or_sync(0xffffffffu, t < C ? rcv[par][t] : 0u);
      __syncwarp();
      if (t == 0) {
        mask[par ^ 1u] = 0u;  // the next exchange's (every warp is past the last one's)
        rcv[par][0] = m;
      }
      if (!ok) s_fail = 1;
    }
    __syncthreads();
    if (s_fail) {
      failed = true;
      break;
    }
    const unsigned m = rcv[par][0];
    ++ep;
    int stop = 0;  // the sweep of this group that met the test
    for (int s = T; s >= 1; --s)
      if (tests && !((m >> (s - 1)) & 1u)) stop = s;
    used = done + (stop ? stop : T);
    if (stop && stop < T) {
      // back to the group's start, then the sweeps up to the stop
      take_kept(hw + (ep & 1u) * 2 * SVOF_T * nx, done == 0, true);  // received before the group
      __syncthreads();
      for (int s = 1; s <= stop; ++s) {
        sweep();
        cur ^= 1;
        __syncthreads();
      }
    }
    if (stop) break;
    done += T;
  }
  if (failed) {
    if (t == 0) *a.status = 1;
    __nanosleep(200000);  // pushes still in flight land before anyone leaves
  } else {
#pragma unroll
    for (int c = 0; c < CPT; ++c)
      if ((own >> c) & 1u) a.out[g.at(col + 1, j0 + q0 + c - hb)] = v[c];
  }
  cl.sync();
  // every ghost of C_smooth from its interior (halo + Neumann); the padding as in craw
  for (long q = rank * (long)blockDim.x + t; q < g.n(); q += (long)C * blockDim.x) {
    const int i = (int)(q % g.P) - 2, j = (int)(q / g.P) - 2;
    if (i >= 1 && i <= nx && j >= 1 && j <= ny) continue;
    if (i < -1 || j < -1 || i > nx + 2 || j > ny + 2) {
      a.out[q] = a.craw[q];
      continue;
    }
    const int mi = (i >= 1 && i <= nx) ? i : (g.px ? (i < 1 ? i + nx : i - nx) : (i < 1 ? 1 - i : 2 * nx + 1 - i));
    const int mj = (j >= 1 && j <= ny) ? j : (g.py ? (j < 1 ? j + ny : j - ny) : (j < 1 ? 1 - j : 2 * ny + 1 - j));
    a.out[q] = __ldcg(a.out + g.at(mi, mj));
  }
  if (rank == 0 && t == 0) *a.iters += used;
}
// the strip's rows, from those built, for rows_per rows and the kept ones (0: too many)
inline int svofc_cpt(int nx, int rows_per) {
  const int strips = SVOFC_TPB / nx, need = (rows_per + 2 * SVOF_T + strips - 1) / strips;
  for (int k : {1, 2, 3, 4, 6, 8, 12, 16})
    if (k >= need) return k;
  return 0;
}
inline const void* svof_cluster_fn(int cpt) {
  switch (cpt) {
    case 1: return (const void*)k_svof_cluster<1>;
    case 2: return (const void*)k_svof_cluster<2>;
    case 3: return (const void*)k_svof_cluster<3>;
    case 4: return (const void*)k_svof_cluster<4>;
    case 6: return (const void*)k_svof_cluster<6>;
    case 8: return (const void*)k_svof_cluster<8>;
    case 12: return (const void*)k_svof_cluster<12>;
    case 16: return (const void*)k_svof_cluster<16>;
  }
  return nullptr;
}

}  // namespace fugu
