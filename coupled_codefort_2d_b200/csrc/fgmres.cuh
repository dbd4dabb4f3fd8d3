// fgmres.cuh -- flexible GMRES(m) with right PCD preconditioning (extension,
// not in the reference): the inner solve of the FP64 defect correction when
// refine = 2.  The reference's BiCGStab(l) needs a fixed preconditioner; PCD
// around a truncated PCG is not one, and BiCGStab(2) diverges on high
// density-ratio bubbles, while flexible GMRES keeps Z_j = M^{-1} V_j and
// minimises the true residual over span(Z).
//
// Device pieces: a multi-vector coupled dot (all projections of one
// Gram-Schmidt pass in one launch), a multi-vector axpy, the scale of a new
// basis vector, and the scalar steps (projections into H, Givens rotations,
// the small triangular solve), which run in the last CTA of the reductions
// like the BiCGStab recurrences do.
#pragma once

#include "pcg_exchange.cuh"
#include "scalars.cuh"

namespace fugu {

// device-resident scalars of one FGMRES cycle (doubles)
struct FgLayout {
  int m;  // Arnoldi steps of the cycle
  __host__ __device__ int H(int i, int j) const { return i + j * (m + 1); }  // (m+1) x m, column-major
  __host__ __device__ int cs() const { return (m + 1) * m; }
  __host__ __device__ int sn() const { return cs() + m; }
  __host__ __device__ int g() const { return sn() + m; }
  __host__ __device__ int y() const { return g() + m + 1; }
  __host__ __device__ int h() const { return y() + m; }  // projections of the current pass
  __host__ __device__ int beta() const { return h() + m + 1; }
  __host__ __device__ int inv() const { return beta() + 1; }  // scale of the next basis vector
  __host__ __device__ int rel() const { return beta() + 2; }
  __host__ __device__ int size() const { return beta() + 3; }
};

enum FgOp {
  FG_BETA = 0,  // beta = |B|; V_0 scale; g[0] = beta; exit when beta == 0
  FG_PROJ1,     // first Gram-Schmidt pass: h = d, H[0..j, j] = 0 + d
  FG_PROJ2,     // second pass: h = d, H[0..j, j] += d
  FG_ROTATE,    // H[j+1, j] = |w|, Givens rotations, g, rel, exit test
};

// FG_BETA and FG_ROTATE by one thread, from copies of H's column j, cs and sn
__device__ inline void fg_op(int op, const double* d, int j, double tol, const FgLayout L, double* st, KState* ks,
                             const double* col, const double* cs, const double* sn, double gj, double beta0) {
  switch (op) {
    case FG_BETA: {
      const double beta = sqrt(d[0]);
      st[L.beta()] = beta;
      st[L.g()] = beta;
      st[L.inv()] = beta > 0.0 ? 1.0 / beta : 0.0;
      st[L.rel()] = beta > 0.0 ? 1.0 : 0.0;
      if (isnan(beta)) ks->nan = 1;
      if (!(beta > 0.0)) kexit(ks, 0);
      break;
    }
    case FG_ROTATE: {
      const double hn = sqrt(d[0]);
      double* H = st + L.H(0, j);
      double* g = st + L.g();
      double b = col[0];
      for (int i = 0; i < j; ++i) {
        const double a = b, n = col[i + 1];
        H[i] = cs[i] * a + sn[i] * n;
        b = -sn[i] * a + cs[i] * n;
      }
      const double a = b;
      b = hn;
      const double rr = sqrt(a * a + b * b);
      const double c = rr > 0.0 ? a / rr : 1.0, s = rr > 0.0 ? b / rr : 0.0;
      st[L.cs() + j] = c;
      st[L.sn() + j] = s;
      H[j] = rr;
      H[j + 1] = 0.0;
      const double gn = -s * gj;
      g[j + 1] = gn;
      g[j] = c * gj;
      const double rel = fabs(gn) / beta0;
      st[L.rel()] = rel;
      st[L.inv()] = hn > 0.0 ? 1.0 / hn : 0.0;
      if (isnan(rel)) ks->nan = 1;
      if (rel < tol || hn == 0.0 || j + 1 == L.m || isnan(rel)) kexit(ks, j + 1);
      break;
    }
  }
}

// coupled dots of w with nvec vectors V_i = V0 + i * stride.  The work items
// are chunks of MDOT_CHUNK consecutive unknowns of one grid row of one
// component (u, v or p rows of the owned interior), so a warp reads contiguous
// memory and maps an item to its row once.  Each CTA keeps one DD partial for
// its vector; the last CTA merges them and does the scalar step.  Launch: grid
// (Gx, nvec) of MDOT_TPB threads, grid row y computing the dot with V_y.
// Latency-bound on the grids of a step: what counts is the dependent chain
// after the products.  The last CTA's warps share the partials of a vector with
// four loads in flight each (a norm has up to four partials per SM, and one
// warp read them a round trip apart), H's column is updated by a thread per
// entry, and the rotation's inputs are read beside the partials.  B200, FP32, mean us
// of the first launches of a step under a profiler: 8.3 -> 7.9 at 64 x 128,
// 13.9 -> 11.9 at 320 x 640.
constexpr int MDOT_TPB = 256;
constexpr int MDOT_CHUNK = 128;
constexpr int MDOT_MAXV = 128;

template <typename T>
struct MdotArgs {
  Geo g;
  long n;  // elements of one component buffer
  const T* w;
  const T* V0;
  long stride;
  int nvec;      // <= MDOT_MAXV
  double vol;
  double* part;  // >= 2 * nvec * gridDim.x
  double* st;
  KState* ks;
  FgLayout L;
  int op, j;
  double tol;
};

// number of work items of a grid (u rows, v rows, p rows in MDOT_CHUNK pieces)
__host__ __device__ inline long mdot_items(const Geo& g) {
  const long cu = (g.imax() + MDOT_CHUNK - 1) / MDOT_CHUNK, cv = (g.nx + MDOT_CHUNK - 1) / MDOT_CHUNK;
  return (long)g.ny * cu + (long)g.jmax() * cv + (long)g.ny * cv;
}

// CTA (bx, by) of a (Gx, Gy = nvec) grid
// a lane's running sum of its products: error-free (double-double) for the
// FP64 parity path; the FP32 inner solve needs only a fixed order, so a plain
// double sum of its (exact) float products serves there at a fraction of the
// dependent FP64 work
template <typename T>
__device__ __forceinline__ void mdot_acc(DD& acc, double x) {
  if constexpr (sizeof(T) == 8) dd_add(acc, x);
  else acc.hi += x;
}
template <typename T>
__device__ __forceinline__ void mdot_body(const MdotArgs<T>& a, int bx, int by, int Gx, int Gy) {
  constexpr int NW = MDOT_TPB / 32;
  __shared__ DD wsum[NW], vsum[MDOT_MAXV];
  __shared__ double dsum[1], rot[3][MDOT_MAXV + 1];
  __shared__ bool last;
  const Geo g = a.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = g.nx, ny = g.ny, imax = g.imax(), jmax = g.jmax();
  const int cu = (imax + MDOT_CHUNK - 1) / MDOT_CHUNK, cv = (nx + MDOT_CHUNK - 1) / MDOT_CHUNK;
  const long iu = (long)ny * cu, iv = (long)jmax * cv, ip = (long)ny * cv;
  const long items = iu + iv + ip;
  const T* V = a.V0 + by * a.stride;  // this grid row's vector
  DD acc{0.0, 0.0};
  for (long it = (long)bx * NW + warp; it < items; it += (long)Gx * NW) {
    long base;
    int len, c;
    if (it < iu) {
      c = (int)(it % cu);
      base = g.at(1, 1 + (int)(it / cu));
      len = imax;
    } else if (it < iu + iv) {
      const long r = it - iu;
      c = (int)(r % cv);
      base = a.n + g.at(1, 1 + (int)(r / cv));
      len = nx;
    } else {
      const long r = it - iu - iv;
      c = (int)(r % cv);
      base = 2 * a.n + g.at(1, 1 + (int)(r / cv));
      len = nx;
    }
    const int i0 = c * MDOT_CHUNK + lane, i1 = min(len, (c + 1) * MDOT_CHUNK);
    if (i1 - c * MDOT_CHUNK == MDOT_CHUNK) {
      // a full chunk: issue the lane's 2 x 4 loads before the dependent
      // double-double chain (same accumulation order as the loop below)
      constexpr int U = MDOT_CHUNK / 32;
      T wv[U], vv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        wv[u] = a.w[base + i0 + 32 * u];
        vv[u] = V[base + i0 + 32 * u];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) mdot_acc<T>(acc, (double(wv[u]) * double(vv[u])) * a.vol);
    } else {
      for (int i = i0; i < i1; i += 32) {
        const long e = base + i;
        mdot_acc<T>(acc, (double(a.w[e]) * double(V[e])) * a.vol);
      }
    }
  }
  acc = rsum_warp<true, 1>(&acc);
  if (lane == 0) wsum[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    DD s = wsum[lane & (NW - 1)];
#pragma unroll
    for (int o = NW / 2; o > 0; o >>= 1) s = rsum_merge<true>(s, rsum_xor<true>(s, o));
    if (lane == 0) {
      put_partial(a.part + 2L * by * Gx, bx, s);
      __threadfence();
      const unsigned int t = atomicAdd(&a.ks->ticket, 1u);
      last = (t == (unsigned int)(Gx * Gy) - 1);
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the rotation's inputs, read beside the partials
  const int t = threadIdx.x;
  double gj = 0.0, beta0 = 0.0;
  if (a.op == FG_ROTATE) {
    for (int i = t; i <= a.j; i += MDOT_TPB) {
      rot[0][i] = a.st[a.L.H(i, a.j)];
      if (i < a.j) {
        rot[1][i] = a.st[a.L.cs() + i];
        rot[2][i] = a.st[a.L.sn() + i];
      }
    }
    gj = a.st[a.L.g() + a.j];
    beta0 = a.st[a.L.beta()];
  }
  // every warp reads: wpv of them share a vector's partials, U loads in flight
  constexpr int U = 4;
  const int wpv = max(1, NW / a.nvec), sub = warp % wpv;
  for (int v = warp / wpv; v < a.nvec; v += NW / wpv) {
    const double2* pv = reinterpret_cast<const double2*>(a.part) + (long)v * Gx;
    DD s{0.0, 0.0};
    for (int k = sub * 32 + lane; k < Gx; k += U * 32 * wpv) {
      double2 q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) q[u] = k + u * 32 * wpv < Gx ? __ldcg(pv + k + u * 32 * wpv) : double2{0.0, 0.0};
#pragma unroll
      for (int u = 0; u < U; ++u) s = rsum_merge<true>(s, DD{q[u].x, q[u].y});
    }
    s = rsum_warp<true, 1>(&s);
    if (lane == 0) vsum[v * wpv + sub] = s;
  }
  __syncthreads();
  for (int v = t; v < a.nvec; v += MDOT_TPB) {
    DD s = vsum[v * wpv];
    for (int k = 1; k < wpv; ++k) s = rsum_merge<true>(s, vsum[v * wpv + k]);
    const double d = s.hi + s.lo;
    if (v == 0) dsum[0] = d;
    if (a.op == FG_PROJ1 || a.op == FG_PROJ2) {
      double& h = a.st[a.L.H(v, a.j)];
      a.st[a.L.h() + v] = d;
      h = (a.op == FG_PROJ1 ? 0.0 : h) + d;
    }
  }
  if (t == 0) {
    a.ks->ticket = 0;
    fg_op(a.op, dsum, a.j, a.tol, a.L, a.st, a.ks, rot[0], rot[1], rot[2], gj, beta0);
  }
}
template <typename T>
__global__ void __launch_bounds__(MDOT_TPB) k_mdot(MdotArgs<T> a) {
  if (!a.ks->active) return;
  mdot_body<T>(a, blockIdx.x, blockIdx.y, gridDim.x, gridDim.y);
}

// w = (...((w + s_0 V_0) + s_1 V_1) ...) + s_{nvec-1} V_{nvec-1}, s_i = sign * coef[i],
// over every element of the triple (whole-array, as the reference's array
// expressions).  Each element takes the same updates in the same order
// however the elements are spread over threads, so the two paths below give
// the same bits.
template <typename T>
__device__ __forceinline__ void maxpy_body(long n3, T* w, const T* V0, long stride, const double* coef, int nvec,
                                           double sign, int b, int G) {
  __shared__ T s[MDOT_MAXV];  // the coefficients, converted once per CTA
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) s[i] = T(sign * coef[i]);
  __syncthreads();
  constexpr int W = VecW<T>::value;
  const long S = (long)G * blockDim.x;
  const bool aligned = ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(V0)) & 15u) == 0;
  if (n3 % W == 0 && stride % W == 0 && aligned) {
    // W consecutive elements per thread with 16-byte loads and stores, the
    // loads of up to eight vectors in flight before their updates: a
    // thread's elements are a few long, wide round trips rather than many
    // short ones (at 2048^2 a one-element-per-thread pass was latency-bound)
    for (long q = (b * (long)blockDim.x + threadIdx.x) * W; q < n3; q += S * W) {
      T x[W];
      ldv(w + q, x);
      for (int i = 0; i < nvec; i += 8) {
        T v[8][W];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (i + u < nvec) ldv(V0 + (i + u) * stride + q, v[u]);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (i + u < nvec) {
#pragma unroll
            for (int e = 0; e < W; ++e) x[e] = madd(s[i + u], v[u][e], x[e]);
          }
      }
      stv(w + q, x);
    }
    return;
  }
  for (long q = b * (long)blockDim.x + threadIdx.x; q < n3; q += S) {
    T x = w[q];
    // the loads of up to 16 vectors in flight together before the (ordered)
    // dependent updates: each group of loads costs one memory round trip,
    // so a projection on up to 16 vectors is one round trip per element
    for (int i = 0; i < nvec; i += 16) {
      T v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) v[u] = i + u < nvec ? V0[(i + u) * stride + q] : T(0);
#pragma unroll
      for (int u = 0; u < 16; ++u)
        if (i + u < nvec) x = madd(s[i + u], v[u], x);
    }
    w[q] = x;
  }
}
template <typename T>
__global__ void k_maxpy(long n3, T* w, const T* V0, long stride, const double* coef, int nvec, double sign,
                        const int* active) {
  if (active && !*active) return;
  maxpy_body<T>(n3, w, V0, stride, coef, nvec, sign, blockIdx.x, gridDim.x);
}

// dst = 0 + s * src (the reference-style array expression of a fresh vector)
template <typename T>
__global__ void k_fg_scale(long n3, T* dst, const T* src, const double* s, const int* active) {
  if (active && !*active) return;
  const T f = T(*s);
  const long S = (long)gridDim.x * blockDim.x;
  for (long q0 = blockIdx.x * (long)blockDim.x + threadIdx.x; q0 < n3; q0 += 4 * S) {
    T a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u * S < n3) a[u] = src[q0 + u * S];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u * S < n3) dst[q0 + u * S] = T(0) + f * a[u];
  }
}

// back substitution R y = g over the k columns used
__device__ __forceinline__ void fg_solve_body(double* st, FgLayout L, int k) {
  const double* g = st + L.g();
  double* y = st + L.y();
  for (int i = k - 1; i >= 0; --i) {
    double s = g[i];
    for (int q = i + 1; q < k; ++q) s -= st[L.H(i, q)] * y[q];
    const double hii = st[L.H(i, i)];
    y[i] = hii != 0.0 ? s / hii : 0.0;
  }
}
__global__ void k_fg_solve(double* st, FgLayout L, int k) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  fg_solve_body(st, L, k);
}

}  // namespace fugu
