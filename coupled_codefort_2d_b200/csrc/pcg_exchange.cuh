// pcg_exchange.cuh -- sums and boundary rows exchanged between the CTAs of a
// resident PCG solve without a barrier.
//
// A barrier followed by a read of the partial sums puts several dependent
// round trips on the critical path of a reduction (a grid barrier: the
// partial's store and its fence, the atomic arrival, the poll that sees the
// last arrival, the read of the partials).  Here the data carries its own
// arrival:
//   cluster  every CTA pushes its sums into the shared memory of all CTAs of
//            its thread-block cluster and its boundary rows into its
//            neighbours' (st.async), and waits on its own mbarrier for the
//            bytes it expects.  On a B200 a bare exchange of 8 bytes takes 357
//            cycles between 16 CTAs (236 between 2), an all-reduce of 16 x 512
//            threads 1,028 (FP32, one sum) to 2,063 (FP64, two sums).
//   grid     8-byte words in global memory hold four bytes of payload and the
//            32-bit number of the exchange, so a reader that sees the
//            expected number has the payload too (an aligned 8-byte access is
//            never torn).  One exchange costs the writer's store and the
//            reader's poll, about 1,300 cycles for 64 CTAs.
// Both alternate two sets of receive buffers by the parity of the exchange: a
// CTA sends exchange e + 2 only after it received every CTA's e + 1, which each
// CTA sends after it has read everything of e, so nothing is overwritten
// before all its readers are done.  The grid's numbers keep growing from
// launch to launch (Exchange::epoch), so nothing is cleared in between.  A launch
// in which a wait gave up leaves words of numbers that a later one would use, and
// a CTA that starts late may add some, so the host clears the buffers after it.
//
// Every wait is bounded: after its limit of polls, or when another CTA has
// flagged an error, allreduce returns false and the kernel unwinds.
#pragma once

#include <cooperative_groups.h>

#include <cstddef>

#include "fugu_internal.cuh"

namespace fugu {

namespace cgc = cooperative_groups;

// ------------------------------------------------------------------- sums
// A value being summed: an error-free pair (DDS; the parity path and the
// grid-wide forms) or a plain double in the high part.
// a + b: the high parts' TwoSum and the sum of the low parts; the pair is
// rounded once at the end, so it is not renormalised at every stage.
template <bool DDS>
__device__ __forceinline__ DD rsum_merge(DD a, DD b) {
  DD r{a.hi + b.hi, 0.0};
  if constexpr (DDS) {
    double e;
    two_sum(a.hi, b.hi, r.hi, e);
    r.lo = (a.lo + b.lo) + e;
  }
  return r;
}
template <bool DDS>
__device__ __forceinline__ DD rsum_xor(DD v, int o) {
  DD r{__shfl_xor_sync(0xffffffffu, v.hi, o), 0.0};
  if constexpr (DDS) r.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
  return r;
}
// Sums of NV (1, 2 or 3) values over a warp.  With several values the first
// stages exchange values instead of repeating the butterfly for each: a
// lane keeps half of its values and sends the other half.  Value q ends in
// lane rsum_lane<NV>(q).  The pairs of lanes added at each stage are those of
// a plain tree over 16, 8, 4, 2, 1.
template <int NV>
__host__ __device__ constexpr int rsum_lane(int q) {
  return NV == 1 ? 0 : NV == 2 ? 16 * q : q == 0 ? 0 : q == 1 ? 8 : 16;
}
template <bool DDS, int NV>
__device__ __forceinline__ DD rsum_warp(const DD* v) {
  const int lane = threadIdx.x & 31;
  DD a;
  int o = 16;
  if constexpr (NV == 1) {
    a = v[0];
  } else if constexpr (NV == 2) {
    const bool h = lane & 16;
    a = rsum_merge<DDS>(h ? v[1] : v[0], rsum_xor<DDS>(h ? v[0] : v[1], 16));
    o = 8;
  } else {
    const bool h = lane & 16, k = lane & 8;
    const DD z{0.0, 0.0};
    const DD p = rsum_merge<DDS>(h ? v[2] : v[0], rsum_xor<DDS>(h ? v[0] : v[2], 16));
    const DD q = rsum_merge<DDS>(h ? z : v[1], rsum_xor<DDS>(h ? v[1] : z, 16));
    a = rsum_merge<DDS>(k ? q : p, rsum_xor<DDS>(k ? p : q, 8));
    o = 4;
  }
  for (; o > 0; o >>= 1) a = rsum_merge<DDS>(a, rsum_xor<DDS>(a, o));
  return a;
}

// ------------------------------------------------------------ cluster form
constexpr int CX_MAXC = 16;  // CTAs of a cluster

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned mapa(unsigned addr, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void push16(unsigned dst, unsigned bar, unsigned a, unsigned b, unsigned c, unsigned d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void push16(unsigned dst, unsigned bar, const float* v) {
  push16(dst, bar, __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
}
__device__ __forceinline__ void push16(unsigned dst, unsigned bar, const double* v) {
  push16(dst, bar, (unsigned)__double2loint(v[0]), (unsigned)__double2hiint(v[0]), (unsigned)__double2loint(v[1]),
         (unsigned)__double2hiint(v[1]));
}
__device__ __forceinline__ void push8(unsigned dst, unsigned bar, double v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void push4(unsigned dst, unsigned bar, float v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(phase)
      : "memory");
  return ok != 0;
}

// the bound of a cluster's waits, in polls (0: FUGU_SPIN_LIMIT); the
// failure-detection test lowers it and expects bytes that nobody sends
struct CxLimit {
  unsigned int spin_limit, extra_bytes;
  __device__ __forceinline__ unsigned polls() const { return spin_limit ? spin_limit : FUGU_SPIN_LIMIT; }
};

template <int TPB>
struct alignas(16) ClusterXSmem {
  double rcv[2][CX_MAXC][4];  // received sums [parity][rank]; first, for push16's 16-byte stores
  DD wp[3][TPB / 32];         // the warps' sums
  double bc[3];               // the totals
  unsigned long long mbar[2];
  int fail;
};
// One CTA's side of the cluster exchange.  start() once (a cluster barrier),
// then pushes and one allreduce per exchange, leave() last (a cluster barrier:
// no CTA goes while another may still push to it).
template <int TPB, bool DDS>
struct ClusterX {
  static constexpr int NP = DDS ? 2 : 1;  // doubles per sum
  static_assert(alignof(ClusterXSmem<TPB>) >= 16 && offsetof(ClusterXSmem<TPB>, rcv) == 0,
                "push16 stores 16 bytes at rcv[parity][rank][q * NP]");
  ClusterXSmem<TPB>& s;
  int rank, G;
  unsigned ep, lim, extra;
  __device__ __forceinline__ ClusterX(ClusterXSmem<TPB>& sm, int r, int g, CxLimit l)
      : s(sm), rank(r), G(g), ep(0), lim(l.polls()), extra(l.extra_bytes) {}
  __device__ __forceinline__ void start() {
    if (threadIdx.x == 0) {
      s.fail = 0;
      for (int b = 0; b < 2; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s.mbar[b])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cgc::this_cluster().sync();
  }
  __device__ __forceinline__ void leave() { cgc::this_cluster().sync(); }
  // after a failed wait: pushes still in flight land before anyone leaves
  __device__ __forceinline__ void abandon() {
    __nanosleep(200000);
    leave();
  }
  __device__ __forceinline__ unsigned parity() const { return ep & 1u; }
  __device__ __forceinline__ unsigned bar(int to) const { return mapa(smem_u32(&s.mbar[ep & 1u]), to); }
  // Sum NV values over the cluster and receive the halo_bytes that the
  // neighbours push in this exchange; between() runs while the data is in
  // flight.  The block's and the cluster's trees add pairs 8, 4, 2, 1 apart.
  template <int NV, typename F>
  __device__ __forceinline__ bool allreduce(const DD* v, double* out, unsigned halo_bytes, F between) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const unsigned par = ep & 1u, mb = smem_u32(&s.mbar[par]);
    if (tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(mb),
                   "r"((unsigned)(G * NV * NP * 8) + halo_bytes + extra)
                   : "memory");
    {
      const DD t = rsum_warp<DDS, NV>(v);
#pragma unroll
      for (int q = 0; q < NV; ++q)
        if (lane == rsum_lane<NV>(q)) s.wp[q][warp] = t;
    }
    __syncthreads();
    // value q over the block's warps by warp q (by warp 0 in a smaller block)
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (warp == (q < nw ? q : 0)) {
        DD t = s.wp[q][lane & (nw - 1)];
#pragma unroll
        for (int o = TPB / 64; o > 0; o >>= 1)
          if (o < nw) t = rsum_merge<DDS>(t, rsum_xor<DDS>(t, o));
        if (lane < G) {
          const unsigned dst = mapa(smem_u32(&s.rcv[par][rank][q * NP]), lane), to = mapa(mb, lane);
          if constexpr (DDS) {
            const double x[2] = {t.hi, t.lo};
            push16(dst, to, x);
          } else {
            push8(dst, to, t.hi);
          }
        }
      }
    between();
    // the merging warps wait; the block barrier passes the arrival on
    bool ok = true;
    if (warp < NV) {
      unsigned spins = 0;
      while (!mbar_test(mb, (ep >> 1) & 1u))
        if (++spins > lim) {
          ok = false;
          break;
        }
#pragma unroll
      for (int q = 0; q < NV; ++q)
        if (warp == (q < nw ? q : 0)) {
          DD t{0.0, 0.0};
          if (lane < G) {
            t.hi = s.rcv[par][lane][q * NP];
            if constexpr (DDS) t.lo = s.rcv[par][lane][q * NP + 1];
          }
#pragma unroll
          for (int o = CX_MAXC / 2; o > 0; o >>= 1) t = rsum_merge<DDS>(t, rsum_xor<DDS>(t, o));
          if (lane == 0) s.bc[q] = t.hi + t.lo;
        }
    }
    if (!ok) s.fail = 1;
    __syncthreads();
    if (s.fail) return false;
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = s.bc[q];
    ++ep;
    return true;
  }
};

// --------------------------------------------------------------- grid form
constexpr int GX_NV = 8;  // word pairs (doubles) per CTA and exchange: a cache line

// the context's exchange buffers (device memory, zero at allocation)
struct Exchange {
  unsigned int* epoch;       // the last epoch used by an earlier launch
  ulonglong2* sum;           // [2][nslots][GX_NV]
  unsigned long long* halo;  // [2][nslots][2 sides][halo_words]
  int nslots;                // CTAs + 1; the last slot is never written
  long halo_words;           // 8-byte words of one boundary row
};

__device__ __forceinline__ unsigned long long gx_word(unsigned int v, unsigned int ep) {
  return (unsigned long long)v | ((unsigned long long)ep << 32);
}
__device__ __forceinline__ void gx_st2(void* p, unsigned long long a, unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void gx_ld2(const void* p, unsigned long long& a, unsigned long long& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
// a double as two words
__device__ __forceinline__ void gx_put(void* p, double x, unsigned int ep) {
  gx_st2(p, gx_word((unsigned)__double2loint(x), ep), gx_word((unsigned)__double2hiint(x), ep));
}
__device__ __forceinline__ bool gx_ready(unsigned long long a, unsigned long long b, unsigned int ep) {
  return (unsigned)(a >> 32) == ep && (unsigned)(b >> 32) == ep;
}
__device__ __forceinline__ double gx_double(unsigned long long a, unsigned long long b) {
  return __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
}

// a segment of a boundary row (four floats or two doubles): two 16-byte
// stores of two words each
__device__ __forceinline__ void gx_put_seg(unsigned long long* p, const float* v, unsigned int ep) {
  gx_st2(p, gx_word(__float_as_uint(v[0]), ep), gx_word(__float_as_uint(v[1]), ep));
  gx_st2(p + 2, gx_word(__float_as_uint(v[2]), ep), gx_word(__float_as_uint(v[3]), ep));
}
__device__ __forceinline__ void gx_put_seg(unsigned long long* p, const double* v, unsigned int ep) {
  gx_put(p, v[0], ep);
  gx_put(p + 2, v[1], ep);
}
struct GxSeg {
  unsigned long long w[4];
  __device__ __forceinline__ void load(const unsigned long long* p) {
    gx_ld2(p, w[0], w[1]);
    gx_ld2(p + 2, w[2], w[3]);
  }
  __device__ __forceinline__ bool ready(unsigned int ep) const { return gx_ready(w[0], w[1], ep) && gx_ready(w[2], w[3], ep); }
  __device__ __forceinline__ void get(float* v) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = __uint_as_float((unsigned)w[e]);
  }
  __device__ __forceinline__ void get(double* v) const {
    v[0] = gx_double(w[0], w[1]);
    v[1] = gx_double(w[2], w[3]);
  }
};

// a bounded wait's bookkeeping: true while the caller may poll again
struct GxWait {
  unsigned int lim, spins;
  int* err;
  __device__ __forceinline__ bool again() {
    if (++spins > lim || ((spins & 255u) == 0u && ld_relaxed_i32(err) != 0)) {
      atomicExch(err, 1);
      return false;
    }
    return true;
  }
};


template <int TPB>
struct GridXSmem {
  DD wp[3][TPB / 32];  // the warps' sums
  DD wr[3][TPB / 32];  // received sums per warp
  int fail;
};
// One CTA's side of the grid exchange (error-free sums).
template <int TPB>
struct GridX {
  GridXSmem<TPB>& s;
  const Exchange& x;
  int rank, G, extra;
  unsigned ep, lim;
  int* err;
  __device__ __forceinline__ GridX(GridXSmem<TPB>& sm, const Exchange& xc, int r, int g, int extra_arrivals,
                                   unsigned spin_limit, int* e)
      : s(sm), x(xc), rank(r), G(g), extra(extra_arrivals), ep(0), lim(spin_limit ? spin_limit : FUGU_SPIN_LIMIT / 16),
        err(e) {}
  __device__ __forceinline__ void start() {
    if (threadIdx.x == 0) s.fail = 0;
    ep = *(volatile unsigned int*)x.epoch + 1u;
    __syncthreads();
  }
  // by one thread, when every CTA has taken part in an exchange of the launch
  __device__ __forceinline__ void finish() { *x.epoch = ep; }
  __device__ __forceinline__ unsigned parity() const { return ep & 1u; }
  __device__ __forceinline__ unsigned long long* outbox(int cta, int side) const {
    return x.halo + (((long)(ep & 1u) * x.nslots + cta) * 2 + side) * x.halo_words;
  }
  // Sum NV values over the grid; halo(wait) receives boundary rows with the
  // wait's bookkeeping (they left before the sums, so usually at once).
  template <int NV, typename H, typename F>
  __device__ __forceinline__ bool allreduce(const DD* v, double* out, H halo, F between) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    {
      const DD t = rsum_warp<true, NV>(v);
#pragma unroll
      for (int q = 0; q < NV; ++q)
        if (lane == rsum_lane<NV>(q)) s.wp[q][warp] = t;
    }
    __syncthreads();
    ulonglong2* sum = x.sum + (long)(ep & 1u) * x.nslots * GX_NV;
    // word pair q of a CTA.  One or two sums: a CTA's words in a line of its
    // own (side by side, the writers meet in one line: FP64 512 x 512 6.7 ->
    // 8.8 us per iteration).  Three sums: word by word, so that a warp's readers
    // share sectors (twice the words: FP32 320 x 640 4.9 -> 4.2).
    auto word = [&](int cta, int q) { return NV == 3 ? q * x.nslots + cta : cta * GX_NV + q; };
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (warp == (q < nw ? q : 0)) {
        DD t = s.wp[q][lane & (nw - 1)];
#pragma unroll
        for (int o = TPB / 64; o > 0; o >>= 1)
          if (o < nw) t = rsum_merge<true>(t, rsum_xor<true>(t, o));
        if (lane < 2) gx_put(sum + word(rank, q * 2 + lane), lane ? t.lo : t.hi, ep);
      }
    between();
    GxWait gw{lim, 0u, err};
    bool ok = halo(gw);
    const int nrecv = G + (extra ? 1 : 0);
    const int nwr = min(min(nw, 8), (nrecv + 31) >> 5);  // warps that receive
    if (warp < nwr) {
      DD acc[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q] = DD{0.0, 0.0};
      for (int c = tid; c < nrecv; c += nwr * 32) {
        unsigned long long w[NV * 2][2];
        while (ok) {
          bool got = true;
#pragma unroll
          for (int q = 0; q < NV * 2; ++q) gx_ld2(sum + word(c, q), w[q][0], w[q][1]);
#pragma unroll
          for (int q = 0; q < NV * 2; ++q) got = got && gx_ready(w[q][0], w[q][1], ep);
          if (got) break;
          ok = gw.again();
        }
        if (!ok) break;
#pragma unroll
        for (int q = 0; q < NV; ++q)
          acc[q] = rsum_merge<true>(acc[q], DD{gx_double(w[2 * q][0], w[2 * q][1]), gx_double(w[2 * q + 1][0], w[2 * q + 1][1])});
      }
      __syncwarp();
      const DD t = rsum_warp<true, NV>(acc);
#pragma unroll
      for (int q = 0; q < NV; ++q)
        if (lane == rsum_lane<NV>(q)) s.wr[q][warp] = t;
    }
    if (!ok) s.fail = 1;
    __syncthreads();
    if (s.fail) return false;
    {
      // each warp adds the receiving warps' sums (at most eight), value q in
      // lanes 8 q ..; in turn by every thread this cost about as much as the
      // exchange (us per iteration with / without: FP32 320 x 640 4.38 / 3.90,
      // 768 x 768 9.18 / 8.35, FP64 320 x 640 6.59 / 6.18, launch included)
      const int q = lane >> 3, k = lane & 7;
      DD t{0.0, 0.0};
      if (q < NV && k < nwr) t = s.wr[q][k];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t = rsum_merge<true>(t, rsum_xor<true>(t, o));
      const double x = t.hi + t.lo;
#pragma unroll
      for (int v = 0; v < NV; ++v) out[v] = __shfl_sync(0xffffffffu, x, 8 * v);
    }
    ++ep;
    return true;
  }
};

// quotient a / b from the correctly rounded reciprocal y of b (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000", 1990):
// with q = a y, the remainder a - q b is exact in one fused operation and
// q + (a - q b) y rounds to the quotient.  Lets a division whose divisor is
// known early leave three operations on the critical path.
__device__ __forceinline__ double quotient(double a, double b, double y) {
  const double q = a * y;
  return __fma_rn(__fma_rn(-q, b, a), y, q);
}

}  // namespace fugu
