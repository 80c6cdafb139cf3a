// ERI kernel templates (one thread per shell quartet) -- included by the eri_g*.cu
// translation units, each of which instantiates a group of classes.
#pragma once
#include <math.h>
#include "common.cuh"
#include "pcg_internal.h"
#include "eri_gen.cuh"

struct PQd {
  double PAx, PAy, PAz, WPx, WPy, WPz, QCx, QCy, QCz, WQx, WQy, WQz, oo2z, oo2e, oo2ze, rz, re;
};
struct PQf {
  float PAx, PAy, PAz, WPx, WPy, WPz, QCx, QCy, QCz, WQx, WQy, WQz, oo2z, oo2e, oo2ze, rz, re;
};

// The tasks of one launch, sorted by decreasing primitive-quartet count: end[i] of them have
// 256, 128, 64, 32, 16, 8 or more (and end[6] = ntask all).  Part i is shared by 2^lg[i] lanes a
// task; a lane takes every 2^lg-th primitive quartet, the partial sums are added by shuffles.
// stride: distance of a block's elements in the store.
#define ERI_PARTS 7
struct EriRange {
  int stride, end[ERI_PARTS], lg[ERI_PARTS];
};

// One warp's FP64 instruction takes its quarter of an SM 64 cycles whatever runs beside it, and a
// quarter's resident warps take turns: a lane with a few times the average share of a quarter
// (mean = all primitive quartets / (608 quarters x 32 lanes)) ends alone, after the launch.  So
// a lane gets at most a twelfth of that share, but not fewer than 4 to 8 primitive quartets: a
// step of the sums over lanes costs a third of one ((dd|dd): 961 accumulators).  (H2O)8, 6-31G,
// FP64 part of a mixed pass: (pp|ps) 188 us with one lane up to 127 primitive quartets, 117 us so;
// C12H26/cc-pVDZ with a half, a quarter, an eighth, a 16th, a 32nd of the share: 62.3, 59.8, 58.8,
// 59.0, 59.5 ms; with at least 2, 4, 8, 16 in a lane 60.8, 58.8, 58.1, 58.9 ms.
static inline EriRange eri_range(int ntask, const int* more) {
  static const int from[ERI_PARTS] = {256, 128, 64, 32, 16, 8, 1}, most[ERI_PARTS] = {1296, 256, 128, 64, 32, 16, 8};
  EriRange r;
  r.stride = ntask;
  double all = 0.0;
  for (int i = 0, prev = 0; i < ERI_PARTS; ++i) {
    r.end[i] = i + 1 < ERI_PARTS ? (more ? more[i] : 0) : ntask;
    all += 1.4 * from[i] * (r.end[i] - prev);
    prev = r.end[i];
  }
  const double share = fmax(8.0, all / (608 * 32 * 12));
  for (int i = 0; i < ERI_PARTS; ++i)
    for (r.lg[i] = 0; i + 1 < ERI_PARTS && r.lg[i] < 5 && most[i] > share * (1 << r.lg[i]);) ++r.lg[i];
  return r;
}
// lanes of a part, rounded up to whole warps
__host__ __device__ static inline long long eri_lanes(int n, int lg) { return (((long long)n << lg) + 31) / 32 * 32; }
static inline unsigned eri_blocks(const EriRange& r, int threads) {
  long long n = 0;
  for (int i = 0; i < ERI_PARTS; ++i) n += eri_lanes(r.end[i] - (i ? r.end[i - 1] : 0), r.lg[i]);
  return (unsigned)((n + threads - 1) / threads);
}

// This lane's task, its place among the lanes of the task, and log2 of their number; lanes
// past the end of a part take part in the shuffles on the last task with no primitive quartet.
struct EriLane {
  int t, g, lg;
  bool on;
};
__device__ __forceinline__ EriLane eri_lane(const EriRange& r) {
  long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int lo = 0, hi = r.end[0], lg = r.lg[0];
#pragma unroll
  for (int i = 1; i < ERI_PARTS; ++i) {
    const long long n = eri_lanes(hi - lo, lg);
    if (x < n || hi == r.end[ERI_PARTS - 1]) break;
    x -= n;
    lo = hi;
    hi = r.end[i];
    lg = r.lg[i];
  }
  EriLane l;
  l.lg = lg;
  const long long t = lo + (x >> lg);
  l.on = t < hi;
  l.g = (int)(threadIdx.x & ((1u << lg) - 1));
  l.t = l.on ? (int)t : r.end[ERI_PARTS - 1] - 1;
  return l;
}

// sums of acc over the lanes of a task (every lane of the warp takes part, with the same lg)
template <int N, class T>
__device__ __forceinline__ void eri_lane_sum(T* acc, int lg) {
  for (int o = 1; o < (1 << lg); o <<= 1)
#pragma unroll
    for (int k = 0; k < N; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
}

// The factors of a primitive quartet that depend on its two exponent sums alone come from a
// table over the molecule's distinct sums (PrimTab): 1/sqrt(zeta + eta), rho, rho/zeta, rho/eta and
// 1/(2 (zeta + eta)), nine FP64 instructions of about 40 in (ps|ss).  A pair without an
// entry (no table, or more sums than it takes) has them computed.  Packed pair data halve the
// gathers: P and K, P - A and 1/(2 zeta) are two 16-byte loads each.
template <class C>
__global__ void __launch_bounds__(128) k_eri(DevPairsExt pr, PrimTab pt, BoysTable bt, const int2* __restrict__ tasks,
                                             EriRange rg, double* __restrict__ store) {
  const EriLane ln = eri_lane(rg);
  const int t = ln.t;
  const int2 tk = tasks[t];
  const int i0 = __ldg(pr.p.ppoff + tk.x), j0 = __ldg(pr.p.ppoff + tk.y), nj = __ldg(pr.p.npp_of + tk.y);
  const int nq = ln.on ? __ldg(pr.p.npp_of + tk.x) * nj : 0;
  double acc[C::NACC];
#pragma unroll
  for (int k = 0; k < C::NACC; ++k) acc[k] = 0.0;
  int i = i0 - 1, jj = ln.g + nj;      // jj: ket primitive plus the bra steps not yet taken
  int zi = -1;
  double Px = 0.0, Py = 0.0, Pz = 0.0, Kp = 0.0;
  PQd q;
  for (int n = ln.g; n < nq; n += 1 << ln.lg, jj += 1 << ln.lg) {
    if (jj >= nj) {
      do { jj -= nj; ++i; } while (jj >= nj);
      if (pt.pk) {
        const double2* b = (const double2*)pt.pk + 4 * (size_t)i;
        const double2 b0 = __ldg(b), b1 = __ldg(b + 1), b2 = __ldg(b + 2), b3 = __ldg(b + 3);
        Px = b0.x; Py = b0.y; Pz = b1.x; Kp = b1.y;
        q.PAx = b2.x; q.PAy = b2.y; q.PAz = b3.x; q.oo2z = b3.y;
        zi = __ldg(pt.zid + i);
      } else {
        Px = __ldg(pr.p.P + 3 * i); Py = __ldg(pr.p.P + 3 * i + 1); Pz = __ldg(pr.p.P + 3 * i + 2);
        Kp = __ldg(pr.p.K + i);
        q.PAx = __ldg(pr.p.PA + 3 * i);
        q.PAy = __ldg(pr.p.PA + 3 * i + 1);
        q.PAz = __ldg(pr.p.PA + 3 * i + 2);
        q.oo2z = __ldg(pr.oo2z + i);
      }
    }
    const int j = j0 + jj;
    double PQx, PQy, PQz, Kq;
    int zj = -1;
    if (pt.pk) {
      const double2* b = (const double2*)pt.pk + 4 * (size_t)j;
      const double2 b0 = __ldg(b), b1 = __ldg(b + 1), b2 = __ldg(b + 2), b3 = __ldg(b + 3);
      PQx = Px - b0.x; PQy = Py - b0.y; PQz = Pz - b1.x;
      Kq = b1.y;
      q.QCx = b2.x; q.QCy = b2.y; q.QCz = b3.x; q.oo2e = b3.y;
      zj = __ldg(pt.zid + j);
    } else {
      PQx = Px - __ldg(pr.p.P + 3 * j);
      PQy = Py - __ldg(pr.p.P + 3 * j + 1);
      PQz = Pz - __ldg(pr.p.P + 3 * j + 2);
      Kq = __ldg(pr.p.K + j);
      q.QCx = __ldg(pr.p.PA + 3 * j);
      q.QCy = __ldg(pr.p.PA + 3 * j + 1);
      q.QCz = __ldg(pr.p.PA + 3 * j + 2);
      q.oo2e = __ldg(pr.oo2z + j);
    }
    double rs, rho;
    if ((zi | zj) >= 0) {
      const double2* e = (const double2*)pt.tab + 3 * ((size_t)zi * pt.nz + zj);
      const double2 e0 = __ldg(e), e1 = __ldg(e + 1), e2 = __ldg(e + 2);
      rs = e0.x; rho = e0.y;
      q.rz = e1.x; q.re = e1.y;
      q.oo2ze = e2.x;
    } else {
      const double zeta = __ldg(pr.p.zeta + i), eta = __ldg(pr.p.zeta + j);
      rs = nr_rsqrt(zeta + eta);
      const double izpe = rs * rs;
      q.rz = eta * izpe;
      q.re = zeta * izpe;
      rho = zeta * q.rz;
      q.oo2ze = 0.5 * izpe;
    }
    double F[C::L + 1];
    boys_eval<C::L>(bt, rho * fma(PQx, PQx, fma(PQy, PQy, PQz * PQz)), F);
    const double pre = Kp * Kq * rs;
    if constexpr (C::L == 0) {
      acc[0] = fma(F[0], pre, acc[0]);
    } else if constexpr (C::LC + C::LD == 0 && C::L <= 2) {
      // all momentum on the bra: rz^m goes with F_m, so that W - P = -rz (P - Q) and the rz of the
      // recursion need no products of their own (27 FP64 instructions instead of 29 for (ps|ss))
      double f = pre;
      F[0] *= f;
#pragma unroll
      for (int m = 1; m <= C::L; ++m) F[m] *= f *= q.rz;
      q.WPx = -PQx; q.WPy = -PQy; q.WPz = -PQz;
      q.rz = 1.0;
      C::prim(q, F, acc);
    } else {
#pragma unroll
      for (int m = 0; m <= C::L; ++m) F[m] *= pre;
      q.WPx = -q.rz * PQx; q.WPy = -q.rz * PQy; q.WPz = -q.rz * PQz;
      q.WQx = q.re * PQx; q.WQy = q.re * PQy; q.WQz = q.re * PQz;
      C::prim(q, F, acc);
    }
  }
  eri_lane_sum<C::NACC>(acc, ln.lg);
  if (ln.g != 0 || !ln.on) return;
  const double ABx = __ldg(pr.p.AB + 3 * tk.x), ABy = __ldg(pr.p.AB + 3 * tk.x + 1), ABz = __ldg(pr.p.AB + 3 * tk.x + 2);
  const double CDx = __ldg(pr.p.AB + 3 * tk.y), CDy = __ldg(pr.p.AB + 3 * tk.y + 1), CDz = __ldg(pr.p.AB + 3 * tk.y + 2);
  C::finish(acc, ABx, ABy, ABz, CDx, CDy, CDz, [&](int k, double v) { store[(size_t)k * rg.stride + t] = v; });
}

// Single-precision variant for quartets whose Schwarz bound is below the mixed
// threshold; the pair data are rounded from the double arrays, results widened.
template <class C>
__global__ void __launch_bounds__(128) k_eri_f(DevPairsExt pr, BoysTable bt, const int2* __restrict__ tasks,
                                               int ntask, double* __restrict__ store) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntask) return;
  const int2 tk = tasks[t];
  const int i0 = __ldg(pr.p.ppoff + tk.x), i1 = i0 + __ldg(pr.p.npp_of + tk.x);
  const int j0 = __ldg(pr.p.ppoff + tk.y), j1 = j0 + __ldg(pr.p.npp_of + tk.y);
  float acc[C::NACC];
#pragma unroll
  for (int k = 0; k < C::NACC; ++k) acc[k] = 0.0f;
  if (pr.p.pf8) {
    // packed FP32 pair table: P - Q = (P - A) - (Q - C) + (A - C), the shell-centre
    // difference A - C formed once per quartet in double precision
    const float ACx = (float)((__ldg(pr.p.P + 3 * i0) - __ldg(pr.p.PA + 3 * i0)) -
                              (__ldg(pr.p.P + 3 * j0) - __ldg(pr.p.PA + 3 * j0)));
    const float ACy = (float)((__ldg(pr.p.P + 3 * i0 + 1) - __ldg(pr.p.PA + 3 * i0 + 1)) -
                              (__ldg(pr.p.P + 3 * j0 + 1) - __ldg(pr.p.PA + 3 * j0 + 1)));
    const float ACz = (float)((__ldg(pr.p.P + 3 * i0 + 2) - __ldg(pr.p.PA + 3 * i0 + 2)) -
                              (__ldg(pr.p.P + 3 * j0 + 2) - __ldg(pr.p.PA + 3 * j0 + 2)));
    for (int i = i0; i < i1; ++i) {
      const float4 a0 = __ldg(pr.p.pf8 + 2 * i), a1 = __ldg(pr.p.pf8 + 2 * i + 1);
      const float zeta = a0.x, Kp = a1.y;
      PQf q;
      q.PAx = a0.y; q.PAy = a0.z; q.PAz = a0.w;
      q.oo2z = a1.x;
      for (int j = j0; j < j1; ++j) {
        const float4 b0 = __ldg(pr.p.pf8 + 2 * j), b1 = __ldg(pr.p.pf8 + 2 * j + 1);
        const float eta = b0.x;
        const float PQx = (q.PAx - b0.y) + ACx;
        const float PQy = (q.PAy - b0.z) + ACy;
        const float PQz = (q.PAz - b0.w) + ACz;
        const float rs = rsqrtf(zeta + eta);
        const float izpe = rs * rs;
        const float rho = zeta * eta * izpe;
        const float T = rho * fmaf(PQx, PQx, fmaf(PQy, PQy, PQz * PQz));
        float F[C::L + 1];
        boys_eval_f<C::L>(bt, T, F);
        const float pre = Kp * b1.y * rs;
#pragma unroll
        for (int m = 0; m <= C::L; ++m) F[m] *= pre;
        const float wp = -eta * izpe, wq = zeta * izpe;
        q.WPx = wp * PQx; q.WPy = wp * PQy; q.WPz = wp * PQz;
        q.WQx = wq * PQx; q.WQy = wq * PQy; q.WQz = wq * PQz;
        q.QCx = b0.y; q.QCy = b0.z; q.QCz = b0.w;
        q.oo2e = b1.x;
        q.oo2ze = 0.5f * izpe;
        q.rz = eta * izpe;
        q.re = zeta * izpe;
        C::prim(q, F, acc);
      }
    }
  } else
  for (int i = i0; i < i1; ++i) {
    const double zd = __ldg(pr.p.zeta + i);
    const float zeta = (float)zd;
    const double Px = __ldg(pr.p.P + 3 * i), Py = __ldg(pr.p.P + 3 * i + 1), Pz = __ldg(pr.p.P + 3 * i + 2);
    const float Kp = __ldg(pr.p.Kf + i);
    PQf q;
    q.PAx = (float)__ldg(pr.p.PA + 3 * i);
    q.PAy = (float)__ldg(pr.p.PA + 3 * i + 1);
    q.PAz = (float)__ldg(pr.p.PA + 3 * i + 2);
    q.oo2z = (float)__ldg(pr.oo2z + i);
    for (int j = j0; j < j1; ++j) {
      const float eta = (float)__ldg(pr.p.zeta + j);
      const float PQx = (float)(Px - __ldg(pr.p.P + 3 * j));
      const float PQy = (float)(Py - __ldg(pr.p.P + 3 * j + 1));
      const float PQz = (float)(Pz - __ldg(pr.p.P + 3 * j + 2));
      const float rs = rsqrtf(zeta + eta);
      const float izpe = rs * rs;
      const float rho = zeta * eta * izpe;
      const float T = rho * fmaf(PQx, PQx, fmaf(PQy, PQy, PQz * PQz));
      float F[C::L + 1];
      boys_eval_f<C::L>(bt, T, F);
      const float pre = Kp * __ldg(pr.p.Kf + j) * rs;
#pragma unroll
      for (int m = 0; m <= C::L; ++m) F[m] *= pre;
      const float wp = -eta * izpe, wq = zeta * izpe;
      q.WPx = wp * PQx; q.WPy = wp * PQy; q.WPz = wp * PQz;
      q.WQx = wq * PQx; q.WQy = wq * PQy; q.WQz = wq * PQz;
      q.QCx = (float)__ldg(pr.p.PA + 3 * j);
      q.QCy = (float)__ldg(pr.p.PA + 3 * j + 1);
      q.QCz = (float)__ldg(pr.p.PA + 3 * j + 2);
      q.oo2e = (float)__ldg(pr.oo2z + j);
      q.oo2ze = 0.5f * izpe;
      q.rz = eta * izpe;
      q.re = zeta * izpe;
      C::prim(q, F, acc);
    }
  }
  const float ABx = (float)__ldg(pr.p.AB + 3 * tk.x), ABy = (float)__ldg(pr.p.AB + 3 * tk.x + 1),
              ABz = (float)__ldg(pr.p.AB + 3 * tk.x + 2);
  const float CDx = (float)__ldg(pr.p.AB + 3 * tk.y), CDy = (float)__ldg(pr.p.AB + 3 * tk.y + 1),
              CDz = (float)__ldg(pr.p.AB + 3 * tk.y + 2);
  C::finish(acc, ABx, ABy, ABz, CDx, CDy, CDz, [&](int k, float v) { store[(size_t)k * ntask + t] = (double)v; });
}

