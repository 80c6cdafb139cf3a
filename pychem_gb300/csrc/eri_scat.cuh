// Electron-scattering integrals (ab|j0(S r12)|cd) -- the operator of
// Methods/properties.py:20-23, integrals of Methods/c_ints/two_electron_scattering.c
// and spherical_bessel_j.c.  The generated VRR/HRR and the task-to-lane map of the
// Coulomb kernels; only the fundamentals differ.  Included by eri_s*.cu.
#pragma once
#include "eri_kernels.cuh"
#include "scat_fund.cuh"

// z^-m j_m(z), m = 0..L, for z^2 = 2x = S^2 R^2.  z < 10: rows of the table over x (as the
// Boys function: 4 FP64 instructions each), the two highest orders from the table and the
// others downwards, f_{m-1} = (2m+1) f_m - 2x f_{m+1}.  10 <= z < 100: sin and cos from
// the grid of 64 points per unit (11 FP64 instructions; |d| <= 1/128, so d^5 and up are
// FP32) and upward recursion f_{m+1} = ((2m+1) f_m - f_{m-1}) / z^2.  From 100 the two-term
// asymptotic form of spherical_bessel_j.c.  A warp whose lanes fall on both sides of
// z = 10 runs both branches; the power series of up to 20 terms with a division each, one
// series an order, that stood here ran at 12 of 32 active lanes and made these integrals 20
// times dearer than 1/r12.
template <int L>
__device__ __forceinline__ void bessel_eval(const BesselTable& bt, double S, double iS, double R2, double* f) {
  const double x = 0.5 * S * S * R2;
  if ((unsigned)__double2hiint(x) < 0x40490000u) {   // 0 <= x < 50, and no NaN
    double d;
    float df;
    const int p = taylor_point(x, d, df);
    f[L] = taylor_row(bt.c + L * BESSEL_NP + p, d, df);
    if (L > 0) {
      f[L - 1] = taylor_row(bt.c + (L - 1) * BESSEL_NP + p, d, df);
      const double x2 = 2.0 * x;
#pragma unroll
      for (int m = L - 1; m > 0; --m) f[m - 1] = fma(-x2, f[m + 1], (2 * m + 1) * f[m]);
    }
    return;
  }
  const double ri = nr_rsqrt(R2);
  const double z = S * R2 * ri, zi = iS * ri;
  if (z < 100.0) {
    double d;
    float df;
    const int p = taylor_point(z, d, df);
    const double2 sc = __ldg(bt.sc + p);
    const double h = -d;                            // z = z_p + h
    const double w = h * h;
    const float wf = df * df;
    const double s1 = fma(h * w, -1.0 / 6.0 + bits_to_double(wf * fmaf(wf, -1.0f / 5040.0f, 1.0f / 120.0f)), h);
    const double c1 = w * (-0.5 + bits_to_double(wf * fmaf(wf, -1.0f / 720.0f, 1.0f / 24.0f)));
    const double sz = fma(sc.x, c1, fma(sc.y, s1, sc.x));
    f[0] = sz * zi;
    if (L > 0) {
      const double cz = fma(sc.y, c1, fma(-sc.x, s1, sc.y));
      const double zi2 = zi * zi;
      f[1] = (f[0] - cz) * zi2;
#pragma unroll
      for (int m = 1; m < L; ++m) f[m + 1] = fma((double)(2 * m + 1), f[m], -f[m - 1]) * zi2;
    }
#pragma unroll
    for (int m = 0; m <= L; ++m)
      if (fabs(f[m]) < 1e-16) f[m] = 0.0;           // as spherical_bessel_j.c
    return;
  }
  sph_bessel_scaled<L>(z, f);
}

// A primitive pair's factor of every integral that it is in.  K_P K_Q carries the
// 2 pi^{5/2}/(zeta eta) of 1/r12; times sqrt(pi) / (2 sqrt(zeta eta)) it is the overlap product
// U_P U_Q.  exp(-S^2/(4 rho)) = exp(-S^2/(4 zeta)) exp(-S^2/(4 eta)), so both split into one
// number a pair, and the exponential and the two roots leave the primitive-quartet loop.
__device__ __forceinline__ double scat_factor(double zeta, double K, double S) {
  // sqrt(sqrt(pi) / 2) = 0.9413962637767148
  return 0.94139626377671481 * K * nr_rsqrt(zeta) * exp(-0.25 * S * S / zeta);
}

// fac: the factors of all primitive pairs (pcg_scattering_factors), or null: formed here.
// The fundamentals in the Obara-Saika form of the generated VRR are (-d/dT)^m of
// exp(-S^2/(4 rho)) j0(S R) at T = rho R^2, i.e. exp(-S^2/(4 rho)) (S^2/(2 rho))^m z^-m j_m(z).
template <class C>
__global__ void __launch_bounds__(128) k_eri_s(DevPairsExt pr, BesselTable bt, const double* __restrict__ fac,
                                               const int2* __restrict__ tasks, EriRange rg, double S,
                                               double* __restrict__ store) {
  const EriLane ln = eri_lane(rg);
  const int t = ln.t;
  const int2 tk = tasks[t];
  const int i0 = __ldg(pr.p.ppoff + tk.x), j0 = __ldg(pr.p.ppoff + tk.y), nj = __ldg(pr.p.npp_of + tk.y);
  const int nq = ln.on ? __ldg(pr.p.npp_of + tk.x) * nj : 0;
  const double iS = 1.0 / S, S2 = S * S;      // iS is used where S > 0 only
  double acc[C::NACC];
#pragma unroll
  for (int k = 0; k < C::NACC; ++k) acc[k] = 0.0;
  int i = i0 - 1, jj = ln.g + nj;
  double zeta = 0.0, Px = 0.0, Py = 0.0, Pz = 0.0, Kp = 0.0;
  PQd q;
  for (int n = ln.g; n < nq; n += 1 << ln.lg, jj += 1 << ln.lg) {
    if (jj >= nj) {
      do { jj -= nj; ++i; } while (jj >= nj);
      zeta = __ldg(pr.p.zeta + i);
      Px = __ldg(pr.p.P + 3 * i); Py = __ldg(pr.p.P + 3 * i + 1); Pz = __ldg(pr.p.P + 3 * i + 2);
      Kp = fac ? __ldg(fac + i) : scat_factor(zeta, __ldg(pr.p.K + i), S);
      q.PAx = __ldg(pr.p.PA + 3 * i);
      q.PAy = __ldg(pr.p.PA + 3 * i + 1);
      q.PAz = __ldg(pr.p.PA + 3 * i + 2);
      q.oo2z = __ldg(pr.oo2z + i);
    }
    const int j = j0 + jj;
    const double PQx = Px - __ldg(pr.p.P + 3 * j);
    const double PQy = Py - __ldg(pr.p.P + 3 * j + 1);
    const double PQz = Pz - __ldg(pr.p.P + 3 * j + 2);
    double F[C::L + 1];
    bessel_eval<C::L>(bt, S, iS, fma(PQx, PQx, fma(PQy, PQy, PQz * PQz)), F);
    const double eta = __ldg(pr.p.zeta + j);
    double pre = Kp * (fac ? __ldg(fac + j) : scat_factor(eta, __ldg(pr.p.K + j), S));
    q.oo2e = __ldg(pr.oo2z + j);
    const double step = S2 * (q.oo2z + q.oo2e);      // S^2 / (2 rho)
    F[0] *= pre;
#pragma unroll
    for (int m = 1; m <= C::L; ++m) {
      pre *= step;
      F[m] *= pre;
    }
    const double rs = nr_rsqrt(zeta + eta);
    const double izpe = rs * rs;
    q.rz = eta * izpe;
    q.re = zeta * izpe;
    q.WPx = -q.rz * PQx; q.WPy = -q.rz * PQy; q.WPz = -q.rz * PQz;
    q.WQx = q.re * PQx; q.WQy = q.re * PQy; q.WQz = q.re * PQz;
    q.QCx = __ldg(pr.p.PA + 3 * j);
    q.QCy = __ldg(pr.p.PA + 3 * j + 1);
    q.QCz = __ldg(pr.p.PA + 3 * j + 2);
    q.oo2ze = 0.5 * izpe;
    C::prim(q, F, acc);
  }
  eri_lane_sum<C::NACC>(acc, ln.lg);
  if (ln.g != 0 || !ln.on) return;
  const double ABx = __ldg(pr.p.AB + 3 * tk.x), ABy = __ldg(pr.p.AB + 3 * tk.x + 1), ABz = __ldg(pr.p.AB + 3 * tk.x + 2);
  const double CDx = __ldg(pr.p.AB + 3 * tk.y), CDy = __ldg(pr.p.AB + 3 * tk.y + 1), CDz = __ldg(pr.p.AB + 3 * tk.y + 2);
  C::finish(acc, ABx, ABy, ABz, CDx, CDy, CDz, [&](int k, double v) { store[(size_t)k * rg.stride + t] = v; });
}
