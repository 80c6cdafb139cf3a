// Boys table, primitive-pair data and one-electron (S, T, V) kernels.
//
// Upstream counterparts: pair data Methods/c_ints/shellpair_quantities.c:5-38 and
// Util/structures.py:918-956; one-electron integrals Methods/integrals.py:220-370 with
// one_electron_{fundamentals,vrr,hrr,kinetic,contract}.c; core/overlap assembly
// Methods/hartree_fock.py:207-224.
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "pcg_internal.h"

// ----------------------------------------------------------------------------------
// Boys table (host build once per device)
// ----------------------------------------------------------------------------------
// In extended precision: the error of a row would otherwise be that of this series, 2e-15 of
// the value, ten times what the evaluation from the row adds.
static void boys_host(int mmax, double T, double* F) {
  // positive series for the top order, downward recursion (stable for all T here,
  // T <= 48 keeps exp(T) finite)
  const long double t2 = 2.0L * T, e = expl(-(long double)T);
  long double term = 1.0L / (2 * mmax + 1), acc = term;
  for (int k = 1; k < 10000; ++k) {
    term *= t2 / (2 * mmax + 2 * k + 1);
    acc += term;
    if (k > 10 && term < 1e-20L * acc) break;
  }
  long double f = e * acc;
  F[mmax] = (double)f;
  for (int m = mmax; m > 0; --m) {
    f = (t2 * f + e) / (2 * m - 1);
    F[m - 1] = (double)f;
  }
}

// z^-m j_m(z), m = 0 .. mmax (z <= 10 < mmax): the power series for the two highest
// orders, where nothing cancels, and f_{m-1} = (2m+1) f_m - z^2 f_{m+1} downwards
static void bessel_host(int mmax, double z, double* f) {
  const long double x = 0.5L * z * z;
  long double up[2];
  for (int m = mmax; m <= mmax + 1; ++m) {
    long double term = 1.0L;
    for (int k = 1; k <= m; ++k) term /= 2 * k + 1;
    long double acc = term;
    for (int k = 1; fabsl(term) > 1e-22L * fabsl(acc); ++k) {
      term *= -x / ((long double)k * (2 * m + 2 * k + 1));
      acc += term;
    }
    up[m - mmax] = acc;
  }
  for (int m = mmax; m >= 0; --m) {
    f[m] = (double)up[0];
    const long double lower = (2 * m + 1) * up[0] - 2.0L * x * up[1];
    up[1] = up[0];
    up[0] = lower;
  }
}

static DeviceState g_dev[16];

DeviceState* pcg_state() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return nullptr;
  return &g_dev[dev];
}

int pcg_ensure_boys(BoysTable* out) {
  DeviceState* st = pcg_state();
  if (!st) { pcg_set_error("no CUDA device"); return PCG_ERR_CUDA; }
  // threads may make their first calls at the same time: none sees some of the tables
  static std::mutex building;
  std::lock_guard<std::mutex> hold(building);
  if (!st->boys_c) {
    std::vector<TaylorRow> c((size_t)BOYS_M * BOYS_ROWS);
    std::vector<double> ex(BOYS_NP);
    std::vector<float> cf((size_t)BOYS_NPF * BOYS_M * BOYS_KF), exf(BOYS_NPF);
    double F[64], fact[BOYS_K];
    fact[0] = 1.0;
    for (int k = 1; k < BOYS_K; ++k) fact[k] = fact[k - 1] * k;
    for (int p = 0; p < BOYS_NP; ++p) {
      const double T = (double)p / BOYS_INV_H;
      boys_host(BOYS_M + BOYS_K, T, F);
      for (int m = 0; m < BOYS_M; ++m) {
        TaylorRow& r = c[(size_t)m * BOYS_ROWS + p];
        for (int k = 0; k < 4; ++k) r.c[k] = F[m + k] / fact[k];
        for (int k = 4; k < BOYS_K; ++k) r.t[k - 4] = (float)(F[m + k] / fact[k]);
        r.t[3] = 0.0f;
      }
      ex[p] = (double)expl(-(long double)T);
      if (p % (BOYS_INV_H / BOYS_INV_HF) == 0) {
        const int q = p / (BOYS_INV_H / BOYS_INV_HF);
        for (int m = 0; m < BOYS_M; ++m)
          for (int k = 0; k < BOYS_KF; ++k) cf[((size_t)q * BOYS_M + m) * BOYS_KF + k] = (float)(F[m + k] / fact[k]);
        exf[q] = (float)ex[p];
      }
    }
    for (int q = 0; q < BOYS_NLOG; ++q) {
      // the middle of the interval whose high words start at BOYS_TMAX_HI + (q << 12)
      const int64_t bits = ((int64_t)(BOYS_TMAX_HI + (q << 12) + 0x800)) << 32;
      double T;
      memcpy(&T, &bits, sizeof(T));
      F[0] = 0.5 * sqrt(M_PI / T);
      for (int m = 0; m < 3 + BOYS_K; ++m) F[m + 1] = (2 * m + 1) * F[m] / (2.0 * T);
      for (int m = 0; m < 3; ++m) {
        TaylorRow& r = c[(size_t)m * BOYS_ROWS + BOYS_NP + q];
        for (int k = 0; k < 4; ++k) r.c[k] = F[m + k] / fact[k];
        for (int k = 4; k < BOYS_K; ++k) r.t[k - 4] = (float)(F[m + k] / fact[k]);
        r.t[3] = 0.0f;
      }
    }
    // j_m(z) / z^m about x_p = p / 64, x = z^2 / 2: its derivative in x is -j_{m+1}(z) / z^{m+1},
    // so the rows have the Boys rows' form
    std::vector<TaylorRow> bj((size_t)BOYS_M * BESSEL_NP);
    std::vector<double2> sc(SINCOS_NP);
    for (int p = 0; p < BESSEL_NP; ++p) {
      bessel_host(BOYS_M + BOYS_K, sqrt(2.0 * p / BOYS_INV_H), F);
      for (int m = 0; m < BOYS_M; ++m) {
        TaylorRow& r = bj[(size_t)m * BESSEL_NP + p];
        for (int k = 0; k < 4; ++k) r.c[k] = F[m + k] / fact[k];
        for (int k = 4; k < BOYS_K; ++k) r.t[k - 4] = (float)(F[m + k] / fact[k]);
        r.t[3] = 0.0f;
      }
    }
    for (int p = 0; p < SINCOS_NP; ++p) sc[p] = make_double2(sin((double)p / BOYS_INV_H), cos((double)p / BOYS_INV_H));
    auto upload = [](auto** dst, const auto& v) {
      const size_t bytes = v.size() * sizeof(v[0]);
      cudaError_t e = cudaMalloc((void**)dst, bytes);
      return e != cudaSuccess ? e : cudaMemcpy((void*)*dst, v.data(), bytes, cudaMemcpyHostToDevice);
    };
    DeviceState n;
    PCG_CUDA(upload(&n.boys_c, c));
    PCG_CUDA(upload(&n.boys_ex, ex));
    PCG_CUDA(upload(&n.boys_cf, cf));
    PCG_CUDA(upload(&n.boys_exf, exf));
    PCG_CUDA(upload(&n.bessel, bj));
    PCG_CUDA(upload(&n.sincos, sc));
    *st = n;
  }
  out->c = st->boys_c; out->ex = st->boys_ex; out->cf = st->boys_cf; out->exf = st->boys_exf;
  return PCG_OK;
}

int pcg_ensure_bessel(BesselTable* out) {
  BoysTable bt;
  if (int rc = pcg_ensure_boys(&bt)) return rc;
  DeviceState* st = pcg_state();
  out->c = st->bessel;
  out->sc = st->sincos;
  return PCG_OK;
}

// ----------------------------------------------------------------------------------
// Primitive-pair data.  A warp takes the primitive pairs of `group` (1 to 32) shell pairs in a
// row, its lanes one each whatever shell pair they belong to: an exponential, two roots and a
// reciprocal are a chain of about a microsecond, and the 36 of an oxygen 1s pair on one
// thread took 171 us.
// ----------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_pair_data(DevBasis b, int npair, int group, const int* __restrict__ pA,
                                                   const int* __restrict__ pB, const int* __restrict__ ppoff,
                                                   double* __restrict__ AB, double* __restrict__ zeta,
                                                   double* __restrict__ P, double* __restrict__ PA,
                                                   double* __restrict__ K, float* __restrict__ Kf,
                                                   double* __restrict__ oo2z) {
  const int lane = threadIdx.x & 31;
  const int p0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * group;
  if (p0 >= npair) return;
  int A = 0, B = 0, k0 = 0, nb = 1, count = 0;       // this lane's shell pair
  if (lane < group && p0 + lane < npair) {
    const int p = p0 + lane;
    A = pA[p];
    B = pB[p];
    k0 = ppoff[p];
    nb = b.sh_nprim[B];
    count = b.sh_nprim[A] * nb;
    for (int d = 0; d < 3; ++d) AB[3 * p + d] = b.sh_xyz[3 * A + d] - b.sh_xyz[3 * B + d];
  }
  int end = count;                                   // primitive pairs up to and with this lane's
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += x;
  }
  const int total = __shfl_sync(0xffffffffu, end, 31);
  for (int it0 = 0; it0 < total; it0 += 32) {
    const int it = it0 + lane;
    int src = 0;                                     // the first lane with end > it
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(0xffffffffu, end, src + o - 1) <= it) src += o;
    src = min(src, 31);
    const int sA = __shfl_sync(0xffffffffu, A, src), sB = __shfl_sync(0xffffffffu, B, src);
    const int snb = __shfl_sync(0xffffffffu, nb, src), sk = __shfl_sync(0xffffffffu, k0, src);
    const int local = it - (__shfl_sync(0xffffffffu, end, src) - __shfl_sync(0xffffffffu, count, src));
    if (it >= total) continue;
    const int i = local / snb, j = local - i * snb, k = sk + local;
    const double ax = b.sh_xyz[3 * sA], ay = b.sh_xyz[3 * sA + 1], az = b.sh_xyz[3 * sA + 2];
    const double bx = b.sh_xyz[3 * sB], by = b.sh_xyz[3 * sB + 1], bz = b.sh_xyz[3 * sB + 2];
    const double dx = ax - bx, dy = ay - by, dz = az - bz;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double a = b.pr_exp[b.sh_prim[sA] + i], ca = b.pr_cc[b.sh_prim[sA] + i];
    const double be = b.pr_exp[b.sh_prim[sB] + j], cb = b.pr_cc[b.sh_prim[sB] + j];
    const double z = a + be, s = 1.0 / z, ps = M_PI * s;
    const double U = ps * sqrt(ps) * exp(-a * be * s * r2);
    const double px = (a * ax + be * bx) * s, py = (a * ay + be * by) * s, pz = (a * az + be * bz) * s;
    zeta[k] = z;
    oo2z[k] = 0.5 * s;
    P[3 * k] = px; P[3 * k + 1] = py; P[3 * k + 2] = pz;
    PA[3 * k] = px - ax; PA[3 * k + 1] = py - ay; PA[3 * k + 2] = pz - az;
    // sqrt(2/sqrt(pi)) = 1.0622519320271968
    const double kk = ca * cb * 1.0622519320271968 * U * sqrt(z);
    K[k] = kk;
    Kf[k] = (float)kk;
  }
}

int pcg_launch_pair_data(const DevBasis& b, int npair, const int* pA, const int* pB, const int* ppoff,
                         double* AB, double* zeta, double* P, double* PA, double* K, float* Kf, double* oo2z,
                         cudaStream_t s) {
  if (npair <= 0) return PCG_OK;
  int group = 1;                                     // about 16 warps on every SM
  while (group < 32 && npair / group > 2432) group *= 2;
  const int warps = (npair + group - 1) / group;
  k_pair_data<<<(warps + 3) / 4, 128, 0, s>>>(b, npair, group, pA, pB, ppoff, AB, zeta, P, PA, K, Kf, oo2z);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

__global__ void k_pair_data_f32(int npp, const double* __restrict__ zeta, const double* __restrict__ PA,
                                const double* __restrict__ oo2z, const float* __restrict__ Kf,
                                float4* __restrict__ pf8) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= npp) return;
  pf8[2 * k] = make_float4((float)zeta[k], (float)PA[3 * k], (float)PA[3 * k + 1], (float)PA[3 * k + 2]);
  pf8[2 * k + 1] = make_float4((float)oo2z[k], Kf[k], 0.0f, 0.0f);
}

int pcg_launch_pair_data_f32(int npp, const double* zeta, const double* PA, const double* oo2z, const float* Kf,
                             float* pf8, cudaStream_t s) {
  if (npp <= 0) return PCG_OK;
  k_pair_data_f32<<<(npp + 255) / 256, 256, 0, s>>>(npp, zeta, PA, oo2z, Kf, (float4*)pf8);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

__global__ void k_pair_ao(DevBasis b, int npair, const int* __restrict__ pA, const int* __restrict__ pB,
                          int4* __restrict__ ao4) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npair) return;
  const int A = pA[p], B = pB[p];
  const long long o = dev_blk(b, A);
  ao4[p] = make_int4(b.sh_ao[A] | (A == B ? 1 << 30 : 0), b.sh_ao[B], (int)(unsigned)(o & 0xFFFFFFFFll),
                     (int)(o >> 32));
}

int pcg_launch_pair_ao(const DevBasis& b, int npair, const int* pA, const int* pB, int* ao4, cudaStream_t s) {
  if (npair <= 0) return PCG_OK;
  k_pair_ao<<<(npair + 127) / 128, 128, 0, s>>>(b, npair, pA, pB, (int4*)ao4);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// ----------------------------------------------------------------------------------
// One-electron integrals
// ----------------------------------------------------------------------------------
// Cartesian -> spherical row coefficient times the component normalisation ratio.
__device__ __forceinline__ double d_sph(int l, int r, int c) {
  if (l <= 1) return r == c ? 1.0 : 0.0;
  // d: xx xy xz yy yz zz; ratio sqrt(3) for the mixed components xy, xz, yz
  const double h = 0.86602540378443864676, s3 = 1.7320508075688772935;
  switch (r) {
    case 0: return c == 0 ? h : (c == 3 ? -h : 0.0);
    case 1: return c == 1 ? s3 : 0.0;
    case 2: return c == 2 ? s3 : 0.0;
    case 3: return c == 4 ? s3 : 0.0;
    default: return c == 0 ? -0.5 : (c == 3 ? -0.5 : (c == 5 ? 1.0 : 0.0));
  }
}

// (x, y, z) of degree d is component s(s+1)/2 + z, s = y + z, of its degree
__host__ __device__ constexpr int oe_ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int oe_first(int l) { return l * (l + 1) * (l + 2) / 6; }
__host__ __device__ constexpr int oe_k(int s, int z) { return s * (s + 1) / 2 + z; }
__host__ __device__ constexpr int oe_up(int s, int z, int i) { return i == 0 ? oe_k(s, z) : oe_k(s + 1, z + (i == 2)); }

// Overlap, kinetic energy and nuclear attraction of the shell pairs of one class
// (Methods/integrals.py:220-370), a warp per pair.  32 primitive pairs at a time, a lane each
// works out one's exponential and centre, leaves them in shared memory and adds its
// overlap and kinetic terms; then the lanes take the (primitive pair, nucleus) items, the loop
// that dominates: the attraction with the whole momentum on the first centre,
// [e|0] for e = LA .. LA + LB (Obara-Saika, in registers), summed before it is shifted to the
// second centre once per pair -- (a|b+1) = (a+1|b) + (A - B)(a|b) holds for contracted
// functions.  FP64 instructions bound it.  C12H26/cc-pVDZ: 1760 us with run-time momenta, the
// recursion's tables in local memory and the exponential per item; 430 us so.
template <int LA, int LB>
__global__ void __launch_bounds__(128) k_one_electron(DevBasis b, BoysTable bt, int npair, const int* __restrict__ pA,
                                                      const int* __restrict__ pB, double* __restrict__ S,
                                                      double* __restrict__ H) {
  constexpr int L = LA + LB, NA = oe_ncart(LA), NB = oe_ncart(LB), NE = oe_first(L + 1) - oe_first(LA);
  __shared__ double prim[4][32][6];                  // P, exponent sum, 1 / (2 sum), factor
  __shared__ double blk[4][2][NA * NB];              // overlap; kinetic energy, then the sum
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double(*pr)[6] = prim[warp];
  double* sS = blk[warp][0];
  double* sH = blk[warp][1];
  for (int p = blockIdx.x * 4 + warp; p < npair; p += gridDim.x * 4) {
    int A = pA[p], B = pB[p];
    if (b.sh_l[A] < b.sh_l[B]) { const int t = A; A = B; B = t; }
    if (b.sh_l[A] != LA || b.sh_l[B] != LB) continue;
    double a0[3], ab[3], r2 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      a0[i] = b.sh_xyz[3 * A + i];
      ab[i] = a0[i] - b.sh_xyz[3 * B + i];
      r2 = fma(ab[i], ab[i], r2);
    }
    const int npb = b.sh_nprim[B], npp = b.sh_nprim[A] * npb;
    const int c0 = b.sh_at0 ? b.sh_at0[A] : 0, nnuc = b.sh_at0 ? b.sh_nat[A] : b.natom;
    double Sc[NA * NB], Tc[NA * NB], Vc[NE];
#pragma unroll
    for (int i = 0; i < NA * NB; ++i) Sc[i] = Tc[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NE; ++i) Vc[i] = 0.0;
    for (int base = 0; base < npp; base += 32) {
      const int cnt = min(32, npp - base);
      __syncwarp();
      if (lane < cnt) {
        const int ia = (base + lane) / npb, ib = base + lane - ia * npb;
        const double al = b.pr_exp[b.sh_prim[A] + ia], be = b.pr_exp[b.sh_prim[B] + ib];
        const double cc = b.pr_cc[b.sh_prim[A] + ia] * b.pr_cc[b.sh_prim[B] + ib];
        const double z = al + be, s = 1.0 / z, ps = M_PI * s, h = 0.5 * s;
        const double U = ps * sqrt(ps) * exp(-al * be * s * r2) * cc;
        double PA[3], PB[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double P = (al * a0[i] + be * (a0[i] - ab[i])) * s;
          PA[i] = P - a0[i];
          PB[i] = PA[i] + ab[i];
          pr[lane][i] = P;
        }
        pr[lane][3] = z;
        pr[lane][4] = h;
        pr[lane][5] = 2.0 * sqrt(z * (1.0 / M_PI)) * U;
        // one-dimensional overlap factors (Obara-Saika)
        double E[3][LA + 1][LB + 3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
          for (int i = 0; i <= LA; ++i)
#pragma unroll
            for (int j = 0; j <= LB + 2; ++j) {
              double v = 1.0;
              if (j == 0 && i > 0) {
                v = PA[d] * E[d][i - 1][0];
                if (i > 1) v += (i - 1) * h * E[d][i - 2][0];
              } else if (j > 0) {
                v = PB[d] * E[d][i][j - 1];
                if (i > 0) v += i * h * E[d][i - 1][j - 1];
                if (j > 1) v += (j - 1) * h * E[d][i][j - 2];
              }
              E[d][i][j] = v;
            }
        // kinetic energy from overlaps [a|b+2], [a|b], [a|b-2] (one_electron_kinetic.c:60-64)
#pragma unroll
        for (int sa = 0; sa <= LA; ++sa)
#pragma unroll
          for (int za = 0; za <= sa; ++za)
#pragma unroll
            for (int sb = 0; sb <= LB; ++sb)
#pragma unroll
              for (int zb = 0; zb <= sb; ++zb) {
                const int x[3] = {LA - sa, sa - za, za}, y[3] = {LB - sb, sb - zb, zb};
                double f[3], t[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                  f[d] = E[d][x[d]][y[d]];
                  t[d] = be * E[d][x[d]][y[d] + 2];
                  if (y[d] > 1) t[d] = fma(0.25 * y[d] * (y[d] - 1) / be, E[d][x[d]][y[d] - 2], t[d]);
                }
                const double sv = f[0] * f[1] * f[2];
                const double q = t[0] * f[1] * f[2] + f[0] * t[1] * f[2] + f[0] * f[1] * t[2];
                const int e = oe_k(sa, za) * NB + oe_k(sb, zb);
                Sc[e] = fma(U, sv, Sc[e]);
                Tc[e] = fma(U * be, fma(-2.0, q, (2 * LB + 3) * sv), Tc[e]);
              }
      }
      __syncwarp();
      for (int item = lane; item < cnt * nnuc; item += 32) {
        const int pp = item / nnuc, c = c0 + item - pp * nnuc;
        const double* q = pr[pp];
        const double z = q[3], h = q[4];
        double PA[3], PC[3], pc2 = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          PA[i] = q[i] - a0[i];
          PC[i] = q[i] - b.at_xyz[3 * c + i];
          pc2 = fma(PC[i], PC[i], pc2);
        }
        double F[L + 1];
        boys_eval<L>(bt, z * pc2, F);
        const double pre = -(double)b.at_z[c] * q[5];
        double V[oe_first(L + 1)][L + 1];            // [component][m]
#pragma unroll
        for (int m = 0; m <= L; ++m) V[0][m] = pre * F[m];
#pragma unroll
        for (int l = 1; l <= L; ++l)
#pragma unroll
          for (int s = 0; s <= l; ++s)
#pragma unroll
            for (int zz = 0; zz <= s; ++zz) {
              const int x = l - s, y = s - zz;
              const int i = x ? 0 : (y ? 1 : 2), n = (i == 0 ? x : i == 1 ? y : zz) - 1;   // one down along i, then two
              const int s1 = s - (i != 0), z1 = zz - (i == 2), s2 = s1 - (i != 0), z2 = z1 - (i == 2);
              const int g = oe_first(l) + oe_k(s, zz), g1 = oe_first(l - 1) + oe_k(s1, z1);
#pragma unroll
              for (int m = 0; m <= L - l; ++m) {
                double v = fma(PA[i], V[g1][m], -PC[i] * V[g1][m + 1]);
                if (n > 0) {
                  const int g2 = oe_first(l - 2) + oe_k(s2, z2);
                  v = fma(n * h, V[g2][m] - V[g2][m + 1], v);
                }
                V[g][m] = v;
              }
            }
#pragma unroll
        for (int i = 0; i < NE; ++i) Vc[i] += V[oe_first(LA) + i][0];
      }
    }
    auto sum = [](double v) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      return v;
    };
#pragma unroll
    for (int i = 0; i < NA * NB; ++i) {
      Sc[i] = sum(Sc[i]);
      Tc[i] = sum(Tc[i]);
    }
#pragma unroll
    for (int i = 0; i < NE; ++i) Vc[i] = sum(Vc[i]);
    // the attraction with LB units on the second centre
#pragma unroll
    for (int sa = 0; sa <= LA; ++sa)
#pragma unroll
      for (int za = 0; za <= sa; ++za)
#pragma unroll
        for (int sb = 0; sb <= LB; ++sb)
#pragma unroll
          for (int zb = 0; zb <= sb; ++zb) {
            const int y = sb - zb;
            const int e = oe_k(sa, za) * NB + oe_k(sb, zb);
            const int o1 = oe_first(LA + 1) - oe_first(LA), o2 = oe_first(LA + 2) - oe_first(LA);
            double v = Vc[oe_k(sa, za)];
            if (LB > 0) {
              const int i = sb < LB ? 0 : (y ? 1 : 2), s1 = sa + (i != 0), z1 = za + (i == 2);
              v = fma(ab[i], v, Vc[o1 + oe_k(s1, z1)]);
              if (LB > 1) {                          // one more along j
                const int j = sb == 0 ? 0 : sb == 1 ? (zb ? 2 : 1) : (zb == 2 ? 2 : zb == 1 ? 2 : 1);
                const int sj = sa + (j != 0), zj = za + (j == 2);
                const double w = fma(ab[i], Vc[o1 + oe_k(sj, zj)], Vc[o2 + oe_up(s1, z1, j)]);
                v = fma(ab[j], v, w);
              }
            }
            if (lane == 0) {
              sS[e] = Sc[e];
              sH[e] = Tc[e] + v;
            }
          }
    __syncwarp();
    // spherical transform, both triangles
    constexpr int SA = 2 * LA + 1, SB = 2 * LB + 1;
    const int oa = b.sh_ao[A], ob = b.sh_ao[B], n = b.ld;
    const long long o = b.sh_blk ? b.sh_blk[A] : 0ll;
    if (lane < SA * SB) {
      const int r = lane / SB, q = lane - r * SB;
      double sv = 0.0, hv = 0.0;
      for (int ka = 0; ka < NA; ++ka) {
        const double ca = d_sph(LA, r, ka);
        if (ca == 0.0) continue;
        for (int kb = 0; kb < NB; ++kb) {
          const double cb = d_sph(LB, q, kb);
          if (cb == 0.0) continue;
          sv += ca * cb * sS[ka * NB + kb];
          hv += ca * cb * sH[ka * NB + kb];
        }
      }
      // a shell with itself: element (q, r) is the mirror of (r, q), written by one lane
      if (A != B || r >= q) {
        const size_t i = (size_t)(oa + r) * n + ob + q, j = (size_t)(ob + q) * n + oa + r;
        S[o + i] = sv;
        S[o + j] = sv;
        H[o + i] = hv;
        H[o + j] = hv;
      }
    }
  }
}

int pcg_launch_one_electron(const DevBasis& b, const BoysTable& bt, int npair, const int* pA, const int* pB,
                            double* S, double* H, cudaStream_t s) {
  if (npair <= 0) return PCG_OK;
  // a launch per class over all pairs: looking at a pair of another class costs little
  const unsigned blocks = (unsigned)min((npair + 3) / 4, 152 * 8);
  k_one_electron<0, 0><<<blocks, 128, 0, s>>>(b, bt, npair, pA, pB, S, H);
  k_one_electron<1, 0><<<blocks, 128, 0, s>>>(b, bt, npair, pA, pB, S, H);
  k_one_electron<1, 1><<<blocks, 128, 0, s>>>(b, bt, npair, pA, pB, S, H);
  k_one_electron<2, 0><<<blocks, 128, 0, s>>>(b, bt, npair, pA, pB, S, H);
  k_one_electron<2, 1><<<blocks, 128, 0, s>>>(b, bt, npair, pA, pB, S, H);
  k_one_electron<2, 2><<<blocks, 128, 0, s>>>(b, bt, npair, pA, pB, S, H);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// ----------------------------------------------------------------------------------
// Packed primitive pairs (64 bytes each) with the index of their exponent sum among the
// nz ascending sums zsum (-1: not there), and the factors of every two sums.
// ----------------------------------------------------------------------------------
__global__ void k_prim_pack(int npp, const double* __restrict__ zeta, const double* __restrict__ P,
                            const double* __restrict__ PA, const double* __restrict__ K, const double* __restrict__ oo2z,
                            int nz, const double* __restrict__ zsum, double* __restrict__ pk, int* __restrict__ zid) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npp) return;
  double2* o = (double2*)pk + 4 * (size_t)i;
  o[0] = make_double2(P[3 * i], P[3 * i + 1]);
  o[1] = make_double2(P[3 * i + 2], K[i]);
  o[2] = make_double2(PA[3 * i], PA[3 * i + 1]);
  o[3] = make_double2(PA[3 * i + 2], oo2z[i]);
  const double z = zeta[i];
  int lo = 0, hi = nz;                 // first sum >= z
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(zsum + mid) < z) lo = mid + 1; else hi = mid;
  }
  zid[i] = lo < nz && __ldg(zsum + lo) == z ? lo : -1;
}

__global__ void k_prim_tab(int nz, const double* __restrict__ zsum, double* __restrict__ tab) {
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= (long long)nz * nz) return;
  const double z = __ldg(zsum + x / nz), e = __ldg(zsum + x % nz), s = z + e;
  const double i = 1.0 / s;
  double2* o = (double2*)tab + 3 * x;
  o[0] = make_double2(1.0 / sqrt(s), z * (e * i));
  o[1] = make_double2(e * i, z * i);
  o[2] = make_double2(0.5 * i, 0.0);
}

int pcg_launch_prim_pack(int npp, const double* zeta, const double* P, const double* PA, const double* K,
                         const double* oo2z, int nz, const double* zsum, double* pk, int* zid, double* tab,
                         cudaStream_t s) {
  if (npp > 0) k_prim_pack<<<(npp + 127) / 128, 128, 0, s>>>(npp, zeta, P, PA, K, oo2z, nz, zsum, pk, zid);
  if (nz > 0) k_prim_tab<<<(unsigned)(((long long)nz * nz + 127) / 128), 128, 0, s>>>(nz, zsum, tab);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
