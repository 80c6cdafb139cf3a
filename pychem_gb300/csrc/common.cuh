// Shared device-side definitions for the pychem_gb300 integral/SCF library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define PCG_MAXL 2               // shells up to d
#define PCG_MAXLT (4 * PCG_MAXL) // highest Boys order for an ERI class
#define PCG_MAXPRIM 16

// status codes of the C ABI (PCG_OK, PCG_ERR_*)
#include "../../include/pychem_gb300.h"

#define PCG_CUDA(call)                                      \
  do {                                                      \
    cudaError_t _e = (call);                                \
    if (_e != cudaSuccess) { pcg_set_cuda_error(_e, #call); \
      return PCG_ERR_CUDA; }                                \
  } while (0)

void pcg_set_cuda_error(cudaError_t e, const char* what);
void pcg_set_error(const char* msg);

// ----------------------------------------------------------------------------------
// Boys function F_m(T), T < BOYS_TMAX: the Taylor series about the nearest grid point
// T_p = p / 64, with d = T_p - T (|d| <= 1/128): F_m(T) = sum_k F_{m+k}(T_p) d^k / k!.
// The FP64 pipe of this GPU issues 2 lanes per clock and SM, 1/64 of the FP32 and
// integer rates, so an integral kernel's time is its count of FP64 instructions and the
// series is arranged to need few of them: the terms d^4 .. d^6, below 2e-10 of the sum,
// are summed in FP32 (their rounding is 1e-17 of the sum), and grid index, grid point and
// the conversions between the two precisions are integer operations.  A row of the
// table holds four doubles and three floats (48 bytes, three 16-byte loads), truncation
// 2e-18.  Order m costs 4 FP64 instructions (the 16-point grid with eight FP64 terms: 7, and
// 5 more for the argument).  Orders up to 2 are each read from the table; above, the lower ones come
// from the downward recursion F_{m-1} = (2T F_m + exp(-T)) / (2m - 1), exp(-T) from the
// same grid.  Beyond BOYS_TMAX: F_0 = sqrt(pi/T)/2 and the upward recursion
// F_{m+1} = (2m+1) F_m / (2T) (exp(-T) < 1e-20 there).  Orders up to 2 have rows to T = 65536
// too, 256 a binade about the middles of their intervals (|d| <= T / 512, truncation 1e-17; beyond, the
// float terms would underflow): the lanes of a warp fall on both sides of 48 as a rule, and
// with one evaluation for both no lane waits for the other formula.
// The range test is on the high word, unsigned: a NaN of either sign (and a negative T) goes past
// the table to the formula for large T.
// The single-precision variant keeps a grid of 16 points per unit and BOYS_KF terms.
// ----------------------------------------------------------------------------------
#define BOYS_TMAX 48.0
#define BOYS_TMAX_HI 0x40480000  // high word of 48.0
#define BOYS_INV_H 64
#define BOYS_NP (48 * BOYS_INV_H + 1)
#define BOYS_LOG_HI 0x40F00000   // high word of 65536.0
#define BOYS_NLOG ((BOYS_LOG_HI - BOYS_TMAX_HI) >> 12)
#define BOYS_ROWS (BOYS_NP + BOYS_NLOG)
#define BOYS_M (PCG_MAXLT + 1)
#define BOYS_K 7
#define BOYS_INV_HF 16
#define BOYS_NPF (48 * BOYS_INV_HF + 1)
#define BOYS_KF 5  // terms for the single-precision variant

// Taylor row of a function of one variable about a grid point: c_0 .. c_3 and c_4 .. c_6
struct __align__(16) TaylorRow {
  double c[4];
  float t[4];
};

struct BoysTable {
  const TaylorRow* c;  // [BOYS_M][BOYS_ROWS] (rows from BOYS_NP on: m <= 2)
  const double* ex;    // exp(-T_p), [BOYS_NP]
  const float* cf;     // [BOYS_NPF][BOYS_M][BOYS_KF]
  const float* exf;    // [BOYS_NPF]
};

// Tables of the j0(S r12) fundamentals: rows of z^-m j_m(z) over x = z^2 / 2 < 50, and
// (sin, cos) at z_p = p / 64 up to z = 100
#define BESSEL_NP (50 * BOYS_INV_H + 1)
#define SINCOS_NP (100 * BOYS_INV_H + 1)
struct BesselTable {
  const TaylorRow* c;  // [BOYS_M][BESSEL_NP]
  const double2* sc;   // [SINCOS_NP]
};

// Double to float and back by integer operations (the conversion instructions use the
// FP64 pipe).  to_float truncates; magnitudes below 2^-126 become (nearly) 0.
// to_double of 0 is 2^-127, far below anything that it is added to here.
__device__ __forceinline__ float bits_to_float(double x) {
  const int hi = __double2hiint(x);
  const int m = max((hi & 0x7fffffff) - (896 << 20), 0);
  return __int_as_float((hi & 0x80000000) | __funnelshift_l(__double2loint(x), m, 3));
}
__device__ __forceinline__ double bits_to_double(float x) {
  const unsigned u = __float_as_uint(x);
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
}

// Reciprocal square root: the hardware's FP64 estimate (about 20 bits) and one
// third-order step y <- y (1 + e/2 + 3 e^2/8), e = 1 - x y^2, whose remainder 5 e^3 / 16 is
// below 2^-58: 5 FP64 instructions.
__device__ __forceinline__ double nr_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// c_0 + c_1 d + ... + c_6 d^6 from a row; df = d in single precision
__device__ __forceinline__ double taylor_row(const TaylorRow* row, double d, float df) {
  const double2 a = __ldg((const double2*)row), b = __ldg((const double2*)row + 1);
  const float4 t = __ldg((const float4*)row + 2);
  const float x = df * fmaf(df, fmaf(df, t.z, t.y), t.x);
  return fma(fma(fma(b.y + bits_to_double(x), d, b.x), d, a.y), d, a.x);
}

// nearest point of a grid of 64 per unit to T in [0, 2^15): its index, and d = T_p - T
__device__ __forceinline__ int taylor_point(double T, double& d, float& df) {
  const float r = fmaf(bits_to_float(T), 64.0f, 12582912.0f);   // 1.5 * 2^23: rounds to an integer
  d = bits_to_double((r - 12582912.0f) * 0.015625f) - T;
  df = bits_to_float(d);
  return __float_as_int(r) - 0x4B400000;
}

template <int L>
__device__ __forceinline__ void boys_eval(const BoysTable& bt, double T, double* F) {
  const int hi = __double2hiint(T);
  if ((unsigned)hi < (unsigned)(L <= 2 ? BOYS_LOG_HI : BOYS_TMAX_HI)) {
    double d;
    float df;
    int p;
    if (L <= 2) {
      const float r = fmaf(bits_to_float(T), 64.0f, 12582912.0f);   // 1.5 * 2^23: rounds to an integer
      const double lin = bits_to_double((r - 12582912.0f) * 0.015625f);
      const bool low = hi < BOYS_TMAX_HI;
      d = __hiloint2double(low ? __double2hiint(lin) : (hi & ~0xfff) | 0x800, low ? __double2loint(lin) : 0) - T;
      df = bits_to_float(d);
      p = low ? __float_as_int(r) - 0x4B400000 : BOYS_NP + ((hi - BOYS_TMAX_HI) >> 12);
#pragma unroll
      for (int m = 0; m <= L; ++m) F[m] = taylor_row(bt.c + m * BOYS_ROWS + p, d, df);
    } else {
      p = taylor_point(T, d, df);
      F[L] = taylor_row(bt.c + L * BOYS_ROWS + p, d, df);
      // exp(-T) = exp(-T_p) (1 + d (1 + d/2 + d^2 (1/6 + ...)))
      const float x = df * fmaf(df, fmaf(df, 1.0f / 720.0f, 1.0f / 120.0f), 1.0f / 24.0f);
      const double u = fma(fma(1.0 / 6.0 + bits_to_double(x), d, 0.5), d, 1.0);
      const double ep = __ldg(bt.ex + p);
      const double e = fma(ep * d, u, ep);
      const double t2 = 2.0 * T;
#pragma unroll
      for (int m = L; m > 0; --m) F[m - 1] = fma(t2, F[m], e) * (1.0 / (2 * m - 1));
    }
  } else {
    const double rs = nr_rsqrt(T);
    F[0] = 0.88622692545275801365 * rs;  // sqrt(pi)/2
    if (L > 0) {
      const double h = 0.5 * rs * rs;      // 1 / (2T)
#pragma unroll
      for (int m = 0; m < L; ++m) F[m + 1] = F[m] * ((2 * m + 1) * h);
    }
  }
}

template <int L>
__device__ __forceinline__ void boys_eval_f(const BoysTable& bt, float T, float* F) {
  if (T < (float)BOYS_TMAX) {
    const int p = __float2int_rn(T * BOYS_INV_HF);
    const float d = (float)p * (1.0f / BOYS_INV_HF) - T;
    const float* row = bt.cf + ((size_t)p * BOYS_M + L) * BOYS_KF;
    float f = __ldg(row + BOYS_KF - 1);
#pragma unroll
    for (int k = BOYS_KF - 2; k >= 0; --k) f = fmaf(f, d, __ldg(row + k));
    F[L] = f;
    if (L > 0) {
      float e = 1.0f / 24.0f;
      e = fmaf(e, d, 1.0f / 6.0f);
      e = fmaf(e, d, 0.5f);
      e = fmaf(e, d, 1.0f);
      e = fmaf(e, d, 1.0f);
      e *= __ldg(bt.exf + p);
      const float t2 = 2.0f * T;
#pragma unroll
      for (int m = L; m > 0; --m) F[m - 1] = fmaf(t2, F[m], e) * (1.0f / (2 * m - 1));
    }
  } else {
    const float rs = rsqrtf(T);
    F[0] = 0.88622692545275801365f * rs;
    if (L > 0) {
      const float h = 0.5f * rs * rs;
#pragma unroll
      for (int m = 0; m < L; ++m) F[m + 1] = F[m] * ((2 * m + 1) * h);
    }
  }
}

// runtime-L dispatch used by the one-electron kernels and fine-grained entry points
__device__ __forceinline__ void boys_eval_rt(const BoysTable& bt, int L, double T, double* F) {
  switch (L) {
    case 0: boys_eval<0>(bt, T, F); break;
    case 1: boys_eval<1>(bt, T, F); break;
    case 2: boys_eval<2>(bt, T, F); break;
    case 3: boys_eval<3>(bt, T, F); break;
    case 4: boys_eval<4>(bt, T, F); break;
    case 5: boys_eval<5>(bt, T, F); break;
    case 6: boys_eval<6>(bt, T, F); break;
    case 7: boys_eval<7>(bt, T, F); break;
    default: boys_eval<8>(bt, T, F); break;
  }
}

// ----------------------------------------------------------------------------------
// Basis and pair data in HBM (structure of arrays).
//   shells:      l, nprim, first primitive, first AO (spherical), atom, centre
//   primitives:  exponent, contraction coefficient times (2a)^{(l+1.5)/2} times the
//                normalisation of the pure-axis Cartesian component
//   shell pairs: oriented A = higher l; primitive pairs of pair p are
//                [ppoff[p], ppoff[p] + npp[p]), row-major over (primA, primB)
//   prim pairs:  zeta, P, P - A, and K = cc_a cc_b (2/sqrt(pi))^{1/2} U sqrt(zeta)
//                with U = (pi/zeta)^{3/2} exp(-ab/zeta |A-B|^2), so that
//                [00|00]^(m) = K_P K_Q F_m(T) / sqrt(zeta + eta)
// ----------------------------------------------------------------------------------
struct DevBasis {
  int nshell, nprim, natom, nbf;
  const int* sh_l;
  const int* sh_nprim;
  const int* sh_prim;
  const int* sh_ao;
  const int* sh_atom;
  const double* sh_xyz;      // [nshell][3]
  const double* pr_exp;
  const double* pr_cc;
  const double* at_xyz;      // [natom][3]
  const double* at_z;
  // matrix layout: element (p, q) of the shell's molecule lives at
  //   blk(shell) + p * ld + q   (p, q local AO indices); a single molecule has
  //   blk = 0, ld = nbf.  Nuclear attraction runs over the molecule's atoms only.
  int ld;
  const long long* sh_blk;   // nullptr: 0 for every shell
  const int* sh_at0;         // nullptr: atoms [0, natom)
  const int* sh_nat;
};

__device__ __forceinline__ long long dev_blk(const DevBasis& b, int sh) {
  return b.sh_blk ? __ldg(b.sh_blk + sh) : 0ll;
}

struct DevPairs {
  int npair, npp;
  const int* A;       // shell index, l_A >= l_B
  const int* B;
  const int* ppoff;
  const int* npp_of;
  const double* AB;   // [npair][3] = A - B
  // primitive-pair SoA
  const double* zeta;
  const double* P;    // [npp][3]
  const double* PA;   // [npp][3]
  const double* K;
  const float* Kf;
  const int4* ao4;    // optional: (AO of A | (A == B) << 30, AO of B, block offset lo, hi)
  const float4* pf8;  // optional: per primitive pair (zeta, PA xyz), (1/(2 zeta), K, 0, 0)
};
