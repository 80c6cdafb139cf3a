// Batched symmetric eigensolver: parallel cyclic Jacobi.
//
// Method: two-sided Jacobi rotations B = J^T A J (Golub & Van Loan, Matrix
// Computations, 4th ed., Alg. 8.5.2 sym.schur2 for the rotation), applied to n/2
// disjoint index pairs at a time in the round-robin ("circle method") order, so one
// sweep is n-1 rounds of n/2 independent rotations.  Rows of A are updated for all
// pairs, then columns of A and of V; the sweep loop stops when the off-diagonal
// Frobenius norm falls below tol times the total norm.
//
// FP64 (n <= 136; the batched small-molecule SCF): up to four matrices to a CTA, or one over
// several CTAs.  FP32 (n <= 334): packed A and V in shared memory too, V's rows spread
// over as many CTAs per matrix as that takes and the GPU has free; the caller refines the
// float result in FP64 (Ogita-Aishima iteration, pychem_gb300/eigen.py), so the O(n^3)
// rotation work runs on the FP32 pipe.
#include <math.h>

#include "../../include/pychem_gb300.h"
#include "common.cuh"
#include "pcg_internal.h"

__device__ __forceinline__ void rot_params(float app, float aqq, float apq, float& c, float& s) {
  if (apq == 0.0f) { c = 1.0f; s = 0.0f; return; }
  const float tau = (aqq - app) / (2.0f * apq);
  float t;
  if (fabsf(tau) > 1e18f) t = 0.5f / tau;
  else t = (tau >= 0.0f ? 1.0f : -1.0f) / (fabsf(tau) + sqrtf(1.0f + tau * tau));
  c = 1.0f / sqrtf(1.0f + t * t);
  s = t * c;
}

__device__ __forceinline__ bool is_zero(double x) {   // without the FP64 pipe
  return ((__double2hiint(x) << 1) | __double2loint(x)) == 0;
}

// The FP64 rotation: c = cos of the angle, t = tan, from a = apq and d = aqq - app, scaled to order one by their exponents; t is the smaller root of
// a t^2 + d t - a = 0: an FP32 root and one Newton step in FP64 with the FP32 slope (relative
// error 1e-13).  No division or root on the FP64 pipe: the chain of dependent instructions is
// what a small matrix's round takes.  The rotation is orthogonal to rounding whatever the
// error of t (c = (1 + t^2)^-1/2); what is left of a_pq is computed, not set to zero.
__device__ __forceinline__ void rot_params(double a0, double d0, double& c, double& t) {
  c = 1.0;
  t = 0.0;
  if (is_zero(a0)) return;
  double d = d0, a = a0;
  const int ed = (__double2hiint(d) >> 20) & 0x7ff, ea = (__double2hiint(a) >> 20) & 0x7ff;
  const int e = max(ed, ea);
  if (e >= 0x7fe || e == 0) {            // infinities, NaNs and subnormal pairs: the plain form
    const double tau = d / (2.0 * a);
    t = fabs(tau) > 1e18 ? 0.5 / tau : (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
    c = 1.0 / sqrt(1.0 + t * t);
    return;
  }
  // exponents to [.., 1023]; what falls below 2^-1022 of the other is zero beside it
  const int k = e - 1023;
  d = ed > k ? __hiloint2double(__double2hiint(d) - (k << 20), __double2loint(d)) : 0.0;
  if (ea <= k) return;
  a = __hiloint2double(__double2hiint(a) - (k << 20), __double2loint(a));
  const float df = bits_to_float(d), af = bits_to_float(a);
  const float w = fmaf(df, df, 4.0f * af * af), rs = rsqrtf(w);
  const float tf = __fdividef(2.0f * af, fmaf(w, rs, fabsf(df)));
  t = bits_to_double(df < 0.0f ? -tf : tf);
  t = fma(-fma(fma(a, t, d), t, -a), bits_to_double(df < 0.0f ? -rs : rs), t);
  c = nr_rsqrt(fma(t, t, 1.0));
}

__device__ __forceinline__ int tri(int i, int j) {  // packed lower triangle, i >= j
  return i * (i + 1) / 2 + j;
}
__device__ __forceinline__ int sym(int i, int j) { return i >= j ? tri(i, j) : tri(j, i); }

// A is held as a packed lower triangle in shared memory.  Each round first computes
// the n/2 rotations, then transforms every 2x2 block (pair k rows, pair k' columns,
// k >= k') as B' = J_k^T B J_k' -- blocks are disjoint, so one pass suffices -- and
// the rows of V as V J.
//
// One matrix may be spread over `split` CTAs: every CTA holds the whole packed A and
// applies the same rotations to it (the same arithmetic in the same order, so the
// copies stay identical and need no communication), and rows [r0, r1) of V, in shared
// memory; rotations act on each row of V separately.  That keeps V out of global
// memory for n up to 334 in FP32.  With use_tab, the (k, k2) pair of every 2x2 block
// is read from a table in shared memory (after V) instead of being decoded with a
// square root per block and round.  Rotations that are the identity (a_pq = 0) skip
// their updates.  Instructions bound a round (n = 208: 5,460 blocks on every CTA); a pair's
// indices with the starts of their rows are one 16-byte word, its cosine and sine one of 8:
// n = 208 0.835 -> 0.800 ms a sweep, 298 2.57 -> 2.28.  A in square storage with odd rows, free
// of bank conflicts, gave 4 % more at 208 and lost 2 % at 64.
__global__ void __launch_bounds__(1024) k_jacobi_f(int n, int m, int split, int rows_per, const double* __restrict__ Ain,
                                                 long long sA, float* __restrict__ Vg, long long sV,
                                                 const float* __restrict__ V0, double* __restrict__ w, long long sw,
                                                 int max_sweeps, double tol, int* __restrict__ info, int use_tab) {
  extern __shared__ unsigned char smem_raw[];
  float* A = (float*)smem_raw;
  const int ntri = m * (m + 1) / 2;
  const int b = blockIdx.x / split, part = blockIdx.x % split;
  const int r0 = part * rows_per, r1 = min(m, r0 + rows_per), nrow = max(0, r1 - r0);
  float* V = A + ((ntri + 1) & ~1);                      // rows r0..r1 of V (nrow x m)
  unsigned* tab = (unsigned*)(V + (((size_t)rows_per * m + 1) & ~(size_t)1));
  constexpr int HMAX = 176;                          // m / 2 <= 167
  __shared__ float2 cs[HMAX];                        // c, s of pair k
  __shared__ int4 pq[HMAX];                          // p, q and the starts of their rows
  __shared__ double red0[32], red1[32];
  __shared__ int stop;
  const double* Ab = Ain + (size_t)b * sA;
  const int nt = blockDim.x, tid = threadIdx.x;
  for (int idx = tid; idx < ntri; idx += nt) {
    int i = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
    while (tri(i + 1, 0) <= idx) ++i;
    while (tri(i, 0) > idx) --i;
    const int j = idx - tri(i, 0);
    A[idx] = (i < n && j < n) ? (float)Ab[(size_t)i * n + j] : (float)0;
  }
  for (int idx = tid; idx < nrow * m; idx += nt) {
    const int i = r0 + idx / m, j = idx % m;
    float v = (float)(i == j);
    if (V0 && i < n && j < n) v = V0[(size_t)b * sV + (size_t)i * m + j];
    V[idx] = v;
  }
  if (tid == 0) stop = 0;
  const int h = m / 2;
  const int nblk = h * (h + 1) / 2;
  if (use_tab)
    for (int k = tid; k < h; k += nt)
      for (int k2 = 0; k2 <= k; ++k2) tab[k * (k + 1) / 2 + k2] = ((unsigned)k << 16) | (unsigned)k2;
  __syncthreads();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    double off = 0.0, tot = 0.0;
    for (int idx = tid; idx < ntri; idx += nt) {
      const double a = (double)A[idx];
      int i = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
      while (tri(i + 1, 0) <= idx) ++i;
      while (tri(i, 0) > idx) --i;
      const bool diag = (idx - tri(i, 0)) == i;
      tot += diag ? a * a : 2.0 * a * a;
      if (!diag) off += 2.0 * a * a;
    }
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_down_sync(0xffffffffu, off, o);
      tot += __shfl_down_sync(0xffffffffu, tot, o);
    }
    if ((tid & 31) == 0) { red0[tid >> 5] = off; red1[tid >> 5] = tot; }
    __syncthreads();
    if (tid == 0) {
      double o2 = 0.0, t2 = 0.0;
      for (int k = 0; k < (nt + 31) / 32; ++k) { o2 += red0[k]; t2 += red1[k]; }
      stop = (o2 <= tol * tol * t2) ? 1 : 0;
    }
    __syncthreads();
    if (stop) break;
    for (int r = 0; r < m - 1; ++r) {
      for (int k = tid; k < h; k += nt) {
        // circle method: position 0 fixed, positions 1..m-1 rotate by r
        const int a0 = (k == 0) ? 0 : 1 + (k - 1 + r) % (m - 1);
        const int a1 = 1 + (m - 2 - k + r) % (m - 1);
        const int p = min(a0, a1), q = max(a0, a1);
        float c, s;
        rot_params(A[tri(p, p)], A[tri(q, q)], A[tri(q, p)], c, s);
        cs[k] = make_float2(c, s);
        pq[k] = make_int4(p, q, tri(p, 0), tri(q, 0));
      }
      __syncthreads();
      for (int it = tid; it < nblk + nrow * h; it += nt) {
        if (it < nblk) {
          int k, k2;  // k >= k2
          if (use_tab) {
            const unsigned e = tab[it];
            k = (int)(e >> 16); k2 = (int)(e & 0xFFFFu);
          } else {
            k = (int)((sqrtf(8.0f * it + 1.0f) - 1.0f) * 0.5f);
            while ((k + 1) * (k + 2) / 2 <= it) ++k;
            while (k * (k + 1) / 2 > it) --k;
            k2 = it - k * (k + 1) / 2;
          }
          const float2 r1 = cs[k], r2 = cs[k2];
          const float c = r1.x, s = r1.y, c2 = r2.x, s2 = r2.y;
          if (s == (float)0 && s2 == (float)0) continue;   // both rotations the identity
          const int4 e1 = pq[k], e2 = pq[k2];
          const int p = e1.x, q = e1.y;
          if (k == k2) {
            const int ip = e1.z + p, iq = e1.w + q, iqp = e1.w + p;
            const float app = A[ip], aqq = A[iq], apq = A[iqp];
            // J^T [[app, apq], [apq, aqq]] J with the rotation that zeroes apq
            A[ip] = c * c * app - (float)2 * c * s * apq + s * s * aqq;
            A[iq] = s * s * app + (float)2 * c * s * apq + c * c * aqq;
            A[iqp] = (float)0;
          } else {
            const int ipp = p >= e2.x ? e1.z + e2.x : e2.z + p, ipq = p >= e2.y ? e1.z + e2.y : e2.w + p;
            const int iqp = q >= e2.x ? e1.w + e2.x : e2.z + q, iqq = q >= e2.y ? e1.w + e2.y : e2.w + q;
            const float b00 = A[ipp], b01 = A[ipq], b10 = A[iqp], b11 = A[iqq];
            // rows: J_k^T B
            const float r00 = c * b00 - s * b10, r01 = c * b01 - s * b11;
            const float r10 = s * b00 + c * b10, r11 = s * b01 + c * b11;
            // columns: (J_k^T B) J_k2
            A[ipp] = c2 * r00 - s2 * r01;
            A[ipq] = s2 * r00 + c2 * r01;
            A[iqp] = c2 * r10 - s2 * r11;
            A[iqq] = s2 * r10 + c2 * r11;
          }
        } else {
          const int t = it - nblk;
          const int i = t / h, k = t % h;            // local row i of V
          const float c = cs[k].x, s = cs[k].y;
          if (s == (float)0) continue;
          const int p = pq[k].x, q = pq[k].y;
          const float vp = V[i * m + p], vq = V[i * m + q];
          V[i * m + p] = c * vp - s * vq;
          V[i * m + q] = s * vp + c * vq;
        }
      }
      __syncthreads();
    }
  }
  if (part == 0) {
    for (int i = tid; i < n; i += nt) w[(size_t)b * sw + i] = (double)A[tri(i, i)];
    if (tid == 0 && info) info[b] = sweep;
  }
  for (int idx = tid; idx < nrow * m; idx += nt) Vg[(size_t)b * sV + (size_t)r0 * m + idx] = V[idx];
}


// FP64.  A warp's FP64 instruction takes its quarter of the SM 64 cycles whatever lanes are on,
// so the time of a round is the number of them: in its first part, one warp's as a rule, only
// the 11 that every other lane waits for (cosine, tangent, sine); in its second part 13 for
// 32 blocks off the diagonal (the tangents applied, then c c2), 4 for 32 pairs of V, and 10 in
// a warp of its own for the diagonal, held apart, with what is left of a_pq.  Zeros are found by
// their bits.  A CTA takes `per` matrices (one if split > 1), because the rotations fill only h
// lanes; each matrix stops by itself.
// 1024 matrices to 1e-15, against a CTA each with whole rotations in the first part,
// 16-instruction blocks and the diagonal among them: n = 7 170 -> 86 us, 13 390 -> 268, 25 1840 ->
// 1162; one matrix: n = 7 105 -> 60 us, 13 218 -> 123, 32 908 -> 451.
__global__ void __launch_bounds__(1024) k_jacobi_d(int n, int m, int batch, int per, int split, int rows_per,
                                                   const double* __restrict__ Ain, long long sA,
                                                   double* __restrict__ Vg, long long sV, const double* __restrict__ V0,
                                                   double* __restrict__ w, long long sw, int max_sweeps, double tol,
                                                   int* __restrict__ info) {
  extern __shared__ double smem_d[];
  const int ntri = m * (m + 1) / 2, npad = (ntri + 1) & ~1;
  const int h = m / 2, nblk = h * (h - 1) / 2;
  const int b0 = blockIdx.x / split * per, part = blockIdx.x % split;
  per = min(per, batch - b0);
  const int r0 = part * rows_per, r1 = min(m, r0 + rows_per), nrow = max(0, r1 - r0);
  // per matrix: the packed lower triangle (its diagonal slots zero), the diagonal, rows of V
  const int mat = npad + m + ((rows_per * m + 1) & ~1);
  double* rot = smem_d + per * mat;                  // c, t, s of every pair (and a gap)
  unsigned* tab = (unsigned*)(rot + 4 * per * h);    // (k, k2) of a block
  unsigned short* pq = (unsigned short*)(tab + nblk);  // p, q of pair k
  __shared__ double red[32];
  __shared__ int done[32], ndone;
  const int nt = blockDim.x, tid = threadIdx.x;
  for (int idx = tid; idx < per * m * m; idx += nt) {
    const int g = idx / (m * m), e = idx - g * m * m, i = e / m, j = e - i * m;
    if (j > i) continue;
    const double a = i < n && j < n ? Ain[(size_t)(b0 + g) * sA + (size_t)i * n + j] : 0.0;
    smem_d[g * mat + tri(i, j)] = i == j ? 0.0 : a;
    if (i == j) smem_d[g * mat + npad + i] = a;
  }
  for (int idx = tid; idx < per * nrow * m; idx += nt) {
    const int g = idx / (nrow * m), e = idx - g * nrow * m, i = r0 + e / m, j = e % m;
    double v = (double)(i == j);
    if (V0 && i < n && j < n) v = V0[(size_t)(b0 + g) * sV + (size_t)i * m + j];
    smem_d[g * mat + npad + m + e] = v;
  }
  for (int k = tid; k < h; k += nt)
    for (int k2 = 0; k2 < k; ++k2) tab[k * (k - 1) / 2 + k2] = ((unsigned)k << 16) | (unsigned)k2;
  if (tid < 32) done[tid] = 0;
  if (tid == 0) ndone = 0;
  __syncthreads();
  const int wpm = (nt / 32) / per, warp = tid >> 5, lane = tid & 31;   // warps per matrix
  const int na = (per * nblk + 31) & ~31, nv = (per * nrow * h + 31) & ~31;
  double tot = 0.0;
  int sweep = 0;
  for (;; ++sweep) {
    // sums of squares off the diagonal, and (unchanged by rotations) in all
    {
      const int g = warp / wpm, sub = (warp - g * wpm) * 32 + lane;
      double off = 0.0, dia = 0.0;
      if (g < per && !done[g]) {
        const double* A = smem_d + g * mat;
        double o1 = 0.0;
        for (int idx = sub; idx < ntri; idx += 64 * wpm) {
          off = fma(A[idx], A[idx], off);
          const int i2 = idx + 32 * wpm;
          if (i2 < ntri) o1 = fma(A[i2], A[i2], o1);
        }
        off = 2.0 * (off + o1);
        if (sweep == 0)
          for (int i = sub; i < m; i += 32 * wpm) dia = fma(A[npad + i], A[npad + i], dia);
      }
      for (int o = 16; o > 0; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
      if (sweep == 0) {
        tot = dia;
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        if (lane == 0) red[warp] = tot + off;
        __syncthreads();
        tot = 0.0;
        if (tid < per)
          for (int k = 0; k < wpm; ++k) tot += red[tid * wpm + k];
        __syncthreads();
      }
      if (lane == 0) red[warp] = off;
    }
    __syncthreads();
    if (tid < per && !done[tid]) {
      double o2 = 0.0;
      for (int k = 0; k < wpm; ++k) o2 += red[tid * wpm + k];
      if (o2 <= tol * tol * tot || sweep == max_sweeps) {
        done[tid] = 1;
        atomicAdd(&ndone, 1);
        if (part == 0 && info) info[b0 + tid] = sweep;
      }
    }
    __syncthreads();
    if (ndone == per) break;
    for (int r = 0; r < m - 1; ++r) {
      for (int it = tid; it < per * h; it += nt) {
        const int g = it / h, k = it - g * h;
        // circle method: position 0 fixed, positions 1..m-1 rotate by r
        int a0 = k - 1 + r, a1 = m - 2 - k + r;
        a0 -= a0 >= m - 1 ? m - 1 : 0;
        a1 -= a1 >= m - 1 ? m - 1 : 0;
        a0 = k == 0 ? 0 : 1 + a0;
        a1 = 1 + a1;
        const int p = min(a0, a1), q = max(a0, a1);
        const double* A = smem_d + g * mat;
        double c, t;
        rot_params(done[g] ? 0.0 : A[tri(q, p)], A[npad + q] - A[npad + p], c, t);
        if (g == 0) *(unsigned*)(pq + 2 * k) = (unsigned)p | ((unsigned)q << 16);
        *(double2*)(rot + 4 * it) = make_double2(c, t);
        rot[4 * it + 2] = t * c;
      }
      __syncthreads();
      for (int it = tid; it < na + nv + per * h; it += nt) {
        if (it < na) {
          const int g = per == 1 ? 0 : it / nblk;
          if (g >= per || it >= per * nblk) continue;
          const unsigned e = tab[it - g * nblk];
          const int k = (int)(e >> 16), k2 = (int)(e & 0xFFFFu);
          const double2 r1 = *(const double2*)(rot + 4 * (g * h + k)), r2 = *(const double2*)(rot + 4 * (g * h + k2));
          const double t = r1.y, t2 = r2.y;
          if (is_zero(t) && is_zero(t2)) continue;   // both rotations the identity
          const int p = pq[2 * k], q = pq[2 * k + 1], p2 = pq[2 * k2], q2 = pq[2 * k2 + 1];
          double* A = smem_d + g * mat;
          const int ipp = sym(p, p2), ipq = sym(p, q2), iqp = sym(q, p2), iqq = sym(q, q2);
          const double b00 = A[ipp], b01 = A[ipq], b10 = A[iqp], b11 = A[iqq], cc = r1.x * r2.x;
          // rows, then columns
          const double r00 = fma(-t, b10, b00), r01 = fma(-t, b11, b01);
          const double r10 = fma(t, b00, b10), r11 = fma(t, b01, b11);
          A[ipp] = cc * fma(-t2, r01, r00);
          A[ipq] = cc * fma(t2, r00, r01);
          A[iqp] = cc * fma(-t2, r11, r10);
          A[iqq] = cc * fma(t2, r10, r11);
        } else if (it < na + nv) {
          const int x = it - na, row = x / h, k = x - row * h, g = per == 1 ? 0 : row / nrow;
          if (row >= per * nrow) continue;
          const double* o = rot + 4 * (g * h + k);
          const double c = o[0], sn = o[2];
          if (is_zero(sn)) continue;
          const unsigned e = *(const unsigned*)(pq + 2 * k);
          double* v = smem_d + g * mat + npad + m + (row - g * nrow) * m;
          double* vp = v + (e & 0xFFFFu);
          double* vq = v + (e >> 16);
          const double x0 = *vp, x1 = *vq;
          *vp = fma(c, x0, -sn * x1);
          *vq = fma(sn, x0, c * x1);
        } else {
          const int x = it - na - nv, g = x / h, k = x - g * h;
          const double c = rot[4 * x], t = rot[4 * x + 1];
          if (is_zero(t)) continue;
          const int p = pq[2 * k], q = pq[2 * k + 1];
          double* A = smem_d + g * mat;
          const double dp = A[npad + p], dq = A[npad + q], a = A[tri(q, p)], d = dq - dp;
          const double c2 = c * c, f = fma(a, t, d), ch = (t * c2) * fma(-t, d, a + a);
          A[npad + p] = dp - ch;
          A[npad + q] = dq + ch;
          A[tri(q, p)] = -c2 * fma(f, t, -a);
        }
      }
      __syncthreads();
    }
  }
  for (int idx = tid; idx < per * m; idx += nt) {
    const int g = idx / m, i = idx - g * m;
    if (part == 0 && i < n) w[(size_t)(b0 + g) * sw + i] = smem_d[g * mat + npad + i];
  }
  for (int idx = tid; idx < per * nrow * m; idx += nt) {
    const int g = idx / (nrow * m), e = idx - g * nrow * m;
    Vg[(size_t)(b0 + g) * sV + (size_t)r0 * m + e] = smem_d[g * mat + npad + m + e];
  }
}

// 227 KB less the static tables.  The launches ask for this limit whatever they use: the attribute
// is the process's, and a thread with a smaller matrix would take it from another's launch.
#define JACOBI_D_SMEM (232448 - 1024)
#define JACOBI_F_SMEM (232448 - 5120)

// bytes of `per` matrices with rows_per rows of V each
static size_t jacobi_bytes_d(int m, int per, int rows_per) {
  const size_t h = m / 2, mat = (((size_t)m * (m + 1) / 2 + 1) & ~(size_t)1) + m + (((size_t)rows_per * m + 1) & ~(size_t)1);
  return per * (mat + 4 * h) * 8 + h * (h - 1) / 2 * 4 + 4 * h + 16;
}

// A round updates m^2 / 8 blocks of A, in every CTA, and m^2 / 2 elements of V: while SMs are
// free, V's rows are shared by up to 16 CTAs (n = 208, FP32: 0.84 ms a sweep with 2 CTAs)
static int jacobi_least(int batch, int m) {
  const int k = 152 / batch < 16 ? 152 / batch : 16;
  return k > m / 8 ? (m / 8 > 1 ? m / 8 : 1) : (k > 1 ? k : 1);
}

struct JacobiPlanD {
  int per, split, rows_per, threads;
  size_t bytes;
};
static JacobiPlanD jacobi_plan_d(int batch, int m, int least) {
  JacobiPlanD p;
  // matrices per CTA: what the rotations leave of a warp, as long as the SMs have 1.5 CTAs each
  // (n = 13, whole rotations in the first part: 1024 matrices 294 us by fours, 338 by twos; 400
  // matrices 238 us one by one, 267 by twos), and at most four: each matrix has a warp of the
  // smallest CTA to itself for its sums
  p.per = 1;
  while (p.per < 4 && 2 * p.per * (m / 2) < 32 && batch / (2 * p.per) >= 228) p.per *= 2;
  for (p.split = least; jacobi_bytes_d(m, 1, (m + p.split - 1) / p.split) > JACOBI_D_SMEM; ++p.split) {}
  p.rows_per = (m + p.split - 1) / p.split;
  p.bytes = jacobi_bytes_d(m, p.per, p.rows_per);
  const long long ctas = (long long)((batch + p.per - 1) / p.per) * p.split;
  // above n = 64 one CTA per SM is resident anyway (shared memory): 1024 threads.  Up to 32, 128
  // threads where that fills the SMs (4096 of n = 13: 621 us) or a round has no more work; else
  // 256 (one matrix of n = 32: 451 us; 478 and 526 with 128 before the diagonal had its warp)
  p.threads = m <= 32 ? (m * p.per <= 8 || ctas > 608 ? 128 : 256) : (m <= 64 ? 256 : 1024);
  return p;
}

extern "C" int pcg_jacobi_plan(int batch, int n, int* plan) {
  if (batch < 1 || n < 1 || n > 136 || !plan) {
    pcg_set_error("pcg_jacobi_plan: bad arguments (n <= 136)");
    return PCG_ERR_ARG;
  }
  const int m = n + (n & 1);
  const JacobiPlanD p = jacobi_plan_d(batch, m, jacobi_least(batch, m));
  plan[0] = p.per; plan[1] = p.split; plan[2] = p.rows_per; plan[3] = p.threads; plan[4] = (int)p.bytes;
  return PCG_OK;
}

// shared-memory plan of one FP32 launch: how many CTAs share a matrix (at least `least`), rows of V
// per CTA, whether the block table fits, and the dynamic bytes
static bool jacobi_plan(int m, int least, int& split, int& rows_per, int& tab, size_t& bytes) {
  const size_t limit = JACOBI_F_SMEM;
  const size_t a_bytes = (size_t)((m * (m + 1) / 2 + 1) & ~1) * sizeof(float);
  const size_t tab_bytes = (size_t)(m / 2) * (m / 2 + 1) / 2 * sizeof(unsigned);
  for (split = least; split <= m; ++split) {
    rows_per = (m + split - 1) / split;
    const size_t v_bytes = (size_t)(((size_t)rows_per * m + 1) & ~(size_t)1) * sizeof(float);
    if (a_bytes + v_bytes <= limit) {
      tab = a_bytes + v_bytes + tab_bytes <= limit;
      bytes = a_bytes + v_bytes + (tab ? tab_bytes : 0);
      return true;
    }
  }
  return false;
}

extern "C" int pcg_jacobi_eigh(int batch, int n, const double* A, double* w, void* V, int fp32, const void* V0,
                               int max_sweeps, double tol, int* info, void* stream) {
  if (batch < 1 || n < 1 || !A || !w || !V || max_sweeps < 1) {
    pcg_set_error("pcg_jacobi_eigh: bad arguments");
    return PCG_ERR_ARG;
  }
  const int m = n + (n & 1);
  if (m / 2 > 512 || m < 2) { pcg_set_error("pcg_jacobi_eigh: n out of range"); return PCG_ERR_UNSUPPORTED; }
  cudaStream_t s = (cudaStream_t)stream;
  {
    const cudaError_t prior = cudaGetLastError();
    if (prior != cudaSuccess) {
      pcg_set_cuda_error(prior, "an earlier asynchronous operation (reported on entry to pcg_jacobi_eigh)");
      return PCG_ERR_CUDA;
    }
  }
  const long long sA = (long long)n * n, sV = (long long)m * m, sw = n;
  // above n = 64 one CTA per SM is resident anyway (shared memory): 1024 threads
  const int threads = m <= 32 ? 128 : (m <= 64 ? 256 : 1024);
  const int least = jacobi_least(batch, m);
  int split = 1, rows_per = m, tab = 0;
  size_t bytes = 0;
  if (!fp32) {
    if (m / 2 > 68) {
      pcg_set_error("pcg_jacobi_eigh: FP64 variant needs n <= 136");
      return PCG_ERR_UNSUPPORTED;
    }
    const JacobiPlanD p = jacobi_plan_d(batch, m, least);
    const long long ctas = (long long)((batch + p.per - 1) / p.per) * p.split;
    if (ctas > 0x7fffffffLL) { pcg_set_error("pcg_jacobi_eigh: batch too large"); return PCG_ERR_ARG; }
    if (32 * p.per > p.threads) { pcg_set_error("pcg_jacobi_eigh: a CTA with more matrices than warps"); return PCG_ERR_UNSUPPORTED; }
    PCG_CUDA(cudaFuncSetAttribute(k_jacobi_d, cudaFuncAttributeMaxDynamicSharedMemorySize, JACOBI_D_SMEM));
    k_jacobi_d<<<(unsigned)ctas, p.threads, p.bytes, s>>>(n, m, batch, p.per, p.split, p.rows_per, A, sA, (double*)V, sV,
                                                 (const double*)V0, w, sw, max_sweeps, tol, info);
  } else {
    if (m / 2 > 167 || !jacobi_plan(m, least, split, rows_per, tab, bytes)) {
      pcg_set_error("pcg_jacobi_eigh: FP32 variant needs n <= 334");
      return PCG_ERR_UNSUPPORTED;
    }
    if ((long long)batch * split > 0x7fffffffLL) { pcg_set_error("pcg_jacobi_eigh: batch too large"); return PCG_ERR_ARG; }
    PCG_CUDA(cudaFuncSetAttribute(k_jacobi_f, cudaFuncAttributeMaxDynamicSharedMemorySize, JACOBI_F_SMEM));
    k_jacobi_f<<<batch * split, threads, bytes, s>>>(n, m, split, rows_per, A, sA, (float*)V, sV,
                                                          (const float*)V0, w, sw, max_sweeps, tol, info, tab);
  }
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
