// Small dense FP64 algebra of the SCF iteration, all on the GPU:
//
//  * pcg_dgemm: batched C = alpha A B + beta C with arbitrary element strides (so any
//    transposes), 8 x 8 output tiles of one thread per element.  GB300's FP64 pipe
//    is thin (about 1.7 FMA per clock per SM), so the SCF's n <= 300 products are
//    spread over many CTAs: 676 for n = 208.  Replaces the numpy.dot /
//    matrix products of Methods/hartree_fock.py:168-184 and
//    Methods/hf_extensions/diis.py:48-54 (X^T F X, the commutator, C = X C').
//  * pcg_oa_correction: the correction matrix of one Ogita-Aishima refinement step of
//    approximate eigenvectors (T. Ogita, K. Aishima, Japan J. Indust. Appl. Math. 35
//    (2018) 1007-1035, Algorithm 1) from S = X^T A X and R = I - X^T X.
//  * DIIS (Methods/hf_extensions/diis.py:32-41,108-112): Fock matrices and residuals
//    in a ring of `cap` slots, the new row of the residual inner-product matrix, the
//    C1 system solved by one CTA (Gaussian elimination with partial pivoting, the
//    oldest vectors dropped while it is singular), and the extrapolation -- no host
//    round trip, so an SCF iteration can be captured in a CUDA graph.
#include <math.h>

#include "../../include/pychem_gb300.h"
#include "common.cuh"
#include "pcg_internal.h"

// 8 x 8 output tiles (one thread per element), K in steps of 32: at n = 208 that is
// 676 CTAs, 4-5 per SM, so the FP64 work is spread evenly over the 152 SMs (with
// 16 x 16 tiles the 169 CTAs left 17 SMs with twice the work of the others).  Larger products and
// batches run at the FP64 rate too (3 x 756 x 406 x 406: 639 us, 1.17 TFLOP/s; 1500^3: 1.22);
// 32 x 32 tiles of 4 x 4 outputs a thread were slower at every shape (858 us and 1.12 TFLOP/s; 64 x 104^3
// 237 us against 153).
#define DG_T 8
#define DG_K 32

// SYM: C is symmetric (M = N): only the tiles on and below the diagonal are formed (grid.x
// counts them) and mirrored, which halves the FP64 work of X^T X, X^T A X and C C^T
// (208^3: 18 -> 12 us).
template <bool SYM>
__global__ void __launch_bounds__(DG_T* DG_T)
    k_dgemm(int M, int N, int K, double alpha, const double* __restrict__ A, long long sAb, long long sAm,
            long long sAk, const double* __restrict__ B, long long sBb, long long sBk, long long sBn, double beta,
            double* __restrict__ C, long long sCb, long long sCm, long long sCn) {
  // two shared-memory stages: the next K step's tile is loaded into registers while
  // the current one is multiplied, so the global-load latency overlaps the FMAs
  __shared__ double As[2][DG_T][DG_K + 1], Bs[2][DG_K][DG_T + 1];
  constexpr int PER = DG_T * DG_K / (DG_T * DG_T);   // elements of each tile per thread
  const int tid = threadIdx.x, tx = tid % DG_T, ty = tid / DG_T;
  const long long b = blockIdx.z;
  int by = blockIdx.y, bx = blockIdx.x;
  if (SYM) {
    by = (int)((sqrtf(8.0f * bx + 1.0f) - 1.0f) * 0.5f);
    while ((by + 1) * (by + 2) / 2 <= bx) ++by;
    while (by * (by + 1) / 2 > bx) --by;
    bx -= by * (by + 1) / 2;
  }
  const int m0 = by * DG_T, n0 = bx * DG_T;
  const int m = m0 + ty, n = n0 + tx;
  A += b * sAb;
  B += b * sBb;
  double ra[PER], rb[PER];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = tid + u * DG_T * DG_T;
      const int mr = m0 + e / DG_K, ka = k0 + e % DG_K;
      ra[u] = (mr < M && ka < K) ? __ldg(A + mr * sAm + ka * sAk) : 0.0;
      const int kb = k0 + e / DG_T, c = n0 + e % DG_T;
      rb[u] = (kb < K && c < N) ? __ldg(B + kb * sBk + c * sBn) : 0.0;
    }
  };
  auto store = [&](int st) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = tid + u * DG_T * DG_T;
      As[st][e / DG_K][e % DG_K] = ra[u];
      Bs[st][e / DG_T][e % DG_T] = rb[u];
    }
  };
  double acc = 0.0;
  load(0);
  store(0);
  __syncthreads();
  int st = 0;
  for (int k0 = 0; k0 < K; k0 += DG_K) {
    const bool more = k0 + DG_K < K;
    if (more) load(k0 + DG_K);
#pragma unroll
    for (int kk = 0; kk < DG_K; ++kk) acc = fma(As[st][ty][kk], Bs[st][kk][tx], acc);
    if (more) store(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
  if (m < M && n < N) {
    double* c = C + b * sCb + m * sCm + n * sCn;
    const double v = beta == 0.0 ? alpha * acc : fma(alpha, acc, beta * *c);
    *c = v;
    if (SYM && bx != by) C[b * sCb + n * sCm + m * sCn] = v;
  }
}

extern "C" int pcg_dgemm(int batch, int M, int N, int K, double alpha, const double* A, long long sAb, long long sAm,
                         long long sAk, const double* B, long long sBb, long long sBk, long long sBn, double beta,
                         double* C, long long sCb, long long sCm, long long sCn, void* stream) {
  if (batch < 1 || M < 0 || N < 0 || K < 0 || batch > 65535 || (M > 0 && N > 0 && (!C || (K > 0 && (!A || !B))))) {
    pcg_set_error("pcg_dgemm: bad arguments");
    return PCG_ERR_ARG;
  }
  if (M == 0 || N == 0) return PCG_OK;
  dim3 grid((N + DG_T - 1) / DG_T, (M + DG_T - 1) / DG_T, batch);
  if (grid.y > 65535) {
    if (grid.x > 65535) { pcg_set_error("pcg_dgemm: M too large"); return PCG_ERR_UNSUPPORTED; }
    // C^T = B^T A^T: the long side along grid.x
    return pcg_dgemm(batch, N, M, K, alpha, B, sBb, sBn, sBk, A, sAb, sAk, sAm, beta, C, sCb, sCn, sCm, stream);
  }
  k_dgemm<false><<<grid, DG_T * DG_T, 0, (cudaStream_t)stream>>>(M, N, K, alpha, A, sAb, sAm, sAk, B, sBb, sBk, sBn, beta,
                                                          C, sCb, sCm, sCn);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_dgemm_sym(int M, int K, double alpha, const double* A, long long sAm, long long sAk, const double* B,
                             long long sBk, long long sBn, double beta, double* C, long long sCm, long long sCn,
                             void* stream) {
  if (M < 0 || K < 0 || M > 32767 * DG_T || (M > 0 && (!C || (K > 0 && (!A || !B))))) {
    pcg_set_error("pcg_dgemm_sym: bad arguments");
    return PCG_ERR_ARG;
  }
  if (M == 0) return PCG_OK;
  const long long t = (M + DG_T - 1) / DG_T;
  k_dgemm<true><<<(unsigned)(t * (t + 1) / 2), DG_T * DG_T, 0, (cudaStream_t)stream>>>(
      M, M, K, alpha, A, 0, sAm, sAk, B, 0, sBk, sBn, beta, C, 0, sCm, sCn);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// ---------------------------------------------------------------------------------
// The reductions of an SCF iteration, two launches instead of about fifteen of tensor
// operations (each 3 to 14 us at n = 208).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ double block_reduce(double v, bool is_max, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmax(v, w) : v + w;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int k = 1; k < (int)(blockDim.x >> 5); ++k) v = is_max ? fmax(v, red[k]) : v + red[k];
  return v;
}
// a maximum that keeps NaNs, as torch's
__device__ __forceinline__ double nan_max(double a, double b) { return (a != a || b != b) ? a + b : fmax(a, b); }

#define SCF_BLOCKS 64
// R = P - P^T (n2 x n2); block partials of sum D (H + F), sum (D - Dold)^2 (n x n) and max |R|;
// Dold = D
__global__ void __launch_bounds__(256) k_scf_stats(int n, int n2, const double* __restrict__ P, const double* __restrict__ D,
                                                   const double* __restrict__ H, const double* __restrict__ F,
                                                   double* __restrict__ Dold, double* __restrict__ R,
                                                   double* __restrict__ part) {
  __shared__ double red[8];
  double e = 0.0, d2 = 0.0, mx = 0.0;
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = t0; i < n * n; i += stride) {
    const double d = D[i], x = d - Dold[i];
    e = fma(d, H[i] + F[i], e);
    d2 = fma(x, x, d2);
    Dold[i] = d;
  }
  bool bad = false;
  for (int i = t0; i < n2 * n2; i += stride) {
    const double r = P[i] - P[(size_t)(i % n2) * n2 + i / n2];
    R[i] = r;
    bad |= r != r;
    mx = fmax(mx, fabs(r));
  }
  e = block_reduce(e, false, red);
  d2 = block_reduce(d2, false, red);
  mx = block_reduce(mx, true, red);
  if (__syncthreads_or(bad)) mx = __longlong_as_double(0x7ff8000000000000ll);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = e;
    part[SCF_BLOCKS + blockIdx.x] = d2;
    part[2 * SCF_BLOCKS + blockIdx.x] = mx;
  }
}

// vals[0] = sum D (H + F), vals[1] = RMS(D - Dold), vals[5] = max |R|, partials in order
__global__ void k_scf_stats_sum(int n, int blocks, const double* __restrict__ part, double* __restrict__ vals) {
  const int w = threadIdx.x;
  if (w > 2) return;
  double v = 0.0;
  for (int k = 0; k < blocks; ++k) v = w == 2 ? nan_max(v, part[2 * SCF_BLOCKS + k]) : v + part[w * SCF_BLOCKS + k];
  if (w == 0) vals[0] = v;
  if (w == 1) vals[1] = sqrt(v / ((double)n * n));
  if (w == 2) vals[5] = v;
}

extern "C" int pcg_scf_stats(int n, int n2, const double* P, const double* D, const double* H, const double* F,
                             double* Dold, double* R, double* part, double* vals, void* stream) {
  if (n < 1 || n > 32767 || n2 < 1 || n2 > n || !P || !D || !H || !F || !Dold || !R || !part || !vals) {
    pcg_set_error("pcg_scf_stats: bad arguments");
    return PCG_ERR_ARG;
  }
  const int want = (n * n + 255) / 256, blocks = want < SCF_BLOCKS ? want : SCF_BLOCKS;
  k_scf_stats<<<blocks, 256, 0, (cudaStream_t)stream>>>(n, n2, P, D, H, F, Dold, R, part);
  k_scf_stats_sum<<<1, 32, 0, (cudaStream_t)stream>>>(n, blocks, part, vals);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// out = (max |R|, max |S_ov| over the occupied-virtual block, max d_occ - min d_virt) of a
// refined basis, d = diag S, NaN for any NaN: first the four maxima of CHECK_ROWS rows by a
// block each, then theirs by one warp.  (n = 208: one block for all took 100 us, the two 9 us.)
#define CHECK_ROWS 8
__global__ void __launch_bounds__(256) k_projector_check(int n, int nocc, const double* __restrict__ S,
                                                         const double* __restrict__ R, double* __restrict__ part) {
  __shared__ double red[32];
  double r = 0.0, c = 0.0, lo = -__longlong_as_double(0x7ff0000000000000ll), hi = lo;
  bool bad = false;
  const int a0 = blockIdx.x * CHECK_ROWS, a1 = min(n, a0 + CHECK_ROWS);
  for (int a = a0; a < a1; ++a)
    for (int b = threadIdx.x; b < n; b += blockDim.x) {
      const double x = R[(size_t)a * n + b];
      bad |= x != x;
      r = fmax(r, fabs(x));
      if ((a < nocc && b >= nocc) || a == b) {
        const double y = S[(size_t)a * n + b];
        bad |= y != y;
        if (a != b) c = fmax(c, fabs(y));
        else if (a < nocc) lo = fmax(lo, y);
        else hi = fmax(hi, -y);
      }
    }
  r = block_reduce(r, true, red);
  c = block_reduce(c, true, red);
  lo = block_reduce(lo, true, red);
  hi = block_reduce(hi, true, red);
  const bool any = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    double* o = part + 4 * blockIdx.x;
    o[0] = any ? __longlong_as_double(0x7ff8000000000000ll) : r;
    o[1] = c;
    o[2] = lo;
    o[3] = hi;
  }
}

__global__ void __launch_bounds__(32) k_projector_check_max(int blocks, const double* __restrict__ part,
                                                            double* __restrict__ out) {
  double r = 0.0, c = 0.0, lo = -__longlong_as_double(0x7ff0000000000000ll), hi = lo;
  for (int k = threadIdx.x; k < blocks; k += 32) {
    r = nan_max(r, part[4 * k]);
    c = fmax(c, part[4 * k + 1]);
    lo = fmax(lo, part[4 * k + 2]);
    hi = fmax(hi, part[4 * k + 3]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    r = nan_max(r, __shfl_xor_sync(0xffffffffu, r, o));
    c = fmax(c, __shfl_xor_sync(0xffffffffu, c, o));
    lo = fmax(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (threadIdx.x == 0) {
    out[0] = r;
    out[1] = r != r ? r : c;
    out[2] = r != r ? r : lo + hi;
  }
}

extern "C" int pcg_projector_check(int n, int nocc, const double* S, const double* R, double* part, double* out,
                                   void* stream) {
  if (n < 1 || n > 32767 || nocc < 1 || nocc >= n || !S || !R || !part || !out) {
    pcg_set_error("pcg_projector_check: bad arguments");
    return PCG_ERR_ARG;
  }
  const int blocks = (n + CHECK_ROWS - 1) / CHECK_ROWS;
  cudaStream_t s = (cudaStream_t)stream;
  k_projector_check<<<blocks, 256, 0, s>>>(n, nocc, S, R, part);
  k_projector_check_max<<<1, 32, 0, s>>>(blocks, part, out);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// E[i][j] for one refinement step X <- X + X E, with lam_i = S_ii / (1 - R_ii):
//   mode 0 (occupied-space projector): pairs with exactly one of i, j below nocc get
//     (S_ij + lam_j R_ij) / (lam_j - lam_i), all others R_ij / 2;
//   mode 1 (full): pairs with |lam_j - lam_i| > delta get that quotient, the others
//     R_ij / 2 (delta: a device scalar from the caller, the cluster threshold of the
//     paper, so that no host round trip is needed).
__global__ void k_oa_correction(int n, int nocc, int mode, const double* __restrict__ delta_p,
                                const double* __restrict__ S, const double* __restrict__ R, double* __restrict__ E,
                                double* __restrict__ lam_out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * n) return;
  const int i = (int)(idx / n), j = (int)(idx % n);
  const double li = __ldg(S + (long long)i * n + i) / (1.0 - __ldg(R + (long long)i * n + i));
  const double lj = __ldg(S + (long long)j * n + j) / (1.0 - __ldg(R + (long long)j * n + j));
  const double dl = lj - li;
  const double delta = delta_p ? *delta_p : 0.0;
  const double num = __ldg(S + idx) + lj * __ldg(R + idx);
  const bool sep = mode == 0 ? ((i < nocc) != (j < nocc)) : (fabs(dl) > delta);
  E[idx] = sep ? num / dl : 0.5 * __ldg(R + idx);
  if (lam_out && j == 0) lam_out[i] = li;
}

extern "C" int pcg_oa_correction(int n, int nocc, int mode, const double* delta, const double* S, const double* R,
                                 double* E, double* lam, void* stream) {
  if (n < 1 || !S || !R || !E || (mode != 0 && mode != 1)) {
    pcg_set_error("pcg_oa_correction: bad arguments");
    return PCG_ERR_ARG;
  }
  const long long total = (long long)n * n;
  k_oa_correction<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, nocc, mode, delta, S, R, E,
                                                                                    lam);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// ---------------------------------------------------------------------------------
// DIIS.  state[0] = number of vectors stored so far (device int).  The new vector goes
// to slot count % cap; Bm (cap x cap) holds inner products between slots.
// ---------------------------------------------------------------------------------
__global__ void k_diis_store(long long len, int cap, const int* __restrict__ state, const double* __restrict__ F,
                             const double* __restrict__ R, double* __restrict__ focks, double* __restrict__ resids) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= len) return;
  const long long slot = state[0] % cap;
  focks[slot * len + e] = F[e];
  resids[slot * len + e] = R[e];
}

// block j: <resid slot j, R> for the slots in use after this store
__global__ void k_diis_dots(long long len, int cap, const int* __restrict__ state, const double* __restrict__ R,
                            const double* __restrict__ resids, double* __restrict__ row) {
  const int j = blockIdx.x;
  const int used = min(state[0] + 1, cap);
  if (j >= used) return;
  const double* rj = resids + (long long)j * len;
  double s = 0.0;
  for (long long e = threadIdx.x; e < len; e += blockDim.x) s = fma(__ldg(rj + e), __ldg(R + e), s);
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) row[j] = s;
  }
}

#define DIIS_MAXCAP 32
#define DIIS_LD (DIIS_MAXCAP + 3)
// One warp solves the C1 system over m vectors, B(a, b) their residual products with the newest
// first: scaled by the largest diagonal element, Gaussian elimination with partial pivoting
// (lanes over rows for the pivot and the multipliers, over columns for the updates), the
// oldest vector dropped while a pivot is not above eps.  M: (DIIS_MAXCAP + 1) rows of DIIS_LD
// doubles in shared memory; the coefficients come in its last column.  Returns the number of
// vectors kept.  (10 vectors: one thread took 41 us, the warp 20 us.)
template <class Get>
__device__ __forceinline__ int diis_solve(int lane, int m, double eps, double* M, Get B) {
  double scale = 0.0;
  for (int a = lane; a < m; a += 32) scale = fabs(B(a, a));
  for (;; --m) {
    double sc = lane < m ? scale : 0.0;
    for (int o = 16; o > 0; o >>= 1) sc = fmax(sc, __shfl_xor_sync(0xffffffffu, sc, o));
    if (sc <= 0.0) sc = 1.0;
    const int rhs = m + 1;
    for (int a = 0; a <= m; ++a)
      for (int k = lane; k <= rhs; k += 32)
        M[a * DIIS_LD + k] = k == rhs ? (a == m ? -1.0 : 0.0) : a == m ? (k == m ? 0.0 : -1.0) : k == m ? -1.0 : B(a, k) / sc;
    __syncwarp();
    bool singular = false;
    for (int col = 0; col <= m && !singular; ++col) {
      // the largest element at or below the diagonal, the first of equals
      double v = -1.0;
      int piv = col;
      for (int r = col + lane; r <= m; r += 32) {
        const double x = fabs(M[r * DIIS_LD + col]);
        if (x > v || (r == col && !(x <= v))) { v = x; piv = r; }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, v, o);
        const int q = __shfl_xor_sync(0xffffffffu, piv, o);
        if (x > v || (x == v && q < piv)) { v = x; piv = q; }
      }
      piv = __shfl_sync(0xffffffffu, piv, 0);
      const double d = M[piv * DIIS_LD + col];
      if (fabs(d) <= eps) { singular = true; break; }
      __syncwarp();
      if (piv != col)
        for (int k = lane; k <= rhs; k += 32) {
          const double t = M[col * DIIS_LD + k];
          M[col * DIIS_LD + k] = M[piv * DIIS_LD + k];
          M[piv * DIIS_LD + k] = t;
        }
      __syncwarp();
      for (int r = col + 1 + lane; r <= m; r += 32) M[r * DIIS_LD + col] /= d;
      __syncwarp();
      for (int k = col + 1 + lane; k <= rhs; k += 32) {
        const double u = M[col * DIIS_LD + k];
        for (int r = col + 1; r <= m; ++r) M[r * DIIS_LD + k] -= M[r * DIIS_LD + col] * u;
      }
      __syncwarp();
    }
    if (singular && m > 1) continue;
    if (singular) {
      if (lane == 0) M[2] = 1.0;
    } else {
      for (int r = m; r >= 0; --r) {           // back substitution, column by column
        if (lane == 0) M[r * DIIS_LD + rhs] /= M[r * DIIS_LD + r];
        __syncwarp();
        const double c = M[r * DIIS_LD + rhs];
        for (int k = lane; k < r; k += 32) M[k * DIIS_LD + rhs] -= M[k * DIIS_LD + r] * c;
        __syncwarp();
      }
    }
    __syncwarp();
    return m;
  }
}

// fold the new row into Bm, solve over the slots in use, write the coefficient of every slot
// (0 for unused) and advance the count
__global__ void __launch_bounds__(32) k_diis_solve(int cap, int* __restrict__ state, const double* __restrict__ row,
                                                   double* __restrict__ Bm, double* __restrict__ coef) {
  __shared__ double M[(DIIS_MAXCAP + 1) * DIIS_LD];
  const int lane = threadIdx.x, count = state[0], slot = count % cap, used = min(count + 1, cap);
  for (int j = lane; j < used; j += 32) {
    Bm[slot * cap + j] = row[j];
    Bm[j * cap + slot] = row[j];
  }
  for (int j = lane; j < cap; j += 32) coef[j] = 0.0;
  __syncthreads();
  const volatile double* Bv = Bm;
  const int m = diis_solve(lane, used, 1e-14, M, [&](int a, int b) {
    return Bv[((slot - a + cap) % cap) * cap + (slot - b + cap) % cap];
  });
  for (int a = lane; a < m; a += 32) coef[(slot - a + cap) % cap] = M[a * DIIS_LD + m + 1];
  if (lane == 0) state[0] = count + 1;
}

// A warp per molecule of an ensemble: Bnew (mn x mn, oldest first) from Bold (mo x mo) and the
// products `row` of the newest residual with the mo older ones and itself, the oldest
// mo + 1 - mn left out; coef: mn coefficients.
__global__ void __launch_bounds__(128) k_diis_batched(int batch, int mo, int mn, const double* __restrict__ Bold,
                                                      const double* __restrict__ row, long long ldrow,
                                                      double* __restrict__ Bnew, double* __restrict__ coef) {
  __shared__ double Ms[4][(DIIS_MAXCAP + 1) * DIIS_LD];
  const int b = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= batch) return;
  const int cut = mo + 1 - mn;
  const double* Bo = Bold + (size_t)b * mo * mo;
  const double* rw = row + b * ldrow;
  double* Bn = Bnew + (size_t)b * mn * mn;
  auto get = [&](int i, int j) {                // of the mo + 1 vectors, oldest first
    return i == mo ? rw[j] : j == mo ? rw[i] : Bo[i * mo + j];
  };
  for (int e = lane; e < mn * mn; e += 32) Bn[e] = get(e / mn + cut, e % mn + cut);
  double* M = Ms[threadIdx.x >> 5];
  const int m = diis_solve(lane, mn, 0.0, M, [&](int a, int c) { return get(mo - a, mo - c); });
  for (int a = lane; a < mn; a += 32) coef[(size_t)b * mn + mn - 1 - a] = a < m ? M[a * DIIS_LD + m + 1] : 0.0;
}

extern "C" int pcg_diis_batched(int batch, int mo, int mn, const double* Bold, const double* row, long long ldrow,
                                double* Bnew, double* coef, void* stream) {
  if (batch < 0 || mo < 0 || mn < 1 || mn > mo + 1 || mn > DIIS_MAXCAP || ldrow < mo + 1 || (mo > 0 && !Bold) || !row ||
      !Bnew || !coef) {
    pcg_set_error("pcg_diis_batched: bad arguments (1 <= mn <= min(mo + 1, 32))");
    return PCG_ERR_ARG;
  }
  if (batch == 0) return PCG_OK;
  k_diis_batched<<<(batch + 3) / 4, 128, 0, (cudaStream_t)stream>>>(batch, mo, mn, Bold, row, ldrow, Bnew, coef);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

__global__ void k_diis_extrapolate(long long len, int cap, const double* __restrict__ coef,
                                   const double* __restrict__ focks, double* __restrict__ Fx) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= len) return;
  double s = 0.0;
  for (int j = 0; j < cap; ++j) {
    const double cj = coef[j];
    if (cj != 0.0) s = fma(cj, focks[(long long)j * len + e], s);
  }
  Fx[e] = s;
}

extern "C" int pcg_diis_step(long long len, int cap, int* state, const double* F, const double* R, double* focks,
                             double* resids, double* Bm, double* row, double* coef, double* Fx, void* stream) {
  if (len < 1 || cap < 1 || cap > DIIS_MAXCAP || !state || !F || !R || !focks || !resids || !Bm || !row || !coef ||
      !Fx) {
    pcg_set_error("pcg_diis_step: bad arguments (1 <= cap <= 32)");
    return PCG_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned blocks = (unsigned)((len + 255) / 256);
  k_diis_store<<<blocks, 256, 0, s>>>(len, cap, state, F, R, focks, resids);
  k_diis_dots<<<cap, 1024, 0, s>>>(len, cap, state, R, resids, row);
  k_diis_solve<<<1, 32, 0, s>>>(cap, state, row, Bm, coef);
  k_diis_extrapolate<<<blocks, 256, 0, s>>>(len, cap, coef, focks, Fx);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

// ------------------------------------------------------------------------------------
// Closed-shell MP2 energy sums over the transformed integrals X(i,a,j,b) = (ia|jb)
// (Methods/mp2.py:71-94), X stored b-major: X(i,a,j,b) at ((b*o + j)*v + a)*o + i, so
// that both X(i,a,j,b) and its exchange partner X(i,b,j,a) are read along i.
//   s1 = sum X(i,a,j,b)^2 / D,  s2 = sum X(i,a,j,b) X(i,b,j,a) / D,
//   D = e_i + e_j - e_a - e_b.
// Both summands are symmetric under (i,a) <-> (j,b); block p = b*o + j takes the
// pairs q = a*o + i <= p, weight 2 below the diagonal.  1/D: the FP32 reciprocal of
// the denominator formed from FP32 copies of the energies, then one Newton step
// against the FP64 denominator (relative error ~ 1e-13).  part[2p], part[2p+1]: the block's
// s1 and s2 (summed on the host side of the call, in a fixed order).
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_mp2_pair_sums(int o, int v, const double* __restrict__ X,
                                                       const double* __restrict__ eo, const double* __restrict__ ev,
                                                       double* __restrict__ part) {
  extern __shared__ double e_sh[];                 // eo (o), then ev (v); then their FP32 copies
  float* ef = (float*)(e_sh + o + v);
  for (int t = threadIdx.x; t < o + v; t += blockDim.x) {
    const double e = t < o ? eo[t] : ev[t - o];
    e_sh[t] = e;
    ef[t] = (float)e;
  }
  __syncthreads();
  const int p = blockIdx.x, b = p / o, j = p % o;
  const double ejb = e_sh[j] - e_sh[o + b];
  const float fjb = ef[j] - ef[o + b];
  const double* Xp = X + (size_t)p * v * o;                       // X(., ., j, b)
  const int step = blockDim.x, da = step / o, di = step % o;
  int a = threadIdx.x / o, i = threadIdx.x % o;
  double s1 = 0.0, s2 = 0.0;
  // every pair q <= p with weight 1; the block total is 2 * sum - (the q = p term)
  for (int q = threadIdx.x; q <= p; q += step) {
    const double x = Xp[q];
    const double xe = X[((size_t)(a * o + j) * v + b) * o + i];   // X(i, b, j, a)
    const double d = (e_sh[i] - e_sh[o + a]) + ejb;
    // FP32 seed from the FP32 energies, one Newton step against the FP64 denominator
    double r = (double)__frcp_rn((ef[i] - ef[o + a]) + fjb);
    r = fma(r, fma(-d, r, 1.0), r);
    const double t = x * r;
    s1 = fma(x, t, s1);
    s2 = fma(xe, t, s2);
    i += di; a += da;
    if (i >= o) { i -= o; ++a; }
  }
  for (int off = 16; off; off >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    s2 += __shfl_xor_sync(0xffffffffu, s2, off);
  }
  __shared__ double red[2][8];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { red[0][w] = s1; red[1][w] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r1 = 0.0, r2 = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { r1 += red[0][k]; r2 += red[1][k]; }
    const double xd = Xp[p];                       // (jb|jb), its own exchange partner
    const double dg = xd * xd / (2.0 * ejb);
    part[2 * (size_t)p] = 2.0 * r1 - dg;
    part[2 * (size_t)p + 1] = 2.0 * r2 - dg;
  }
}

extern "C" int pcg_mp2_pair_sums(int o, int v, const double* X, const double* eo, const double* ev, double* part,
                                 void* stream) {
  if (o < 1 || v < 1 || !X || !eo || !ev || !part || (long long)o * v > 0x7fffffffLL ||
      (size_t)(o + v) * (sizeof(double) + sizeof(float)) > 200 * 1024) {
    pcg_set_error("pcg_mp2_pair_sums: bad arguments");
    return PCG_ERR_ARG;
  }
  const size_t sh = (size_t)(o + v) * (sizeof(double) + sizeof(float));
  if (sh > 48 * 1024) PCG_CUDA(cudaFuncSetAttribute(k_mp2_pair_sums, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
  k_mp2_pair_sums<<<o * v, 256, sh, (cudaStream_t)stream>>>(o, v, X, eo, ev, part);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
