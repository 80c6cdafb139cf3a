// Coulomb and exchange matrices of many co-densities from the dense integral tensor:
//   J[W]_ab = sum_cd (ab|cd) W_cd,  K[W]_ad = sum_bc (ab|cd) W_cb
// (Methods/hartree_fock.py:345-347, applied by Methods/noci.py:261-318).
//
// With pairs a >= b both are products of packed densities with pair matrices.  J depends on
// W + W^T alone; K of the symmetric part is symmetric and K of the antisymmetric part
// antisymmetric, so
//   J_ab = sum_{c>=d} (ab|cd) (W_cd + W_dc)         (W_cc on the diagonal)
//   S_ad = sum_{b>=c} [(ab|cd) + (ac|bd)] (W_cb + W_bc) / 2    (W_bb / 2 on the diagonal)
//   A_ad = sum_{b>c}  [(ab|cd) - (ac|bd)] (W_cb - W_bc) / 2,   K_ad = S_ad + A_ad, K_da = S_ad - A_ad:
// three nd x np products with np x np matrices, np = n (n + 1) / 2, 3 np^2 FP64 instructions a
// density against 10 an integral (10 np^2 / 2) and 10 or more FP64 atomics a shell quartet's
// element in the digestion.  C2 / cc-pVDZ (n = 28), 756 co-densities: 3.84 ms by digestion.
#include "../../include/pychem_gb300.h"
#include "common.cuh"
#include "pcg_internal.h"

// pair p = a (a + 1) / 2 + b, a >= b
__device__ __forceinline__ void pair_of(int p, int& a, int& b) {
  a = (int)((sqrtf(8.0f * p + 1.0f) - 1.0f) * 0.5f);
  while ((a + 1) * (a + 2) / 2 <= p) ++a;
  while (a * (a + 1) / 2 > p) --a;
  b = p - a * (a + 1) / 2;
}

// the three pair matrices, [row pair][column pair]: (ab|cd), and for row (a, d), column (b, c)
// the symmetric and antisymmetric exchange combinations
__global__ void k_pair_matrices(int n, int np, const double* __restrict__ eri, double* __restrict__ M) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x, row = blockIdx.y;
  if (col >= np) return;
  int a, d, b, c;
  pair_of(row, a, d);
  pair_of(col, b, c);
  const long long N = n, sq = (long long)np * np, o = (long long)row * np + col;
  // rows (a, d), columns (b, c): the Coulomb matrix needs (ad|bc)
  M[o] = eri[((a * N + d) * N + b) * N + c];
  const double x = eri[((a * N + b) * N + c) * N + d], y = eri[((a * N + c) * N + b) * N + d];
  M[sq + o] = x + y;
  M[2 * sq + o] = x - y;
}

// packed densities, [which][density][pair]: W_cd + W_dc (W_cc), and for column (b, c) the same
// and W_cb - W_bc
__global__ void k_pack_densities(int n, int np, int nd, const double* __restrict__ W, double* __restrict__ P) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (p >= np) return;
  int b, c;
  pair_of(p, b, c);
  const double* w = W + (long long)q * n * n;
  const double x = w[c * n + b], y = w[b * n + c];
  const long long len = (long long)nd * np, o = (long long)q * np + p;
  P[o] = P[len + o] = b == c ? x : x + y;
  P[2 * len + o] = x - y;
}

__global__ void k_unpack_jk(int n, int np, int nd, const double* __restrict__ P, double* __restrict__ J,
                            double* __restrict__ K) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (p >= np) return;
  int a, d;
  pair_of(p, a, d);
  const long long len = (long long)nd * np, o = (long long)q * np + p, base = (long long)q * n * n;
  const double j = P[o], s = P[len + o], t = P[2 * len + o];
  J[base + a * n + d] = J[base + d * n + a] = j;
  K[base + a * n + d] = 0.5 * (s + t);
  K[base + d * n + a] = 0.5 * (s - t);
}

extern "C" size_t pcg_coulomb_exchange_workspace(int n, int nd) {
  if (n < 1 || nd < 1) return 0;
  const size_t np = (size_t)n * (n + 1) / 2;
  return (3 * np * np + 6 * (size_t)nd * np) * sizeof(double);
}

extern "C" int pcg_coulomb_exchange(int n, int nd, const double* eri, const double* W, double* J, double* K,
                                    void* workspace, size_t ws_bytes, void* stream) {
  if (n < 1 || n > 255 || nd < 1 || nd > 65535 || !eri || !W || !J || !K) {
    pcg_set_error("pcg_coulomb_exchange: bad arguments (n <= 255, nd <= 65535)");
    return PCG_ERR_ARG;
  }
  if (!workspace || ((size_t)workspace & 7) || ws_bytes < pcg_coulomb_exchange_workspace(n, nd)) {
    pcg_set_error("pcg_coulomb_exchange: workspace missing, misaligned or too small (query pcg_coulomb_exchange_workspace)");
    return PCG_ERR_CAPACITY;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int np = n * (n + 1) / 2;
  const long long sq = (long long)np * np, len = (long long)nd * np;
  double *M = (double*)workspace, *P = M + 3 * sq, *R = P + 3 * len;
  const unsigned bx = (unsigned)((np + 127) / 128);
  k_pair_matrices<<<dim3(bx, np), 128, 0, s>>>(n, np, eri, M);
  k_pack_densities<<<dim3(bx, nd), 128, 0, s>>>(n, np, nd, W, P);
  PCG_CUDA(cudaGetLastError());
  // R[which][density][row] = sum_col P[which][density][col] M[which][row][col]
  if (int rc = pcg_dgemm(3, nd, np, np, 1.0, P, len, np, 1, M, sq, 1, np, 0.0, R, len, np, 1, stream)) return rc;
  k_unpack_jk<<<dim3(bx, nd), 128, 0, s>>>(n, np, nd, R, J, K);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
