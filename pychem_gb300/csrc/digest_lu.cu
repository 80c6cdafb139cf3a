// Unrestricted Fock digestion of all lists (see digest_lists.cuh) and the Fock matrices.
#include "digest_lists.cuh"

int pcg_launch_digest_lists_u(int nlist, const int* cls, const int* const* tasks, const int* ntask,
                              const double* const* stores, const DevBasis& b, const DevPairsExt& pr, const double* Da,
                              const double* Db, double* GJ, double* GKa, double* GKb, cudaStream_t s) {
  return launch_digest_lists<2>(nlist, cls, tasks, ntask, stores,
                                DigestArgs{b, pr, nullptr, 0, 1, nullptr, {Da, Db}, GJ, {GKa, GKb}, 0}, s);
}

// F_s = H + (GJ + GK_s + its transpose) / 2 for both spins
__global__ void k_fock_u(int n, const double* __restrict__ H, const double* __restrict__ GJ,
                         const double* __restrict__ GKa, const double* __restrict__ GKb, double* __restrict__ Fa,
                         double* __restrict__ Fb) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n * n) return;
  const size_t tr = (size_t)(idx % n) * n + idx / n;
  const double h = H[idx], j = GJ[idx], jt = GJ[tr];
  Fa[idx] = h + 0.5 * ((j + GKa[idx]) + (jt + GKa[tr]));
  Fb[idx] = h + 0.5 * ((j + GKb[idx]) + (jt + GKb[tr]));
}

int pcg_launch_fock_u(int n, const double* H, const double* GJ, const double* GKa, const double* GKb, double* Fa,
                      double* Fb, cudaStream_t s) {
  if (n <= 0) return PCG_OK;
  k_fock_u<<<(n * n + 127) / 128, 128, 0, s>>>(n, H, GJ, GKa, GKb, Fa, Fb);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
