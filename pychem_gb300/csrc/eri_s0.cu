// Electron-scattering integral classes 0..13 (see eri_scat.cuh); split for parallel compilation.
#include "eri_scat.cuh"

int pcg_launch_eri_s0(int cls, const DevPairsExt& pr, const BesselTable& bt, const double* fac,
                      const int2* tasks, int ntask, const int* more, double S, double* store,
                      cudaStream_t s) {
  const int threads = 128;
  const EriRange rg = eri_range(ntask, more);
  switch (cls) {
      case 0: k_eri_s<Eri0000><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 1: k_eri_s<Eri1000><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 2: k_eri_s<Eri1010><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 3: k_eri_s<Eri1100><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 4: k_eri_s<Eri1110><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 5: k_eri_s<Eri1111><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 6: k_eri_s<Eri2000><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 7: k_eri_s<Eri2010><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 8: k_eri_s<Eri2011><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 9: k_eri_s<Eri2020><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 10: k_eri_s<Eri2100><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 11: k_eri_s<Eri2110><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 12: k_eri_s<Eri2111><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 13: k_eri_s<Eri2120><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
    default: return PCG_ERR_ARG;
  }
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

__global__ void k_scat_factors(int npp, const double* __restrict__ zeta, const double* __restrict__ K, double S,
                               double* __restrict__ fac) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < npp) fac[i] = scat_factor(zeta[i], K[i], S);
}

int pcg_launch_scattering_factors(int npp, const double* zeta, const double* K, double S, double* fac, cudaStream_t s) {
  if (npp <= 0) return PCG_OK;
  k_scat_factors<<<(npp + 127) / 128, 128, 0, s>>>(npp, zeta, K, S, fac);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
