// Electron-scattering integral classes 14..17 (see eri_scat.cuh); split for parallel compilation.
#include "eri_scat.cuh"

int pcg_launch_eri_s1(int cls, const DevPairsExt& pr, const BesselTable& bt, const double* fac,
                      const int2* tasks, int ntask, const int* more, double S, double* store,
                      cudaStream_t s) {
  const int threads = 128;
  const EriRange rg = eri_range(ntask, more);
  switch (cls) {
      case 14: k_eri_s<Eri2121><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 15: k_eri_s<Eri2200><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 16: k_eri_s<Eri2210><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
      case 17: k_eri_s<Eri2211><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
    default: return PCG_ERR_ARG;
  }
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
