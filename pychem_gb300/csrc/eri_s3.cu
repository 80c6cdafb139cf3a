// Electron-scattering integral classes 20 (see eri_scat.cuh); split for parallel compilation.
#include "eri_scat.cuh"

int pcg_launch_eri_s3(int cls, const DevPairsExt& pr, const BesselTable& bt, const double* fac,
                      const int2* tasks, int ntask, const int* more, double S, double* store,
                      cudaStream_t s) {
  const int threads = 128;
  const EriRange rg = eri_range(ntask, more);
  switch (cls) {
      case 20: k_eri_s<Eri2222><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, bt, fac, tasks, rg, S, store); break;
    default: return PCG_ERR_ARG;
  }
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
