// ERI class 20, (dd|dd), double precision (see eri_kernels.cuh); its own translation
// unit because it is the largest straight-line kernel.
#include "eri_kernels.cuh"

int pcg_launch_eri_g4(int cls, const DevPairsExt& pr, const PrimTab& pt, const BoysTable& bt, const int2* tasks, int ntask,
                      const int* more, double* store, int precision, cudaStream_t s) {
  const int threads = 128;
  const EriRange rg = eri_range(ntask, more);
  if (cls != 20 || precision != 0) return PCG_ERR_ARG;
  k_eri<Eri2222><<<eri_blocks(rg, threads), threads, 0, s>>>(pr, pt, bt, tasks, rg, store);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
