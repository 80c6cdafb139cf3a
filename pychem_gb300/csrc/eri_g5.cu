// ERI class 20, (dd|dd), single precision (see eri_kernels.cuh).
#include "eri_kernels.cuh"

int pcg_launch_eri_g5(int cls, const DevPairsExt& pr, const PrimTab& pt, const BoysTable& bt, const int2* tasks, int ntask,
                      const int* more, double* store, int precision, cudaStream_t s) {
  (void)more;
  (void)pt;
  const int threads = 128, blocks = (ntask + threads - 1) / threads;
  if (cls != 20 || precision == 0) return PCG_ERR_ARG;
  k_eri_f<Eri2222f><<<blocks, threads, 0, s>>>(pr, bt, tasks, ntask, store);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
