// Co-density digestion, one class a launch for up to 65,535 densities (see digest.cuh).
#include "digest.cuh"

int pcg_launch_digest_co(int cls, const DevBasis& b, const DevPairsExt& pr, const int2* tasks, int ntask,
                         const double* store, int nd, const double* W, double* GJ, double* GK, cudaStream_t s) {
  for (int d0 = 0; d0 < nd; d0 += 65535) {
    const DigestArgs a{b, pr, tasks, ntask, 1, store, {W, W}, GJ, {GK, GK}, (unsigned)d0};
    if (int rc = launch_digest<2, true>(cls, a, s, nd - d0 < 65535 ? nd - d0 : 65535)) return rc;
  }
  return PCG_OK;
}
