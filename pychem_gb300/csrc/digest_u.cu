// Unrestricted Fock digestion and co-density digestion, one class a launch (see digest.cuh).
#include "digest.cuh"

int pcg_launch_digest_args_u(int cls, const DigestArgs& a, cudaStream_t s) { return launch_digest<2>(cls, a, s); }

int pcg_launch_digest_u(int cls, const DevBasis& b, const DevPairsExt& pr, const int2* tasks, int ntask,
                        const double* store, const double* Da, const double* Db, double* GJ, double* GKa,
                        double* GKb, cudaStream_t s) {
  return launch_digest<2>(cls, DigestArgs{b, pr, tasks, ntask, 1, store, {Da, Db}, GJ, {GKa, GKb}, false, 0}, s);
}

int pcg_launch_digest_co(int cls, const DevBasis& b, const DevPairsExt& pr, const int2* tasks, int ntask,
                         const double* store, int nd, const double* W, double* GJ, double* GK, cudaStream_t s) {
  for (int d0 = 0; d0 < nd; d0 += 65535) {
    DigestArgs a{b, pr, tasks, ntask, 1, store, {W, W}, GJ, {GK, GK}, true, (unsigned)d0};
    if (int rc = launch_digest<2>(cls, a, s, nd - d0 < 65535 ? nd - d0 : 65535)) return rc;
  }
  return PCG_OK;
}
