// Unrestricted Fock digestion, one class a launch (see digest.cuh).
#include "digest.cuh"

int pcg_launch_digest_args_u(int cls, const DigestArgs& a, cudaStream_t s) { return launch_digest<2>(cls, a, s); }

int pcg_launch_digest_u(int cls, const DevBasis& b, const DevPairsExt& pr, const int2* tasks, int ntask,
                        const double* store, const double* Da, const double* Db, double* GJ, double* GKa,
                        double* GKb, cudaStream_t s) {
  return launch_digest<2>(cls, DigestArgs{b, pr, tasks, ntask, 1, store, {Da, Db}, GJ, {GKa, GKb}, 0}, s);
}
