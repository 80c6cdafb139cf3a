// Closed-shell Fock digestion, one class a launch (see digest.cuh).
#include "digest.cuh"

int pcg_launch_digest_args(int cls, const DigestArgs& a, cudaStream_t s) { return launch_digest<1>(cls, a, s); }

int pcg_launch_digest(int cls, const DevBasis& b, const DevPairsExt& pr, const int2* tasks, int ntask,
                      const double* store, const double* D, double* G, cudaStream_t s) {
  return launch_digest<1>(cls, DigestArgs{b, pr, tasks, ntask, 1, store, {D, nullptr}, G, {G, nullptr}, 0}, s);
}
