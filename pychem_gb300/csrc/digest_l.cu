// Closed-shell Fock digestion of all lists (see digest_lists.cuh).
#include "digest_lists.cuh"

int pcg_launch_digest_lists(int nlist, const int* cls, const int* const* tasks, const int* ntask,
                            const double* const* stores, const DevBasis& b, const DevPairsExt& pr, const double* D,
                            double* G, cudaStream_t s) {
  return launch_digest_lists<1>(nlist, cls, tasks, ntask, stores,
                                DigestArgs{b, pr, nullptr, 0, 1, nullptr, {D, nullptr}, G, {G, nullptr}, 0}, s);
}
