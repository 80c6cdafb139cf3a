// Co-density digestion, one quartet a thread (see digest.cuh, digest_co.cu).
#include "digest.cuh"

int pcg_launch_digest_co1(int cls, const DigestArgs& a, unsigned ndens, cudaStream_t s) {
  return launch_digest<2, true, true>(cls, a, s, ndens);
}
