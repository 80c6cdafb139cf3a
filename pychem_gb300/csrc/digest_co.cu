// Co-density digestion, one class a launch for up to 65,535 densities (see digest.cuh).
#include "digest.cuh"

int pcg_launch_digest_co1(int cls, const DigestArgs& a, unsigned ndens, cudaStream_t s);

int pcg_launch_digest_co(int cls, const DevBasis& b, const DevPairsExt& pr, const int2* tasks, int ntask,
                         const double* store, int nd, const double* W, double* GJ, double* GK, cudaStream_t s) {
  for (int d0 = 0; d0 < nd; d0 += 65535) {
    const DigestArgs a{b, pr, tasks, ntask, 1, store, {W, W}, GJ, {GK, GK}, (unsigned)d0};
    const unsigned k = nd - d0 < 65535 ? nd - d0 : 65535;
    // nothing is kept from a quartet to the next where a thread has one: fewer registers (one density
    // of four waters in cc-pVDZ 1.30 ms; 1.76 in the kernel of runs, 1.58 before there were runs)
    const int rc = digest_run((long long)ntask * k) == 1 ? pcg_launch_digest_co1(cls, a, k, s)
                                                         : launch_digest<2, true>(cls, a, s, k);
    if (rc) return rc;
  }
  return PCG_OK;
}
