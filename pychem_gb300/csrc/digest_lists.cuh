// Fock digestion of all quartet lists, one launch for all of them where the quartets are few
// -- included by digest_l.cu and digest_lu.cu.
#pragma once
#include "digest.cuh"

int pcg_launch_digest_args(int cls, const DigestArgs& a, cudaStream_t s);
int pcg_launch_digest_args_u(int cls, const DigestArgs& a, cudaStream_t s);

// Several lists in one launch, each with its blocks [first, next list's first).
#define DIGEST_LISTS 42        // 21 classes, two precision parts
#define DIGEST_SHARED 15       // classes from (dd|ss) on keep their own launches (code size)
struct DigestLists {
  DigestArgs a;                // densities and accumulators; tasks, ntask, store per list
  int nlist;
  unsigned first[DIGEST_LISTS];
  int cls[DIGEST_LISTS], ntask[DIGEST_LISTS];
  const int2* tasks[DIGEST_LISTS];
  const double* store[DIGEST_LISTS];
};

template <int S>
__global__ void __launch_bounds__(128) k_digest_lists(const __grid_constant__ DigestLists ls) {
  int q = 0;
  while (q + 1 < ls.nlist && ls.first[q + 1] <= blockIdx.x) ++q;
  DigestArgs a = ls.a;
  a.tasks = ls.tasks[q];
  a.ntask = ls.ntask[q];
  a.store = ls.store[q];
  const unsigned blk = blockIdx.x - ls.first[q];
  switch (ls.cls[q]) {
#define X(id, na, nb, nc, nd) \
  case id: if constexpr (id < DIGEST_SHARED) digest_block<na, nb, nc, nd, S, false, false>(a, blk); break;
    PCG_SHAPE_CASES(X)
#undef X
  }
}

// Every list.  Few quartets (below 2,000 a SM): one launch for all classes below (dd|ss), largest
// blocks first, one quartet a thread -- the launches of a small molecule would each leave most SMs
// idle and their times, 10 to 40 us, add up.  Otherwise one launch a class: the shared
// kernel has the registers of the largest class, 255 a thread, which costs the common ones
// their occupancy.
template <int S>
static int launch_digest_lists(int nlist, const int* cls, const int* const* tasks, const int* ntask,
                               const double* const* stores, DigestArgs a, cudaStream_t s) {
  long long total = 0;
  for (int q = 0; q < nlist; ++q) total += ntask[q];
  const bool few = total <= 152 * 2000 && nlist <= DIGEST_LISTS;
  for (int q = 0; q < nlist; ++q) {
    if (few && cls[q] < DIGEST_SHARED) continue;
    a.tasks = (const int2*)tasks[q];
    a.ntask = ntask[q];
    a.store = stores[q];
    const int rc = S == 1 ? pcg_launch_digest_args(cls[q], a, s) : pcg_launch_digest_args_u(cls[q], a, s);
    if (rc) return rc;
  }
  if (!few) return PCG_OK;
  DigestLists ls;
  ls.a = a;
  ls.a.run = 1;
  ls.nlist = 0;
  unsigned blocks = 0;
  for (int c = DIGEST_SHARED - 1; c >= 0; --c)          // higher class ids have larger blocks
    for (int q = 0; q < nlist; ++q) {
      if (cls[q] != c || ntask[q] <= 0) continue;
      const int k = ls.nlist++;
      ls.first[k] = blocks;
      ls.cls[k] = c;
      ls.ntask[k] = ntask[q];
      ls.tasks[k] = (const int2*)tasks[q];
      ls.store[k] = stores[q];
      blocks += (unsigned)((ntask[q] + 127) / 128);
    }
  if (!blocks) return PCG_OK;
  k_digest_lists<S><<<blocks, 128, 0, s>>>(ls);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
