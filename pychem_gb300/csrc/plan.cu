// Screened canonical quartet lists (the quartet loop, the Schwarz test Q_ab Q_cd > threshold
// and the always-computed diagonal quartet of Methods/hartree_fock.py:241-312).
//
// Shell pairs are sorted by (kind, molecule, A, B), a kind being a pair class with one
// count of primitive pairs; a bucket is a bra kind with a ket kind <= it, and a row one bra
// pair of a bucket with all its kets: the bra molecule's segment of the ket kind, up to the
// bra itself where the kinds are equal.  Buckets are ordered by (class, decreasing primitive
// quartets a task, bra kind, ket kind), so rows in order fill the class lists in order.  All
// of that depends on the pairs alone and comes as tables; one warp a row counts the kets that
// pass, and after a prefix sum over the rows another pass writes them.  Kets stay in (A, B)
// order inside a row, so that neighbouring tasks of a list share A and read neighbouring
// columns of the density.
//
// Bound: two FP64 instructions (product, comparison) per candidate and pass; 54 M candidates
// of a 16-water cluster are 0.2 ms a pass.  The sort and bisection on 200,000 rows that this
// replaces took 120 launches of tensor operations, 5 ms of host time whatever the size.
#include "../../include/pychem_gb300.h"
#include "common.cuh"
#include "pcg_internal.h"

// FILL = false: cnt[r + 1] (FP64 part) and, mixed, cnt[nrow + r + 1] (FP32 part) = tasks of
// row r.  FILL = true: the tasks themselves, at the offsets off (the prefix sums of cnt).
template <bool FILL>
__global__ void __launch_bounds__(256) k_plan(const pcg_plan_t p, const double* __restrict__ Qs, double thr, double thr32,
                                              long long* __restrict__ cnt, const long long* __restrict__ off,
                                              int2* __restrict__ tasks) {
  const int lane = threadIdx.x & 31;
  const bool mixed = thr32 > 0.0;
  for (long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r < p.nrow; r += (long long)gridDim.x * 8) {
    int lo = 0, hi = p.nbucket - 1;    // the bucket: last b with row0[b] <= r
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(p.row0 + mid) <= r) lo = mid; else hi = mid - 1;
    }
    const int kb = __ldg(p.bra_kind + lo), kk = __ldg(p.ket_kind + lo);
    const int pos = __ldg(p.kind0 + kb) + (int)(r - __ldg(p.row0 + lo));
    const int* seg = p.seg0 + (long long)kk * p.nmol + __ldg(p.mol + pos);
    const int first = __ldg(seg), last = kk == kb ? pos + 1 : __ldg(seg + 1);
    const int bra = __ldg(p.order + pos);
    const double qb = __ldg(Qs + pos);
    long long n64 = 0, n32 = 0;
    const long long o64 = FILL ? off[r] : 0, o32 = FILL && mixed ? off[p.nrow + r] : 0;
    for (int base = first; base < last; base += 32) {
      const int q = base + lane;
      bool in64 = false, in32 = false;
      if (q < last) {
        const double b = qb * __ldg(Qs + q);
        const bool pass = b > thr;
        in64 = pass ? !mixed || b > thr32 : (kk == kb && q == pos);
        in32 = pass && !in64;
      }
      const unsigned m64 = __ballot_sync(0xffffffffu, in64), m32 = __ballot_sync(0xffffffffu, in32);
      if (FILL) {
        const unsigned below = (1u << lane) - 1u;
        if (in64) tasks[o64 + n64 + __popc(m64 & below)] = make_int2(bra, __ldg(p.order + q));
        if (in32) tasks[o32 + n32 + __popc(m32 & below)] = make_int2(bra, __ldg(p.order + q));
      }
      n64 += __popc(m64);
      n32 += __popc(m32);
    }
    if (!FILL && lane == 0) {
      cnt[r + 1] = n64;
      if (mixed) cnt[p.nrow + r + 1] = n32;
      if (r == 0) cnt[0] = 0;
    }
  }
}

static int plan_check(const pcg_plan_t* p, const double* Qs, const char* msg) {
  if (!p || !Qs || p->nrow < 1 || p->nbucket < 1 || p->nmol < 1 || !p->row0 || !p->bra_kind || !p->ket_kind || !p->kind0 ||
      !p->seg0 || !p->order || !p->mol) {
    pcg_set_error(msg);
    return PCG_ERR_ARG;
  }
  return PCG_OK;
}

static unsigned plan_blocks(long long nrow) {
  const long long b = (nrow + 7) / 8;
  return (unsigned)(b < 152LL * 64 ? b : 152LL * 64);
}

extern "C" int pcg_plan_count(const pcg_plan_t* plan, const double* Qs, double thr, double thr32, long long* cnt,
                              void* stream) {
  if (int rc = plan_check(plan, Qs, "pcg_plan_count: bad arguments")) return rc;
  if (!cnt) { pcg_set_error("pcg_plan_count: no output"); return PCG_ERR_ARG; }
  k_plan<false><<<plan_blocks(plan->nrow), 256, 0, (cudaStream_t)stream>>>(*plan, Qs, thr, thr32, cnt, nullptr, nullptr);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_plan_fill(const pcg_plan_t* plan, const double* Qs, double thr, double thr32, const long long* off,
                             int* tasks, void* stream) {
  if (int rc = plan_check(plan, Qs, "pcg_plan_fill: bad arguments")) return rc;
  if (!off || !tasks) { pcg_set_error("pcg_plan_fill: no offsets or output"); return PCG_ERR_ARG; }
  k_plan<true><<<plan_blocks(plan->nrow), 256, 0, (cudaStream_t)stream>>>(*plan, Qs, thr, thr32, nullptr, off, (int2*)tasks);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
