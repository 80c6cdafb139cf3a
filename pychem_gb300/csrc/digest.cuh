// Fock digestion kernels (closed shell, unrestricted, co-densities) -- included by digest.cu,
// digest_u.cu, digest_co.cu and digest_co1.cu, one translation unit each so that the class
// instantiations compile in parallel.
//
// For every stored quartet block, with the shell-level degeneracy d = (A!=B ? 2:1)
// (C!=D ? 2:1)(AB!=CD ? 2:1) and v' = d (ab|cd),
//   GJ_ab += D_cd v', GJ_cd += D_ab v',
//   GK_ac -= D_bd v'/4, GK_bd -= D_ac v'/4, GK_ad -= D_bc v'/4, GK_bc -= D_ad v'/4.
// Closed shell (S = 1): GJ = GK = G; the caller's F = H + (G + G^T)/2 equals H + 2J[D] - K[D]
// with D the alpha density -- upstream's H + J[D_a + D_b] - K[D_a] (hartree_fock.py:345-355).
// Unrestricted (S = 2): GJ from (D_a + D_b)/2 and one GK per spin, so that
// F_s = H + sym(GJ + GK_s) = H + J[D_a + D_b] - K[D_s].  Co-densities W of non-orthogonal CI
// (Methods/noci.py:243-300, hartree_fock.py:345-347 for non-symmetric densities) are the
// unrestricted case with D_a = W and D_b = W^T, the D_a exchange blocks written transposed:
// GK then holds G[W^T] + G[W]^T, J[W] = (GJ + GJ^T)/4 and K[W] = -GK/2 with K_ad = sum_bc
// (ab|cd) W_cb; blockIdx.y selects the density.  They are instances of their own (CO): with both
// in one kernel each address was a choice of two ((dd|dd): 39 KB of stack instead of 8), and an
// unrestricted build of C10H22 / cc-pVDZ took 5.80 ms instead of 5.47, of four waters 1.61 instead
// of 1.40.
//
// Bound: the FP64 pipe, six instructions an integral (0.48 ms for the 42 M integrals of
// (H2O)16 / 6-31G), and the load/store queue, which one gather and one reduction a density
// element and quartet fills (1.25 ms).  A thread therefore takes `run` consecutive quartets: lists
// run through the kets (C, D) of one bra in order, so D_ab, D_ac, D_bc are loaded and G_ab,
// G_ac, G_bc written once a run of equal (A, B) and C, and the lanes of a warp touch neighbouring
// columns (run = 1, 2, 4, 8: 1.64, 1.06, 0.92, 1.00 ms).  All factors are powers of two and are
// applied to exponents by integer operations, off the FP64 pipe.
#pragma once
#include "common.cuh"
#include "pcg_internal.h"

struct DigestArgs {
  DevBasis b;
  DevPairsExt pr;
  const int2* tasks;
  int ntask, run;              // quartets, and consecutive quartets per thread
  const double* store;
  const double* D[2];
  double* GJ;
  double* GK[2];
  unsigned d0;                 // first density of the launch
};

// x 2^k, |k| <= 3, by its exponent; zero, infinities and NaNs stay what they are, below 2^-1015
// is zero and from 2^1021 on unscaled.  Selects, no branch: a branch an integral would keep the
// loads of a block from being in flight together (1.6 times the time).
__device__ __forceinline__ double dg_scale(double x, int k) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  const bool small = e < 8u, usual = e - 8u < 0x7f4u;
  return __hiloint2double(small ? 0 : (usual ? hi + (k << 20) : hi), small ? 0 : lo);
}

template <int R, int C>
__device__ __forceinline__ void dg_load(const double* __restrict__ M, int r0, int c0, int n, double (&v)[R][C],
                                        bool tr = false) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) v[i][j] = __ldg(M + (tr ? (size_t)(c0 + j) * n + r0 + i : (size_t)(r0 + i) * n + c0 + j));
}
// M += v 2^k, or -= if neg; clears v
template <int R, int C>
__device__ __forceinline__ void dg_add(double* __restrict__ M, int r0, int c0, int n, int k, bool neg,
                                       double (&v)[R][C], bool tr = false) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const double x = k ? dg_scale(v[i][j], k) : v[i][j];
      atomicAdd(M + (tr ? (size_t)(c0 + j) * n + r0 + i : (size_t)(r0 + i) * n + c0 + j), neg ? -x : x);
      v[i][j] = 0.0;
    }
}

// the quartets of block blk: 128 threads of a.run consecutive ones, or of one (ONE)
template <int NA, int NB, int NC, int ND, int S, bool CO, bool ONE>
__device__ __forceinline__ void digest_block(const DigestArgs& a, unsigned blk) {
  const int run = ONE ? 1 : a.run;
  const long long first = ((long long)blk * blockDim.x + threadIdx.x) * run;
  if (first >= a.ntask) return;
  const int t1 = ONE ? (int)first + 1 : (int)(first + run < a.ntask ? first + run : a.ntask);
  constexpr int JK = S == 2 ? -1 : 0;      // the J density is the sum of both spins: half of it
  const int n = a.b.ld;
  const long long dens = CO ? (long long)(a.d0 + blockIdx.y) * n * n : 0;
  int bra = -1, oa = 0, ob = 0, oc = -1;
  long long o = dens;
  bool sab = false;
  double Jab[NA][NB], gab[NA][NB] = {};
  double Dac[S][NA][NC], Dbc[S][NB][NC], gac[S][NA][NC] = {}, gbc[S][NB][NC] = {};
  auto flush_c = [&]() {
    if (oc < 0) return;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      dg_add(a.GK[s] + o, oa, oc, n, -2, true, gac[s], CO && s == 0);
      dg_add(a.GK[s] + o, ob, oc, n, -2, true, gbc[s], CO && s == 0);
    }
  };
  auto load_j = [&](int r0, int c0, auto& v) {
    dg_load(a.D[0] + o, r0, c0, n, v);
    if constexpr (S == 2) {
      constexpr int R = sizeof(v) / sizeof(v[0]), C = sizeof(v[0]) / sizeof(double);
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) v[i][j] += __ldg(a.D[1] + o + (CO ? (size_t)(c0 + j) * n + r0 + i : (size_t)(r0 + i) * n + c0 + j));
    }
  };
  // the next quartet and its ket (AO of C | (C == D) << 30, AO of D, block offset) are loaded
  // while this one is digested
  int2 next = __ldg(a.tasks + (int)first);
  int4 pn = a.pr.p.ao4 ? __ldg(a.pr.p.ao4 + next.y) : make_int4(0, 0, 0, 0);
  for (int t = (int)first; t < t1; ++t) {
    const int2 tk = next;
    const int4 pk = pn;
    if (t + 1 < t1) {
      next = __ldg(a.tasks + t + 1);
      if (a.pr.p.ao4) pn = __ldg(a.pr.p.ao4 + next.y);
    }
    int c, d;
    bool scd;
    if (a.pr.p.ao4) {
      c = pk.x & 0x3FFFFFFF; d = pk.y; scd = (pk.x >> 30) & 1;
    } else {
      const int C = __ldg(a.pr.p.A + tk.y), Dd = __ldg(a.pr.p.B + tk.y);
      c = __ldg(a.b.sh_ao + C); d = __ldg(a.b.sh_ao + Dd); scd = C == Dd;
    }
    if (tk.x != bra) {
      flush_c();
      if (bra >= 0) dg_add(a.GJ + o, oa, ob, n, JK, false, gab);
      bra = tk.x;
      if (a.pr.p.ao4) {
        const int4 pb = __ldg(a.pr.p.ao4 + bra);
        oa = pb.x & 0x3FFFFFFF; ob = pb.y; sab = (pb.x >> 30) & 1;
        o = dens + ((long long)(unsigned)pb.z | ((long long)pb.w << 32));
      } else {
        const int A = __ldg(a.pr.p.A + bra), B = __ldg(a.pr.p.B + bra);
        o = dens + dev_blk(a.b, A);
        oa = __ldg(a.b.sh_ao + A); ob = __ldg(a.b.sh_ao + B); sab = A == B;
      }
      load_j(oa, ob, Jab);
      oc = -1;
    }
    if (c != oc) {
      flush_c();
      oc = c;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        dg_load(a.D[s] + o, oa, oc, n, Dac[s], CO && s == 1);
        dg_load(a.D[s] + o, ob, oc, n, Dbc[s], CO && s == 1);
      }
    }
    const int deg = !sab + !scd + (tk.x != tk.y);      // log2 of the degeneracy
    double Jcd[NC][ND], gcd[NC][ND] = {};
    double Dad[S][NA][ND], Dbd[S][NB][ND], gad[S][NA][ND] = {}, gbd[S][NB][ND] = {};
    load_j(oc, d, Jcd);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      dg_load(a.D[s] + o, oa, d, n, Dad[s], CO && s == 1);
      dg_load(a.D[s] + o, ob, d, n, Dbd[s], CO && s == 1);
    }
    const double* st = a.store + t;
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int k = 0; k < NC; ++k)
#pragma unroll
          for (int l = 0; l < ND; ++l) {
            const double v = dg_scale(__ldg(st + (size_t)(((i * NB + j) * NC + k) * ND + l) * a.ntask), deg);
            gab[i][j] = fma(Jcd[k][l], v, gab[i][j]);
            gcd[k][l] = fma(Jab[i][j], v, gcd[k][l]);
#pragma unroll
            for (int s = 0; s < S; ++s) {
              gac[s][i][k] = fma(Dbd[s][j][l], v, gac[s][i][k]);
              gbd[s][j][l] = fma(Dac[s][i][k], v, gbd[s][j][l]);
              gad[s][i][l] = fma(Dbc[s][j][k], v, gad[s][i][l]);
              gbc[s][j][k] = fma(Dad[s][i][l], v, gbc[s][j][k]);
            }
          }
    dg_add(a.GJ + o, oc, d, n, JK, false, gcd);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      dg_add(a.GK[s] + o, ob, d, n, -2, true, gbd[s], CO && s == 0);
      dg_add(a.GK[s] + o, oa, d, n, -2, true, gad[s], CO && s == 0);
    }
  }
  flush_c();
  dg_add(a.GJ + o, oa, ob, n, JK, false, gab);
}

template <int NA, int NB, int NC, int ND, int S, bool CO, bool ONE>
__global__ void __launch_bounds__(128) k_digest(const DigestArgs a) {
  digest_block<NA, NB, NC, ND, S, CO, ONE>(a, blockIdx.x);
}

// consecutive quartets per thread: up to 4, fewer where that would leave less than 1,024
// threads an SM, over all densities of the launch (six waters in 6-31G, 15 co-densities: 1.27 ms, 2.02
// one by one; one co-density 0.26 against 0.38 with four)
static inline int digest_run(long long quartets) {
  const long long r = quartets / (152 * 1024);
  return r < 1 ? 1 : (r > 4 ? 4 : (int)r);
}

template <int S, bool CO = false, bool ONE = false>
static int launch_digest(int cls, DigestArgs a, cudaStream_t s, unsigned ndens = 1) {
  if (a.ntask <= 0) return PCG_OK;
  a.run = ONE ? 1 : digest_run((long long)a.ntask * ndens);
  const int threads = 128;
  const unsigned blocks = (unsigned)(((long long)a.ntask + (long long)threads * a.run - 1) / ((long long)threads * a.run));
  switch (cls) {
#define X(id, na, nb, nc, nd) \
  case id: k_digest<na, nb, nc, nd, S, CO, ONE><<<dim3(blocks, ndens), threads, 0, s>>>(a); break;
    PCG_SHAPE_CASES(X)
#undef X
    default: pcg_set_error("digestion: class id out of range"); return PCG_ERR_ARG;
  }
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}
