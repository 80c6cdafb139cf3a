// FP64-accurate GEMM on the tcgen05 tensor cores, every Ozaki level in one kernel.
//
//   C[m*sCm + n*sCn] (+)= sum_k X[m*ldx + k] * Y[k*sYk + n*sYn]      (all FP64)
//
// The scheme is the one of ozaki.cu (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, Numer.
// Algorithms 59 (2012) 95-118): each row of X and column of Y gets a power-of-two
// scale and NS signed 7-bit digits (exact in BF16); products of digit slices are exact
// integers in FP32; the level sums P_L = sum_{p+q=L} X_p Y_q are combined exactly in
// int64.  What this kernel changes is where the work happens:
//
//  * X, the large operand (millions of rows in the MP2 transforms), is read once as
//    FP64 from global memory and split on the fly: sixteen producer warps load a 128-row
//    by 32-column chunk, cut it into NS digit slices and store them BF16, K-major and
//    64-byte swizzled, straight into the shared-memory operand tiles (no BF16 copy of
//    X in global memory).  The exponent of each row comes from a first pass over the
//    tile's rows, column by column beside the chunks of the tile before (the re-read is
//    served by L2; as a pass of its own it was a third of the time).
//  * Y, the small operand (C_occ or C_vir: a few hundred columns), is split once by
//    k_ozt_split_y into K-major BF16 slices in the caller's workspace (slice-major,
//    [p][n][k]) and brought into shared memory tile by tile by the tensor memory
//    accelerator (cp.async.bulk.tensor, 64-byte swizzle, completion counted on the
//    stage's mbarrier).
//  * One warp issues tcgen05.mma (M = 128, N = BN, K = 16, BF16 in, FP32 out) for
//    every slice pair with p + q <= NS + 1 into NS accumulators in tensor memory, one
//    per level (NS * BN <= 512 columns), over a two-stage mbarrier pipeline.
//  * Eight epilogue warps then read the level accumulators (tcgen05.ld), combine them in
//    int64, scale by 2^{eX + eY} and write FP64 C with any strides (sCm = 1 gives
//    coalesced stores of the transposed product, which is how the MP2 transforms chain).
//
// Level sums are exact while K (NS + 2) < 4096.  Every mbarrier wait is bounded; a CTA
// that gives up sets the error flag in the workspace, drains its MMAs, frees its
// tensor memory and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <stdio.h>

#include "../../include/pychem_gb300.h"
#include "common.cuh"
#include "ozaki_common.cuh"
#include "pcg_internal.h"
#include "umma.cuh"

#define OZT_BM 128
#define OZT_BK 32
#define OZT_PROD_WARPS 16
#define OZT_PROD (OZT_PROD_WARPS * 32)
#define OZT_EPI 256                          // threads of the epilogue warps
#define OZT_THREADS (OZT_PROD + 32 + OZT_EPI)
#define OZT_WAIT (1u << 24)

template <int NS, int BN>
struct OztCfg {
  static constexpr int XT = OZT_BM * OZT_BK * 2;  // one X slice tile (bytes)
  static constexpr int YT = BN * OZT_BK * 2;      // one Y slice tile
  static constexpr int STAGE = NS * (XT + YT);
  static constexpr int SMEM = 2 * STAGE + 1024 + 2304;  // two stages, alignment slack, barriers and exponents
  static_assert(NS * BN <= 512, "level accumulators exceed tensor memory");
  static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256, "MMA N");
  static_assert(YT % 512 == 0, "Y tiles must stay 512-byte aligned");
};

struct OztWs {  // workspace header (device): error flag, then exponents of Y and its slices
  int err;
};

// Y slices: ys[(p * Npad + n) * Kp + k] (BF16, zero for k >= K and n >= N), ey[n]: one
// warp per column n, lanes over k.
template <int NS>
__global__ void k_ozt_split_y(const double* __restrict__ Y, long long sYk, long long sYn, int K, int N, int Npad,
                              int Kp, __nv_bfloat16* __restrict__ ys, int* __restrict__ ey) {
  const int n = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (n >= Npad) return;
  __nv_bfloat16* out = ys + (size_t)n * Kp;
  const size_t pstride = (size_t)Npad * Kp;
  if (n >= N) {
    for (int i = lane; i < NS * Kp; i += 32) out[(i / Kp) * pstride + i % Kp] = __float2bfloat16(0.0f);
    if (lane == 0) ey[n] = 0;
    return;
  }
  unsigned long long mx = 0;
  for (int k = lane; k < K; k += 32) mx = max(mx, oz_absbits(__ldg(Y + k * sYk + n * sYn)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int emax = (int)(mx >> 52);
  if (lane == 0) ey[n] = emax ? emax - 1022 : 0;
  for (int k = lane; k < Kp; k += 32) {
    int d[NS];
    if (k < K) {
      oz_digits<NS>(__ldg(Y + k * sYk + n * sYn), emax, d);
    } else {
#pragma unroll
      for (int p = 0; p < NS; ++p) d[p] = 0;
    }
#pragma unroll
    for (int p = 0; p < NS; ++p) out[p * pstride + k] = __int2bfloat16_rn(d[p]);
  }
}

// the 8 consecutive FP64 values of row m from column kb (zero outside [0, K) or m >= M)
__device__ __forceinline__ void ozt_load8(const double* __restrict__ X, long long ldx, long long m, long long M, int kb,
                                          int K, bool vec, double (&v)[8]) {
  if (m < M && vec && kb + 8 <= K) {
    const double2* src = (const double2*)(X + m * ldx + kb);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const double2 q = __ldg(src + h);
      v[2 * h] = q.x;
      v[2 * h + 1] = q.y;
    }
  } else if (m < M) {
    const double* src = X + m * ldx + kb;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (kb + j < K) ? __ldg(src + j) : 0.0;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.0;
  }
}

// the high words of the same values
__device__ __forceinline__ void ozt_load_hi8(const double* __restrict__ X, long long ldx, long long m, long long M, int kb,
                                             int K, unsigned (&h)[8]) {
  const unsigned* src = (const unsigned*)(X + m * ldx + kb) + 1;
#pragma unroll
  for (int j = 0; j < 8; ++j) h[j] = (m < M && kb + j < K) ? __ldg(src + 2 * j) : 0u;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// One CTA an SM works through the row tiles blockIdx.x, + gridDim.x, ...: the producers go on to
// the next tile's exponents and digits while the tensor core finishes a tile and eight epilogue
// warps read its accumulators; the next tile's first MMA waits for them (the levels fill tensor
// memory, so there is one set).  With a CTA a tile each of these phases was exposed, with the
// launch and the tensor-memory allocation: 22 us a 128-row tile of K = 104 (2.4 us of MMAs).
template <int NS, int BN>
__global__ void __launch_bounds__(OZT_THREADS, 1)
    k_ozt_gemm(long long M, int N, int K, int Kp, int Npad, const double* __restrict__ X, long long ldx,
               const __grid_constant__ CUtensorMap ymap, const int* __restrict__ ey, double* __restrict__ C,
               long long sCm, long long sCn, int accumulate, int* __restrict__ err) {
  using Cfg = OztCfg<NS, BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = sm;                                        // [stage][X slices | Y slices]
  uint64_t* bars = (uint64_t*)(sm + 2 * Cfg::STAGE);  // full[2], empty[2], acc full, drain, ycopy[2], acc empty
  uint32_t* tmem_slot = (uint32_t*)(bars + 9);
  volatile int* abort_s = (volatile int*)(tmem_slot + 1);
  // exponent fields of a tile's 128 rows.  Four sets: while the epilogue of tile i reads its
  // own, two stages let the producers start tile i + 3 at most
  int* ex_s = (int*)(tmem_slot + 6);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  // the N tiles of one row tile are adjacent (they share its X rows in L2)
  const int ntn = (N + BN - 1) / BN;
  const long long ntile = (M + OZT_BM - 1) / OZT_BM * ntn;
  const int nchunk = Kp / OZT_BK;

  if (threadIdx.x == 0) {
    // full: one arrival a producer warp (512 on one barrier are 512 turns at its address); ycopy: the expect_tx arrival of the thread that issues
    // the Y copies, completed by their bytes
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars[i], OZT_PROD_WARPS);
      mbar_init(&bars[2 + i], 1);
      mbar_init(&bars[6 + i], 1);
    }
    mbar_init(&bars[4], 2);
    mbar_init(&bars[5], 1);
    mbar_init(&bars[8], OZT_EPI / 32);
    *abort_s = 0;
    mbar_fence_init();
  }
  if (warp == OZT_PROD_WARPS) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < OZT_PROD_WARPS) {
    const int t = threadIdx.x;
    const bool vec = (ldx % 2 == 0) && (((uintptr_t)X & 15) == 0);
    // this thread's 8-column item of every chunk: row r, column group g
    const int g = t & 3, r = t >> 2;
    const uint32_t off = sw64_offset(r, g);
    bool ok = true;
    int ycopies[2] = {0, 0};  // Y copies issued per stage (thread 0)
    unsigned cc = 0;          // chunks so far
    int set = 0;
    // largest high word of this thread's items; a row's four threads are neighbours
    unsigned mx = 0;
    {
      const long long m = (long long)blockIdx.x / ntn * OZT_BM + r;
      for (int c = 0; c < nchunk; ++c) {
        unsigned h[8];
        ozt_load_hi8(X, ldx, m, M, c * OZT_BK + 8 * g, K, h);
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = max(mx, h[j] & 0x7fffffffu);
      }
    }
    for (long long tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x, set = (set + 1) & 3) {
      const long long m0 = tile / ntn * OZT_BM;
      const int n0 = (int)(tile % ntn) * BN;
      const bool more = tile + gridDim.x < ntile;
      const long long mnext = (tile + gridDim.x) / ntn * OZT_BM + r;
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const int emax = (int)(mx >> 20);
      if (g == 0) ex_s[set * OZT_BM + r] = emax;
      mx = 0;
      double v[8], nv[8];
      ozt_load8(X, ldx, m0 + r, M, 8 * g, K, vec, nv);
      for (int c = 0; c < nchunk; ++c, ++cc) {
        const int st = cc & 1;
        const int k0 = c * OZT_BK;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = nv[j];
        // while this chunk is split: the next one's values, and the same columns of the next
        // tile for its exponents (which also brings the tile to L2)
        if (c + 1 < nchunk) ozt_load8(X, ldx, m0 + r, M, k0 + OZT_BK + 8 * g, K, vec, nv);
        unsigned h[8];
        if (more) ozt_load_hi8(X, ldx, mnext, M, k0 + 8 * g, K, h);
        if (cc >= 2 && !mbar_wait(&bars[2 + st], ((cc >> 1) + 1) & 1, OZT_WAIT, abort_s)) ok = false;
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        uint8_t* xt = tiles + st * Cfg::STAGE;
        uint8_t* yt = xt + NS * Cfg::XT;
        if (t == 0) {  // Y slices of this chunk by TMA
          ++ycopies[st];
          mbar_arrive_expect_tx(&bars[6 + st], NS * Cfg::YT);
#pragma unroll 1
          for (int p = 0; p < NS; ++p) tma_load_2d(smem_u32(yt + p * Cfg::YT), &ymap, k0, p * Npad + n0, &bars[6 + st]);
        }
        unsigned w[4][NS];
#pragma unroll
        for (int hh = 0; hh < 4; ++hh) oz_digits_bf16x2<NS>(v[2 * hh], v[2 * hh + 1], emax, w[hh]);
#pragma unroll
        for (int p = 0; p < NS; ++p)
          *(uint4*)(xt + p * Cfg::XT + off) = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[st]);
        if (more) {
#pragma unroll
          for (int j = 0; j < 8; ++j) mx = max(mx, h[j] & 0x7fffffffu);
        }
      }
    }
    if (!ok) { *abort_s = 1; atomicExch(err, 1); }
    // the last copies land before the CTA exits: the MMA warp has waited for them unless a
    // wait gave up
    if (t == 0 && *abort_s) {
      volatile int keep_waiting = 0;
      for (int i = 0; i < 2; ++i)
        if (ycopies[i]) mbar_wait(&bars[6 + i], (ycopies[i] - 1) & 1, OZT_WAIT, &keep_waiting);
    }
  } else if (warp == OZT_PROD_WARPS) {
    // ---- MMA issuer: the whole warp keeps in step, its leading lane issues
    const uint32_t idesc = idesc_bf16_f32(OZT_BM, BN);
    const uint32_t lead = elect_one();
    const uint64_t xd0 = sdesc_k_sw64(smem_u32(tiles));
    bool ok = true;
    unsigned cc = 0, it = 0;
    for (long long tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x, ++it) {
      if (it && !mbar_wait(&bars[8], (it - 1) & 1, OZT_WAIT, abort_s)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      for (int c = 0; c < nchunk && ok; ++c, ++cc) {
        const int st = cc & 1;
        ok = mbar_wait(&bars[st], (cc >> 1) & 1, OZT_WAIT, abort_s) &&
             mbar_wait(&bars[6 + st], (cc >> 1) & 1, OZT_WAIT, abort_s);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        // descriptors count 16-byte units in their low bits
        const uint64_t xd = xd0 + (uint64_t)(st * (Cfg::STAGE >> 4));
        const uint64_t yd = xd + (NS * Cfg::XT >> 4);
#pragma unroll
        for (int kk = 0; kk < OZT_BK / 16; ++kk) {
#pragma unroll
          for (int p = 0; p < NS; ++p)
#pragma unroll
            for (int q = 0; q < NS - p; ++q)      // level L = p + q is first reached with p = 0
              umma_bf16_lead(lead, tmem + (p + q) * BN, xd + ((p * Cfg::XT + kk * 32) >> 4),
                             yd + ((q * Cfg::YT + kk * 32) >> 4), idesc, (c | kk | p) != 0);
        }
        umma_commit_lead(lead, &bars[2 + st]);
      }
      if (ok) {
        umma_commit_lead(lead, &bars[4]);
        if (lead) mbar_arrive(&bars[4]);      // and the producers' exponents, seen by this thread
      }
      __syncwarp();
    }
    if (!ok) {
      *abort_s = 1;
      if (lead) atomicExch(err, 2);
      umma_commit_lead(lead, &bars[5]);  // drain what was issued before freeing tensor memory
      volatile int keep_waiting = 0;
      mbar_wait(&bars[5], 0, OZT_WAIT, &keep_waiting);
      __syncwarp();
    }
  } else {
    // ---- epilogue: wait for a tile's last MMAs, combine the levels, write C
    const int lg = warp & 3, half = (warp - OZT_PROD_WARPS - 1) >> 2;
    const int re = 32 * lg + lane;
    const uint32_t trow = tmem + ((uint32_t)(32 * lg) << 16);
    unsigned it = 0;
    for (long long tile = blockIdx.x; tile < ntile; tile += gridDim.x, ++it) {
      const long long m = tile / ntn * OZT_BM + re;
      const int n0 = (int)(tile % ntn) * BN;
      if (!warp_all(mbar_wait(&bars[4], it & 1, OZT_WAIT, abort_s))) {
        *abort_s = 1;
        atomicExch(err, 1);
        break;
      }
      tc_fence_after();
      const int eme = ex_s[(it & 3) * OZT_BM + re];
      const int ex = (eme ? eme - 1022 : 0) - OZ_BETA * (NS + 1);
#pragma unroll 1
      for (int cb = 8 * half; cb < BN; cb += 16) {
        float P[NS][8];
        __syncwarp();                  // the loads want every lane, also those past the last row
#pragma unroll
        for (int L = 0; L < NS; ++L) tmem_ld8(trow + L * BN + cb, P[L]);
        tmem_wait_ld();
        if (cb + 16 >= BN) {           // the last reads: the next tile may overwrite
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[8]);
        }
        if (m < M) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int n = n0 + cb + j;
            if (n >= N) break;
            // sum of P_L 2^{7 (NS - 1 - L)}: three levels at a time by 32 x 32 + 64-bit
            // multiply-adds
            long long hi = 0, acc = 0;
#pragma unroll
            for (int L = 0; L < NS; ++L) {
              const int q = __float2int_rn(P[L][j]);
              if (L < NS - 3) hi = (long long)q * (1 << (OZ_BETA * (NS - 4 - L))) + hi;
              else acc = (long long)q * (1 << (OZ_BETA * (NS - 1 - L))) + acc;
            }
            acc += hi << (3 * OZ_BETA);
            const double val = oz_ll_scaled(acc, ex + __ldg(ey + n));
            double* cp = C + m * sCm + (long long)n * sCn;
            *cp = accumulate ? *cp + val : val;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == OZT_PROD_WARPS) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------
static size_t al256(size_t x) { return (x + 255) / 256 * 256; }

struct OztLayout {
  int BN, Kp, Npad;
  size_t off_ey, off_ys, total;
};

static int ozt_bn(int nslice, int N) {
  if (nslice == 6) return N <= 64 ? 64 : (N <= 80 ? 80 : (N % 80 == 0 || N % 64 != 0 ? 80 : 64));
  return 64;
}

static OztLayout ozt_layout(int N, int K, int nslice) {
  OztLayout L;
  L.BN = ozt_bn(nslice, N);
  L.Kp = (K + OZT_BK - 1) / OZT_BK * OZT_BK;
  L.Npad = (N + L.BN - 1) / L.BN * L.BN;
  L.off_ey = 256;
  L.off_ys = al256(L.off_ey + (size_t)L.Npad * 4);
  L.total = al256(L.off_ys + (size_t)L.Npad * nslice * L.Kp * 2);
  return L;
}

typedef CUresult (*PcgEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int get_encode_tiled(PcgEncodeTiled* fn) {
  static PcgEncodeTiled cached = nullptr;
  if (!cached) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p) {
      pcg_set_error("cuTensorMapEncodeTiled not available from the driver");
      return PCG_ERR_CUDA;
    }
    cached = (PcgEncodeTiled)p;
  }
  *fn = cached;
  return PCG_OK;
}

template <int NS, int BN>
static int ozt_run(long long M, int N, int K, const double* X, long long ldx, const double* Y, long long sYk, long long sYn,
                   double* C, long long sCm, long long sCn, int accumulate, char* ws, const OztLayout& L,
                   cudaStream_t s) {
  using Cfg = OztCfg<NS, BN>;
  int* err = (int*)ws;
  int* ey = (int*)(ws + L.off_ey);
  __nv_bfloat16* ys = (__nv_bfloat16*)(ws + L.off_ys);
  k_ozt_split_y<NS><<<(L.Npad + 7) / 8, 256, 0, s>>>(Y, sYk, sYn, K, N, L.Npad, L.Kp, ys, ey);
  PCG_CUDA(cudaGetLastError());
  // Y slices as a 2-D tensor [NS * Npad rows][Kp columns] of BF16; boxes of 32 columns
  // (64 bytes, the swizzle span) by BN rows; k0 is a multiple of 32, so every copy
  // starts on a 64-byte boundary
  PcgEncodeTiled encode;
  if (int rc = get_encode_tiled(&encode)) return rc;
  CUtensorMap ymap;
  const cuuint64_t gdim[2] = {(cuuint64_t)L.Kp, (cuuint64_t)NS * L.Npad};
  const cuuint64_t gstride[1] = {(cuuint64_t)L.Kp * 2};
  const cuuint32_t box[2] = {OZT_BK, BN};
  const cuuint32_t estr[2] = {1, 1};
  if (encode(&ymap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)ys, gdim, gstride, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
    pcg_set_error("pcg_ozaki_gemm_tc: cuTensorMapEncodeTiled rejected the Y slice layout");
    return PCG_ERR_CUDA;
  }
  static bool attr_set[64];
  int dev = 0;
  PCG_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    PCG_CUDA(cudaFuncSetAttribute(k_ozt_gemm<NS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM));
    attr_set[dev] = true;
  }
  int sms = 0;
  PCG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const long long tiles = (long long)(L.Npad / BN) * ((M + OZT_BM - 1) / OZT_BM);
  const long long blocks = tiles < sms ? tiles : sms;
  k_ozt_gemm<NS, BN><<<(unsigned)blocks, OZT_THREADS, Cfg::SMEM, s>>>(M, N, K, L.Kp, L.Npad, X, ldx, ymap, ey, C, sCm,
                                                                    sCn, accumulate, err);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" size_t pcg_ozaki_tc_workspace(int N, int K, int nslice) {
  if (N < 1 || K < 1 || (nslice != 6 && nslice != 7)) return 0;
  return ozt_layout(N, K, nslice).total;
}

extern "C" int pcg_ozaki_gemm_tc(long long M, int N, int K, const double* X, long long ldx, const double* Y, long long sYk,
                                 long long sYn, double* C, long long sCm, long long sCn, int nslice, int accumulate,
                                 void* workspace, size_t ws_bytes, void* stream) {
  if (M < 1 || N < 1 || K < 1 || !X || !Y || !C || ldx < K) {
    pcg_set_error("pcg_ozaki_gemm_tc: bad arguments");
    return PCG_ERR_ARG;
  }
  if (nslice != 6 && nslice != 7) {
    pcg_set_error("pcg_ozaki_gemm_tc: nslice must be 6 or 7");
    return PCG_ERR_UNSUPPORTED;
  }
  if ((long long)K * (nslice + 2) >= 4096) {
    pcg_set_error("pcg_ozaki_gemm_tc: K too large for exact FP32 level sums (need K * (nslice + 2) < 4096)");
    return PCG_ERR_UNSUPPORTED;
  }
  const OztLayout L = ozt_layout(N, K, nslice);
  if ((M + OZT_BM - 1) / OZT_BM * (long long)(L.Npad / L.BN) >= (1ll << 31)) {
    pcg_set_error("pcg_ozaki_gemm_tc: M too large for one launch");
    return PCG_ERR_UNSUPPORTED;
  }
  if (!workspace || ws_bytes < L.total || ((size_t)workspace & 255)) {
    pcg_set_error("pcg_ozaki_gemm_tc: workspace missing, too small or not 256-byte aligned (query pcg_ozaki_tc_workspace)");
    return PCG_ERR_CAPACITY;
  }
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  PCG_CUDA(cudaMemsetAsync(ws, 0, 4, s));
  if (nslice == 7) return ozt_run<7, 64>(M, N, K, X, ldx, Y, sYk, sYn, C, sCm, sCn, accumulate, ws, L, s);
  if (L.BN == 80) return ozt_run<6, 80>(M, N, K, X, ldx, Y, sYk, sYn, C, sCm, sCn, accumulate, ws, L, s);
  return ozt_run<6, 64>(M, N, K, X, ldx, Y, sYk, sYn, C, sCm, sCn, accumulate, ws, L, s);
}

// Error flag of the last pcg_ozaki_gemm_tc call that used this workspace (0: no CTA
// gave up on a wait); synchronises the stream.
extern "C" int pcg_ozaki_tc_status(const void* workspace, void* stream) {
  int h = 0;
  PCG_CUDA(cudaMemcpyAsync(&h, workspace, 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  PCG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  return h;
}
