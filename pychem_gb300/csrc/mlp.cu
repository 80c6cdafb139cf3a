// Kernels of the learned initial-guess network: dense layers with BF16 weights and
// FP32 accumulation, SiLU activation, masked squared-error loss and Adam.
//
// One tensor-core GEMM (tcgen05) serves the forward pass and both backward products:
//   C[m][n] (+)= sum_k A(m, k) B(k, n),  A(m, k) = A[m*sam + k*sak] (FP32),
//   B(k, n) = B[k*sbk + n*sbn] (FP32 or BF16), C row-major with ldc.
// FP32 operands keep all their bits: x = x0 + x1 + x2 with BF16 terms of 8 bits each (the
// top 16 bits of x, of what is left, and the rest), so a product with a BF16 weight is three
// exact BF16 products and one of two FP32 operands the eight with p + q <= 3 (the others are
// below 2^-32 of it).  The tensor core truncates each FP32 partial sum, so a long chain in
// one accumulator drifts (5e-7 of the result at K = 256, more than FP32 cores lose): the
// leading products x0 y0 go round three accumulators in tensor memory and the corrections have
// a fourth, added once at the end.
//
// A CTA owns a 128 x 64 (or, with many tiles, 128 x 128) tile; sixteen producer warps load 32 columns of K at a time (16-byte
// loads where the operand is contiguous along k and aligned, coalesced along m or n where it
// is contiguous there), split and store them K-major and 64-byte swizzled through three
// stages, one warp issues the MMAs.  64 columns give 132 CTAs at 4,097 rows x 256, one
// wave of the 152 SMs; the split of A is repeated for each of the 4 column tiles, which costs
// less than idle SMs.  The weight gradient contracts over the rows: its few output tiles
// (8 for 256 x 256) are split along the rows into partial sums, as many as fill the GPU,
// added in a fixed order by a second kernel; the bias gradient is summed by the same producers.
// 10,989 rows, 256 x 256: 1.5 ms with 16 CTAs of a 64 x 64 FP32-core GEMM.
#include <cuda_bf16.h>
#include <math.h>

#include "../../include/pychem_gb300.h"
#include "common.cuh"
#include "pcg_internal.h"
#include "umma.cuh"

#define ML_BM 128
#define ML_BK 32
#define ML_PROD 512
#define ML_THREADS (ML_PROD + 32)
#define ML_STAGES 3
#define ML_WAIT (1u << 24)

// set when a wait of the GEMM gave up (its part of the tile is then NaNs); read and cleared by
// pcg_mlp_status
static __device__ int g_mlp_err;

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// high halves of two words as one BF16 pair (first in the low half)
__device__ __forceinline__ unsigned pack_hi(unsigned a, unsigned b) { return __byte_perm(a, b, 0x7632); }

// the three BF16 terms of eight floats; an infinity or NaN is its first term alone (x - x0 is
// then a NaN, seen once for all eight)
__device__ __forceinline__ void split3(const float (&x)[8], uint4 (&s)[3]) {
  unsigned h[3][8];
  float nan = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const unsigned u = __float_as_uint(x[j]);
    const float r1 = x[j] - __uint_as_float(u & 0xffff0000u);
    nan = fmaf(r1, 0.0f, nan);
    const unsigned u1 = __float_as_uint(r1);
    h[0][j] = u;
    h[1][j] = u1;
    h[2][j] = __float_as_uint(r1 - __uint_as_float(u1 & 0xffff0000u));
  }
  if (nan != nan) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned u = __float_as_uint(x[j]);
      if ((u & 0x7f800000u) != 0x7f800000u) continue;
      h[0][j] = u | (u << 9 ? 0x00400000u : 0u);       // a NaN stays one in its upper half
      h[1][j] = h[2][j] = 0u;
    }
  }
#pragma unroll
  for (int p = 0; p < 3; ++p)
    s[p] = make_uint4(pack_hi(h[p][0], h[p][1]), pack_hi(h[p][2], h[p][3]), pack_hi(h[p][4], h[p][5]),
                      pack_hi(h[p][6], h[p][7]));
}

// eight consecutive k of one row of an operand, zero outside; vec: contiguous along k with
// 16-byte aligned rows (k is a multiple of 8)
__device__ __forceinline__ void load8(const float* __restrict__ p, long long sr, long long sk, long long r, long long R,
                                      int k, int K, bool vec, float (&v)[8]) {
  if (r < R && vec && k + 8 <= K) {
    const float4 a = __ldg((const float4*)(p + r * sr + k)), b = __ldg((const float4*)(p + r * sr + k) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else if (r < R && k + 8 <= K) {
    const float* q = p + r * sr + k * sk;
#pragma unroll
    for (int j = 0; j < 8; ++j, q += sk) v[j] = __ldg(q);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (r < R && k + j < K) ? __ldg(p + r * sr + (k + j) * sk) : 0.0f;
  }
}
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* __restrict__ p, long long sr, long long sk, long long r,
                                       long long R, int k, int K, bool vec) {
  const unsigned short* u = (const unsigned short*)p;
  if (r < R && vec && k + 8 <= K) return __ldg((const uint4*)(u + r * sr + k));
  unsigned h[8];
  if (r < R && k + 8 <= K) {
    const unsigned short* q = u + r * sr + k * sk;
#pragma unroll
    for (int j = 0; j < 8; ++j, q += sk) h[j] = (unsigned)__ldg(q);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = (r < R && k + j < K) ? (unsigned)__ldg(u + r * sr + (k + j) * sk) : 0u;
  }
  return make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
}

// one item of a tile of `rows` rows x 4 groups of eight k: consecutive threads along the
// groups of a row, or along the rows where those are contiguous in memory
__device__ __forceinline__ void tile_item(int t, int rows, bool along_rows, int& r, int& g) {
  if (along_rows) { r = t % rows; g = t / rows; } else { r = t >> 2; g = t & 3; }
}

template <bool BF, int BN>
struct MlCfg {
  static constexpr int SB = BF ? 1 : 3;            // BF16 terms of B
  static constexpr int AT = ML_BM * ML_BK * 2;     // bytes of one term of the A tile
  static constexpr int BT = BN * ML_BK * 2;
  static constexpr int STAGE = 3 * AT + SB * BT;
  static constexpr int SMEM = ML_STAGES * STAGE + 2048;   // 1 KB alignment slack, barriers
};

struct MlArgs {
  int M, N, K;
  const float* A;
  long long sam, sak;
  const void* B;
  long long sbk, sbn;
  float* C;
  int ldc, accumulate;
  const float* bias;
  float* Z;
  int act;                 // 1: C = silu(C), pre-activation to Z; 2: C *= silu'(Z)
  int splits;              // > 1: partial sums of a range of K to C + split * M * N, ldc = N
  float* colsum;           // partial sums of B over k per split (wgrad), or null
};

// one element of the product over k0 <= k < k1 in FP32
template <bool BF>
__device__ __forceinline__ float plain_dot(const MlArgs& a, int m, int n, int k0, int k1) {
  float s = 0.0f;
  for (int k = k0; k < k1; ++k) {
    const float x = __ldg(a.A + m * a.sam + k * a.sak);
    const float y = BF ? __bfloat162float(((const __nv_bfloat16*)a.B)[k * a.sbk + n * a.sbn]) : __ldg((const float*)a.B + k * a.sbk + n * a.sbn);
    s = fmaf(x, y, s);
  }
  return s;
}

template <bool BF, int BN>
__global__ void __launch_bounds__(ML_THREADS, BN == 64 ? 2 : 1) k_gemm(const MlArgs a) {
  using Cfg = MlCfg<BF, BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(sm + ML_STAGES * Cfg::STAGE);     // full[3], empty[3], done
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * ML_STAGES + 1);
  volatile int* abort_s = (volatile int*)(tmem_slot + 1);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int ntn = (a.N + BN - 1) / BN;
  const int m0 = (int)(blockIdx.x / ntn) * ML_BM, n0 = (int)(blockIdx.x % ntn) * BN;
  const int nall = (a.K + ML_BK - 1) / ML_BK;
  const int c0 = (int)((long long)nall * blockIdx.y / a.splits), c1 = (int)((long long)nall * (blockIdx.y + 1) / a.splits);
  if (threadIdx.x == 0) {
    for (int i = 0; i < ML_STAGES; ++i) {
      mbar_init(&bars[i], ML_PROD / 32);
      mbar_init(&bars[ML_STAGES + i], 1);
    }
    mbar_init(&bars[2 * ML_STAGES], 1);
    *abort_s = 0;
    mbar_fence_init();
  }
  if (warp == ML_PROD / 32) tmem_alloc(tmem_slot, 4 * BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < ML_PROD / 32) {
    const int t = threadIdx.x;
    const bool a_rows = a.sam == 1 && a.sak != 1, b_rows = a.sbn == 1 && a.sbk != 1;
    const bool a_vec = a.sak == 1 && a.sam % 4 == 0 && ((uintptr_t)a.A & 15) == 0;
    const bool b_vec = a.sbk == 1 && a.sbn % (BF ? 8 : 4) == 0 && ((uintptr_t)a.B & 15) == 0;
    // one item of A a thread, and one of B (BN = 64: in the upper half of the threads)
    int ra, ga, rb, gb;
    const bool has_b = t >= ML_PROD - 4 * BN;
    tile_item(t, ML_BM, a_rows, ra, ga);
    tile_item(t & (4 * BN - 1), BN, b_rows, rb, gb);
    float csum = 0.0f;
    bool ok = true;
    float va[8], vb[8], na[8], nb[8];
    uint4 wb = make_uint4(0, 0, 0, 0), wn = wb;
    auto fetch = [&](int c) {
      const int k0 = c * ML_BK;
      load8(a.A, a.sam, a.sak, (long long)m0 + ra, a.M, k0 + 8 * ga, a.K, a_vec, na);
      if (has_b) {
        if (BF) wn = load8((const __nv_bfloat16*)a.B, a.sbn, a.sbk, (long long)n0 + rb, a.N, k0 + 8 * gb, a.K, b_vec);
        else load8((const float*)a.B, a.sbn, a.sbk, (long long)n0 + rb, a.N, k0 + 8 * gb, a.K, b_vec, nb);
      }
    };
    fetch(c0);
    for (int c = c0; c < c1; ++c) {
      const int it = c - c0, st = it % ML_STAGES;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        va[j] = na[j];
        if (!BF) vb[j] = nb[j];
      }
      wb = wn;
      if (c + 1 < c1) fetch(c + 1);        // in flight while this step is split
      if (it >= ML_STAGES && !mbar_wait(&bars[ML_STAGES + st], (it / ML_STAGES + 1) & 1, ML_WAIT, abort_s)) ok = false;
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      uint8_t* at = sm + st * Cfg::STAGE;
      uint8_t* bt = at + 3 * Cfg::AT;
      {
        uint4 s[3];
        split3(va, s);
#pragma unroll
        for (int p = 0; p < 3; ++p) *(uint4*)(at + p * Cfg::AT + sw64_offset(ra, ga)) = s[p];
      }
      if (has_b && BF) *(uint4*)(bt + sw64_offset(rb, gb)) = wb;
      if (has_b && !BF) {
        uint4 s[3];
        split3(vb, s);
#pragma unroll
        for (int p = 0; p < Cfg::SB; ++p) *(uint4*)(bt + p * Cfg::BT + sw64_offset(rb, gb)) = s[p];
        if (a.colsum) {
#pragma unroll
          for (int j = 0; j < 8; ++j) csum += vb[j];
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[st]);
    }
    if (!ok) { *abort_s = 1; atomicExch(&g_mlp_err, 1); }
    if (warp_all(ok && mbar_wait(&bars[2 * ML_STAGES], 0, ML_WAIT, abort_s) && !*abort_s)) {
      tc_fence_after();
      const int m = m0 + 32 * (warp & 3) + lane;
      const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
      float* C = a.C + (a.splits > 1 ? (long long)blockIdx.y * a.M * a.N : 0ll);
      const bool cvec = a.ldc % 4 == 0 && ((uintptr_t)C & 15) == 0 && (!a.Z || ((uintptr_t)a.Z & 15) == 0);
#pragma unroll 1
      for (int cb = 8 * (warp >> 2); cb < BN; cb += 32) {
        // the accumulators in use: three only from three K steps of 16 on
        const int lead = min(3, (c1 - c0) * (ML_BK / 16));
        float v[8], w[8], u[8], x3[8];
        if (m0 + ML_BM > a.M) __syncwarp();   // the loads want every lane, also those past the last row
        tmem_ld8(trow + cb, v);
        tmem_ld8(trow + BN + cb, u);
        tmem_ld8(trow + 2 * BN + cb, x3);
        tmem_ld8(trow + 3 * BN + cb, w);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          w[j] += lead > 2 ? x3[j] : 0.0f;
          v[j] += u[j];
        }
        const int n = n0 + cb;
        if (m >= a.M || n >= a.N) continue;
        const long long o = (long long)m * a.ldc + n;
        const bool full = cvec && n + 8 <= a.N;
        float z[8];
        if (a.act == 2) {
#pragma unroll
          for (int j = 0; j < 8; ++j) z[j] = n + j < a.N ? a.Z[o + j] : 0.0f;
        }
        unsigned top = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] += w[j];
          top = max(top, __float_as_uint(v[j]) & 0x7fffffffu);
        }
        // a second or third term of zero times an infinity of the other operand is a NaN that the
        // FP32 product does not have: such elements are summed plainly (the test costs 1.3 % of a
        // 256 x 256 layer; beside the splits, for BF16 weights, it would cost the producers more)
        if (top > 0x7f800000u) {
#pragma unroll 1
          for (int j = 0; j < 8; ++j) {
            float x = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) x = i == j ? v[i] : x;
            if (x == x || n + j >= a.N) continue;
            x = plain_dot<BF>(a, m, n + j, c0 * ML_BK, min(a.K, c1 * ML_BK));
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = i == j ? x : v[i];
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const bool in = n + j < a.N;
          float x = v[j];
          if (a.accumulate && in) x += C[o + j];
          if (a.bias && in) x += __ldg(a.bias + n + j);
          if (a.act == 2) x *= dsilu(z[j]);
          else z[j] = x;
          v[j] = a.act == 1 ? silu(x) : x;
        }
        if (full) {
          if (a.Z && a.act != 2) {
            *(float4*)(a.Z + o) = make_float4(z[0], z[1], z[2], z[3]);
            *(float4*)(a.Z + o + 4) = make_float4(z[4], z[5], z[6], z[7]);
          }
          *(float4*)(C + o) = make_float4(v[0], v[1], v[2], v[3]);
          *(float4*)(C + o + 4) = make_float4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (n + j < a.N) {
              if (a.Z && a.act != 2) a.Z[o + j] = z[j];
              C[o + j] = v[j];
            }
        }
      }
      // the MMAs have read the last tiles, so the stages are free for the four groups' sums
      if (a.colsum && m0 == 0 && has_b) ((float*)sm)[gb * BN + rb] = csum;
    } else {
      // given up: NaNs for what this warp would have stored
      *abort_s = 1;
      atomicExch(&g_mlp_err, 1);
      const int m = m0 + 32 * (warp & 3) + lane;
      float* C = a.C + (a.splits > 1 ? (long long)blockIdx.y * a.M * a.N : 0ll);
      for (int cb = 8 * (warp >> 2); cb < BN; cb += 32)
        for (int n = n0 + cb; m < a.M && n < min(a.N, n0 + cb + 8); ++n) {
          C[(long long)m * a.ldc + n] = __int_as_float(0x7fffffff);
          if (a.Z && a.act != 2) a.Z[(long long)m * a.ldc + n] = __int_as_float(0x7fffffff);
        }
    }
    if (a.colsum && m0 == 0) {
      const float* red = (const float*)sm;
      asm volatile("bar.sync 1, %0;" ::"r"(ML_PROD) : "memory");
      if (t < BN && n0 + t < a.N)
        a.colsum[(long long)blockIdx.y * a.N + n0 + t] =
            *abort_s ? __int_as_float(0x7fffffff) : (red[t] + red[BN + t]) + (red[2 * BN + t] + red[3 * BN + t]);
    }
  } else {
    const uint32_t idesc = idesc_bf16_f32(ML_BM, BN);
    const uint32_t lead = elect_one();
    const uint64_t xd0 = sdesc_k_sw64(smem_u32(sm));
    bool ok = true;
    unsigned have = 0;       // accumulators that hold a sum; 3: the corrections
    for (int it = 0; it < c1 - c0; ++it) {
      const int st = it % ML_STAGES;
      ok = mbar_wait(&bars[st], (it / ML_STAGES) & 1, ML_WAIT, abort_s);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint64_t xd = xd0 + (uint64_t)(st * (Cfg::STAGE >> 4)), yd = xd + (3 * Cfg::AT >> 4);
#pragma unroll
      for (int kk = 0; kk < ML_BK / 16; ++kk) {
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int q = 0; q < Cfg::SB; ++q) {
            if (p + q > 3) continue;
            const int acc = p + q == 0 ? (it * (ML_BK / 16) + kk) % 3 : 3;
            umma_bf16_lead(lead, tmem + acc * BN, xd + ((p * Cfg::AT + kk * 32) >> 4),
                           yd + ((q * Cfg::BT + kk * 32) >> 4), idesc, (have >> acc) & 1u);
            have |= 1u << acc;
          }
      }
      umma_commit_lead(lead, &bars[ML_STAGES + st]);
    }
    if (!ok) {               // before the commit: the epilogue looks at the flag after its wait
      *abort_s = 1;
      __threadfence_block();
      if (lead) atomicExch(&g_mlp_err, 2);
      __syncwarp();
    }
    umma_commit_lead(lead, &bars[2 * ML_STAGES]);
    if (!ok) {
      volatile int keep_waiting = 0;
      mbar_wait(&bars[2 * ML_STAGES], 0, ML_WAIT, &keep_waiting);   // drain before tensor memory is freed
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == ML_PROD / 32) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 4 * BN);
  }
}

// dW = sum of the partial products, db = sum of the partial column sums, splits in order
__global__ void k_wgrad_sum(long long len, int N, int splits, const float* __restrict__ part,
                            const float* __restrict__ cpart, float* __restrict__ dW, float* __restrict__ db) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < len) {
    float s = 0.0f;
#pragma unroll 8
    for (int k = 0; k < splits; ++k) s += __ldg(part + k * len + i);
    dW[i] = s;
  } else if (i < len + N) {
    float s = 0.0f;
#pragma unroll 8
    for (int k = 0; k < splits; ++k) s += __ldg(cpart + (long long)k * N + (i - len));
    db[i - len] = s;
  }
}

// G = dY * silu'(Z) elementwise (in place on dY)
__global__ void k_dsilu(long long n, float* __restrict__ dY, const float* __restrict__ Z) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dY[i] *= dsilu(Z[i]);
}

// column sums: db[n] = sum_m G[m][n]; one block per 32 columns, 32 rows at a time
__global__ void __launch_bounds__(1024) k_colsum(int M, int N, const float* __restrict__ G, float* __restrict__ db) {
  __shared__ float red[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, n = blockIdx.x * 32 + tx;
  float s = 0.0f;
  if (n < N)
    for (int m = ty; m < M; m += 32) s += __ldg(G + (long long)m * N + n);
  red[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && n < N) {
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += red[k][tx];
    db[n] = t;
  }
}

// masked squared error: loss partial sums and dY = 2 (Y - T) mask / count, count from
// *cnt (a device value) when given.  One atomic per block.
__global__ void __launch_bounds__(256) k_mse(long long n, const float* __restrict__ Y, const float* __restrict__ T,
                                             const float* __restrict__ mask, float inv_count,
                                             const float* __restrict__ cnt, float* __restrict__ dY,
                                             float* __restrict__ loss) {
  const float inv = cnt ? (float)(1.0 / fmax((double)*cnt, 1.0)) : inv_count;
  float l = 0.0f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float d = (Y[i] - T[i]) * mask[i];
    dY[i] = 2.0f * d * inv;
    l += d * d * inv;
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  __shared__ float red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) l += red[k];
    atomicAdd(loss, l);
  }
}

// Adam on FP32 master weights, refreshing the BF16 copy used by the GEMMs; all tensors of
// a network in one launch (blockIdx.y: the tensor)
__global__ void k_adam(pcg_adam_t ts, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int k = blockIdx.y;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ts.n[k]) return;
  float *w = ts.w[k], *m = ts.m[k], *v = ts.v[k];
  __nv_bfloat16* wb = (__nv_bfloat16*)ts.w_bf16[k];
  const float gi = ts.g[k][i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  w[i] = wi;
  if (wb) wb[i] = __float2bfloat16_rn(wi);
}

template <bool BF, int BN>
static int run_gemm(const MlArgs& a, cudaStream_t s) {
  const long long tiles = (long long)((a.M + ML_BM - 1) / ML_BM) * ((a.N + BN - 1) / BN);
  if (tiles > 0x7fffffffLL) { pcg_set_error("pcg_mlp_gemm: too many tiles for one launch"); return PCG_ERR_UNSUPPORTED; }
  PCG_CUDA(cudaFuncSetAttribute(k_gemm<BF, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, MlCfg<BF, BN>::SMEM));
  k_gemm<BF, BN><<<dim3((unsigned)tiles, a.splits), ML_THREADS, MlCfg<BF, BN>::SMEM, s>>>(a);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_mlp_gemm(int M, int N, int K, const float* A, long long sam, long long sak, const void* B,
                            int b_bf16, long long sbk, long long sbn, float* C, int ldc, int accumulate,
                            const float* bias, float* Z, int act, void* stream) {
  if (M < 1 || N < 1 || K < 1 || !A || !B || !C || (act == 2 && !Z)) {
    pcg_set_error("pcg_mlp_gemm: bad arguments");
    return PCG_ERR_ARG;
  }
  const MlArgs a = {M, N, K, A, sam, sak, B, sbk, sbn, C, ldc, accumulate, bias, Z, act, 1, nullptr};
  // 128 columns a CTA once 64-column tiles come to more than one an SM: A is split for half as
  // many tiles (256 x 256 layer, 5,000 rows 18.8 -> 12.5 us, 65,536 rows 115 -> 97 us); below that
  // the wide tiles leave SMs idle
  const bool wide = N > 64 && (long long)((M + ML_BM - 1) / ML_BM) * ((N + 63) / 64) > 152;
  cudaStream_t s = (cudaStream_t)stream;
  if (wide) return b_bf16 ? run_gemm<true, 128>(a, s) : run_gemm<false, 128>(a, s);
  return b_bf16 ? run_gemm<true, 64>(a, s) : run_gemm<false, 64>(a, s);
}

extern "C" int pcg_mlp_forward(int nlayer, const int* dims, int M, const float* X, const void* const* W_bf16,
                               const float* const* b, float* const* out, float* const* Z, void* stream) {
  if (nlayer < 1 || !dims || !W_bf16 || !b || !out) { pcg_set_error("pcg_mlp_forward: bad arguments"); return PCG_ERR_ARG; }
  const float* A = X;
  for (int k = 0; k < nlayer; ++k) {
    const int K = dims[k], N = dims[k + 1], act = k < nlayer - 1 ? 1 : 0;
    if (int rc = pcg_mlp_gemm(M, N, K, A, K, 1, W_bf16[k], 1, N, 1, out[k], N, 0, b[k], Z ? Z[k] : nullptr, act, stream))
      return rc;
    A = out[k];
  }
  return PCG_OK;
}

// columns a CTA of the weight gradient takes, and its row splits: one CTA an SM, but at least four
// 32-row steps each
static int wgrad_bn(int N) { return N > 64 ? 128 : 64; }
static int wgrad_splits(int M, int K, int N) {
  const long long tiles = (long long)((K + ML_BM - 1) / ML_BM) * ((N + wgrad_bn(N) - 1) / wgrad_bn(N));
  const long long most = (M + 4 * ML_BK - 1) / (4 * ML_BK), want = 152 / tiles;
  const long long k = want < most ? want : most;
  return k < 1 ? 1 : (int)k;
}

extern "C" size_t pcg_mlp_wgrad_workspace(int M, int K, int N) {
  if (M < 1 || K < 1 || N < 1) return 0;
  return (size_t)wgrad_splits(M, K, N) * ((size_t)K * N + N) * sizeof(float);
}

extern "C" int pcg_mlp_wgrad(int M, int K, int N, const float* A, const float* G, float* dW, float* db, void* workspace,
                             size_t ws_bytes, void* stream) {
  if (M < 1 || K < 1 || N < 1 || !A || !G || !dW || !db) { pcg_set_error("pcg_mlp_wgrad: bad arguments"); return PCG_ERR_ARG; }
  if (!workspace || ((size_t)workspace & 15) || ws_bytes < pcg_mlp_wgrad_workspace(M, K, N)) {
    pcg_set_error("pcg_mlp_wgrad: workspace missing, misaligned or too small (query pcg_mlp_wgrad_workspace)");
    return PCG_ERR_CAPACITY;
  }
  const int splits = wgrad_splits(M, K, N);
  const long long len = (long long)K * N;
  float* part = (float*)workspace;
  float* cpart = part + splits * len;
  MlArgs a = {K, N, M, A, 1, K, G, N, 1, part, N, 0, nullptr, nullptr, 0, splits, cpart};
  if (int rc = wgrad_bn(N) == 128 ? run_gemm<false, 128>(a, (cudaStream_t)stream)
                                  : run_gemm<false, 64>(a, (cudaStream_t)stream)) return rc;
  k_wgrad_sum<<<(unsigned)((len + N + 255) / 256), 256, 0, (cudaStream_t)stream>>>(len, N, splits, part, cpart, dW, db);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_mlp_status(void* stream) {
  int h = 0;
  PCG_CUDA(cudaMemcpyFromSymbolAsync(&h, g_mlp_err, sizeof(int), 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  PCG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  if (h) {
    const int zero = 0;
    PCG_CUDA(cudaMemcpyToSymbolAsync(g_mlp_err, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, (cudaStream_t)stream));
    PCG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  }
  return h;
}

extern "C" int pcg_mlp_dsilu(long long n, float* dY, const float* Z, void* stream) {
  k_dsilu<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, dY, Z);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_mlp_colsum(int M, int N, const float* G, float* db, void* stream) {
  k_colsum<<<(N + 31) / 32, 1024, 0, (cudaStream_t)stream>>>(M, N, G, db);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

static int run_mse(long long n, const float* Y, const float* T, const float* mask, float inv_count, const float* cnt,
                   float* dY, float* loss, cudaStream_t s) {
  const long long blocks = (n + 1023) / 1024;
  k_mse<<<(unsigned)(blocks < 1 ? 1 : (blocks < 608 ? blocks : 608)), 256, 0, s>>>(n, Y, T, mask, inv_count, cnt, dY, loss);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_mlp_mse(long long n, const float* Y, const float* T, const float* mask, float inv_count,
                           float* dY, float* loss, void* stream) {
  return run_mse(n, Y, T, mask, inv_count, nullptr, dY, loss, (cudaStream_t)stream);
}

extern "C" int pcg_mlp_mse_counted(long long n, const float* Y, const float* T, const float* mask, const float* count,
                                   float* dY, float* loss, void* stream) {
  if (!count) { pcg_set_error("pcg_mlp_mse_counted: no count"); return PCG_ERR_ARG; }
  return run_mse(n, Y, T, mask, 0.0f, count, dY, loss, (cudaStream_t)stream);
}

extern "C" int pcg_mlp_adam_all(int ntensor, const pcg_adam_t* tensors, float lr, float b1, float b2, float eps,
                                int step, void* stream) {
  if (ntensor < 1 || ntensor > PCG_ADAM_MAX || !tensors) {
    pcg_set_error("pcg_mlp_adam_all: bad arguments");
    return PCG_ERR_ARG;
  }
  long long most = 1;
  for (int k = 0; k < ntensor; ++k) most = tensors->n[k] > most ? tensors->n[k] : most;
  const float c1 = 1.0f / (1.0f - powf(b1, (float)step)), c2 = 1.0f / (1.0f - powf(b2, (float)step));
  k_adam<<<dim3((unsigned)((most + 255) / 256), ntensor), 256, 0, (cudaStream_t)stream>>>(*tensors, lr, b1, b2, eps, c1, c2);
  PCG_CUDA(cudaGetLastError());
  return PCG_OK;
}

extern "C" int pcg_mlp_adam(long long n, float* w, const float* g, float* m, float* v, void* w_bf16, float lr,
                            float b1, float b2, float eps, int step, void* stream) {
  pcg_adam_t t = {};
  t.n[0] = n; t.w[0] = w; t.g[0] = g; t.m[0] = m; t.v[0] = v; t.w_bf16[0] = w_bf16;
  return pcg_mlp_adam_all(1, &t, lr, b1, b2, eps, step, stream);
}
