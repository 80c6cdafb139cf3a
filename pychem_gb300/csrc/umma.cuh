// Blackwell (sm_103a) tensor-core primitives in inline PTX: mbarriers, tensor memory
// (TMEM) allocation and loads, shared-memory matrix descriptors, tcgen05.mma with
// BF16 operands and FP32 accumulation, and the async-proxy fences between them.
//
// Conventions used by the kernels of this library:
//  * one CTA per SM (tensor memory and shared memory sized for that), cta_group::1;
//  * operands K-major in shared memory with the 64-byte swizzle: a tile of R rows is
//    R x 64 bytes (32 BF16 along K), row r at byte r*64 with its four 16-byte chunks
//    permuted, chunk c stored at c ^ ((r >> 1) & 3); groups of 8 rows are 512 bytes
//    apart (the descriptor's stride offset); tiles start on 512-byte boundaries;
//  * the accumulator of an M = 128 MMA: row m in TMEM lane m, column n in column
//    base + n (FP32).
// Every wait on an mbarrier is bounded (see mbar_wait): a kernel that gives up sets an
// error flag and unwinds instead of spinning forever.
#pragma once
#include <stdint.h>

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// make barrier initialisation visible to the async proxy (tcgen05.commit arrivals)
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for the phase of parity `parity` to complete, at most `limit` polls (each
// try_wait itself suspends for a bounded, implementation-defined time); also gives up
// when *abort becomes nonzero.  Returns false if it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit, volatile int* abort) {
  for (uint32_t it = 0; it < limit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && *abort) return false;
  }
  return false;
}

// Whether x holds in every lane of the warp.  A vote of its own: after __all_sync the compiler
// takes what follows for converged and keeps addresses of a later loop in registers, which spilled
// the network GEMM's epilogue (367 -> 371 us a training step).
__device__ __forceinline__ bool warp_all(bool x) {
  uint32_t m;
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n vote.sync.ballot.b32 %0, p, 0xffffffff;\n}" : "=r"(m) : "r"((int)x));
  return m == 0xffffffffu;
}

// make generic-proxy shared-memory writes visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Tensor memory: allocate / free ncols columns (a power of two >= 32); warp-wide.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 8 consecutive FP32 columns of this thread's lane (warp w reads lanes 32 (w % 4) ..)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major, 64-byte-swizzled tile starting at
// shared address saddr: start address (>> 4) in bits 0-13, leading-dimension offset
// 16 B (not used by swizzled K-major layouts) in bits 16-29, stride offset 512 B
// (8 rows x 64 B) in bits 32-45, the fixed descriptor version 0b001 in bits 46-48,
// base offset 0 (512-byte aligned tiles), swizzle mode 4 (64 B) in bits 61-63.
__device__ __forceinline__ uint64_t sdesc_k_sw64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// Instruction descriptor of tcgen05.mma kind::f16: FP32 accumulator (bits 4-5 = 1),
// BF16 A and B (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 in bits
// 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, from a warp that runs its issue loop converged, with
// warp-uniform operands, and one leading lane: descriptors then stay in uniform registers.  Issued by a single diverged thread,
// each MMA moves its operands there first, about 250 cycles an MMA whatever its size.
__device__ __forceinline__ void umma_bf16_lead(uint32_t lead, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// arrive once on the mbarrier when every MMA that the leading lane issued has completed
__device__ __forceinline__ void umma_commit_lead(uint32_t lead, uint64_t* bar) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
      " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_u32(bar)),
      "r"(lead)
      : "memory");
}
// 1 in one lane of a converged warp
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
  return r;
}
// this thread's warp, as a warp-uniform value
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// byte offset of the 16-byte chunk c (0..3) of row r in a 64-byte-swizzled K-major tile
__device__ __forceinline__ uint32_t sw64_offset(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }
