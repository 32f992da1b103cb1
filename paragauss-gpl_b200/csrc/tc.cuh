// tc.cuh -- Blackwell (sm_100a) fifth-generation tensor core primitives:
// TMEM allocation, tcgen05.mma issue/commit, TMEM loads, shared-memory matrix
// descriptors for the canonical no-swizzle layouts, and bounded mbarrier waits.
//
// Canonical no-swizzle ("interleaved") K-major layout: a core matrix is 8
// rows (along M or N) of 16 bytes (consecutive K elements) stored contiguously
// (128 B); LBO = byte distance between the two 16-byte K halves of one MMA's
// 32-byte K slab, SBO = byte distance between 8-row groups.
#pragma once

#include <cstdint>

namespace pgxc {
namespace tc {

// Iteration bound of every mbarrier wait (each try_wait may itself suspend
// for a hardware-defined interval): a wait that runs out sets the error flag
// and the kernel winds down instead of spinning for ever.
constexpr long long kWaitLimit = 1ll << 24;

// The tensor-core kernels (tcgen05 + TMEM) claim a whole SM: 16 warps and all
// of its shared memory, so that no CTA of another kernel is placed beside them.
// With other CTAs on the same SM (builds running concurrently on the GPU) their
// epilogue warps were seen to read wrong accumulator rows in whole 32-lane
// quarters; alone on the SM they are exact.  Warps beyond a kernel's roles
// idle until the final barrier.
constexpr int kWholeSmThreads = 512;
constexpr int kWholeSmSmem = 227 * 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- shared-memory matrix descriptor (sm_100 format, version 1) -----------
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // version
  // base offset 0, lbo mode 0, layout type 0 (no swizzle)
  return d;
}

// ---- instruction descriptor: kind::i8, S8 x S8 -> S32 ---------------------
__host__ __device__ constexpr uint32_t idesc_s8(int M, int N) {
  return (2u << 4)                          // D format S32
         | (1u << 7)                        // A signed 8-bit
         | (1u << 10)                       // B signed 8-bit
         | ((uint32_t)(N >> 3) << 17)       // N / 8   (A, B K-major)
         | ((uint32_t)(M >> 4) << 24);      // M / 16
}

// ---- TMEM -----------------------------------------------------------------
// Called by one whole warp; writes the TMEM base address to *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
               "r"(ncols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy shared-memory writes -> visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem], signed 8-bit operands, exact 32-bit integer accumulation.
__device__ __forceinline__ void mma_s8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"((uint32_t)accumulate));
}

// Arrive once on the mbarrier when all previously issued MMAs of this thread complete.
__device__ __forceinline__ void mma_commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(mbar))
               : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns: thread t of the warp gets lane
// (warp%4)*32 + t, columns col..col+15 of the addressed region.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 lanes x 8 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// 32 lanes x 4 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
// 32 lanes x 16 consecutive 32-bit columns, raw bits
__device__ __forceinline__ void tmem_ld16u(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// tcgen05.ld writes its registers asynchronously: they hold the data only
// after tcgen05.wait::ld, but nothing in the wait names them, so the compiler
// may schedule their first uses before it.  An empty asm that reads and
// rewrites each register, placed after the wait, makes every later use depend
// on it (volatile asm statements keep their order).
template <int N>
__device__ __forceinline__ void tmem_regs_ready(uint32_t (&r)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
template <int N>
__device__ __forceinline__ void tmem_regs_ready(float (&r)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+f"(r[i]));
}

// ---- mbarrier ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(bytes), "r"(smem_u32(mbar))
               : "memory");
}
// 1-D bulk copy global -> shared (16-byte aligned, size a multiple of 16);
// completes `bytes` of the mbarrier's transaction count.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(mbar))
               : "memory");
}

// Bulk prefetch of global memory into L2 (16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// Bounded wait for the phase with the given parity to complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity) {
  const uint32_t a = smem_u32(mbar);
  for (long long i = 0; i < kWaitLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// The same wait by every thread of a warp, returning the warp's common verdict
// with the warp converged.  The threads of a warp leave the spin loop at
// different polls; the .sync.aligned tcgen05 instructions that follow a wait
// (tcgen05.ld, tcgen05.wait::ld) must be executed by the whole warp together.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* mbar, uint32_t parity) {
  const bool ok = __all_sync(0xffffffffu, mbar_wait(mbar, parity));
  __syncwarp();
  return ok;
}

// Before a CTA ends, also one whose waits ran out, its asynchronous work has ended:
// the copies into its shared memory (uses 0 .. n - 1 of a ring of barriers, the last
// of each slot), and the products that read it and write TMEM (drain: a barrier of
// one arrival, used by the issuer alone).  Bounded like every wait.
__device__ __forceinline__ void copies_land(uint64_t* full, int ring, int n) {
  for (int j = n > ring ? n - ring : 0; j < n; ++j) mbar_wait(&full[j % ring], (j / ring) & 1);
}
__device__ __forceinline__ void products_end(uint64_t* drain) {
  mma_commit(drain);
  mbar_wait(drain, 0);
}

}  // namespace tc
}  // namespace pgxc
