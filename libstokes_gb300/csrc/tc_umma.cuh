// tc_umma.cuh -- minimal tcgen05 (5th-generation tensor core) helpers for
// sm_103a: TMEM allocation, shared-memory matrix descriptors, the f16 MMA,
// commit to an mbarrier, bounded mbarrier waits and TMEM loads.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lsg {
namespace umma {

// descriptor of a K-major tile in the 128-byte swizzled layout that a TMA
// load with CU_TENSOR_MAP_SWIZZLE_128B writes: rows of 128 bytes (64 f16
// values), 8-row groups 1024 bytes apart (SBO), the 16-byte chunks of row r
// permuted by r % 8; the tile must start on a 1024-byte boundary.  The k-th
// K step of 16 values starts 32 k bytes in (the swizzle is applied to the
// address, so the start moves within the atom).  LBO is unused in this mode.
__device__ __forceinline__ uint64_t
smem_desc_sw128 (uint32_t saddr)
{
  uint64_t d = 0;
  d |= (uint64_t) ((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t) 1u << 16;                 // LBO (ignored): 16 bytes
  d |= (uint64_t) (1024u >> 4) << 32;       // SBO: 1024 bytes
  d |= (uint64_t) 1u << 46;                 // descriptor version
  d |= (uint64_t) 2u << 61;                 // layout: 128-byte swizzle
  return d;
}

// instruction descriptor, kind::f16: D f32, A/B f16, both K-major
__host__ __device__ __forceinline__ uint32_t
idesc_f16 (uint32_t M, uint32_t N)
{
  return (1u << 4)            // D format: f32 (A and B format 0: f16)
    | ((N >> 3) << 17)        // N / 8
    | ((M >> 4) << 24);       // M / 16
}

__device__ __forceinline__ uint32_t
smem_u32 (const void *p)
{
  return (uint32_t) __cvta_generic_to_shared (p);
}

// TMEM allocation by one full warp; the column address lands in *slot
__device__ __forceinline__ void
tmem_alloc (uint32_t *slot, uint32_t ncols)
{
  asm volatile ("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                :: "r"(smem_u32 (slot)), "r"(ncols) : "memory");
  asm volatile ("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void
tmem_dealloc (uint32_t taddr, uint32_t ncols)
{
  asm volatile ("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                :: "r"(taddr), "r"(ncols) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, f16 operands (K = 16 per instruction),
// called by a whole converged warp: one elected lane issues it.  The descriptors
// are then warp uniform and live in uniform registers; issued from a branch on
// one lane each MMA first moved them there (about 115 clocks an MMA instead of
// the 32 to 96 that the tensor pipe takes).
__device__ __forceinline__ void
mma_f16 (uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
  asm volatile (
    "{\n\t.reg .pred p, q;\n\t"
    "elect.sync _|q, 0xffffffff;\n\t"
    "setp.ne.b32 p, %4, 0;\n\t"
    "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
    :: "r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// arrive on an mbarrier once all MMAs issued so far are done, from a whole
// converged warp (the lane that mma_f16 elects)
__device__ __forceinline__ void
mma_commit_warp (uint64_t *mbar)
{
  asm volatile ("{\n\t.reg .pred q;\n\t"
                "elect.sync _|q, 0xffffffff;\n\t"
                "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
                :: "r"(smem_u32 (mbar)) : "memory");
}

__device__ __forceinline__ void
mbar_init (uint64_t *mbar, uint32_t count)
{
  asm volatile ("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32 (mbar)), "r"(count)
                : "memory");
}

__device__ __forceinline__ void
fence_mbar_init ()
{
  asm volatile ("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// one arrival on an mbarrier (release at CTA scope)
__device__ __forceinline__ void
mbar_arrive (uint64_t *mbar)
{
  asm volatile ("{\n\t.reg .b64 st;\n\t"
                "mbarrier.arrive.shared::cta.b64 st, [%0];\n\t}"
                :: "r"(smem_u32 (mbar)) : "memory");
}

// wait for phase `parity`, giving up early when *abort (a CTA-wide error flag
// in shared memory) becomes non-zero; returns false when the wait did not
// complete.  Each poll lets the thread sleep until the phase completes or
// about 20 us pass (the try_wait suspend-time hint), so waiting warps do not
// take issue slots from working ones; `limit` polls bound the wait to about
// limit x 20 us.
__device__ __forceinline__ bool
mbar_wait_or_abort (uint64_t *mbar, uint32_t parity, uint32_t limit, volatile int *abort)
{
  const uint32_t a = smem_u32 (mbar);
  for (uint32_t it = 0; it < limit; it++)
    {
      uint32_t done;
      asm volatile (
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(a), "r"(parity), "r"(20000u) : "memory");
      if (done) return true;
      if (*abort) return false;
    }
  *abort = 1;
  return false;
}

// arrive once on an mbarrier and add `bytes` to the transaction count its
// current phase waits for (the TMA loads that follow complete them)
__device__ __forceinline__ void
mbar_expect_tx (uint64_t *mbar, uint32_t bytes)
{
  asm volatile ("{\n\t.reg .b64 st;\n\t"
                "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
                :: "r"(smem_u32 (mbar)), "r"(bytes) : "memory");
}

// 3-d tiled TMA load of one box at coordinates (c0, c1, c2) into shared
// memory, completing `bytes of the box` on the mbarrier; tmap: the address of
// a __grid_constant__ CUtensorMap kernel parameter
__device__ __forceinline__ void
tma_load_3d (void *dst, const void *tmap, int c0, int c1, int c2, uint64_t *mbar)
{
  asm volatile (
    "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
    " [%0], [%1, {%2, %3, %4}], [%5];"
    :: "r"(smem_u32 (dst)), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32 (mbar))
    : "memory");
}

__device__ __forceinline__ void
tma_prefetch_desc (const void *tmap)
{
  asm volatile ("prefetch.tensormap [%0];" :: "l"(tmap) : "memory");
}

// generic-proxy smem writes -> visible to the tensor core (async proxy)
__device__ __forceinline__ void
fence_async_smem ()
{
  asm volatile ("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void
fence_before_sync ()
{
  asm volatile ("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void
fence_after_sync ()
{
  asm volatile ("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane (32x32b shape): warp w
// of a warpgroup reads lanes 32 w .. 32 w + 31; v holds them after tmem_ld_wait (v)
__device__ __forceinline__ void
tmem_ld16_issue (uint32_t taddr, float v[16])
{
  asm volatile (
    "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
    "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
    : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
      "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]),
      "=f"(v[14]), "=f"(v[15])
    : "r"(taddr));
}

// every issued load of this thread is complete; the operands tie the loaded
// registers to the wait
__device__ __forceinline__ void
tmem_ld_wait (float v[16])
{
  asm volatile ("tcgen05.wait::ld.sync.aligned;"
                : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]),
                  "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]),
                  "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                :: "memory");
}

}  // namespace umma
}  // namespace lsg
