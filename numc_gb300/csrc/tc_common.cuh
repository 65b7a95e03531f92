// Blackwell (sm_100a/sm_103a) building blocks as inline PTX: mbarriers with
// bounded waits, TMA tile loads, TMEM allocation, tcgen05.mma (kind::f16),
// tcgen05.commit and tcgen05.ld.  Written against the PTX ISA 8.7+
// descriptions of these instructions.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "status.h"

namespace numc_k {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- mbarrier ---------------------------------------------------------------

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Wait for the phase of `bar` with parity `parity` to complete, giving up
// after `limit_ns`.  On timeout the first failing thread records `code` in
// the device status word; the caller abandons its work and returns.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity,
                                                  unsigned *status, unsigned code,
                                                  uint64_t limit_ns = 2000000000ull) {
#pragma unroll 1
  for (int i = 0; i < 4096; i++)
    if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    __nanosleep(128);
    if (globaltimer_ns() - t0 > limit_ns) {
      if (status) atomicCAS(status, 0u, code);
      return false;
    }
  }
}

// ---- programmatic dependent launch ---------------------------------------------
// A kernel launched with cudaLaunchAttributeProgrammaticStreamSerialization
// may start while the previous kernel in the stream still runs; it calls
// griddep_wait() before touching anything that kernel writes (the wait
// returns once that grid has completed and its writes are visible; it is a
// no-op for a kernel launched without the attribute).  The previous kernel
// calls griddep_launch_dependents() once all of its blocks are resident, so
// the dependent grid's launch and prologue overlap its tail.
__device__ __forceinline__ void griddep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---- TMA ----------------------------------------------------------------------

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)m) : "memory");
}

// 2-D tiled load of box {x (innermost), y} into shared memory, completing
// `bytes` on `bar`.  x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *m, uint32_t bar,
                                            int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"((uint64_t)m), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// 3-D tiled load: box {x, y, 1} at (x, y, z); z selects a plane.
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *m, uint32_t bar,
                                            int32_t x, int32_t y, int32_t z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"((uint64_t)m), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Order earlier writes of a tensor map in global memory (made by copies
// before this kernel) before its use by TMA through the tensormap proxy.
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap *m) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"((uint64_t)m)
               : "memory");
}

// Contiguous copy of `bytes` (a multiple of 16) into shared memory, counted by
// the mbarrier `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"((uint64_t)__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
      : "memory");
}

// ---- TMEM ---------------------------------------------------------------------

// Executed by one full warp.  Writes the TMEM base address to *dst_smem.
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- UMMA descriptors ---------------------------------------------------------

// Shared-memory matrix descriptor for a K-major operand tile stored in the
// 128-byte swizzle layout written by TMA with CU_TENSOR_MAP_SWIZZLE_128B:
// rows of 128 bytes, 8-row atoms of 1024 bytes (stride byte offset), tile
// base 1024-byte aligned.  Fields: start address >> 4 [0,14), leading byte
// offset >> 4 [16,30) (unused for swizzled K-major), stride byte offset >> 4
// [32,46), descriptor version 1 at [46,48), swizzle mode [61,64) = 2.
__device__ __forceinline__ uint64_t sdesc_k128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor of tcgen05.mma kind::f16 with BF16 A and B (both
// K-major), FP32 accumulation, shape M x N: D format [4,6) = 1 (F32),
// A format [7,10) = 1 (BF16), B format [10,13) = 1 (BF16), N >> 3 at
// [17,23), M >> 4 at [24,29).
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

// Same with F16 A and B: formats [7,10) and [10,13) = 0 (both operands must
// have the same type).
__host__ __device__ constexpr uint32_t idesc_f16_f32(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// 32 lanes x 32 bits, 32 consecutive columns: thread t of the warp gets
// row (lane base + t), columns [col, col + 32).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
}

// Same with 16 consecutive columns.
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// Same with 8 consecutive columns.
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- Issue by a whole warp -----------------------------------------------------
//
// A loop of one lane that builds descriptors and issues MMAs moves every
// operand into uniform registers one MMA at a time: some 100 cycles an MMA,
// more than MMAs of up to 128 columns take.  With the whole warp in the loop
// and the instruction predicated on an elected lane the operands stay in
// uniform registers.

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok));
  return ok != 0;
}

// D (+)= A B^T, kind::f16 (operand types in idesc), by the lane with `lead`;
// CTAS = 2: on a CTA pair, called by the even CTA's warp.
template <int CTAS = 1>
__device__ __forceinline__ void mma_f16_lead(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t accumulate, bool lead) {
  if constexpr (CTAS == 1)
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"((uint32_t)lead)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"((uint32_t)lead)
        : "memory");
}

// Arrive once on `bar` (CTAS = 2: of the CTAs in `mask`) when the leading
// lane's earlier MMAs have completed.
template <int CTAS = 1>
__device__ __forceinline__ void mma_commit_lead(uint32_t bar, bool lead, uint16_t mask = 0x3) {
  if constexpr (CTAS == 1)
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
            bar),
        "r"((uint32_t)lead)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
        " [%0], %2;\n}\n" ::"r"(bar),
        "r"((uint32_t)lead), "h"(mask)
        : "memory");
}

// Bounded wait by a whole warp; all lanes agree on the outcome.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, unsigned *status,
                                               unsigned code, uint64_t limit_ns) {
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, status, code, limit_ns));
}

// ---- CTA pairs: clusters of two CTAs sharing one tcgen05 MMA ------------------
//
// With .cta_group::2 one thread of the even CTA issues an MMA of M = 256
// rows: each CTA of the pair holds 128 rows of A and half of the N columns
// of B in its own shared memory at the same offsets, and receives its 128
// accumulator rows in its own TMEM.  Every tcgen05 instruction of such a
// kernel that takes .cta_group uses ::2.

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// All threads of both CTAs; orders earlier shared-memory writes (barrier
// initialisation included) before the peer's later accesses.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The two halves of cluster_sync, for work between them: arrive (release:
// this thread's earlier accesses, reads of peers' shared memory included,
// are done before a peer passes its wait) and wait (acquire).
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// shared::cluster address of the object at shared::cta address `addr` in
// the CTA of cluster rank `rank`.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// 32-bit load from distributed shared memory (a shared::cluster address).
__device__ __forceinline__ uint32_t ld_shared_cluster_u32(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}

// Arrive on an mbarrier given by its shared::cluster address (possibly in
// the peer CTA), releasing this thread's earlier memory operations.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}

// The same without release semantics: for a consumer whose reads are
// complete before it arrives (tcgen05.ld followed by tcgen05.wait::ld), so
// the arrive orders nothing and needs no cluster-scope fence.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                   cluster_addr)
               : "memory");
}

// 3-D tiled load into this CTA's shared memory whose completion is counted
// on an mbarrier of either CTA of the pair (shared::cluster address).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *m,
                                                 uint32_t bar_cluster, int32_t x, int32_t y,
                                                 int32_t z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"((uint64_t)m), "r"(bar_cluster), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// One warp of EACH CTA of the pair executes these collectively.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

}  // namespace tc

// Host: encode a 2-D bf16 K-major tensor map (rows x cols, row pitch in
// elements) with a box of box_cols x box_rows and 128-byte swizzle.
// Defined in tma_host.cpp.
cudaError_t make_tmap_2d(CUtensorMap *m, const void *base, CUtensorMapDataType dtype,
                         int elem_bytes, uint64_t rows, uint64_t cols, uint64_t pitch_elems,
                         uint32_t box_rows, uint32_t box_cols);

// Host: `planes` stacked row-major rows x cols matrices (plane pitch
// rows * pitch_elems elements) as one 3-D tensor map with box
// {box_cols, box_rows, 1} and 128-byte swizzle; out-of-range rows of a
// plane read as zero.
cudaError_t make_tmap_3d(CUtensorMap *m, const void *base, CUtensorMapDataType dtype,
                         int elem_bytes, uint64_t planes, uint64_t rows, uint64_t cols,
                         uint64_t pitch_elems, uint32_t box_rows, uint32_t box_cols);

}  // namespace numc_k
