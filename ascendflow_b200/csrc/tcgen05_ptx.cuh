// Thin inline-PTX wrappers for the Blackwell (sm_100a) tensor path: mbarriers with bounded
// waits, tensor memory allocation, tcgen05.mma issue / commit, tcgen05.ld / st, and the shared
// memory and instruction descriptors those instructions take.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sm100 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- programmatic dependent launch -------------------------------------------------------------

// A kernel launched with programmatic stream serialisation may start while the kernel before it in
// the stream is still running. Nothing that kernel writes (or reads, if this one overwrites it) is
// touched before `wait_for_predecessor`: it returns when that kernel has completed and its memory
// is visible.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
// The kernel behind this one may be started (it waits by itself for this one's completion).
__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

__device__ __forceinline__ void prefetch_l2(const void* at) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(at)); }

// Launch `kernel` so that its start overlaps its predecessor's end.
template <typename Kernel, typename... Arguments>
inline cudaError_t launch_overlapped(Kernel kernel, int grid, int threads, size_t shared_bytes, cudaStream_t stream, const Arguments&... arguments) {
  cudaLaunchAttribute overlap = {};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(grid));
  config.blockDim = dim3(unsigned(threads));
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  config.attrs = &overlap;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, arguments...);
}

// ---- barriers of some of a block's warps --------------------------------------------------------

__device__ __forceinline__ void named_barrier_sync(int id, int threads) { asm volatile("barrier.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void named_barrier_arrive(int id, int threads) { asm volatile("barrier.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }

// In how many of `threads` threads (whole warps), all of which come here, `flag` is set.
__device__ __forceinline__ uint32_t named_barrier_count(int id, int threads, bool flag) {
  uint32_t count;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "barrier.red.popc.u32 %0, %2, %3, p;\n"
      "}\n"
      : "=r"(count) : "r"(uint32_t(flag)), "r"(id), "r"(threads) : "memory");
  return count;
}

// ---- mbarrier -----------------------------------------------------------------------------

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// Arrive, and expect `bytes` of bulk copies in the current phase besides.
__device__ __forceinline__ void mbar_arrive_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
// kCluster: what completes the phase are stores and copies of other blocks of the cluster. They release at cluster
// scope, and a wait synchronises with them only if it acquires at that scope (the default is the block's own).
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  if constexpr (kCluster) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  } else {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  }
  return done != 0;
}

// Wait for the phase with the given parity, giving up after `limit` SM clock cycles or as soon
// as `*abort_flag` (shared memory) is non-zero. Returns false when it gave up; the caller must
// then leave its loop and go to the kernel's common exit.
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          long long limit = (1ll << 31)) {
  if (mbar_try_wait<kCluster>(bar, parity)) return true;
  const long long start = clock64();
  int spins = 0;
  while (!mbar_try_wait<kCluster>(bar, parity)) {
    if ((++spins & 63) == 0) {
      if (*abort_flag != 0) return false;
      if (clock64() - start > limit) { *abort_flag = 1; return false; }
    }
  }
  return true;
}

// ---- proxies and tcgen05 ordering ------------------------------------------------------------

// Make generic-proxy shared memory writes that happened before (this thread's own, and those that a
// barrier has ordered before it) visible to the async proxy (tcgen05.mma operand reads, TMA).
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// ---- clusters and distributed shared memory ------------------------------------------------------------

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  return rank;
}
// The cluster's barrier, executed by every thread of every block: first arrive, then wait.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
// The same for threads whose writes nobody in the cluster reads behind the barrier.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }
// Address of this block's shared-memory word `address` in the block of rank `rank`.
__device__ __forceinline__ uint32_t cluster_address(uint32_t address, uint32_t rank) {
  uint32_t mapped;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(mapped) : "r"(address), "r"(rank));
  return mapped;
}
// Store to another block; counts as four bytes on that block's barrier `bar`.
__device__ __forceinline__ void cluster_store_async(uint32_t address, float value, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n"
               ::"r"(address), "r"(__float_as_uint(value)), "r"(bar) : "memory");
}
// Copy shared memory of this block to another block of the cluster (16-byte aligned addresses, a
// multiple of 16 bytes); counts as `bytes` on that block's barrier.
__device__ __forceinline__ void bulk_copy_to_block(uint32_t target, uint32_t source, uint32_t bytes, uint32_t target_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(target), "r"(source), "r"(bytes), "r"(target_bar) : "memory");
}

// ---- tensor memory ---------------------------------------------------------------------------

// Warp-collective. Writes the base address of `columns` (power of two, >= 32) to `*slot` in smem.
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(columns) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(columns) : "memory");
}

// ---- descriptors -----------------------------------------------------------------------------

// Shared memory matrix descriptor, 128-byte swizzle. `lbo` / `sbo` in bytes.
//  K-major operand (rows of 128 bytes, 8-row groups `sbo` apart): lbo is ignored by the hardware.
//  MN-major operand (64 contiguous MN elements per 128-byte row, rows are K): lbo = distance
//  between 64-element MN blocks, sbo = distance between 8-row K groups.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= uint64_t((addr & 0x3FFFF) >> 4);
  d |= uint64_t((lbo >> 4) & 0x3FFF) << 16;
  d |= uint64_t((sbo >> 4) & 0x3FFF) << 32;
  d |= uint64_t(1) << 46;  // descriptor version for sm_100
  d |= uint64_t(2) << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16 with FP32 accumulation. format: 0 = f16, 1 = bf16.
// a_mn / b_mn: 1 when that operand is MN-major in shared memory. kSparseA: A is 2:4 sparse.
constexpr uint32_t kSparseA = 1u << 2;
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n, int format, int a_mn, int b_mn) {
  return (1u << 4) | (uint32_t(format) << 7) | (uint32_t(format) << 10) | (uint32_t(a_mn) << 15) |
         (uint32_t(b_mn) << 16) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

// ---- MMA issue (one thread) ------------------------------------------------------------------

// True in one thread of the warp, always the same one. Who issues products is chosen by this and not by a comparison of the thread index, from
// which the compiler cannot tell that a single thread runs. Measured against `lane == 0`: one token 10.6 -> 9.3 us,
// 16 tokens 11.0 -> 9.6, 256 tokens at 4K 30.6 -> 29.9, prefill of 8K tokens 824 -> 809, 23 mixed requests 163.9 -> 160.2.
__device__ __forceinline__ bool elect_one() {
  uint32_t elected;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(elected));
  return elected != 0;
}

// The accumulate flag is a template argument: no predicate set-up per instruction, and the issuing
// thread's unrolled sequences carry nothing but immediates.
//
// The form with a 2:4 sparse A: of every four neighbours along K a row of A holds two, and the metadata (two
// bits for each of these: its place among the four) lies in tensor memory at `meta_tmem`. K = 32 per instruction.
template <bool kAccumulate>
__device__ __forceinline__ void mma_sparse_ts_c(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t meta_tmem, uint32_t idesc) {
  if constexpr (kAccumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.eq.b32 p, 0, 0;\n"
        "tcgen05.mma.sp.cta_group::1.kind::f16 [%0], [%1], %2, [%3], %4, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(meta_tmem), "r"(idesc) : "memory");
  } else {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, 0, 0;\n"
        "tcgen05.mma.sp.cta_group::1.kind::f16 [%0], [%1], %2, [%3], %4, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(meta_tmem), "r"(idesc) : "memory");
  }
}
// Weight-stationary form (tcgen05.mma.ws): with M = 64 the accumulator spreads over all 128
// tensor-memory lanes (lanes 0-63 hold rows 0-63 x columns [0, N/2), lanes 64-127 hold the same
// rows x columns [N/2, N); N/2 tensor-memory columns), and the instruction runs at 80 % of the
// M = 128 rate where the plain M = 64 form runs at 50 %.
template <bool kAccumulate>
__device__ __forceinline__ void mma_ws_ss_c(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  if constexpr (kAccumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.eq.b32 p, 0, 0;\n"
        "tcgen05.mma.ws.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc) : "memory");
  } else {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, 0, 0;\n"
        "tcgen05.mma.ws.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc) : "memory");
  }
}
// Arrive on `bar` once all tcgen05.mma issued so far by this thread have completed.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

// ---- tensor memory loads / stores (warp-collective; lane i of warp w touches TMEM lane
// 32*(w%4)+i, `taddr` carries that lane base in bits 31:16) --------------------------------------

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// Two 16-lane accesses in one load: threads 0-15 of the warp receive 16 consecutive columns of the
// 16 lanes at `taddr`'s lane, threads 16-31 receive the 16 columns kSplit further right of the SAME
// 16 lanes (`taddr`'s lane field is the warp's lane base + 0 or + 16).
template <int kSplit>
__device__ __forceinline__ void tmem_ld16_halves(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x32bx2.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16], %17;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr), "n"(kSplit) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 32 columns of 16 lanes (`taddr`'s lane field is the warp's lane base + 0 or + 16). Of every eight columns thread t
// gives four: 2 (t % 4) and 2 (t % 4) + 1 of lane t / 4, then the same of lane t / 4 + 8.
__device__ __forceinline__ void tmem_st_16x256b(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

}  // namespace sm100
