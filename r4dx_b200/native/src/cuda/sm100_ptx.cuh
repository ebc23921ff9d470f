// Thin inline-PTX layer for the Blackwell (sm_100a) asynchronous machinery used by the GEMM
// kernels: mbarrier, TMA (cp.async.bulk / cp.async.bulk.tensor, never with cluster multicast),
// tcgen05 (TMEM allocation, UMMA issue, commit, TMEM loads) and the UMMA descriptors.
//
// Every wait is bounded: a spin that runs out sets a status word and returns false so that the
// kernel can unwind (free TMEM, return) instead of hanging the GPU.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace r4dxb {
namespace ptx {

__device__ __forceinline__ uint32_t SmemAddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// ---- mbarrier ------------------------------------------------------------------------------------
__device__ __forceinline__ void MbarInit(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void MbarFenceInit() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void MbarArrive(uint64_t* bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(SmemAddr(bar)) : "memory");
}
__device__ __forceinline__ void MbarArriveExpectTx(uint64_t* bar, uint32_t bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(SmemAddr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool MbarTryWait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(SmemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool MbarTestWait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(SmemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// try_wait that lets the hardware park the thread for up to `hint_ns` before it answers "not yet": a waiting
// thread then costs an issue slot every few microseconds instead of every few dozen clocks.
__device__ __forceinline__ bool MbarTryWaitHint(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(SmemAddr(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Bounded wait.  `abort_flag` is a shared-memory word any role sets when it gives up; everyone who
// sees it leaves too.  Returns false on abort / timeout (about a second of SM clocks).
// (A suspend-time hint on try_wait - MbarTryWaitHint - was measured too: it changed neither the weight-streaming
// kernel nor the GEMM, so the plain form stays.)
constexpr int kSpinLimit = 1 << 22;
constexpr long long kWaitClocks = 2000000000ll;
__device__ __forceinline__ bool MbarWait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  if (MbarTestWait(bar, parity)) return true;      // the common case in a well-fed pipeline: no suspension at all
  const long long t0 = clock64();
  for (;;) {
    if (MbarTryWait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitClocks) break;
  }
  *abort_flag = code;
  return false;
}
// The same for a whole (converged) warp: one lane polls, the others sleep in the shuffle.  Thirty-two lanes
// polling one barrier word serialise in the shared-memory pipe and slow down every other barrier
// operation of the SM (measured: a satisfied test_wait of another warp went from 15 to ~300 clocks).
__device__ __forceinline__ bool WarpMbarWait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = MbarWait(bar, parity, abort_flag, code) ? 1 : 0;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// The same operations on shared-memory addresses the caller keeps in registers: converting a generic pointer costs about ten
// instructions each time, which a producer that issues several small copies per stage cannot afford.
__device__ __forceinline__ void MbarArriveAt(uint32_t bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void MbarArriveExpectTxAt(uint32_t bar, uint32_t bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool MbarTryWaitAt(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool MbarTestWaitAt(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool MbarWaitAt(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
  if (MbarTryWaitAt(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (MbarTryWaitAt(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitClocks) break;
  }
  *abort_flag = code;
  return false;
}
__device__ __forceinline__ void BulkLoadAt(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(bar) : "memory");
}

// ---- pairs of floats ------------------------------------------------------------------------------------
__device__ __forceinline__ float2 Add2(float2 a, float2 b) {
  float2 d;
  asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z; }"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 Fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{ .reg .b64 x, y, z, w; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 z, {%6, %7}; fma.rn.f32x2 w, x, y, z; mov.b64 {%0, %1}, w; }"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// ---- clusters ------------------------------------------------------------------------------------------
// Barrier over every thread of the cluster; shared-memory writes before it are visible to the peers after it.
__device__ __forceinline__ void ClusterSync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t ClusterRank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The shared-memory address `addr` (of this CTA's window) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t MapToRank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Arrival at a barrier of another CTA (`bar` from MapToRank).  With the default scope: what the arrival announces are operands of a
// paired product, which the writers have handed to the async proxy (fence.proxy.async) or which a TMA load has written; an arrival
// with cluster scope took 1300 to 1900 clocks in the product's main loop.
__device__ __forceinline__ void MbarArriveRemote(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// 16 bytes at the shared-memory address `addr` (of this CTA's window) in CTA `rank` of the cluster.
__device__ __forceinline__ float4 LoadRemote4(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile("{ .reg .b32 a; mapa.shared::cluster.u32 a, %4, %5; ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a]; }"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}

// ---- proxies / fences ------------------------------------------------------------------------------
__device__ __forceinline__ void FenceProxyAsyncShared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void TcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void TcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- TMA ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void PrefetchTensorMap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load into shared memory of this CTA; completion on `bar` (complete_tx bytes).
// x is the innermost coordinate: x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void TmaLoad2D(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(SmemAddr(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(SmemAddr(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void TmaLoad2DAt(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// Untiled bulk copy global -> shared; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void BulkLoad(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(SmemAddr(smem_dst)), "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(SmemAddr(bar))
      : "memory");
}

// Untiled bulk copy shared -> global (of this GPU), both 16-byte aligned, in the issuing thread's bulk groups; the generic writes it
// reads were made visible with FenceProxyAsyncShared.
__device__ __forceinline__ void BulkStore(void* gdst, uint32_t smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(reinterpret_cast<uint64_t>(gdst)), "r"(smem_src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void BulkStoreCommit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void BulkStoreWaitRead() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void BulkStoreWait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- tensor memory ------------------------------------------------------------------------------------
// CTAs of a cluster that hold tensor memory while they wait for each other can lock up: one waits for columns that a CTA of another
// such cluster (of a launch on another stream) holds, whose partner waits for columns that the first one's partner holds.  Shared
// memory keeps them apart: an SM has 228 KB, 1 KB of it reserved per CTA.
//   prefill attention, pairs: kClusterAlone or more (all tensor memory)
//   trellis product, pairs and splits: kProductAlone or more
//   plain linears with a split of K: kClusterShared or more, so two at most on an SM, and none beside the others
// The sizes are the last ones below a step of the split of 228 KB between shared memory and L1 (132 and, for two CTAs, 196 KB): with
// 112 KB a w4a16 linear of 5120 x 17408, whose weights are read through the L1, took 72 us at 64 rows where it takes 67.
// (The waits of the weight-streaming kernel of trellis_gemv_mma.cu for its cluster are bounded: beside it a launch may be late, never stuck.)
constexpr size_t kClusterAlone = 131 * 1024, kProductAlone = 176 * 1024, kClusterShared = 96 * 1024;
static_assert(kClusterAlone + kClusterShared + 2 * 1024 > 228 * 1024 && 2 * (kClusterShared + 1024) <= 228 * 1024 &&
              kClusterAlone <= kProductAlone, "none of the first two kinds meets one of the three");
// Whole-warp calls (.sync.aligned).  Columns: power of two, 32..512.
__device__ __forceinline__ void TmemAlloc(uint32_t* smem_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(smem_result)), "r"(columns)
               : "memory");
}
__device__ __forceinline__ void TmemRelinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void TmemDealloc(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}

// The same for a pair of CTAs (cta_group::2): a warp of each takes part, and both get the same columns.
__device__ __forceinline__ void TmemAllocPair(uint32_t* smem_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(smem_result)), "r"(columns)
               : "memory");
}
__device__ __forceinline__ void TmemRelinquishPair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void TmemDeallocPair(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}

// ---- UMMA --------------------------------------------------------------------------------------------------
// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, rows of 128 bytes, 8-row
// groups 1024 bytes apart (tile base must be 1024-byte aligned).
__device__ __forceinline__ uint64_t UmmaDescSw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);        // start address
  d |= static_cast<uint64_t>(1) << 16;                            // leading byte offset (unused with swizzle)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                    // stride byte offset between 8-row groups
  d |= static_cast<uint64_t>(1) << 46;                            // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;                            // SWIZZLE_128B
  return d;
}
// Instruction descriptor, kind::f16: fp16 (or bf16) A and B, both K-major, fp32 accumulate.
__host__ __device__ constexpr uint32_t UmmaInstrDescF16(int M, int N, bool bf16) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}
// D[tmem] (+)= A[smem] * B[smem]^T, issued by ONE thread.
__device__ __forceinline__ void UmmaF16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same over a pair of CTAs, issued by ONE thread of the first: A rows 0..127 and the first half of the B rows come from the
// first CTA's shared memory, the others from the second's (same addresses); each CTA's tensor memory gets its 128 rows of D.
__device__ __forceinline__ void UmmaF16Pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// kind::f8f6f4 with e4m3 A and B (format code 0 for both), both K-major, fp32 accumulate; K = 32 per instruction.
__host__ __device__ constexpr uint32_t UmmaInstrDescE4m3(int M, int N) {
  return (1u << 4) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}
__device__ __forceinline__ void UmmaF8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p; }"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives once on `bar` when every MMA issued so far by this thread has finished.
__device__ __forceinline__ void UmmaCommit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(SmemAddr(bar)) : "memory");
}
__device__ __forceinline__ void UmmaCommitAt(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// For a pair: arrives on the barrier at the same address in every CTA of the mask (bit = rank in the cluster).
__device__ __forceinline__ void UmmaCommitPairAt(uint32_t bar, uint16_t ctas) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(ctas) : "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread t of the warp reads TMEM lane (base lane + t).
__device__ __forceinline__ void TmemLoad32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void TmemLoad32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void TmemLoadWait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 lanes x 16 consecutive 32-bit columns: thread t of the warp writes TMEM lane (base lane + t).
__device__ __forceinline__ void TmemStore32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void TmemStoreWait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major operand without swizzle: 8-row x 16-byte core matrices
// (128 contiguous bytes each); `lbo` = bytes between the two core matrices that are adjacent in K,
// `sbo` = bytes between 8-row groups.  The start address needs 16-byte alignment only.
__device__ __forceinline__ uint64_t UmmaDescNoSwizzle(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(lbo >> 4) << 16;
  d |= static_cast<uint64_t>(sbo >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;                            // descriptor version (Blackwell)
  return d;
}
// Instruction descriptor, kind::i8: unsigned 8-bit A, signed 8-bit B, both K-major, int32 accumulate.
__host__ __device__ constexpr uint32_t UmmaInstrDescU8S8(int M, int N) {
  return (2u << 4) | (0u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}
// D[tmem] (+)= A[tmem] * B[smem]^T on 8-bit integers (K = 32 per instruction), issued by ONE thread.
// A: lane = row, 8 consecutive 32-bit columns = the row's 32 K bytes.
__device__ __forceinline__ void UmmaI8FromTmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p; }"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]^T on fp16 inputs (K = 16 per instruction), fp32 accumulate, issued by ONE
// thread.  A: lane = row, 8 consecutive 32-bit columns = the row's 16 K values as half2 pairs.
__device__ __forceinline__ void UmmaF16FromTmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same over a pair of CTAs (see UmmaF16Pair): A rows 0..127 from the first CTA's tensor memory, the others from the second's.
__device__ __forceinline__ void UmmaF16PairFromTmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                                    uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p; }"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 32 lanes x 8 consecutive 32-bit columns.
__device__ __forceinline__ void TmemStore32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

__device__ __forceinline__ bool ElectOne() {
  uint32_t pred;
  asm volatile(
      "{ .reg .b32 r; .reg .pred p; elect.sync r|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(pred)::"memory");
  return pred != 0;
}

}  // namespace ptx

// ---- host: tensor map creation through the driver entry point (no link against libcuda) ---------------
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline PFN_encodeTiled GetEncodeTiled() {
  static PFN_encodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
    return reinterpret_cast<PFN_encodeTiled>(p);
  }();
  return fn;
}

// 2-D row-major tensor [rows, cols] of 2-byte elements, box [box_rows, box_cols], 128-byte swizzle.
// 2-D map over a row-major matrix of bytes (8-bit activations) with the 128-byte swizzle: box_cols bytes x box_rows rows.
inline int MakeTensorMap2D8(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols) {
  PFN_encodeTiled enc = GetEncodeTiled();
  if (!enc) return 10004;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 10005;
}

inline int MakeTensorMap2D16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows,
                             uint32_t box_cols, bool is_bf16) {
  PFN_encodeTiled enc = GetEncodeTiled();
  if (!enc) return 10004;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 10005;
}

}  // namespace r4dxb
