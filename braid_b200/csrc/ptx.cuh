// Thin inline-PTX wrappers for the sm_100a features the kernels use:
// mbarrier, TMA (cp.async.bulk.tensor), tcgen05 (MMA / TMEM / commit) and
// thread-block-cluster shared memory.  Every wait here is bounded.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace bq {

// Status codes mirrored from include/braid_b200.h (kept numerically identical).
constexpr int kOk = 0;
constexpr int kErrBadArg = 1;
constexpr int kErrUnsupported = 2;
constexpr int kErrLaunch = 3;
constexpr int kErrWorkspace = 4;
constexpr int kErrDeviceWait = 5;
constexpr int kErrNoDriver = 6;
constexpr int kErrTooLarge = 7;

// Upper bound of any device-side spin, in SM clock cycles (~0.5 s at 1.9 GHz).
// A wait that runs out records an error and the kernel unwinds; it never hangs.
constexpr long long kSpinLimitCycles = 1000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// ---- mbarrier -------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t issue, uint32_t bar, uint32_t bytes) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "setp.ne.b32 e, %2, 0;\n"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n"
      "}\n" ::"r"(bar), "r"(bytes), "r"(issue)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Has the phase completed?  Never suspends the thread.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait on an mbarrier phase.  Returns false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > kSpinLimitCycles) return false;
  }
  return true;
}

// ---- L2 cache policies ------------------------------------------------------
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// ---- instructions that one thread issues ------------------------------------------
// TMA copies, MMAs and commits take an `issue` operand and are predicated on it: the whole warp walks the
// issuing loop in step and one elected lane issues.  Their operands live in uniform registers; inside
// `if (elect_one())` every descriptor was moved there lane-wise first.  Clocks of the MMA warp per K block of the
// K-sliced decode kernel, all tiles in shared memory: 390 inside the branch (50 for an MMA, 45 for the commit, 60 for
// each of two barriers that had completed), 275 in step (16, 40, 85), of which the barriers are taken off the
// path by looking at the next block's before this one's MMAs.  Four graphed decoder layers of hidden 4096:
// 1 row 233.0 -> 216.5 us, 27 rows 277.9 -> 265.2, 128 rows 317.4 -> 313.2.

// ---- TMA --------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* tm) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tm) : "memory");
}
// 2-D tiled load into this CTA's shared memory; x is the innermost (K, bytes for
// u8 tensors) coordinate and must be a multiple of 16.
__device__ __forceinline__ void tma_load_2d(uint32_t issue, uint32_t dst, const CUtensorMap* tm, uint32_t bar,
                                            int x, int y, uint64_t policy) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "setp.ne.b32 e, %6, 0;\n"
      "@e cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      ".L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;\n"
      "}\n"
      ::"r"(dst), "l"(tm), "r"(bar), "r"(x), "r"(y), "l"(policy), "r"(issue)
      : "memory");
}

// Untiled bulk copy of `bytes` contiguous bytes from global memory into this CTA's shared
// memory, completion counted on an mbarrier.  Both addresses 16-byte aligned, `bytes` a
// multiple of 16.
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar,
                                             uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1], %2, [%3], %4;"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}

// 2-D tiled store from this CTA's shared memory (bulk async-group completion); the part of the
// box outside the tensor is not written.  x is the innermost coordinate: x * element size must
// be a multiple of 16 bytes, and no coordinate may be negative.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(tm), "r"(src), "r"(x), "r"(y)
               : "memory");
}

// ---- tcgen05 ----------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_result),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
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
// D[tmem] (+)= A[smem] * B[smem], e4m3 x e4m3 -> fp32; one thread issues.
__device__ __forceinline__ void mma_f8(uint32_t issue, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 e, %5, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], 16-bit x 16-bit (f16 or bf16, per the instruction descriptor)
// -> fp32; K = 16 elements per instruction.
__device__ __forceinline__ void mma_f16(uint32_t issue, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 e, %5, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}
// Arrive on an mbarrier once every MMA issued so far by this thread has retired.
__device__ __forceinline__ void mma_commit(uint32_t issue, uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "setp.ne.b32 e, %1, 0;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(bar), "r"(issue)
      : "memory");
}
// 16 consecutive fp32 columns of this warp's 32 TMEM lanes -> registers.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major operand tile whose rows are one
// 128-byte swizzle span (TMA SWIZZLE_128B): 8-row groups are 1024 bytes apart.
//   bits [0,14)  start address >> 4          bits [16,30) leading byte offset >> 4 (1: unused)
//   bits [32,46) stride byte offset >> 4     bits [46,48) descriptor version (1 on sm_100)
//   bits [61,64) layout type (2 = 128-byte swizzle)
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// Instruction descriptor for kind::f8f6f4, e4m3 x e4m3 -> fp32, both K-major.
//   bits [4,6) D format (1 = f32)   [7,10) A format (0 = e4m3)   [10,13) B format
//   bit 15/16 A/B major (0 = K)     [17,23) N >> 3               [24,29) M >> 4
__host__ __device__ constexpr uint32_t idesc_e4m3(int mma_m, int mma_n) {
  return (1u << 4) | (static_cast<uint32_t>(mma_n >> 3) << 17) |
         (static_cast<uint32_t>(mma_m >> 4) << 24);
}

// Instruction descriptor for kind::f16 with both operands of one 16-bit type (fmt 0 = f16,
// 1 = bf16), fp32 accumulation, both K-major; same field positions as above.
__host__ __device__ constexpr uint32_t idesc_f16(int mma_m, int mma_n, int fmt) {
  return (1u << 4) | (static_cast<uint32_t>(fmt) << 7) | (static_cast<uint32_t>(fmt) << 10) |
         (static_cast<uint32_t>(mma_n >> 3) << 17) | (static_cast<uint32_t>(mma_m >> 4) << 24);
}

// ---- CTA pairs (cta_group::2): one MMA spans two SMs ---------------------------------
// In a cluster of two, bit 24 of a shared-memory address selects the CTA of the pair;
// clearing it names the same offset in the even (leader) CTA.
constexpr uint32_t kPeerBitMask = 0xFEFFFFFFu;

// 2-D tiled load into THIS CTA's shared memory whose completion is counted on the
// mbarrier at the same offset in the pair's leader CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t issue, uint32_t dst, const CUtensorMap* tm,
                                                 uint32_t bar_in_leader, int x, int y,
                                                 uint64_t policy) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "setp.ne.b32 e, %6, 0;\n"
      "@e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      ".L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;\n"
      "}\n"
      ::"r"(dst), "l"(tm), "r"(bar_in_leader & kPeerBitMask), "r"(x), "r"(y), "l"(policy), "r"(issue)
      : "memory");
}
// 3-D form of the same.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t issue, uint32_t dst, const CUtensorMap* tm, uint32_t bar_in_leader, int x,
                                                 int y, int z, uint64_t policy) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "setp.ne.b32 e, %7, 0;\n"
      "@e cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      ".L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;\n"
      "}\n"
      ::"r"(dst), "l"(tm), "r"(bar_in_leader & kPeerBitMask), "r"(x), "r"(y), "r"(z), "l"(policy), "r"(issue)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_result),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// D[256 x N] (+)= A[256 x 32] * B[N x 32]^T over the pair: each CTA holds 128 rows of A,
// N/2 rows of B and 128 rows of D.  Issued by one thread of the leader CTA.
__device__ __forceinline__ void mma_f8_pair(uint32_t issue, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 e, %5, 0;\n"
      "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}
// The same for one 16-bit type (f16 or bf16, per the instruction descriptor), K = 16 elements.
__device__ __forceinline__ void mma_f16_pair(uint32_t issue, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 e, %5, 0;\n"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}
// Arrive on the mbarrier at this offset in BOTH CTAs of the pair once every pair MMA issued so far by this
// thread has retired.
__device__ __forceinline__ void mma_commit_pair(uint32_t issue, uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      ".reg .b16 both;\n"
      "mov.b16 both, 3;\n"
      "setp.ne.b32 e, %1, 0;\n"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], both;\n"
      "}\n" ::"r"(bar), "r"(issue)
      : "memory");
}
// Plain arrival on an mbarrier that may live in another CTA of the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr)
               : "memory");
}

// ---- programmatic dependent launch -------------------------------------------------
// Lets the next kernel in the stream begin (its own set-up, loads that do not depend on
// this kernel) before this one has finished.
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Blocks until every kernel this one depends on has completed and its writes are visible.
// A no-op when the kernel was launched without the programmatic attribute.
__device__ __forceinline__ void pdl_wait_prior_grids() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// What an earlier kernel writes, read behind that wait.  `__ldg` would tell the compiler that nobody
// writes it, and the load could be moved above the wait; volatile keeps it in its place.  Through
// the L1, which serves the twelve warps of a CTA that read one word: with `ld.global.cg` for the
// activation scale and the residual, four graphed decoder layers of 1 row took 257 us, not 254.
__device__ __forceinline__ float ld_coherent4(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_coherent8(const void* p) {
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ld_coherent16(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// ---- phase stamps (development builds only: -DBQ_PHASES) ------------------------------------
// A build with BQ_PHASES records nanosecond stamps (%globaltimer) of the phases of every CTA of
// the decode-regime kernels into a ring in device memory; the shipped library compiles none of
// it.  Ring layout: [launch % kPhaseLaunches][cta < kPhaseCtas][kPhaseWords] of u64; word 8 is
// the SM id, word 9 is (grid << 8 | kind) with kind 0 = GEMM, 1 = quantizer.
constexpr int kPhaseLaunches = 1024, kPhaseCtas = 256, kPhaseWords = 10;
#ifdef BQ_PHASES
unsigned long long* phase_ring_for_launch(int* seq_out);   // host; cabi.cu
__device__ __forceinline__ void phase_stamp(unsigned long long* ring, int seq, int idx) {
  if (ring == nullptr || blockIdx.x >= kPhaseCtas) return;
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  ring[((size_t)(seq % kPhaseLaunches) * kPhaseCtas + blockIdx.x) * kPhaseWords + idx] = t;
}
__device__ __forceinline__ void phase_meta(unsigned long long* ring, int seq, int kind) {
  if (ring == nullptr || blockIdx.x >= kPhaseCtas) return;
  unsigned int smid;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
  unsigned long long* at = ring + ((size_t)(seq % kPhaseLaunches) * kPhaseCtas + blockIdx.x) * kPhaseWords;
  at[8] = smid;
  at[9] = ((unsigned long long)gridDim.x << 8) | (unsigned long long)kind;
}
#define BQ_STAMP(p, idx) ::bq::phase_stamp((p).phase_ring, (p).phase_seq, (idx))
#define BQ_STAMP_META(p, kind) ::bq::phase_meta((p).phase_ring, (p).phase_seq, (kind))
#else
#define BQ_STAMP(p, idx) ((void)0)
#define BQ_STAMP_META(p, kind) ((void)0)
#endif

// ---- thread-block clusters ----------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
// The two halves of it; the first one orders nothing.
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory offset inside CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
__device__ __forceinline__ void st_cluster_f1(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// A word into another CTA's shared memory, its four bytes counted on a barrier there.
__device__ __forceinline__ void st_async_cluster(uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar)
               : "memory");
}
// mbar_wait for a barrier that other CTAs of the cluster complete with what they stored.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok != 0) return true;
    if (clock64() - t0 > kSpinLimitCycles) return false;
  }
}
__device__ __forceinline__ float ld_cluster_f1(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

}  // namespace bq
