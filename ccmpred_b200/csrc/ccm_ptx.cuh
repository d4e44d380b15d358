// Inline-PTX wrappers for sm_100a: mbarriers, TMA tile loads, tcgen05 MMA,
// TMEM allocation and TMEM loads.  Every wait here is bounded: it gives up
// after a clock budget and reports failure to the caller, which records an
// error flag and leaves its loop instead of spinning forever.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace ccm {

// ~2 s at 2 GHz.  A legitimate wait in these kernels is at most one tile of
// MMAs plus one tile epilogue (well under a millisecond).
constexpr long long kWaitBudgetCycles = 4000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ----------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the phase with the given parity to complete; false once `budget`
// clock cycles have passed without it.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          long long budget = kWaitBudgetCycles) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > budget) return false;
  }
  return true;
}

// ---------------------------------------------------------------------- TMA
// 2-D tiled bulk tensor load global -> shared, completion signalled on `bar`
// as transaction bytes.  x is the innermost coordinate (elements).
__device__ __forceinline__ void tma_load_2d(void *smem_dst, const CUtensorMap *map, uint64_t *bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// Programmatic dependent launch.  griddep_wait: block until the previous kernel
// of the stream has completed and its writes are visible (a no-op for a kernel
// launched without the attribute); every kernel of the evaluation calls it before
// its first global-memory access.  griddep_launch: every CTA issues it when it
// starts; the next kernel of the stream is scheduled once all CTAs of this one
// have (its CTAs then take free SMs and wait in griddep_wait), so it never holds
// a slot that a CTA of this kernel still needs.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Make this thread's generic-proxy shared-memory writes visible to the async
// proxy (TMA, tcgen05.mma operand reads).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ------------------------------------------------------------------ tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
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

// D[tmem] (+)= A[smem] * B[smem], kind::f16 (bf16 inputs, f32 accumulate).
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive once on `bar` when all previously issued tcgen05 ops of this thread complete.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 lanes x 32 columns of 32-bit: thread i of the warp receives lane (base+i),
// columns [col, col+32).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
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
      : "r"(taddr)
      : "memory");
}

// Shared-memory matrix descriptor for a 128-byte-swizzled canonical layout
// (tcgen05 "shared memory descriptor": start>>4 @0, LBO>>4 @16, SBO>>4 @32,
// version 1 @46, swizzle mode 2 = 128B @61).
//  K-major:  rows of 128 B (64 bf16 along K), 8-row groups SBO apart; LBO unused.
//  MN-major: 64 MN-contiguous elements per 128 B row, one row per K index;
//            8-row K groups SBO apart, 64-element MN chunks LBO apart.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr, uint32_t lbo_bytes,
                                                uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// Same for the 64-byte swizzle (layout type 4): K-major rows of 64 B (32 bf16),
// 8-row groups of 512 B.
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr, uint32_t lbo_bytes,
                                               uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(4) << 61;
  return d;
}

// Instruction descriptor, kind::f16 with bf16 A/B and f32 D.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N, int a_mn_major,
                                                      int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_mn_major) << 15) |
         (static_cast<uint32_t>(b_mn_major) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

// Named barrier among `nthreads` threads (ids 1..15; 0 is __syncthreads).
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Named barrier with an OR-reduction of `pred` over the participating threads.
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred p, %2, %3, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)pred), "r"(id), "r"(nthreads)
      : "memory");
  return r != 0;
}

// Add v to *p if pred: a predicated reduction, without a branch (a branch per add
// costs a reconvergence, ~40 cycles of a warp's issue).
__device__ __forceinline__ void red_add_if(float *p, float v, bool pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "@p red.global.add.f32 [%0], %1;\n\t}\n" ::"l"(p),
      "f"(v), "r"((uint32_t)pred)
      : "memory");
}

// Four consecutive adds; p is 16-byte aligned.
__device__ __forceinline__ void red_add4_if(float *p, float4 v, bool pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %5, 0;\n\t"
      "@p red.global.add.v4.f32 [%0], {%1,%2,%3,%4};\n\t}\n" ::"l"(p),
      "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"((uint32_t)pred)
      : "memory");
}

// Register split between the warpgroups of a block (all four warps of a warpgroup
// execute one of these; the shares must add up to at most the launch's total).
template <int R> __device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R> __device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}

// 32-byte global store (one full sector); `p` must be 32-byte aligned.
__device__ __forceinline__ void st_global_v8(void *p, const uint32_t (&r)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// ------------------------------------------------------- CTA pairs (clusters of 2)
// A pair of CTAs (cluster ranks 0 and 1) shares one tcgen05 MMA of M = 256:
// each CTA holds half of A (its 128 rows) and half of B (128 of the N columns)
// in its own shared memory and half of D in its own TMEM; rank 0 (the leader)
// issues the MMAs.  Every tcgen05 instruction of such a kernel uses
// .cta_group::2.  No load in this file uses a multicast qualifier.

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// shared::cluster address of the same shared-memory offset in CTA `rank`.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}

// Arrive on an mbarrier given by its shared::cluster address.  The CTA-scope release
// (the default) is enough for what these barriers hand over, tensor memory read or
// written under tcgen05.wait and tcgen05.fence; a cluster-scope release takes about a
// thousand cycles.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// Whole-cluster barrier (all threads of both CTAs).  The non-.aligned form:
// threads of one warp may arrive from different branches.
__device__ __forceinline__ void cluster_sync() {
  asm volatile(
      "barrier.cluster.arrive.release;\n\t"
      "barrier.cluster.wait.acquire;" ::
          : "memory");
}

// 2-D tile load into this CTA's shared memory whose completion bytes are
// signalled on the mbarrier at shared::cluster address `bar` (the leader's).
__device__ __forceinline__ void tma_load_2d_pair(void *smem_dst, const CUtensorMap *map,
                                                 uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// Issued by the same warp in both CTAs; both receive the same TMEM address.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
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

// Pair MMA (leader only): D[tmem of both CTAs] (+)= A * B, kind::f16, M = 256.
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive once on the mbarrier at the same offset in every CTA of `cta_mask`
// when all previously issued tcgen05 ops of this thread complete.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar, uint16_t cta_mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;" ::"r"(smem_u32(bar)),
      "h"(cta_mask)
      : "memory");
}

// ------------------------------------------------------- integer MMA (kind::i8)
// Instruction descriptor, kind::i8 with s32 D: c_format 2 @4, A/B signedness
// (0 = u8, 1 = s8) @7/@10, A/B major @15/@16, N>>3 @17, M>>4 @24.
__host__ __device__ constexpr uint32_t idesc_i8_s32(int M, int N, int a_signed, int b_signed,
                                                    int a_mn_major, int b_mn_major) {
  return (2u << 4) | (static_cast<uint32_t>(a_signed) << 7) |
         (static_cast<uint32_t>(b_signed) << 10) | (static_cast<uint32_t>(a_mn_major) << 15) |
         (static_cast<uint32_t>(b_mn_major) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

// Pair MMA (leader only): D[s32, tmem of both CTAs] (+)= A * B, 8-bit integers, K = 32.
__device__ __forceinline__ void umma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ------------------------------------------------ sparse integer MMA (2:4 on A)
// Instruction descriptor bit 2: A is 2:4 structured-sparse, its metadata in TMEM.
constexpr uint32_t kIdescSparse = 1u << 2;

// Shared-memory descriptor, 32-byte swizzle (layout type 6).  MN-major: 32
// MN-contiguous bytes per row, one row per K index; 8-row K groups SBO apart,
// 32-byte MN atoms LBO apart.
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t saddr, uint32_t lbo_bytes,
                                               uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(6) << 61;
  return d;
}

// Shared-memory descriptor without swizzle (layout type 0): core matrices of
// 8 rows x 16 bytes stored as 128 contiguous bytes; 8-row groups SBO apart, core
// matrices along K LBO apart.
__device__ __forceinline__ uint64_t sdesc_noswz(uint32_t saddr, uint32_t lbo_bytes,
                                                uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}

// Leader only: copy 128 rows x 16 bytes from shared memory (descriptor `src`, in
// each CTA of the pair) to TMEM lanes 0..127, columns [taddr, taddr + 4), of the
// same CTA.  Ordered with the MMAs issued after it by the same thread.
__device__ __forceinline__ void tmem_cp_pair_128x128b(uint32_t taddr, uint64_t src) {
  asm volatile("tcgen05.cp.cta_group::2.128x128b [%0], %1;" ::"r"(taddr), "l"(src) : "memory");
}

// Pair MMAs (leader only) with 2:4-sparse A: D (+)= A * B, 8-bit integers, K = 64 logical
// each (32 stored bytes of A per row), metadata at TMEM column `meta` (two columns per
// instruction: 4 bits per group of four logical K).  One block of 128 logical K of the
// three digit products: hi += A1 B0, lo += A128 B1 + A1 B2 (the first ones overwrite
// unless `accumulate`).  a, b: low words of the descriptors of A x1 and of digit 0
// (k = 0); kA, kB: from there to A x128 and to the next digit; kAK, kBK: to k = 1.
// One asm statement: the sparse MMAs do not queue behind one another, so every
// instruction of the issuing thread between them is tensor time lost.
template <int kA, int kAK, int kB, int kBK>
__device__ __forceinline__ void umma_i8sp_block(uint32_t hi, uint32_t lo, uint32_t a, uint32_t a_top,
                                                uint32_t b, uint32_t b_top, uint32_t idesc,
                                                uint32_t meta, uint32_t accumulate) {
#define CCM_AT(D, FROM, OFF, TOP) "add.u32 w, " FROM ", " OFF ";\n\tmov.b64 " D ", {w, " TOP "};\n\t"
#define CCM_MMA(D, A, B, M, P) \
  "tcgen05.mma.sp.cta_group::2.kind::i8 [" D "], " A ", " B ", [" M "], %6, " P ";\n\t"
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b32 w, m1;\n\t"
      ".reg .b64 a0, a1, c0, c1, b00, b01, b10, b11, b20, b21;\n\t"
      "setp.ne.b32 p, %8, 0;\n\tsetp.eq.b32 q, %8, %8;\n\t"
      "add.u32 m1, %7, 2;\n\t"
      CCM_AT("a0", "%2", "0", "%3") CCM_AT("b00", "%4", "0", "%5")
      CCM_MMA("%0", "a0", "b00", "%7", "p")
      CCM_AT("c0", "%2", "%9", "%3") CCM_AT("b10", "%4", "%11", "%5")
      CCM_MMA("%1", "c0", "b10", "%7", "p")
      CCM_AT("b20", "%4", "%12", "%5")
      CCM_MMA("%1", "a0", "b20", "%7", "q")
      CCM_AT("a1", "%2", "%10", "%3") CCM_AT("b01", "%4", "%13", "%5")
      CCM_MMA("%0", "a1", "b01", "m1", "q")
      CCM_AT("c1", "%2", "%14", "%3") CCM_AT("b11", "%4", "%15", "%5")
      CCM_MMA("%1", "c1", "b11", "m1", "q")
      CCM_AT("b21", "%4", "%16", "%5")
      CCM_MMA("%1", "a1", "b21", "m1", "q")
      "}\n" ::"r"(hi), "r"(lo), "r"(a), "r"(a_top), "r"(b), "r"(b_top), "r"(idesc), "r"(meta),
      "r"(accumulate), "n"(kA), "n"(kAK), "n"(kB), "n"(2 * kB), "n"(kBK), "n"(kA + kAK),
      "n"(kB + kBK), "n"(2 * kB + kBK)
      : "memory");
#undef CCM_AT
#undef CCM_MMA
}

// The two words of a shared-memory descriptor (sdesc_* above): the low one moves with the
// address (in units of 16 bytes), the high one is a constant of the layout.
__host__ __device__ constexpr uint32_t sdesc_low(uint32_t saddr, uint32_t lbo_bytes) {
  return (saddr >> 4) | (lbo_bytes >> 4) << 16;
}
__host__ __device__ constexpr uint32_t sdesc_high(uint32_t sbo_bytes, uint32_t layout) {
  return (sbo_bytes >> 4) | 1u << 14 | layout << 29;
}

// 32 lanes x 32 columns of 32-bit, registers -> TMEM (the inverse of tmem_ld32).
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
      "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// 32 lanes x 16 columns of 32-bit (thread i: lane base+i, columns [col, col+16)).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

}  // namespace ccm
