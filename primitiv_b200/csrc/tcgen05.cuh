// Device-side building blocks of the tcgen05 kernels (gemm_tc.cu, gemm_direct.cu): mbarriers with bounded
// waits, TMA loads, MMA issue, tensor-memory loads, CTA pairs.
#ifndef PRIMITIV_B200_CSRC_TCGEN05_CUH_
#define PRIMITIV_B200_CSRC_TCGEN05_CUH_

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace b200 {
namespace {

constexpr uint32_t kKSteps = 4;  // MMAs per 128-byte k-block: 32 bytes of k each (8 tf32 / 16 fp16)
constexpr long long kWaitLimitCycles = 4000000000ll;  // about 2 s at boost clock, 4 s at the lowest

// Shared-memory descriptor fields of one operand plane: high half, fixed bits of the low half, and the
// advance per k-step in 16-byte units.
struct MixDesc {
  uint32_t hi, lo_fixed, kstep;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done;
}

// Bounded wait.  Returns false if the CTA is aborting or the limit ran out (in
// which case it raises the abort flag itself).  The limit is counted in SM clock
// cycles (%clock64 is a few cycles to read; %globaltimer costs hundreds of nanoseconds
// per read and, on the path every pipeline stage takes, was itself the bottleneck),
// and the clock is only consulted after a run of failed polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *s_abort,
                                          uint32_t sleep_ns = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  uint32_t spins = 0;
  long long t0 = 0;
  for (;;) {
    if (mbar_try_wait(bar, parity)) return true;
    if (sleep_ns) __nanosleep(sleep_ns);  // leave the issue slots to the warps that are not waiting
    if (++spins == 256u) t0 = clock64();
    if (spins > 256u && (spins & 255u) == 0u) {
      if (*s_abort) return false;
      if (clock64() - t0 > kWaitLimitCycles) {
        *s_abort = 1;
        return false;
      }
    }
  }
}

// A whole warp waits, but only lane 0 polls the barrier (32 pollers per warp on one
// shared-memory word slow everyone else's barrier traffic down).
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *s_abort, uint32_t lane) {
  uint32_t ok = 1u;
  if (lane == 0) {
    // The epilogue waits for a whole chunk of main loop: sleep between polls so that the
    // MMA issuer, which shares a scheduler with two epilogue warps, keeps its issue slots.
    ok = mbar_wait(bar, parity, s_abort, 256u) ? 1u : 0u;
  }
  return __shfl_sync(0xffffffffu, ok, 0) != 0u;
}

// Wait used only on the abort path: never raises anything, just gives up.
__device__ __forceinline__ void mbar_wait_quiet(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > kWaitLimitCycles / 4) return;
  }
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// One tcgen05.mma.  The 64-bit shared-memory descriptors are passed as 32-bit halves and
// assembled inside the asm block: the high half (stride offset, version, swizzle) never
// changes during a launch and the low half only advances by a constant per k-step, so the
// issuing thread spends a handful of instructions per MMA.  (With the descriptors rebuilt
// from scratch for every MMA the single issuing thread, sharing its scheduler with polling
// warps, could not feed the tensor core: ~190 ns per MMA whatever the tile width.)
#define B200_MMA_ASM(GROUP, KIND)                                                      \
  asm volatile(                                                                        \
      "{\n\t"                                                                          \
      ".reg .pred p, e;\n\t"                                                           \
      ".reg .b64 da, db;\n\t"                                                          \
      "elect.sync _|e, 0xffffffff;\n\t"                                                \
      "setp.ne.b32 p, %6, 0;\n\t"                                                      \
      "mov.b64 da, {%1, %2};\n\t"                                                      \
      "mov.b64 db, {%3, %4};\n\t"                                                      \
      "@e tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], da, db, %5, p;\n\t"    \
      "}\n" ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) \
      : "memory")

// Called by ALL 32 lanes of the converged MMA warp with warp-uniform arguments; the
// instruction itself is issued by the one lane elect.sync picks (the same lane every
// time for a full mask, so tcgen05.commit from that lane tracks these MMAs).
template <int kCtas, bool kF16>
__device__ __forceinline__ void mma_issue(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                          uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  if constexpr (kCtas == 2) {
    if constexpr (kF16) B200_MMA_ASM("2", "f16"); else B200_MMA_ASM("2", "tf32");
  } else {
    if constexpr (kF16) B200_MMA_ASM("1", "f16"); else B200_MMA_ASM("1", "tf32");
  }
}

// Runs the k-steps (and, for 3xTF32, the three hi/lo pass combinations) of one pipeline stage.
// Runs the k-steps (and, for 3xTF32, the three hi/lo pass combinations) of one k-block as
// straight-line code: every transfer of control between two MMAs showed up as a gap in the
// tensor pipe, so a pipeline stage is one basic block of 8 (single-pass, two k-blocks) or 12
// (3xTF32) MMAs.
template <int kCtas, bool kF16, int kPasses>
__device__ __forceinline__ void mma_stage(uint32_t d_tmem, uint32_t sa, uint32_t sb, uint32_t a_plane, uint32_t b_plane,
                                          uint32_t a_hi, uint32_t b_hi, uint32_t a_lo_fixed, uint32_t b_lo_fixed,
                                          uint32_t kstep_a, uint32_t kstep_b, uint32_t idesc, bool first) {
  uint32_t acc = first ? 0u : 1u;
#pragma unroll
  for (int ps = 0; ps < kPasses; ++ps) {
    // 3xTF32: (lo, hi), (hi, lo), (hi, hi) -- small terms first
    const uint32_t ia = (kPasses == 3 && ps == 0) ? a_plane : 0u;
    const uint32_t ib = (kPasses == 3 && ps == 1) ? b_plane : 0u;
    uint32_t a_lo = a_lo_fixed | (((sa + ia) & 0x3FFFFu) >> 4);
    uint32_t b_lo = b_lo_fixed | (((sb + ib) & 0x3FFFFu) >> 4);
#pragma unroll
    for (uint32_t ks = 0; ks < kKSteps; ++ks) {
      mma_issue<kCtas, kF16>(d_tmem, a_lo, a_hi, b_lo, b_hi, idesc, acc);
      acc = 1u;
      a_lo += kstep_a;  // in 16-byte units; never carries out of the 14-bit address field within a stage
      b_lo += kstep_b;
    }
  }
}

// One k-block of the fp32 mode with bf16 correction passes (kind 4), as one basic block of
// 8 MMAs: (lo8, hi8) and (hi8, lo8) on the bf16 pipe, two k-steps of 16 each, then (hi, hi) in
// TF32, four k-steps of 8 -- small terms first, all into the same fp32 accumulator.  A stage
// holds [A hi | A hi8 | A lo8 | B hi | B hi8 | B lo8]; the bf16 planes are K-major rows of 64
// bytes under the 64-byte swizzle (descriptor layout 4, 8-row groups 512 bytes apart).
template <int kCtas>
__device__ __forceinline__ void mma_stage_mix(uint32_t d_tmem, uint32_t sa, uint32_t sb, uint32_t a_plane,
                                              uint32_t b_plane, uint32_t a8, uint32_t b8, const MixDesc &a32,
                                              const MixDesc &ad8, const MixDesc &b32, const MixDesc &bd8,
                                              uint32_t idesc, uint32_t idesc8, bool first) {
  uint32_t acc = first ? 0u : 1u;
  {
    uint32_t a_lo = ad8.lo_fixed | (((sa + a_plane + a8) & 0x3FFFFu) >> 4);   // A lo8
    uint32_t b_lo = bd8.lo_fixed | (((sb + b_plane) & 0x3FFFFu) >> 4);        // B hi8
#pragma unroll
    for (uint32_t ks = 0; ks < 2u; ++ks) {
      mma_issue<kCtas, true>(d_tmem, a_lo, ad8.hi, b_lo, bd8.hi, idesc8, acc);
      acc = 1u;
      a_lo += ad8.kstep;
      b_lo += bd8.kstep;
    }
  }
  {
    uint32_t a_lo = ad8.lo_fixed | (((sa + a_plane) & 0x3FFFFu) >> 4);        // A hi8
    uint32_t b_lo = bd8.lo_fixed | (((sb + b_plane + b8) & 0x3FFFFu) >> 4);   // B lo8
#pragma unroll
    for (uint32_t ks = 0; ks < 2u; ++ks) {
      mma_issue<kCtas, true>(d_tmem, a_lo, ad8.hi, b_lo, bd8.hi, idesc8, 1u);
      a_lo += ad8.kstep;
      b_lo += bd8.kstep;
    }
  }
  {
    uint32_t a_lo = a32.lo_fixed | ((sa & 0x3FFFFu) >> 4);                    // A hi
    uint32_t b_lo = b32.lo_fixed | ((sb & 0x3FFFFu) >> 4);                    // B hi
#pragma unroll
    for (uint32_t ks = 0; ks < kKSteps; ++ks) {
      mma_issue<kCtas, false>(d_tmem, a_lo, a32.hi, b_lo, b32.hi, idesc, 1u);
      a_lo += a32.kstep;
      b_lo += b32.kstep;
    }
  }
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "{\n\t"
      ".reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The same load without the wait, and the wait as a statement that "produces" the registers, so
// that nothing which uses them can be scheduled in front of it: several loads can then be in
// flight behind one wait.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// ---- CTA-pair (cta_group::2) forms.  Two CTAs of a cluster share one MMA: the leader
// (cluster rank 0) issues it for both, each CTA stages its own 128 rows of A and its own
// half of B's rows, and holds the 128 accumulator rows of its half of M in its own TMEM. ----

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// shared::cluster address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// TMA load whose completion is signalled on a barrier that may live in the peer CTA.
// The data itself lands only in the issuing CTA's shared memory: every CTA fetches its own tiles.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster_addr,
                                                 int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1),
        "r"(c2)
      : "memory");
}

// arrives (once) on the barrier at this shared-memory offset in BOTH CTAs of the pair when
// the MMAs issued so far have retired
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  asm volatile(
      "{\n\t"
      ".reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t"
      "}\n" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

}  // namespace
}  // namespace b200

#endif  // PRIMITIV_B200_CSRC_TCGEN05_CUH_
