// tcgen05 product of the fp32 modes that feeds its tiles itself: for products of a few microseconds.
//
//   C[g] = (acc ? C[g] : 0) + sum_{r<red} opA(A[g*a_gs + r*a_rs]) . opB(B[g*b_gs + r*b_rs])
//
// gemm_tc.cu wants the operands split into planes first, a launch and a pass over memory each, and
// another launch to add the slices of a split contraction: half of the time of a small product.
// gemm_mma.cuh needs none of that but splits every fragment once per warp that uses it (0.9 us per 128 x 32 x 32
// step).  Here eight warps fetch operands with ordinary loads, of any alignment, split each element
// once, and store the planes where the tensor core reads them; the same warps write the result.
//
// A step of 128 x 64 x 32 takes 0.68 us.  48 KB of planes are stored and read again by the tensor core and 24 KB of
// operands come in: at 128 bytes per clock 960 clocks, 0.49 us, of what shared memory moves; what the other quarter
// waits for has not been measured.  TMA-fed planes need half of those bytes, so large products stay with gemm_tc.cu.  Measured back to back, planes and reduction included, against
// gemm_tc.cu: 800 x 200 x 784 14.9 -> 11.2 us, 800 x 784 x 200 12.9 -> 8.5, 512^3 16.0 -> 8.4, 256 x 1024 x 256
// 12.3 -> 8.2 (gemm_mma.cuh: 17.5, 18.3, 13.0, 9.0).  Slices follow gemm_fixed_slices; tiles of 96 columns let
// the 5 slices of 800 x 200 run at once (21 clusters, 26 fit; 64 columns make 28), tiles of 32 give unsplit
// products more CTAs.  (128-column tiles, and the same kernel for halves and TF32, were built too and were
// never the fastest.)
//
// The corrections of the default fp32 mode are bf16, with gemm_tc.cu's bits (off by 0.7 to 1.4e-6).  The 3xFP16 mode
// promises 22 bits: its corrections are TF32 and have an accumulator of their own, and chunks are two k-blocks:
// 2e-7 whatever the length, where its planes lose 2.8e-7 at 86 terms and 1.5e-6 at 784.
//
// Thread roles (288 threads): warps 0-7 feed stages and later drain the accumulator, warp 8 issues the MMAs.
// A stage is one k-block of 32: [A hi | A hi8 | A lo8 | B hi | B hi8 | B lo8], hi in TF32, the correction operands
// in bf16, in the layouts and swizzles of gemm_tc.cu; operands keep the major-ness they have in memory.
// Loads run two k-blocks ahead in registers, stores as far ahead as there are stages.
//
// The contraction of a tile may be cut over the CTAs of a cluster; their tiles meet through distributed
// shared memory and are added in rank order: the same bits every run.  The accumulator is added to registers
// every few k-blocks (the tensor core truncates when it accumulates, see gemm_tc.cu), one chunk behind the
// feeding so that it never waits.
#include <cuda_bf16.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

#include "ctx.h"
#include "tcgen05.cuh"

namespace b200 {
namespace {

struct DirectParams {
  const float *A, *B;
  float *C;                         // column-major m x n, ld = m
  uint32_t m, n, k;
  uint32_t tiles_m, tiles_n, groups;
  uint32_t splits;                  // CTAs of a cluster that share a tile's contraction
  uint32_t kb, red;                 // k-blocks of one matrix pair, and pairs
  uint32_t kb_all, kb_per;          // k-blocks in all (red * kb), and of one split
  uint32_t chunk;                   // k-blocks that the tensor core accumulates before their sum goes to registers: even
  unsigned long long lda, ldb;      // elements from one line to the next
  unsigned long long a_gs, a_rs, b_gs, b_rs, c_gs;
  uint32_t wide_a, wide_b;          // every line starts on 16 bytes
  uint32_t accumulate;
  int *status;
};

constexpr uint32_t kDirectM = 128, kDirectK = 32;   // (a tile has 32, 64 or 96 columns)
constexpr uint32_t kFeedThreads = 256, kFeedWarps = 8;

// One operand's tile: geometry of the shared-memory planes and of the feeding threads' share.
// kFull: the second plane is x - hi in TF32 instead of two in bf16.
template <bool kKMajor, uint32_t ROWS, bool kFull>
struct Feed {
  static constexpr uint32_t kUnits = ROWS * 8u / kFeedThreads;          // units of four floats per thread and k-block
  static constexpr uint32_t kPlane = ROWS * 128u;                       // bytes of the main plane, of a bf16 plane
  static constexpr uint32_t kPlane8 = (!kKMajor && ROWS < 64u ? 64u : ROWS) * 64u;   // (a line of 32 fills half of the swizzle's 128 bytes)
  static constexpr uint32_t kBytes = kPlane + 2u * kPlane8;
  static constexpr uint32_t kLineUnits = kKMajor ? 8u : ROWS / 4u;    // units per line in memory
  static constexpr uint32_t kLineStep = kFeedThreads / kLineUnits;      // lines from one of a thread's units to the next

  const float *from;         // this thread's first unit of the next k-block
  unsigned long long pitch;  // floats from line to line
  uint32_t line, lines;      // its first line and the number there are: rows (K-major) or k (MN-major)
  uint32_t at, inner;        // its position along the line, and the line's length
  bool wide;
  uint32_t to, to8;          // byte offsets in the planes

  __device__ __forceinline__ void start(const float *matrix, unsigned long long ld, uint32_t mn0, uint32_t k0, uint32_t mn, uint32_t k,
                                        bool w) {
    const uint32_t l = threadIdx.x / kLineUnits, c = threadIdx.x % kLineUnits;
    pitch = ld;
    line = (kKMajor ? mn0 : k0) + l;
    lines = kKMajor ? mn : k;
    at = (kKMajor ? k0 : mn0) + c * 4u;
    inner = kKMajor ? k : mn;
    wide = w;
    from = matrix + line * pitch + at;
    if constexpr (kKMajor) {
      to = l * 128u + ((c ^ (l & 7u)) << 4);
      to8 = l * 64u + (((c >> 1) ^ ((l >> 1) & 3u)) << 4) + (c & 1u) * 8u;   // 64-byte swizzle
    } else {
      // 128 bytes of mn by 32 lines per block; TF32 wants the 128-byte pattern on 32-byte units
      to = (c >> 3) * (kDirectK * 128u) + l * 128u + (((c & 7u) ^ ((l & 3u) << 1)) << 4);
      to8 = (c >> 4) * (kDirectK * 128u) + l * 128u + ((((c & 15u) >> 1) ^ (l & 7u)) << 4) + (c & 1u) * 8u;
    }
  }
  static constexpr uint32_t kToStep = kLineStep * 128u, kTo8Step = kLineStep * (kKMajor ? 64u : 128u);

  __device__ __forceinline__ void load(float4 (&raw)[kUnits]) {
#pragma unroll
    for (uint32_t i = 0; i < kUnits; ++i) {
      const float *p = from + i * kLineStep * pitch;
      raw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (line + i * kLineStep < lines && at < inner) {
        const uint32_t left = inner - at;
        if (wide && left >= 4u) {
          raw[i] = *reinterpret_cast<const float4 *>(p);
        } else {
          raw[i].x = p[0];
          if (left > 1u) raw[i].y = p[1];
          if (left > 2u) raw[i].z = p[2];
          if (left > 3u) raw[i].w = p[3];
        }
      }
    }
    // on to the next k-block
    if constexpr (kKMajor) {
      at += kDirectK;
      from += kDirectK;
    } else {
      line += kDirectK;
      from += kDirectK * pitch;
    }
  }

  // Stores the units, split, into a stage whose planes for this operand begin at `base`.
  __device__ __forceinline__ void store(const float4 (&raw)[kUnits], uint32_t base) const {
#pragma unroll
    for (uint32_t i = 0; i < kUnits; ++i) {
      const float4 x = raw[i], hi = make_float4(round(x.x), round(x.y), round(x.z), round(x.w));
      asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(base + to + i * kToStep), "f"(hi.x), "f"(hi.y), "f"(hi.z), "f"(hi.w) : "memory");
      if constexpr (kFull) {
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(base + kPlane + to + i * kToStep), "f"(round_rest(x.x - hi.x)), "f"(round_rest(x.y - hi.y)),
                     "f"(round_rest(x.z - hi.z)), "f"(round_rest(x.w - hi.w)) : "memory");
        continue;
      }
      sts64(base + kPlane + to8 + i * kTo8Step, bf16x2(x.x, x.y), bf16x2(x.z, x.w));
      sts64(base + kPlane + kPlane8 + to8 + i * kTo8Step, bf16x2(x.x - hi.x, x.y - hi.y), bf16x2(x.z - hi.z, x.w - hi.w));
    }
  }

 private:
  // Nearest TF32, ties away, as in pack.cu.  Inf passes through; a nan can become anything, but x - hi is then the one
  // that arithmetic makes, 0x7fffffff: bf16 keeps it, and so does this rounding of the rest (the plain one would make
  // it -0; see gemm_mma.cuh).
  static __device__ __forceinline__ float round(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }
  static __device__ __forceinline__ float round_rest(float x) {
    const int u = __float_as_int(x);
    return __uint_as_float(static_cast<uint32_t>(__viaddmax_s32(u, 0x1000, u)) & 0xffffe000u);
  }
  static __device__ __forceinline__ uint32_t bf16x2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
  }
  static __device__ __forceinline__ void sts64(uint32_t to, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(to), "r"(a), "r"(b) : "memory");
  }
};

// Descriptor fields of a TF32 plane or a bf16 one; see gemm_tc.cu.
template <bool kKMajor>
__device__ __forceinline__ MixDesc plane_desc(bool tf32) {
  const uint32_t sbo = kKMajor == tf32 ? 1024u : 512u;
  const uint32_t layout = kKMajor ? (tf32 ? 2u : 4u) : (tf32 ? 1u : 2u);
  MixDesc d;
  d.hi = ((sbo >> 4) & 0x3FFFu) | (1u << 14) | (layout << 29);
  d.lo_fixed = ((kKMajor ? 0u : kDirectK * 128u) >> 4) << 16;
  d.kstep = (kKMajor ? 32u : tf32 ? 1024u : 2048u) >> 4;
  return d;
}

template <bool KA, bool KB, uint32_t N>
constexpr uint32_t kDirectStage = Feed<KA, kDirectM, false>::kBytes + Feed<KB, N, false>::kBytes;   // 40 to 56 KB
constexpr uint32_t kDirectStages = 4;
constexpr uint32_t kDirectPitch = kDirectM + 4u;                  // floats per column of the result tile
template <bool KA, bool KB, uint32_t N>
constexpr uint32_t kDirectSmem = kDirectStages * kDirectStage<KA, KB, N> + 1024u;   // (the result tile fits in it)

template <bool KA, bool KB, uint32_t kDirectN, bool kFull>
__global__ void __launch_bounds__(kFeedThreads + 32, 1) gemm_direct_kernel(const __grid_constant__ DirectParams p) {
  using FA = Feed<KA, kDirectM, kFull>;
  using FB = Feed<KB, kDirectN, kFull>;
  constexpr uint32_t kStages = kDirectStages, kHalfCols = kDirectN / 2u;
  constexpr uint32_t kSums = kFull ? 3u : 2u;   // accumulators: two in turn, one of the small terms
  constexpr uint32_t kCols = kSums * kDirectN <= 64u ? 64u : kSums * kDirectN <= 128u ? 128u : kSums * kDirectN <= 256u ? 256u : 512u;
  constexpr uint32_t kStageBytes = kDirectStage<KA, KB, kDirectN>;
  static_assert(kDirectN == 32u || kDirectN == 64u || (kDirectN == 96u && KB), "what the feeding threads divide evenly");
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t acc_full_bar[2];
  __shared__ __align__(8) uint64_t acc_empty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;

  pdl_release_next();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  volatile int *abort_flag = &s_abort;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (uint32_t s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), kFeedWarps);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (uint32_t b = 0; b < 2u; ++b) {
      mbar_init(smem_u32(&acc_full_bar[b]), 1);
      mbar_init(smem_u32(&acc_empty_bar[b]), kFeedWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kFeedWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  const uint32_t rank = p.splits > 1u ? cluster_ctarank() : 0u;
  const uint32_t tile = blockIdx.x / p.splits;
  const uint32_t per_group = p.tiles_m * p.tiles_n;
  const uint32_t g = tile / per_group, rem = tile - g * per_group;
  const uint32_t m0 = (rem % p.tiles_m) * kDirectM, n0 = (rem / p.tiles_m) * kDirectN;
  const uint32_t kb0 = rank * p.kb_per;
  const uint32_t count = kb0 + p.kb_per < p.kb_all ? p.kb_per : p.kb_all - kb0;   // > 0: the host makes no empty split
  const uint32_t chunks = (count + p.chunk - 1u) / p.chunk;

  const uint32_t quarter = warp & 3u, half = warp >> 2;            // tensor-memory lanes and columns of a feeding warp
  const uint32_t taddr = tmem + ((quarter * 32u) << 16) + half * kHalfCols;
  float sum[kHalfCols];

  if (warp < kFeedWarps) {
    pdl_wait_previous();
    uint32_t r = kb0 / p.kb, kb = kb0 - r * p.kb;   // matrix pair and k-block of the next load
    FA fa;
    FB fb;
    auto begin = [&](uint32_t k_block) {
      fa.start(p.A + g * p.a_gs + r * p.a_rs, p.lda, m0, k_block * kDirectK, p.m, p.k, p.wide_a != 0u);
      fb.start(p.B + g * p.b_gs + r * p.b_rs, p.ldb, n0, k_block * kDirectK, p.n, p.k, p.wide_b != 0u);
    };
    begin(kb);
    auto fetch = [&](float4 (&ra)[FA::kUnits], float4 (&rb)[FB::kUnits]) {
      fa.load(ra);
      fb.load(rb);
      if (++kb == p.kb) {   // the next matrix pair of the reduction axis
        kb = 0;
        ++r;
        if (r < p.red) begin(0);
      }
    };
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    auto put = [&](const float4 (&ra)[FA::kUnits], const float4 (&rb)[FB::kUnits]) {
      ok = ok && mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1u, abort_flag);
      if (ok) {
        const uint32_t at = base + stage * kStageBytes;
        fa.store(ra, at);
        fb.store(rb, at + FA::kBytes);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor core reads through the async proxy
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full_bar[stage]));
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1u;
      }
    };
    auto add = [&](uint32_t cols, bool first) {
      if constexpr (kHalfCols >= 32u) {
        uint32_t v[32];
        tmem_ld32(taddr + cols, v);
#pragma unroll
        for (uint32_t i = 0; i < 32u; ++i) sum[i] = first ? __uint_as_float(v[i]) : sum[i] + __uint_as_float(v[i]);
      }
      if constexpr (kHalfCols % 32u != 0u) {
        constexpr uint32_t at = kHalfCols - 16u;
        uint32_t v[16];
        tmem_ld16(taddr + cols + at, v);
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) sum[at + i] = first ? __uint_as_float(v[i]) : sum[at + i] + __uint_as_float(v[i]);
      }
    };
    // adds chunk c of the accumulator to the registers
    auto drain = [&](uint32_t c) {
      const uint32_t buf = c & 1u;
      ok = __all_sync(0xffffffffu, ok && mbar_wait(smem_u32(&acc_full_bar[buf]), (c >> 1) & 1u, abort_flag));
      if (!ok) return;
      tc_fence_after();
      add(buf * kDirectN, c == 0u);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[buf]));
    };

    float4 a0[FA::kUnits], b0[FB::kUnits], a1[FA::kUnits], b1[FB::kUnits];
    fetch(a0, b0);
    if (count > 1u) fetch(a1, b1);
    uint32_t drained = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < count; i += 2u) {
      put(a0, b0);
      if (i + 2u < count) fetch(a0, b0);
      if (i + 1u < count) {
        put(a1, b1);
        if (i + 3u < count) fetch(a1, b1);
      }
      // (chunks are an even number of k-blocks) one whole chunk is ahead of the one drained here
      if (i + 2u == (drained + 2u) * p.chunk) drain(drained++);
    }
#pragma unroll 1
    while (drained < chunks) drain(drained++);
    if constexpr (kFull) {
      if (ok) add(2u * kDirectN, false);
    }
  } else {
    const MixDesc da = plane_desc<KA>(true), db = plane_desc<KB>(true), da8 = plane_desc<KA>(false), db8 = plane_desc<KB>(false);
    constexpr uint32_t kShape = (1u << 4) | ((KA ? 0u : 1u) << 15) | ((KB ? 0u : 1u) << 16) | ((kDirectN >> 3) << 17) | ((kDirectM >> 4) << 24);
    constexpr uint32_t kIdesc = kShape | (2u << 7) | (2u << 10), kIdesc8 = kShape | (1u << 7) | (1u << 10);
    uint32_t stage = 0, phase = 0, left = count;
    bool ok = true;
#pragma unroll 1
    for (uint32_t c = 0; ok && c < chunks; ++c) {
      const uint32_t buf = c & 1u;
      if (c >= 2u) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_empty_bar[buf]), ((c >> 1) & 1u) ^ 1u, abort_flag));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem + buf * kDirectN;
      const uint32_t n = left > p.chunk ? p.chunk : left;
      left -= n;
#pragma unroll 1
      for (uint32_t i = 0; i < n; ++i) {
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = base + stage * kStageBytes, sb = sa + FA::kBytes;
        if constexpr (kFull) {
          const uint32_t small = tmem + 2u * kDirectN;
          mma_stage<1, false, 1>(small, sa + FA::kPlane, sb, 0u, 0u, da.hi, db.hi, da.lo_fixed, db.lo_fixed, da.kstep, db.kstep, kIdesc, c + i == 0u);
          mma_stage<1, false, 1>(small, sa, sb + FB::kPlane, 0u, 0u, da.hi, db.hi, da.lo_fixed, db.lo_fixed, da.kstep, db.kstep, kIdesc, false);
          mma_stage<1, false, 1>(d, sa, sb, 0u, 0u, da.hi, db.hi, da.lo_fixed, db.lo_fixed, da.kstep, db.kstep, kIdesc, i == 0u);
        } else
          mma_stage_mix<1>(d, sa, sb, FA::kPlane, FB::kPlane, FA::kPlane8, FB::kPlane8, da, da8, db, db8, kIdesc, kIdesc8, i == 0u);
        mma_commit(smem_u32(&empty_bar[stage]));
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) mma_commit(smem_u32(&acc_full_bar[buf]));
    }
    if (*abort_flag) {   // retire what was issued before shared and tensor memory are given up
      __syncwarp();
      mma_commit(smem_u32(&acc_full_bar[0]));
      const long long t0 = clock64();
      while (clock64() - t0 < 100000ll) {}
    }
  }

  float *C = p.C + g * p.c_gs;
  const bool give_up = s_abort != 0;
  if (p.splits == 1u) {
    if (warp < kFeedWarps && !give_up) {
      const uint32_t row = m0 + quarter * 32u + lane, col = n0 + half * kHalfCols;
      if (row < p.m && col < p.n) {
        const uint32_t cols = p.n - col < kHalfCols ? p.n - col : kHalfCols;
        float *q = C + row + static_cast<unsigned long long>(col) * p.m;
        if (p.accumulate) {
#pragma unroll
          for (uint32_t j = 0; j < kHalfCols; ++j)
            if (j < cols) sum[j] += q[static_cast<unsigned long long>(j) * p.m];
        }
        if (cols == kHalfCols) {
#pragma unroll
          for (uint32_t j = 0; j < kHalfCols; ++j) q[static_cast<unsigned long long>(j) * p.m] = sum[j];
        } else {
#pragma unroll
          for (uint32_t j = 0; j < kHalfCols; ++j)
            if (j < cols) q[static_cast<unsigned long long>(j) * p.m] = sum[j];
        }
      }
    }
  } else {
    // every accumulator value has been read: the stages' memory now takes this CTA's part of the tile
    __syncthreads();
    if (warp < kFeedWarps) {
      const uint32_t out = base + (half * kHalfCols * kDirectPitch + quarter * 32u + lane) * 4u;
#pragma unroll
      for (uint32_t j = 0; j < kHalfCols; ++j)
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(out + j * kDirectPitch * 4u), "f"(sum[j]) : "memory");
    }
    cluster_sync_all();
    if (warp < kFeedWarps && !give_up) {
      // every CTA of the cluster finishes its share of the columns' quarters of four rows
#pragma unroll 1
      for (uint32_t q = threadIdx.x + rank * kFeedThreads; q < (kDirectM / 4u) * kDirectN; q += kFeedThreads * p.splits) {
        const uint32_t nn = q / (kDirectM / 4u), mm = (q % (kDirectM / 4u)) * 4u;
        const uint32_t gm = m0 + mm, gn = n0 + nn;
        if (gm >= p.m || gn >= p.n) continue;
        const uint32_t at = base + (nn * kDirectPitch + mm) * 4u;
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        for (uint32_t s = 0; s < p.splits; ++s) {
          float4 w;
          asm volatile(
              "{\n\t.reg .u32 a;\n\t"
              "mapa.shared::cluster.u32 a, %4, %5;\n\t"
              "ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [a];\n\t}\n"
              : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w) : "r"(at), "r"(s) : "memory");
          x[0] += w.x; x[1] += w.y; x[2] += w.z; x[3] += w.w;
        }
        float *c = C + gm + static_cast<unsigned long long>(gn) * p.m;
        if (gm + 4u <= p.m && (reinterpret_cast<unsigned long long>(c) & 15u) == 0) {
          if (p.accumulate) {
            const float4 o = *reinterpret_cast<const float4 *>(c);
            x[0] += o.x; x[1] += o.y; x[2] += o.z; x[3] += o.w;
          }
          *reinterpret_cast<float4 *>(c) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
          for (uint32_t e = 0; e < 4u; ++e)
            if (gm + e < p.m) c[e] = x[e] + (p.accumulate ? c[e] : 0.f);
        }
      }
    }
    cluster_sync_all();   // nobody leaves while another CTA still reads its tile
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) report_status(p.status, B200_ERR_KERNEL_TIMEOUT);
  if (warp == kFeedWarps) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
}

template <bool KA, bool KB, uint32_t N, bool kFull>
int direct_launch(b200_ctx *ctx, const DirectParams &p, cudaStream_t stream) {
  auto kernel = gemm_direct_kernel<KA, KB, N, kFull>;
  constexpr uint32_t kSmem = kDirectSmem<KA, KB, N>;
  static std::atomic<unsigned long long> done{0};   // opted in to large shared memory, one bit per device
  const unsigned long long bit = 1ull << (ctx->device & 63);
  if (!(done.load(std::memory_order_relaxed) & bit)) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem));
    if (e != cudaSuccess) return static_cast<int>(e);
    done.fetch_or(bit, std::memory_order_relaxed);
  }
  const unsigned grid = p.tiles_m * p.tiles_n * p.groups * p.splits;
  b200::launch(ctx, kernel, dim3(grid), dim3(kFeedThreads + 32u), kSmem, stream, p.splits, p);
  return static_cast<int>(cudaGetLastError());
}

template <bool KA, bool KB, bool kFull>
int direct_launch(b200_ctx *ctx, const DirectParams &p, uint32_t cols, cudaStream_t stream) {
  if constexpr (KB) {
    if (cols == 96u) return direct_launch<KA, true, 96u, kFull>(ctx, p, stream);
  }
  return cols == 32u ? direct_launch<KA, KB, 32u, kFull>(ctx, p, stream) : direct_launch<KA, KB, 64u, kFull>(ctx, p, stream);
}

template <bool kFull>
int direct_launch(b200_ctx *ctx, const DirectParams &p, bool ka, bool kb, uint32_t cols, cudaStream_t stream) {
  if (ka) return kb ? direct_launch<true, true, kFull>(ctx, p, cols, stream) : direct_launch<true, false, kFull>(ctx, p, cols, stream);
  return kb ? direct_launch<false, true, kFull>(ctx, p, cols, stream) : direct_launch<false, false, kFull>(ctx, p, cols, stream);
}

struct DirectChoice {
  uint32_t cols, splits;
  double us;
};

// One CTA fits on an SM; a k-block takes 0.56, 0.68 or 1.0 us (more where loads are single floats), a tile 2 us
// besides, 2.9 where others follow it, adding up a split 1.7 us: fitted to 60 products.  A cluster has to fit a
// GPC: of 28 clusters of five only 26 run at a time (ctx->cluster_room).
DirectChoice choose(const b200_ctx *ctx, const GemmArgs &g, bool wide) {
  static const struct { uint32_t cols; double wide, narrow; } kTiles[] = {{64, 0.68, 0.8}, {96, 1.0, 1.1}, {32, 0.56, 0.7}};
  const uint64_t kb = static_cast<uint64_t>((g.k + kDirectK - 1) / kDirectK) * g.red;
  const uint32_t fixed = gemm_fixed_slices(ctx, g);
  DirectChoice best{64, fixed > 8u ? 8u : fixed ? fixed : 1u, 1e30};   // (more slices than a cluster has CTAs: not this kernel's)
  for (const auto &t : kTiles) {
    if (t.cols == 96u && g.trans_b) continue;   // (a line of 96 columns does not divide among the threads)
    const double tiles = static_cast<double>((g.m + kDirectM - 1) / kDirectM) * ((g.n + t.cols - 1) / t.cols) * g.groups;
    for (uint32_t s = 1; s <= 8u && s <= kb; ++s) {
      const double room = ctx->cluster_room[s];
      if (fixed ? s != fixed : (s > 1u && tiles > room)) continue;
      const double waves = static_cast<double>(static_cast<uint64_t>((tiles + room - 1) / room));
      const double us = 1.5 + waves * (static_cast<double>((kb + s - 1) / s) * (wide ? t.wide : t.narrow) + (waves > 1.0 ? 2.9 : 2.0) + (s > 1u ? 1.7 : 0.0));
      if (us < best.us) best = {t.cols, s, us};
    }
  }
  return best;
}

bool all_wide(const void *ptr, uint64_t ld, uint64_t gs, uint32_t groups, uint64_t rs, uint32_t red) {
  return reinterpret_cast<uintptr_t>(ptr) % 16 == 0 && ld % 4 == 0 && (groups == 1 || gs % 4 == 0) && (red == 1 || rs % 4 == 0);
}
bool wide_a(const GemmArgs &g) { return all_wide(g.A, g.trans_a ? g.k : g.m, g.a_gs, g.groups, g.a_rs, g.red); }
bool wide_b(const GemmArgs &g) { return all_wide(g.B, g.trans_b ? g.n : g.k, g.b_gs, g.groups, g.b_rs, g.red); }

}  // namespace

double gemm_direct_estimate(const b200_ctx *ctx, const GemmArgs &g) {
  if (g.mode != B200_MODE_FP32_3XTF32 && g.mode != B200_MODE_FP32_3XFP16) return 1e30;
  if (ctx->correction_policy == 1) return 1e30;   // the caller wants TF32 planes throughout
  if (has_fp32_sums(g)) return 1e30;
  // (half planes lose less than this kernel where the sum is that short: 1.2e-7 against 1.6e-7 at 48 terms)
  if (g.mode == B200_MODE_FP32_3XFP16 && static_cast<uint64_t>(g.k) * g.red < 64u) return 1e30;
  return choose(ctx, g, wide_a(g) && wide_b(g)).us;
}

int gemm_direct(b200_ctx *ctx, const GemmArgs &g, cudaStream_t stream) {
  if (g.mode != B200_MODE_FP32_3XTF32 && g.mode != B200_MODE_FP32_3XFP16) return B200_ERR_INVALID_ARG;
  DirectParams p;
  std::memset(&p, 0, sizeof(p));
  p.A = static_cast<const float *>(g.A);
  p.B = static_cast<const float *>(g.B);
  p.C = static_cast<float *>(g.C);
  p.m = g.m; p.n = g.n; p.k = g.k;
  p.groups = g.groups;
  p.red = g.red;
  p.lda = g.trans_a ? g.k : g.m;
  p.ldb = g.trans_b ? g.n : g.k;
  p.a_gs = g.a_gs; p.a_rs = g.a_rs; p.b_gs = g.b_gs; p.b_rs = g.b_rs; p.c_gs = g.c_gs;
  p.wide_a = wide_a(g);
  p.wide_b = wide_b(g);
  p.accumulate = g.accumulate ? 1u : 0u;
  p.status = ctx->d_status;
  p.kb = (g.k + kDirectK - 1) / kDirectK;
  const uint64_t all = static_cast<uint64_t>(p.kb) * g.red;
  if (all > 0x7fffffffull) return B200_ERR_TOO_LARGE;
  p.kb_all = static_cast<uint32_t>(all);
  p.tiles_m = (g.m + kDirectM - 1) / kDirectM;
  const DirectChoice c = choose(ctx, g, p.wide_a && p.wide_b);
  uint32_t splits = c.splits, cols = c.cols;
#ifdef PRIMITIV_B200_DEV_KNOBS
  if (const char *e = std::getenv("PRIMITIV_B200_DIRECT_COLS")) cols = std::atoi(e) == 32 ? 32u : std::atoi(e) == 96 && !g.trans_b ? 96u : 64u;
  if (const char *e = std::getenv("PRIMITIV_B200_DIRECT_SPLITS")) splits = std::atoi(e);
#endif
  p.tiles_n = (g.n + cols - 1) / cols;
  // (longer chunks truncate more: where the order is not fixed, shorter ones cost next to nothing)
  p.chunk = g.mode == B200_MODE_FP32_3XFP16 ? 2u : gemm_fixed_slices(ctx, g) ? 8u : 4u;
  p.kb_per = (p.kb_all + splits - 1) / splits;
  p.splits = (p.kb_all + p.kb_per - 1) / p.kb_per;   // no empty splits
  if (static_cast<uint64_t>(p.tiles_m) * p.tiles_n * g.groups * p.splits > 0x7fffffffull) return B200_ERR_TOO_LARGE;
  ProfScope prof(ctx, kProfGemmTc, stream);
  ++ctx->launches;
  if (g.mode == B200_MODE_FP32_3XFP16) return direct_launch<true>(ctx, p, g.trans_a != 0, g.trans_b == 0, cols, stream);
  return direct_launch<false>(ctx, p, g.trans_a != 0, g.trans_b == 0, cols, stream);
}

}  // namespace b200
