// Matrix product for what is too small, too thin or too ragged for the tcgen05 kernel: mma.sync on
// operands read where they lie.
//
//   C[g] = (acc ? C[g] : 0) + sum_{r<red} opA(A[g*a_gs + r*a_rs]) . opB(B[g*b_gs + r*b_rs])
//
// The tcgen05 kernel (gemm_tc.cu) is three times faster per tensor-core operation, and pays for it at
// both ends of a product: operands that TMA can address (repacked first if they are not, split
// into planes first in the fp32 modes), tiles of at least 128 x 64, tensor memory, a separate launch
// to add the slices of a split contraction.  A product of a few microseconds is all ends.  Here
//   - operands are fetched as they lie: with TMA where its alignment rules allow (one thread issues a
//     k-tile), else with 4-byte cp.async, or single elements for halves on odd addresses;
//   - the fp32 modes split x = hi + lo in registers, both in TF32, so nothing is written or read twice.
//     The smallest came from the CUDA cores, and their sums have to stay as good: with bf16 corrections, as
//     the planes of pack.cu have them, 48 x 336 x 88 was off by 7.9e-7 where those had 1.7e-7;
//   - a contraction is cut over the CTAs of a cluster, which add their tiles through distributed
//     shared memory in rank order: one launch, no scratch, the same bits every run;
//   - tiles go down to 128 x 8, so a handful of columns against a large matrix streams that matrix
//     at memory speed.
// What bounds a small product is the instruction cache as much as anything: with the loads of three
// copy widths unrolled into one kernel, two thirds of all stalls of a 256 x 1024 x 256 product were
// instruction fetches.  Hence one kernel per way of loading, and one place each that loads and computes.
//
// Layouts in shared memory.  A tile of a K-major operand is [row][128 bytes of k]; of an MN-major
// operand [block of 128 bytes of mn][k][128 bytes], or [k][rows] where the tile is narrower.  16-byte
// chunks are permuted within a line (chunk_swizzle) as TMA does it, so that fragment loads are free of
// bank conflicts (two-way for floats in MN-major tiles of 16): ldmatrix where the line direction matches
// the fragment's (halves in either major-ness through .trans, floats only K-major), 32-bit loads for
// MN-major floats, under the pattern on 32-byte units.
//
// The tensor core truncates when it adds into its accumulator (see gemm_tc.cu); the fp32 modes
// therefore promote their accumulators to a second set of registers after every k-tile, and keep the small
// terms out of them.  Halves, which the CUDA cores summed without that bias, are promoted every kMmaHalfRun k-tiles: a
// thousand terms lose 2e-6 of their sum, where the result is rounded to 2e-4 (a million terms in one run lost 7.5e-4 to 6e-3).
#ifndef PRIMITIV_B200_CSRC_GEMM_MMA_CUH_
#define PRIMITIV_B200_CSRC_GEMM_MMA_CUH_

#include <cuda_fp16.h>

#include <atomic>
#include <type_traits>

#include "gemm_mma.h"
#include "mbar.cuh"

namespace b200 {
namespace {   // each translation unit instantiates its own kernels

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// Shape of one operand's tile.
template <bool kKMajor, int kES, int ROWS>
struct Layout {
  static constexpr uint32_t kLine = kKMajor ? 128u : (ROWS * kES < 128 ? ROWS * kES : 128);   // bytes
  static constexpr uint32_t kLines = kKMajor ? ROWS : 128u / kES;
  static constexpr uint32_t kBlock = kLine * kLines;
  static constexpr uint32_t kBlocks = kKMajor ? 1u : ROWS * kES / kLine;
  static constexpr uint32_t kBytes = kBlock * kBlocks;
  // Where chunk c (16 bytes) of a line lies: what TMA's swizzle modes do to lines of 128, 64 and 32
  // bytes, and the 128-byte mode on 32-byte units for MN-major floats.
  static __device__ __forceinline__ uint32_t chunk(uint32_t c, uint32_t line) {
    if constexpr (kLine == 128u) {
      if constexpr (!kKMajor && kES == 4) return c ^ ((line & 3u) << 1);
      else return c ^ (line & 7u);
    } else if constexpr (kLine == 64u) {
      return c ^ ((line >> 1) & 3u);
    } else if constexpr (kLine == 32u && kES == 2) {
      return c ^ ((line >> 2) & 1u);
    } else {
      return c;
    }
  }
  // byte offset of chunk c (over the whole extent along the line) of a line
  static __device__ __forceinline__ uint32_t at(uint32_t c, uint32_t line) {
    constexpr uint32_t kPer = kLine / 16u;
    const uint32_t block = kBlocks == 1u ? 0u : c / kPer;
    return block * kBlock + line * kLine + (chunk(kBlocks == 1u ? c : c % kPer, line) << 4);
  }
};

// One k-tile of one operand into shared memory without TMA.  `src` is the matrix, mn0 / k0 the tile's
// origin, mn / k the matrix's extents.  W: bytes per copy, 4 or 2 (single halves, stored in pairs).
template <bool kKMajor, int kES, int ROWS, int NT, int W>
__device__ __forceinline__ void load_tile(uint32_t dst, const char *src, unsigned long long ld, uint32_t mn0, uint32_t k0,
                                          uint32_t mn, uint32_t k) {
  using L = Layout<kKMajor, kES, ROWS>;
  constexpr uint32_t kPerLine = L::kLine * L::kBlocks / 4u, kUnits = L::kLines * kPerLine;
  const uint32_t first = kKMajor ? mn0 : k0, lines = kKMajor ? mn : k;      // slow axis
  const uint32_t inner0 = kKMajor ? k0 : mn0, inner = kKMajor ? k : mn;     // contiguous axis
#pragma unroll 4
  for (uint32_t u = threadIdx.x; u < kUnits; u += NT) {
    const uint32_t line = u / kPerLine, at = (u % kPerLine) * 4u;           // `at`: bytes along the line
    const uint32_t e = inner0 + at / kES;
    const uint32_t to = dst + L::at(at >> 4, line) + (at & 15u);
    uint32_t bytes = 0;
    const char *from = src;
    if (first + line < lines && e < inner) {
      bytes = (inner - e) * kES < 4u ? (inner - e) * kES : 4u;
      from = src + (static_cast<unsigned long long>(first + line) * ld + e) * kES;
    }
    if constexpr (W == 2) {
      const unsigned short *h = reinterpret_cast<const unsigned short *>(from);
      const uint32_t lo = bytes >= 2u ? h[0] : 0u, hi = bytes >= 4u ? h[1] : 0u;
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(to), "r"(lo | (hi << 16)) : "memory");
    } else {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(bytes) : "memory");
    }
  }
}

// ... and with TMA: the boxes of one tile, by one thread.
template <bool kKMajor, int kES, int ROWS>
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap *map, uint32_t bar, uint32_t mn0, uint32_t k0, uint32_t z) {
  using L = Layout<kKMajor, kES, ROWS>;
#pragma unroll
  for (uint32_t b = 0; b < L::kBlocks; ++b) {
    const int c0 = static_cast<int>(kKMajor ? k0 : mn0 + b * (L::kLine / kES)), c1 = static_cast<int>(kKMajor ? mn0 : k0);
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst + b * L::kBlock), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(static_cast<int>(z))
        : "memory");
  }
}

__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm2(uint32_t (&r)[2], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm2t(uint32_t (&r)[2], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Fragments of one 32-byte k-step (16 halves / 8 floats), `ks` counting them inside the k-tile.
//   A: rows r0 .. r0+15 -> {(g, k lo), (g+8, k lo), (g, k hi), (g+8, k hi)}, g = lane / 4
template <bool kKMajor, int kES, int ROWS>
__device__ __forceinline__ void frag_a(uint32_t (&a)[4], uint32_t base, uint32_t r0, uint32_t ks, uint32_t lane) {
  using L = Layout<kKMajor, kES, ROWS>;
  if constexpr (kKMajor) {
    const uint32_t row = r0 + (lane & 15u), c = ks * 2u + (lane >> 4);
    ldm4(a, base + L::at(c, row));
  } else if constexpr (kES == 2) {
    const uint32_t kk = ks * 16u + (lane & 7u) + ((lane >> 4) << 3), c = (r0 >> 3) + ((lane >> 3) & 1u);
    ldm4t(a, base + L::at(c, kk));
  } else {
    const uint32_t g = lane >> 2, t = lane & 3u;
#pragma unroll
    for (uint32_t h = 0; h < 2u; ++h) {
      const uint32_t kk = ks * 8u + t + h * 4u;
#pragma unroll
      for (uint32_t q = 0; q < 2u; ++q) {
        const uint32_t row = r0 + g + q * 8u;
        a[h * 2u + q] = lds32(base + L::at(row >> 2, kk) + ((row & 3u) << 2));
      }
    }
  }
}

//   B: columns c0 .. c0+7 -> {(k lo, g), (k hi, g)}, for NB neighbouring groups of eight columns
template <bool kKMajor, int kES, int ROWS, int NB>
__device__ __forceinline__ void frag_b(uint32_t (&b)[NB][2], uint32_t base, uint32_t c0, uint32_t ks, uint32_t lane) {
  using L = Layout<kKMajor, kES, ROWS>;
  if constexpr (kKMajor || kES == 2) {
    if constexpr (NB == 1) {
      const uint32_t l = lane & 15u;   // lanes 16-31 of an x2 load give no address, but a valid one
      if constexpr (kKMajor) {
        const uint32_t row = c0 + (l & 7u), c = ks * 2u + (l >> 3);
        ldm2(b[0], base + L::at(c, row));
      } else {
        const uint32_t kk = ks * 16u + l, c = c0 >> 3;
        ldm2t(b[0], base + L::at(c, kk));
      }
    } else {
#pragma unroll
      for (int j = 0; j < NB; j += 2) {
        uint32_t r[4];
        if constexpr (kKMajor) {
          const uint32_t row = c0 + j * 8u + (lane & 7u) + ((lane >> 4) << 3), c = ks * 2u + ((lane >> 3) & 1u);
          ldm4(r, base + L::at(c, row));
        } else {
          const uint32_t kk = ks * 16u + (lane & 15u), c = (c0 >> 3) + j + (lane >> 4);
          ldm4t(r, base + L::at(c, kk));
        }
        b[j][0] = r[0]; b[j][1] = r[1];
        b[j + 1][0] = r[2]; b[j + 1][1] = r[3];
      }
    }
  } else {
    const uint32_t g = lane >> 2, t = lane & 3u;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const uint32_t row = c0 + j * 8u + g;
#pragma unroll
      for (uint32_t h = 0; h < 2u; ++h) {
        const uint32_t kk = ks * 8u + t + h * 4u;
        b[j][h] = lds32(base + L::at(row >> 2, kk) + ((row & 3u) << 2));
      }
    }
  }
}

// x rounded to TF32, nearest with ties away, as in pack.cu.  Inf passes through (the carry stays inside
// the mantissa); a nan can become anything here, -0 and inf among it.
__device__ __forceinline__ uint32_t round_tf32(uint32_t u) { return (u + 0x1000u) & 0xffffe000u; }
// The single-pass mode rounds its operands (the tensor core would cut them off, at three times the error).
__device__ __forceinline__ uint32_t nearest_tf32(uint32_t u) {
  uint32_t v;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(v) : "f"(__uint_as_float(u)));
  return v;
}
// The same for x - hi.  Where x is a nan that is the nan which arithmetic makes, 0x7fffffff: the carry would take it to
// -0, so the larger of both integers stays, which for every other value is the sum (the intrinsic's addition wraps, and
// it is one instruction: a 2088-wide TF32 layer over two items 10.4 us, by cvt.rna.tf32, which keeps nans too, 11.7).
__device__ __forceinline__ uint32_t round_rest(float x) {
  const int u = __float_as_int(x);
  return static_cast<uint32_t>(__viaddmax_s32(u, 0x1000, u)) & 0xffffe000u;
}
// The fp32 modes' fragments: x = hi + lo, both TF32.
template <int N>
__device__ __forceinline__ void split_fp32(uint32_t (&x)[N], uint32_t (&lo)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t hi = round_tf32(x[i]);
    lo[i] = round_rest(__uint_as_float(x[i]) - __uint_as_float(hi));
    x[i] = hi;
  }
}

template <typename T>
__device__ __forceinline__ float load_as_float(const T *p) {
  if constexpr (sizeof(T) == 2) return __half2float(*p);
  else return *p;
}
template <typename T>
__device__ __forceinline__ void store_from_float(T *p, float v) {
  if constexpr (sizeof(T) == 2) *p = __float2half_rn(v);
  else *p = v;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .u32 a;\n\t"
      "mapa.shared::cluster.u32 a, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [a];\n\t}\n"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}

// An infinite operand makes x - hi a nan, or meets the zero it left of another one.  Products that are the CUDA
// cores' by their numerics (has_fp32_sums) sum elements that are not finite again in plain fp32: four rows i .. i + 3 of
// column j, by a whole warp with its lanes side by side in k (K-major A), or by each lane for itself, whose
// neighbours have the rows beside its own.  Bound by latency, hence many loads in flight: of nothing but nans 64 x 8 x 65536
// takes 5.8 ms (3.6 with K-major A) and 1000 x 12 x 20000 2.9; one element and one load at a time it was 41 (14.7) and 26,
// on the CUDA cores 4.9 (5.5) and 1.9.
template <bool KA, bool KB>
__device__ __noinline__ float4 plain_sums(const MmaParams &p, uint32_t g, uint32_t i, uint32_t j) {
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  unsigned long long row[4];
#pragma unroll
  for (uint32_t e = 0; e < 4u; ++e) row[e] = (i + e < p.m ? i + e : p.m - 1u) * (KA ? p.lda : 1ull);
  for (uint32_t r = 0; r < p.kt / p.kb; ++r) {
    const float *a = static_cast<const float *>(p.A) + g * p.a_gs + r * p.a_rs;
    const float *b = static_cast<const float *>(p.B) + g * p.b_gs + r * p.b_rs + j * (KB ? p.ldb : 1ull);
#pragma unroll KA ? 8 : 16
    for (uint32_t k = KA ? threadIdx.x & 31u : 0u; k < p.k; k += KA ? 32u : 1u) {
      const float y = b[k * (KB ? 1ull : p.ldb)];
#pragma unroll
      for (uint32_t e = 0; e < 4u; ++e) v[e] = fmaf(a[row[e] + k * (KA ? 1ull : p.lda)], y, v[e]);
    }
  }
  if constexpr (KA) {
#pragma unroll
    for (uint32_t o = 16; o > 0u; o >>= 1) {
#pragma unroll
      for (uint32_t e = 0; e < 4u; ++e) v[e] += __shfl_xor_sync(0xffffffffu, v[e], o);
    }
  }
  return make_float4(v[0], v[1], v[2], v[3]);
}
// Called by whole warps; `inside`: this lane's v is of the result.
template <bool KA, bool KB>
__device__ __forceinline__ void mend(float4 &v, bool inside, const MmaParams &p, uint32_t g, uint32_t i, uint32_t j) {
  const bool odd = inside && !(fabsf(v.x) + fabsf(v.y) + fabsf(v.z) + fabsf(v.w) <= 3e38f);
  float4 w = v;
  if constexpr (KA) {
#pragma unroll 1
    for (uint32_t left = __ballot_sync(0xffffffffu, odd); left != 0u; left &= left - 1u) {
      const int lane = __ffs(left) - 1;
      const float4 sums = plain_sums<KA, KB>(p, g, __shfl_sync(0xffffffffu, i, lane), __shfl_sync(0xffffffffu, j, lane));
      if ((threadIdx.x & 31u) == static_cast<uint32_t>(lane)) w = sums;
    }
  } else {
    if (odd) w = plain_sums<KA, KB>(p, g, i, j);
  }
  if (!(fabsf(v.x) <= 3e38f)) v.x = w.x;
  if (!(fabsf(v.y) <= 3e38f)) v.y = w.y;
  if (!(fabsf(v.z) <= 3e38f)) v.z = w.z;
  if (!(fabsf(v.w) <= 3e38f)) v.w = w.w;
}

template <int KIND, int BM, int BN, int WM, int WN, int STAGES>
struct MmaTile {
  static constexpr int kES = KIND == kMmaHalf ? 2 : 4;
  static constexpr int kWarps = (BM / WM) * (BN / WN);
  static constexpr int kThreads = kWarps * 32;
  static constexpr int kBK = 128 / kES;
  static constexpr uint32_t kBytesA = BM * 128u, kBytesB = BN * 128u, kStage = kBytesA + kBytesB;
  static constexpr uint32_t kPitch = BM + 4;   // floats; 4 modulo 32 keeps the accumulators' stores free of conflicts
  static constexpr uint32_t kOut = kPitch * BN * 4u;
  static constexpr uint32_t kSmem = (STAGES * kStage > kOut ? STAGES * kStage : kOut) + 1024u;   // + alignment of the swizzles
};

// KA / KB: operand K-major (true) or MN-major.  LOAD: how operands are fetched.  RUNS (halves): sums longer than
// kMmaHalfRun k-tiles; a kernel of its own, as the second set of registers costs a thin product of 640 terms 0.2 us.
template <int KIND, int BM, int BN, int WM, int WN, int STAGES, bool KA, bool KB, int LOAD, bool RUNS>
__global__ void __launch_bounds__(MmaTile<KIND, BM, BN, WM, WN, STAGES>::kThreads) gemm_mma_kernel(const __grid_constant__ MmaParams p) {
  using Tile = MmaTile<KIND, BM, BN, WM, WN, STAGES>;
  using T = typename std::conditional<KIND == kMmaHalf, __half, float>::type;
  constexpr int kES = Tile::kES, NT = Tile::kThreads, MT = WM / 16, NB = WN / 8;
  constexpr bool kSums = KIND == kMmaFp32 || RUNS;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ int s_abort;
  const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t wm = (warp % (BM / WM)) * WM, wn = (warp / (BM / WM)) * WN;

  const uint32_t rank = p.splits > 1u ? cluster_rank() : 0u;
  const uint32_t tile = blockIdx.x / p.splits;
  const uint32_t per_group = p.tiles_m * p.tiles_n;
  const uint32_t g = tile / per_group, rem = tile - g * per_group;
  const uint32_t m0 = (rem % p.tiles_m) * BM, n0 = (rem / p.tiles_m) * BN;
  const uint32_t kt0 = rank * p.kt_per;
  const uint32_t kt1 = kt0 + p.kt_per < p.kt ? kt0 + p.kt_per : p.kt;   // kt0 < kt: the host makes no empty split

  pdl_release_next();
  if (LOAD == kMmaTma && threadIdx.x == 0) {
    // the maps are parameters: their fetch need not wait for the grid in front
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(&p.map_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(&p.map_b)) : "memory");
    s_abort = 0;
    for (uint32_t i = 0; i < STAGES; ++i) ring::init(smem_addr(&full_bar[i]), 1);
    ring::fence_init();
  }

  float acc[MT][NB][4];
  float sum[kSums ? MT : 1][kSums ? NB : 1][4], cor[KIND == kMmaFp32 ? MT : 1][KIND == kMmaFp32 ? NB : 1][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[i][j][q] = 0.f;
        if constexpr (kSums) sum[i][j][q] = 0.f;
        if constexpr (KIND == kMmaFp32) cor[i][j][q] = 0.f;
      }

  pdl_wait_previous();
  // The loop fetches STAGES - 1 rounds ahead: round `it` fetches k-tile kt0 + it and computes the one
  // STAGES - 1 before it.
  const uint32_t count = kt1 - kt0;
  uint32_t r = kt0 / p.kb, kb = kt0 - r * p.kb;   // matrix pair and k-tile of the next fetch
  uint32_t to = 0, from = 0, phase = 0;
#pragma unroll 1
  for (uint32_t it = 0; it < count + STAGES - 1u; ++it) {
    const bool compute = it >= STAGES - 1u;
    if constexpr (LOAD != kMmaTma) {
      if (compute) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    }
    __syncthreads();   // everyone is done with the stage that is fetched next (and, without TMA, sees the one computed next)
    if (it < count) {
      const uint32_t at = base + to * Tile::kStage;
      if constexpr (LOAD == kMmaTma) {
        if (threadIdx.x == 0) {
          const uint32_t bar = smem_addr(&full_bar[to]);
          ring::arrive_expect_tx(bar, Tile::kStage);
          tma_tile<KA, kES, BM>(at, &p.map_a, bar, m0, kb * Tile::kBK, g * p.a_gmul + r * p.a_rmul);
          tma_tile<KB, kES, BN>(at + Tile::kBytesA, &p.map_b, bar, n0, kb * Tile::kBK, g * p.b_gmul + r * p.b_rmul);
        }
      } else {
        const char *A = static_cast<const char *>(p.A) + (g * p.a_gs + r * p.a_rs) * kES;
        const char *B = static_cast<const char *>(p.B) + (g * p.b_gs + r * p.b_rs) * kES;
        load_tile<KA, kES, BM, NT, LOAD>(at, A, p.lda, m0, kb * Tile::kBK, p.m, p.k);
        load_tile<KB, kES, BN, NT, LOAD>(at + Tile::kBytesA, B, p.ldb, n0, kb * Tile::kBK, p.n, p.k);
      }
      if (++kb == p.kb) {
        kb = 0;
        ++r;
      }
      if (++to == STAGES) to = 0;
    }
    if constexpr (LOAD != kMmaTma) asm volatile("cp.async.commit_group;" ::: "memory");
    if (!compute) continue;
    // a wait that runs out is reported below; the walk goes on, so every copy is waited for
    if constexpr (LOAD == kMmaTma) ring::wait(smem_addr(&full_bar[from]), phase, &s_abort);
    const uint32_t sa = base + from * Tile::kStage, sb = sa + Tile::kBytesA;
    if (++from == STAGES) {
      from = 0;
      phase ^= 1u;
    }
    if constexpr (KIND == kMmaFp32) {
#pragma unroll
      for (uint32_t ks = 0; ks < 4u; ++ks) {
        uint32_t bh[NB][2], bl[NB][2], ah[MT][4], al[MT][4];
        frag_b<KB, kES, BN, NB>(bh, sb, wn, ks, lane);
#pragma unroll
        for (int j = 0; j < NB; ++j) split_fp32<2>(bh[j], bl[j]);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          frag_a<KA, kES, BM>(ah[i], sa, wm + i * 16u, ks, lane);
          split_fp32<4>(ah[i], al[i]);
        }
        // one pass over all accumulators at a time, so that neighbouring instructions do not wait for each
        // other's sums
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NB; ++j) mma_tf32(cor[i][j], al[i], bh[j]);
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NB; ++j) mma_tf32(acc[i][j], ah[i], bh[j]);
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NB; ++j) mma_tf32(cor[i][j], ah[i], bl[j]);
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            sum[i][j][q] += acc[i][j][q];
            acc[i][j][q] = 0.f;
          }
    } else {
#pragma unroll
      for (uint32_t ks = 0; ks < 4u; ++ks) {
        uint32_t b[NB][2];
        frag_b<KB, kES, BN, NB>(b, sb, wn, ks, lane);
        if constexpr (KIND == kMmaTf32) {
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            b[j][0] = nearest_tf32(b[j][0]);
            b[j][1] = nearest_tf32(b[j][1]);
          }
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          uint32_t a[4];
          frag_a<KA, kES, BM>(a, sa, wm + i * 16u, ks, lane);
          if constexpr (KIND == kMmaTf32) {
#pragma unroll
            for (int q = 0; q < 4; ++q) a[q] = nearest_tf32(a[q]);
          }
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            if constexpr (KIND == kMmaHalf) mma_f16(acc[i][j], a, b[j]);
            else mma_tf32(acc[i][j], a, b[j]);
          }
        }
      }
      if constexpr (RUNS) {
        if ((it - (STAGES - 2u)) % kMmaHalfRun == 0u) {   // that many k-tiles are in
#pragma unroll
          for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                sum[i][j][q] += acc[i][j][q];
                acc[i][j][q] = 0.f;
              }
        }
      }
    }
  }
  if constexpr (LOAD != kMmaTma) asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();   // the pipeline's memory now takes this CTA's part of the tile: [BN][kPitch] floats
  if (LOAD == kMmaTma && threadIdx.x == 0 && s_abort) report_status(p.status, B200_ERR_KERNEL_TIMEOUT);

  float *out = reinterpret_cast<float *>(smem_raw + (base - smem_addr(smem_raw)));
  {
    const uint32_t gq = lane >> 2, t = lane & 3u;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t mm = wm + i * 16u + gq + ((q >> 1) << 3), nn = wn + j * 8u + t * 2u + (q & 1);
          float v = acc[i][j][q];
          if constexpr (KIND == kMmaFp32) v = sum[i][j][q] + cor[i][j][q];
          if constexpr (RUNS) v += sum[i][j][q];
          out[nn * Tile::kPitch + mm] = v;
        }
  }
  if (p.splits > 1u) cluster_barrier();
  else __syncthreads();

  // Every CTA of the cluster finishes its share of the tile, in rounds of whole warps (32 divides the tile's quads).
  T *C = static_cast<T *>(p.C) + g * p.c_gs;
  const bool along_m = p.c_m == 1u;
  if (along_m) {
    // four rows of a column per thread; lanes walk down the column
    constexpr uint32_t kQuads = BM / 4;
    #pragma unroll 1
    for (uint32_t q = threadIdx.x + rank * NT; q < kQuads * BN; q += NT * p.splits) {
      const uint32_t nn = q / kQuads, mm = (q % kQuads) * 4u;
      const uint32_t gm = m0 + mm, gn = n0 + nn;
      const bool inside = gn < p.n && gm < p.m;
      if (!inside && (KIND != kMmaFp32 || !p.mend)) continue;   // (warps stay whole where elements may be summed again)
      const uint32_t at = base + (nn * Tile::kPitch + mm) * 4u;
      float4 v;
      if (p.splits > 1u) {
        v = ld_cluster(at, 0u);
        for (uint32_t s = 1; s < p.splits; ++s) {
          const float4 w = ld_cluster(at, s);
          v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
      } else {
        v = *reinterpret_cast<const float4 *>(out + nn * Tile::kPitch + mm);
      }
      if constexpr (KIND == kMmaFp32) {
        if (p.mend) mend<KA, KB>(v, inside, p, g, gm, gn);
        if (!inside) continue;
      }
      T *c = C + gm + gn * p.c_n;
      const bool whole = gm + 4u <= p.m && (reinterpret_cast<unsigned long long>(c) & (4u * kES - 1u)) == 0;
      if (whole) {
        if constexpr (kES == 4) {
          if (p.accumulate) {
            const float4 o = *reinterpret_cast<const float4 *>(c);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
          }
          *reinterpret_cast<float4 *>(c) = v;
        } else {
          if (p.accumulate) {
            const uint2 o = *reinterpret_cast<const uint2 *>(c);
            const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&o.x)), hi = __half22float2(*reinterpret_cast<const __half2 *>(&o.y));
            v.x += lo.x; v.y += lo.y; v.z += hi.x; v.w += hi.y;
          }
          const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
          *reinterpret_cast<uint2 *>(c) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
        }
      } else {
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t e = 0; e < 4u; ++e)
          if (gm + e < p.m) store_from_float(c + e, x[e] + (p.accumulate ? load_as_float(c + e) : 0.f));
      }
    }
  } else {
    // operands were exchanged: n runs fastest in C
    #pragma unroll 1
    for (uint32_t q = threadIdx.x + rank * NT; q < (BM / 4) * BN; q += NT * p.splits) {
      const uint32_t nn = q % BN, mm = (q / BN) * 4u;
      const uint32_t gm = m0 + mm, gn = n0 + nn;
      const bool inside = gn < p.n && gm < p.m;
      if (!inside && (KIND != kMmaFp32 || !p.mend)) continue;   // (warps stay whole where elements may be summed again)
      const uint32_t at = base + (nn * Tile::kPitch + mm) * 4u;
      float4 v;
      if (p.splits > 1u) {
        v = ld_cluster(at, 0u);
        for (uint32_t s = 1; s < p.splits; ++s) {
          const float4 w = ld_cluster(at, s);
          v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
      } else {
        v = *reinterpret_cast<const float4 *>(out + nn * Tile::kPitch + mm);
      }
      if constexpr (KIND == kMmaFp32) {
        if (p.mend) mend<KA, KB>(v, inside, p, g, gm, gn);
        if (!inside) continue;
      }
      T *c = C + gm * p.c_m + gn;
      const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (uint32_t e = 0; e < 4u; ++e)
        if (gm + e < p.m) store_from_float(c + e * p.c_m, x[e] + (p.accumulate ? load_as_float(c + e * p.c_m) : 0.f));
    }
  }
  if (p.splits > 1u) cluster_barrier();   // nobody leaves while another CTA still reads its tile
}

// Launches one instance.
template <int KIND, int BM, int BN, int WM, int WN, int STAGES, bool KA, bool KB, int LOAD, bool RUNS>
int mma_launch(b200_ctx *ctx, const MmaParams &p, cudaStream_t stream) {
  using Tile = MmaTile<KIND, BM, BN, WM, WN, STAGES>;
  auto kernel = gemm_mma_kernel<KIND, BM, BN, WM, WN, STAGES, KA, KB, LOAD, RUNS>;
  if (Tile::kSmem > 48u * 1024u) {   // opt in once per device
    static std::atomic<unsigned long long> done{0};
    const unsigned long long bit = 1ull << (ctx->device & 63);
    if (!(done.load(std::memory_order_relaxed) & bit)) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Tile::kSmem));
      if (e != cudaSuccess) return static_cast<int>(e);
      done.fetch_or(bit, std::memory_order_relaxed);
    }
  }
  const unsigned grid = p.tiles_m * p.tiles_n * p.groups * p.splits;
  b200::launch(ctx, kernel, dim3(grid), dim3(Tile::kThreads), Tile::kSmem, stream, p.splits, p);
  return static_cast<int>(cudaGetLastError());
}

template <int KIND, int BM, int BN, int WM, int WN, int STAGES, int LOAD, bool RUNS>
int mma_launch_layout(b200_ctx *ctx, const MmaParams &p, bool ka, bool kb, cudaStream_t stream) {
  if (ka) return kb ? mma_launch<KIND, BM, BN, WM, WN, STAGES, true, true, LOAD, RUNS>(ctx, p, stream)
                    : mma_launch<KIND, BM, BN, WM, WN, STAGES, true, false, LOAD, RUNS>(ctx, p, stream);
  return kb ? mma_launch<KIND, BM, BN, WM, WN, STAGES, false, true, LOAD, RUNS>(ctx, p, stream)
            : mma_launch<KIND, BM, BN, WM, WN, STAGES, false, false, LOAD, RUNS>(ctx, p, stream);
}

template <int KIND, int BM, int BN, int WM, int WN, int STAGES, bool RUNS>
int mma_launch_load(b200_ctx *ctx, const MmaParams &p, bool ka, bool kb, cudaStream_t stream) {
  if (p.load == kMmaTma) return mma_launch_layout<KIND, BM, BN, WM, WN, STAGES, kMmaTma, RUNS>(ctx, p, ka, kb, stream);
  if constexpr (KIND == kMmaHalf) {
    if (p.load == kMmaSingle) return mma_launch_layout<KIND, BM, BN, WM, WN, STAGES, kMmaSingle, RUNS>(ctx, p, ka, kb, stream);
  }
  return mma_launch_layout<KIND, BM, BN, WM, WN, STAGES, kMmaWord, RUNS>(ctx, p, ka, kb, stream);
}

template <int KIND, int BM, int BN, int WM, int WN, int STAGES>
int mma_launch_runs(b200_ctx *ctx, const MmaParams &p, bool ka, bool kb, cudaStream_t stream) {
  if constexpr (KIND == kMmaHalf) {
    if (p.kt_per > kMmaHalfRun) return mma_launch_load<KIND, BM, BN, WM, WN, STAGES, true>(ctx, p, ka, kb, stream);
  }
  return mma_launch_load<KIND, BM, BN, WM, WN, STAGES, false>(ctx, p, ka, kb, stream);
}

// The tiles of one kind.
template <int KIND>
int mma_launch_tile(b200_ctx *ctx, const MmaParams &p, int tile, bool ka, bool kb, cudaStream_t stream) {
  switch (tile) {
    case kTile128x8: return mma_launch_runs<KIND, 128, 8, 32, 8, 6>(ctx, p, ka, kb, stream);
    case kTile128x16: return mma_launch_runs<KIND, 128, 16, 32, 16, 5>(ctx, p, ka, kb, stream);
    case kTile128x32: return mma_launch_runs<KIND, 128, 32, 32, 32, 5>(ctx, p, ka, kb, stream);
    case kTile64x64: return mma_launch_runs<KIND, 64, 64, 32, 32, 4>(ctx, p, ka, kb, stream);
    case kTile128x64: return mma_launch_runs<KIND, 128, 64, 32, 32, 4>(ctx, p, ka, kb, stream);
    default:
      // (a second set of accumulators does not leave the registers for it: not for the fp32 kinds, nor for runs)
      if constexpr (KIND != kMmaFp32) return mma_launch_load<KIND, 128, 128, 64, 32, 3, false>(ctx, p, ka, kb, stream);
      else return B200_ERR_INVALID_ARG;
  }
}

}  // namespace
}  // namespace b200

#endif  // PRIMITIV_B200_CSRC_GEMM_MMA_CUH_
