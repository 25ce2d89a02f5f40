// CUDA-core matrix product: the path for operands the tensor-core kernel cannot
// take (leading dimensions or pointers not 16-byte aligned, e.g. 123x123 or
// {10,1024}) and for problems too small to fill a 128-row MMA tile.
//
//   C[g] = (acc ? C[g] : 0) + sum_{r<red} opA(A[g*a_gs + r*a_rs]) . opB(B[g*b_gs + r*b_rs])
//
// 64x64 output tile per CTA, 16-deep k slices staged in shared memory, 4x4
// outputs per thread, fp32 FMA accumulation for both float and half storage;
// half results are rounded once on store.  The reduction over `red` runs inside
// the k loop, so a broadcast operand's gradient is summed without atomics and
// without the serial per-batch GEMM loop of the reference
// (primitiv/devices/cuda/ops/matmul.cu:113-123).
#include <cuda_fp16.h>

#include "ctx.h"

namespace b200 {
namespace {

constexpr int TM = 64, TN = 64, TK = 16, NT = 256;

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
__device__ __forceinline__ void from_f32(float &d, float v) { d = v; }
__device__ __forceinline__ void from_f32(__half &d, float v) { d = __float2half_rn(v); }

template <typename T, bool kTA, bool kTB>
__global__ void __launch_bounds__(NT) gemm_simt_kernel(
    const T *__restrict__ A, const T *__restrict__ B, T *__restrict__ C,
    uint32_t m, uint32_t n, uint32_t k, uint32_t red,
    uint64_t a_gs, uint64_t a_rs, uint64_t b_gs, uint64_t b_rs, uint64_t c_gs,
    int accumulate, uint32_t tiles_m, uint32_t tiles_n) {
  pdl_enter();
  __shared__ float As[TK][TM + 1];
  __shared__ float Bs[TK][TN + 1];

  const uint32_t tile = blockIdx.x;
  const uint32_t g = tile / (tiles_m * tiles_n);
  const uint32_t rem = tile - g * tiles_m * tiles_n;
  const uint32_t m0 = (rem % tiles_m) * TM;
  const uint32_t n0 = (rem / tiles_m) * TN;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (uint32_t r = 0; r < red; ++r) {
    const T *Ag = A + g * a_gs + r * a_rs;
    const T *Bg = B + g * b_gs + r * b_rs;
    for (uint32_t k0 = 0; k0 < k; k0 += TK) {
#pragma unroll
      for (int i = 0; i < (TM * TK) / NT; ++i) {
        const int e = tid + i * NT;
        int mm, kk;
        if (kTA) { kk = e % TK; mm = e / TK; } else { mm = e % TM; kk = e / TM; }
        const uint32_t gm = m0 + mm, gk = k0 + kk;
        float v = 0.f;
        if (gm < m && gk < k)
          v = to_f32(kTA ? Ag[(uint64_t)gk + (uint64_t)gm * k] : Ag[(uint64_t)gm + (uint64_t)gk * m]);
        As[kk][mm] = v;
      }
#pragma unroll
      for (int i = 0; i < (TN * TK) / NT; ++i) {
        const int e = tid + i * NT;
        int nn, kk;
        if (kTB) { nn = e % TN; kk = e / TN; } else { kk = e % TK; nn = e / TK; }
        const uint32_t gn = n0 + nn, gk = k0 + kk;
        float v = 0.f;
        if (gn < n && gk < k)
          v = to_f32(kTB ? Bg[(uint64_t)gn + (uint64_t)gk * n] : Bg[(uint64_t)gk + (uint64_t)gn * k]);
        Bs[kk][nn] = v;
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < TK; ++kk) {
        float av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = As[kk][tx + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[j] = Bs[kk][ty + 16 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
      __syncthreads();
    }
  }

  T *Cg = C + g * c_gs;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t gn = n0 + ty + 16 * j;
    if (gn >= n) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t gm = m0 + tx + 16 * i;
      if (gm >= m) continue;
      T *p = Cg + (uint64_t)gm + (uint64_t)gn * m;
      float v = acc[i][j];
      if (accumulate) v += to_f32(*p);
      from_f32(*p, v);
    }
  }
}

template <typename T>
int launch(b200_ctx *ctx, const GemmArgs &a, cudaStream_t s) {
  const uint32_t tiles_m = (a.m + TM - 1) / TM, tiles_n = (a.n + TN - 1) / TN;
  const uint64_t tiles = (uint64_t)tiles_m * tiles_n * a.groups;
  if (tiles == 0) return B200_OK;
  if (tiles > 0x7fffffffull) return B200_ERR_TOO_LARGE;
  const dim3 grid((unsigned)tiles), block(NT);
  const T *A = static_cast<const T *>(a.A);
  const T *B = static_cast<const T *>(a.B);
  T *C = static_cast<T *>(a.C);
  ProfScope prof(ctx, kProfGemmSimt, s);
#define B200_SIMT_LAUNCH(TA, TB)                                                              \
  b200::launch(ctx, gemm_simt_kernel<T, TA, TB>, dim3(grid), dim3(block), 0, s, 1u, A, B, C, a.m, a.n, a.k, a.red, a.a_gs, \
                                                     a.a_rs, a.b_gs, a.b_rs, a.c_gs,        \
                                                     a.accumulate, tiles_m, tiles_n)
  if (a.trans_a) {
    if (a.trans_b) B200_SIMT_LAUNCH(true, true); else B200_SIMT_LAUNCH(true, false);
  } else {
    if (a.trans_b) B200_SIMT_LAUNCH(false, true); else B200_SIMT_LAUNCH(false, false);
  }
#undef B200_SIMT_LAUNCH
  ++ctx->launches;
  return (int)cudaGetLastError();
}

// The same sums in the same order (fused multiply-adds by rising k, so the same bits) for a few thousand outputs:
// one output per thread, 8 x 16 tiles, k in slices of 128 that are fetched while the one before is summed.
// Bound by the latency of a slice.  A 64 x 64 tile in steps of 16 leaves 10 x 200 x 800 to 4 CTAs that wait for
// memory 50 times: 69 us, 8.0 here.
constexpr uint32_t SM = 8, SN = 16, SK = 128, ST = SM * SN;

template <bool kTA, bool kTB>
__global__ void __launch_bounds__(ST) gemm_serial_kernel(const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ C, uint32_t m,
                                                         uint32_t n, uint32_t k, uint32_t red, uint64_t a_gs, uint64_t a_rs, uint64_t b_gs,
                                                         uint64_t b_rs, uint64_t c_gs, int accumulate, uint32_t tiles_m, uint32_t tiles_n) {
  pdl_enter();
  __shared__ __align__(16) float As[2][SM][SK + 4], Bs[2][SN][SK + 4];
  const uint32_t g = blockIdx.x / (tiles_m * tiles_n), rem = blockIdx.x - g * tiles_m * tiles_n;
  const uint32_t m0 = (rem % tiles_m) * SM, n0 = (rem / tiles_m) * SN, t = threadIdx.x, i = t % SM, j = t / SM;
  float ra[SM], rb[SN];   // this thread's elements of the next slice
  auto fetch = [&](uint32_t r, uint32_t k0) {
    const float *Ag = A + g * a_gs + r * a_rs, *Bg = B + g * b_gs + r * b_rs;
#pragma unroll
    for (uint32_t u = 0; u < SM; ++u) {
      const uint32_t e = t + u * ST, mm = kTA ? e / SK : e % SM, kk = kTA ? e % SK : e / SM, gm = m0 + mm, gk = k0 + kk;
      ra[u] = gm < m && gk < k ? Ag[kTA ? gk + static_cast<uint64_t>(gm) * k : gm + static_cast<uint64_t>(gk) * m] : 0.f;
    }
#pragma unroll
    for (uint32_t u = 0; u < SN; ++u) {
      const uint32_t e = t + u * ST, nn = kTB ? e % SN : e / SK, kk = kTB ? e / SN : e % SK, gn = n0 + nn, gk = k0 + kk;
      rb[u] = gn < n && gk < k ? Bg[kTB ? gn + static_cast<uint64_t>(gk) * n : gk + static_cast<uint64_t>(gn) * k] : 0.f;
    }
  };
  float acc = 0.f;
  uint32_t r = 0, k0 = 0, buf = 0;
  fetch(0, 0);
  for (;;) {
#pragma unroll
    for (uint32_t u = 0; u < SM; ++u) {
      const uint32_t e = t + u * ST;
      As[buf][kTA ? e / SK : e % SM][kTA ? e % SK : e / SM] = ra[u];
    }
#pragma unroll
    for (uint32_t u = 0; u < SN; ++u) {
      const uint32_t e = t + u * ST;
      Bs[buf][kTB ? e % SN : e / SK][kTB ? e / SN : e % SK] = rb[u];
    }
    __syncthreads();   // (a buffer is written again only after the next slice's barrier)
    const uint32_t count = k - k0 < SK ? k - k0 : SK;
    bool more = true;
    k0 += SK;
    if (k0 >= k) {
      k0 = 0;
      more = ++r < red;
    }
    if (more) fetch(r, k0);
#pragma unroll 8
    for (uint32_t q = 0; q < count; q += 4u) {
      const float4 a = *reinterpret_cast<const float4 *>(&As[buf][i][q]), b = *reinterpret_cast<const float4 *>(&Bs[buf][j][q]);
      acc = fmaf(a.x, b.x, acc);
      acc = fmaf(a.y, b.y, acc);
      acc = fmaf(a.z, b.z, acc);
      acc = fmaf(a.w, b.w, acc);
    }
    if (!more) break;
    buf ^= 1u;
  }
  if (m0 + i < m && n0 + j < n) {
    float *c = C + g * c_gs + (m0 + i) + static_cast<uint64_t>(n0 + j) * m;
    *c = accumulate ? acc + *c : acc;
  }
}

}  // namespace

int gemm_simt(b200_ctx *ctx, const GemmArgs &a, cudaStream_t s) {
  if (a.mode == B200_MODE_FP16) return launch<__half>(ctx, a, s);
  return launch<float>(ctx, a, s);
}

// A launch and 1.3 us per step of 16 terms, more where CTAs share an SM: fitted to 220 products of up to 1200 terms, off by 17 %
// on average.
double gemm_simt_estimate(const b200_ctx *ctx, const GemmArgs &a) {
  const double steps = static_cast<double>((a.k + TK - 1) / TK) * a.red;
  const double waves = static_cast<double>((a.m + TM - 1) / TM) * ((a.n + TN - 1) / TN) * a.groups / ctx->sm_count;
  return 2.25 + steps * (waves > 1.625 ? 0.8 * waves : 1.3) + (waves > 1.0 ? 0.3 * (waves - 1.0) : 0.0);
}

// A launch and 0.95 us per slice of k, while four CTAs fit an SM: fitted to 18 products (2.1 us for 64^3, 9.3 for
// 200 x 8 x 1000, 24.8 for 20 x 30 x 3000).
double gemm_serial_estimate(const b200_ctx *ctx, const GemmArgs &a) {
  if (a.mode == B200_MODE_FP16) return 1e30;
  const double tiles = static_cast<double>((a.m + SM - 1) / SM) * ((a.n + SN - 1) / SN) * a.groups, waves = tiles / (4.0 * ctx->sm_count);
  return 1.3 + 0.95 * ((a.k + SK - 1) / SK) * a.red * (waves > 1.0 ? waves : 1.0);
}

int gemm_serial(b200_ctx *ctx, const GemmArgs &a, cudaStream_t s) {
  if (a.mode == B200_MODE_FP16) return B200_ERR_INVALID_ARG;
  const uint32_t tiles_m = (a.m + SM - 1) / SM, tiles_n = (a.n + SN - 1) / SN;
  const uint64_t tiles = static_cast<uint64_t>(tiles_m) * tiles_n * a.groups;
  if (tiles > 0x7fffffffull) return B200_ERR_TOO_LARGE;
  ProfScope prof(ctx, kProfGemmSimt, s);
  auto kernel = a.trans_a ? (a.trans_b ? gemm_serial_kernel<true, true> : gemm_serial_kernel<true, false>)
                          : (a.trans_b ? gemm_serial_kernel<false, true> : gemm_serial_kernel<false, false>);
  b200::launch(ctx, kernel, dim3(static_cast<unsigned>(tiles)), dim3(ST), 0, s, 1u, static_cast<const float *>(a.A), static_cast<const float *>(a.B),
               static_cast<float *>(a.C), a.m, a.n, a.k, a.red, a.a_gs, a.a_rs, a.b_gs, a.b_rs, a.c_gs, a.accumulate, tiles_m, tiles_n);
  ++ctx->launches;
  return static_cast<int>(cudaGetLastError());
}

}  // namespace b200
