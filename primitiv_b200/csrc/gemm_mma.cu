// Picks tile, split and copy widths of the mma.sync matrix product (gemm_mma.cuh).
#include "gemm_mma.h"

#include <cstdlib>
#include <cstring>
#include <utility>

namespace b200 {
namespace {

struct MmaOperand {
  const void *ptr;
  uint32_t mn;
  bool k_major;
  uint64_t ld, gs, rs;
  bool tma_ok(uint32_t groups, uint32_t red, int es) const {
    const bool g_on = groups > 1 && gs != 0, r_on = red > 1 && rs != 0;
    if (g_on && r_on) return false;   // two batch axes
    return (reinterpret_cast<uintptr_t>(ptr) | ld * es | (g_on ? gs * es : 0) | (r_on ? rs * es : 0)) % 16 == 0;
  }
};

// A product as the kernels take it.
struct MmaProblem {
  MmaOperand a, b;
  bool exchanged;
  int kind, es;
  uint32_t kb;      // k-tiles of one matrix pair
  uint64_t kt;      // and of the whole contraction
  uint32_t load;
};

MmaProblem describe(const GemmArgs &g) {
  MmaProblem p;
  p.kind = g.mode == B200_MODE_FP16 ? kMmaHalf : g.mode == B200_MODE_TF32 && !has_fp32_sums(g) ? kMmaTf32 : kMmaFp32;
  p.es = elem_bytes(g.mode);
  p.a = {g.A, g.m, g.trans_a != 0, g.trans_a ? g.k : g.m, g.a_gs, g.a_rs};
  p.b = {g.B, g.n, g.trans_b == 0, g.trans_b ? g.n : g.k, g.b_gs, g.b_rs};
  p.exchanged = g.m < g.n && g.m <= 32u;   // few rows: the transposed product, whose few columns have tiles of their own
  if (p.exchanged) std::swap(p.a, p.b);
  const uint32_t bk = 128u / p.es;
  p.kb = (g.k + bk - 1) / bk;
  p.kt = static_cast<uint64_t>(p.kb) * g.red;
  if (p.a.tma_ok(g.groups, g.red, p.es) && p.b.tma_ok(g.groups, g.red, p.es)) {
    p.load = kMmaTma;
  } else {
    uint64_t all = reinterpret_cast<uintptr_t>(p.a.ptr) | reinterpret_cast<uintptr_t>(p.b.ptr) | p.a.ld * p.es | p.b.ld * p.es;
    if (g.groups > 1) all |= (p.a.gs | p.b.gs) * p.es;
    if (g.red > 1) all |= (p.a.rs | p.b.rs) * p.es;
    p.load = all % 4 ? kMmaSingle : kMmaWord;
  }
  return p;
}

struct MmaChoice {
  int tile;
  uint32_t splits;
  double us;
};

constexpr uint32_t kTileM[] = {128, 128, 128, 64, 128, 128}, kTileN[] = {8, 16, 32, 64, 64, 128};

// Tile and split by an estimate fitted to 87 products (extents 1 to 4096, all tiles, splits 1 to 8): a CTA takes
// `step` us per k-tile (latency: each k-tile is fetched, waited for and multiplied by a handful of warps) and
// `ends` us besides, two CTAs of the small tiles and one of the large ones run at full speed on an SM, and
// adding up a split costs 1.8 us.  Within 6 % of the best choice on average.
MmaChoice choose(const b200_ctx *ctx, const GemmArgs &g, const MmaProblem &p) {
  static const double kStep[3][6] = {{0.40, 0.48, 0.54, 0.59, 0.60, 0.95}, {0.52, 0.55, 0.60, 0.66, 0.70, 0.95}, {0.75, 0.86, 1.0, 1.15, 1.25, 0.0}};
  static const double kEnds[3][6] = {{1.8, 2.0, 2.5, 2.1, 3.0, 4.4}, {2.0, 2.2, 2.9, 2.4, 3.3, 5.0}, {2.2, 2.4, 3.2, 2.7, 4.2, 0.0}};
  MmaChoice best{kTile64x64, 1, 1e30};
  for (int t = 0; t < 6; ++t) {
    if (p.kind == kMmaFp32 && t == kTile128x128) continue;
    if (t > kTile128x8 && kTileN[t] / 2u >= p.b.mn) continue;   // half the columns or more would be padding
    double step = kStep[p.kind][t];
    if (p.load == kMmaWord && step < 1.8) step = 1.8;     // narrow copies bound a k-tile instead
    if (p.load == kMmaSingle && step < 6.0) step = 6.0;
    const double tiles = static_cast<double>((p.a.mn + kTileM[t] - 1) / kTileM[t]) * ((p.b.mn + kTileN[t] - 1) / kTileN[t]) * g.groups;
    const int *clusters = t <= kTile64x64 ? ctx->cluster_room_two : ctx->cluster_room;
    for (uint32_t s = 1; s <= 8u && s <= p.kt; ++s) {
      if (t == kTile128x128 && p.kind == kMmaHalf && (p.kt + s - 1) / s > kMmaHalfRun) continue;   // (it has no second set of registers)
      // A cluster has to find its SMs free in one GPC.  Of clusters of eight with two CTAs to an SM 33 fit an
      // idle GPU, but a layer of 4096 halves over 8 columns that needs 32 of them waits for what the kernel in
      // front still holds: 14 us in a chain, 9 with seven.  Hence a tenth in reserve.
      const double waves = tiles / (s > 1u ? 0.9 * clusters[s] : clusters[s]);
      const double whole = static_cast<double>(static_cast<uint64_t>(waves + 0.999));
      // (what is bound by arithmetic, or comes in clusters, pays for a started wave)
      const double load = waves <= 1.0 ? 1.0 : (p.kind == kMmaFp32 || s > 1u) ? 0.5 * (waves + whole) : waves;
      const double us = load * (static_cast<double>((p.kt + s - 1) / s) * step + kEnds[p.kind][t]) + (s > 1u ? 1.8 : 0.0);
      if (us < best.us) best = {t, s, us};
    }
  }
  return best;
}

// Never launched: what the driver is asked about.
__global__ void room_kernel() { pdl_enter(); }

// Tensor map of an operand for tiles of `rows`: the box and swizzle that gemm_mma.cuh's Layout describes.
bool make_map(const b200_ctx *ctx, const MmaOperand &o, uint32_t k, uint32_t groups, uint32_t red, int es, uint32_t rows,
              CUtensorMap *map, uint32_t *gmul, uint32_t *rmul) {
  const bool g_on = groups > 1 && o.gs != 0, r_on = red > 1 && o.rs != 0;
  *gmul = g_on;
  *rmul = r_on;
  const uint32_t inner = o.k_major ? k : o.mn, outer = o.k_major ? o.mn : k;
  const uint64_t count = g_on ? groups : r_on ? red : 1, stride = g_on ? o.gs : r_on ? o.rs : o.ld * outer;
  const uint32_t line = o.k_major ? 128u : (rows * es < 128u ? rows * es : 128u);
  cuuint64_t dims[3] = {inner, outer, count}, strides[2] = {o.ld * es, stride * es};
  cuuint32_t box[3] = {line / es, o.k_major ? rows : 128u / es, 1}, step[3] = {1, 1, 1};
  CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE;
  if (line == 128u) swizzle = (!o.k_major && es == 4) ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B;
  else if (line == 64u) swizzle = CU_TENSOR_MAP_SWIZZLE_64B;
  else if (line == 32u && es == 2) swizzle = CU_TENSOR_MAP_SWIZZLE_32B;
  return ctx->encode_tiled(map, es == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                           const_cast<void *>(o.ptr), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

int gemm_find_rooms(b200_ctx *ctx) {
  for (unsigned s = 1; s <= 8u; ++s) {
    for (int two = 0; two < 2; ++two) {
      const unsigned smem = (two ? 106u : 200u) * 1024u;   // two CTAs of the smaller tiles fit an SM, one of everything else
      B200_CUDA_TRY(cudaFuncSetAttribute(room_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = s;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.gridDim = dim3(s);
      cfg.blockDim = dim3(128);
      cfg.dynamicSmemBytes = smem;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int *room = two ? &ctx->cluster_room_two[s] : &ctx->cluster_room[s];
      B200_CUDA_TRY(cudaOccupancyMaxActiveClusters(room, room_kernel, &cfg));
      if (*room < 1) *room = 1;
    }
  }
  return B200_OK;
}

double gemm_mma_estimate(const b200_ctx *ctx, const GemmArgs &g) {
  // (half planes lose less than TF32 ones where the sum is that short, see gemm_direct_estimate; this kernel takes
  // what cannot have them, two batch axes among it)
  if (g.mode == B200_MODE_FP32_3XFP16 && static_cast<uint64_t>(g.k) * g.red < 64u && !has_fp32_sums(g)) return 1e30;
  const MmaProblem p = describe(g);
  // (the fixed part was fitted with the rest: `ends` has it)
  return choose(ctx, g, p).us + 0.5;
}

int gemm_mma(b200_ctx *ctx, const GemmArgs &g, cudaStream_t stream) {
  const MmaProblem q = describe(g);
  MmaChoice c = choose(ctx, g, q);
#ifdef PRIMITIV_B200_DEV_KNOBS
  if (const char *e = std::getenv("PRIMITIV_B200_MMA_TILE")) c.tile = std::atoi(e);
  if (const char *e = std::getenv("PRIMITIV_B200_MMA_SPLITS")) c.splits = std::atoi(e);
  if (q.kind == kMmaFp32 && c.tile == kTile128x128) c.tile = kTile128x64;
#endif
  if (q.kt > 0x7fffffffull) return B200_ERR_TOO_LARGE;
  MmaParams p;
  std::memset(&p, 0, sizeof(p));
  p.C = g.C;
  p.c_gs = g.c_gs;
  p.c_m = q.exchanged ? g.m : 1;
  p.c_n = q.exchanged ? 1 : g.m;
  p.m = q.a.mn;
  p.n = q.b.mn;
  p.k = g.k;
  p.groups = g.groups;
  p.accumulate = g.accumulate ? 1u : 0u;
  p.status = ctx->d_status;
  p.load = q.load;
  if (q.load == kMmaTma) {
    if (!make_map(ctx, q.a, g.k, g.groups, g.red, q.es, kTileM[c.tile], &p.map_a, &p.a_gmul, &p.a_rmul) ||
        !make_map(ctx, q.b, g.k, g.groups, g.red, q.es, kTileN[c.tile], &p.map_b, &p.b_gmul, &p.b_rmul))
      return B200_ERR_DRIVER;
  }
  p.A = q.a.ptr; p.lda = q.a.ld; p.a_gs = q.a.gs; p.a_rs = q.a.rs;
  p.B = q.b.ptr; p.ldb = q.b.ld; p.b_gs = q.b.gs; p.b_rs = q.b.rs;
  p.mend = q.kind == kMmaFp32 && has_fp32_sums(g) ? 1u : 0u;
  p.tiles_m = (p.m + kTileM[c.tile] - 1) / kTileM[c.tile];
  p.tiles_n = (p.n + kTileN[c.tile] - 1) / kTileN[c.tile];
  p.kb = q.kb;
  p.kt = static_cast<uint32_t>(q.kt);
  p.kt_per = (p.kt + c.splits - 1) / c.splits;
  p.splits = (p.kt + p.kt_per - 1) / p.kt_per;   // no empty splits
  if (static_cast<uint64_t>(p.tiles_m) * p.tiles_n * g.groups * p.splits > 0x7fffffffull) return B200_ERR_TOO_LARGE;
  ProfScope prof(ctx, kProfGemmSimt, stream);
  ++ctx->launches;
  if (q.kind == kMmaHalf) return mma_launch_half(ctx, p, c.tile, q.a.k_major, q.b.k_major, stream);
  if (q.kind == kMmaTf32) return mma_launch_tf32(ctx, p, c.tile, q.a.k_major, q.b.k_major, stream);
  return mma_launch_fp32(ctx, p, c.tile, q.a.k_major, q.b.k_major, stream);
}

}  // namespace b200
