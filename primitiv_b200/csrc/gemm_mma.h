// Host side of the mma.sync matrix product (gemm_mma.cuh): what crosses between the code that picks a
// tile and the translation units that hold the kernels, one per kind.
#ifndef PRIMITIV_B200_CSRC_GEMM_MMA_H_
#define PRIMITIV_B200_CSRC_GEMM_MMA_H_

#include "ctx.h"

namespace b200 {

enum : int { kMmaHalf = 0, kMmaTf32 = 1, kMmaFp32 = 2 };   // storage and arithmetic
// How a kernel fetches its operands: TMA (both meet its alignment rules), 4-byte copies, single halves.
enum : int { kMmaTma = 16, kMmaWord = 4, kMmaSingle = 2 };
enum : int { kTile128x8 = 0, kTile128x16, kTile128x32, kTile64x64, kTile128x64, kTile128x128 };
constexpr uint32_t kMmaHalfRun = 16;   // k-tiles of 64 halves that the tensor core accumulates before their sum goes to registers

struct alignas(64) MmaParams {
  CUtensorMap map_a, map_b;      // load == kMmaTma: dims {contiguous axis, other axis, matrix}
  const void *A, *B;
  void *C;
  uint32_t m, n, k;
  uint32_t tiles_m, tiles_n, groups;
  uint32_t splits;               // CTAs of a cluster that share a tile's contraction
  uint32_t kb;                   // k-tiles of one matrix pair
  uint32_t kt, kt_per;           // k-tiles in all (red * kb), and of one split
  unsigned long long lda, ldb;   // elements from one line to the next
  unsigned long long a_gs, a_rs, b_gs, b_rs, c_gs;
  unsigned long long c_m, c_n;   // element (i, j) of C is at i * c_m + j * c_n; one of the two is 1
  uint32_t a_gmul, a_rmul, b_gmul, b_rmul;   // matrix (g, r) of an operand is number g * gmul + r * rmul of its map
  uint32_t load;
  uint32_t accumulate;
  uint32_t mend;                 // elements that are not finite are summed again, as the CUDA cores would
  int *status;
};

// ka / kb: the operand is K-major.
int mma_launch_half(b200_ctx *ctx, const MmaParams &p, int tile, bool ka, bool kb, cudaStream_t stream);
int mma_launch_tf32(b200_ctx *ctx, const MmaParams &p, int tile, bool ka, bool kb, cudaStream_t stream);
int mma_launch_fp32(b200_ctx *ctx, const MmaParams &p, int tile, bool ka, bool kb, cudaStream_t stream);

}  // namespace b200

#endif  // PRIMITIV_B200_CSRC_GEMM_MMA_H_
