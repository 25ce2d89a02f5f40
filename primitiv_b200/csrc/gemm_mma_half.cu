#include "gemm_mma.cuh"

namespace b200 {

int mma_launch_half(b200_ctx *ctx, const MmaParams &p, int tile, bool ka, bool kb, cudaStream_t stream) {
  return mma_launch_tile<kMmaHalf>(ctx, p, tile, ka, kb, stream);
}

}  // namespace b200
