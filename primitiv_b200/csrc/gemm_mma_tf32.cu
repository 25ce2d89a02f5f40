#include "gemm_mma.cuh"

namespace b200 {

int mma_launch_tf32(b200_ctx *ctx, const MmaParams &p, int tile, bool ka, bool kb, cudaStream_t stream) {
  return mma_launch_tile<kMmaTf32>(ctx, p, tile, ka, kb, stream);
}

}  // namespace b200
