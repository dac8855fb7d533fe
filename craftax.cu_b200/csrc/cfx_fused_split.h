// Launcher of the small-batch form of the fused forward (cfx_fused_split.cu).
#pragma once
#include "cfx_fused_common.cuh"

namespace cfx {
namespace fused {

// Sets the kernel for clusters of S CTAs up on the current device; *max_clusters: how many run at once (0: not
// built for the shape, or not with the registers it needs).
int split_prepare(int precision, int game, int H, int S, int sm_count, int* max_clusters);
// One cluster of S CTAs for each of `tiles` tiles of P.tile_rows rows (32, 64 or 128) from row 128 P.tile_begin on;
// P.state_map: boxes of 32 rows x 32 units.
int split_launch(int precision, int game, int H, int S, int tiles, const Params& P, cudaStream_t st);

}  // namespace fused
}  // namespace cfx
