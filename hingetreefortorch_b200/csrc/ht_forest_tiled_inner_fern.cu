// Ferns on inputs with inner positions.
#include "ht_forest_tiled_inner.cuh"

namespace ht {
namespace tile {

int launch_inner_ferns(int depth, const TilePlan &plan, const TiledArgs &a, dim3 grid, cudaStream_t stream) {
  return launch_inner_kind<FERN>(depth, plan, a, grid, stream);
}

}  // namespace tile
}  // namespace ht
