#include "lbgb_tile.cuh"

namespace lbgb {
template int launch_tile<LBGB_F64>(const TileCall &c, cudaStream_t s);
template int launch_tile_batch<LBGB_F64>(const BatchCall &c, cudaStream_t s);
}  // namespace lbgb
