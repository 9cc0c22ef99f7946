#include "lbgb_march.cuh"
#include "lbgb_tile.cuh"

namespace lbgb {
template int launch_march<LBGB_F16DEV>(const MarchCall &c, cudaStream_t s);
template int launch_tile<LBGB_F16DEV>(const TileCall &c, cudaStream_t s);
template int launch_tile_batch<LBGB_F16DEV>(const BatchCall &c, cudaStream_t s);
}  // namespace lbgb
