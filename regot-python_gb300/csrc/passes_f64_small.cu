// Dense passes over FP64 M with the tiles of small problems (tile_rows).
#include "dense_pass.cuh"

namespace regot {
template void launch_pass_cfg<double, kSmallCfg>(int, const PassParams&, cudaStream_t, int);
template int occupancy_cfg<double, kSmallCfg>(int);
}  // namespace regot
