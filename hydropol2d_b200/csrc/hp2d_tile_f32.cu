// Instantiations of the tile step (hp2d_tile.cuh) for float.
#define HP2D_TILE_INSTANTIATE
#include "hp2d_tile.cuh"

namespace hp2d {
template void launch_tile_step<float>(const FusedArgs<float>&, int, bool, bool, bool, int, cudaStream_t);
template void launch_tile_li<float>(const FusedArgs<float>&, const LiArgs<float>&, bool, bool, int, cudaStream_t);
}
