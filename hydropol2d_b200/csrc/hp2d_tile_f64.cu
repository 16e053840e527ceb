// Instantiations of the tile step (hp2d_tile.cuh) for double.
#define HP2D_TILE_INSTANTIATE
#include "hp2d_tile.cuh"

namespace hp2d {
template void launch_tile_step<double>(const FusedArgs<double>&, int, bool, bool, bool, int, cudaStream_t);
template void launch_tile_li<double>(const FusedArgs<double>&, const LiArgs<double>&, bool, bool, int, cudaStream_t);
}
