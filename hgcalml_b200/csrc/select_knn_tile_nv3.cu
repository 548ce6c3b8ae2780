// Instantiates the tile search for hits of 3 packed float4 record(s).
#include "select_knn_tile.cuh"
namespace hgc {
template int launch_tile_nv<3>(const TileKnnArgs &, int, cudaStream_t);
}
