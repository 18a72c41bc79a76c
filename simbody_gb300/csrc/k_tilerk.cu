// k_tilerk.cu -- FP64 fixed-step RK-Merson on the tile driver, one launch per
// call.
#include "tilerk_device.cuh"

namespace sbg {

void rkTiles(const KArgs& a, const TileSet& S, cudaStream_t s) {
    if (S.tt.ys == kTile) rkTilesWith<kTile>(a, S, s);
    else rkTilesMixed(a, S, s);
}

}  // namespace sbg
