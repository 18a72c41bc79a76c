// k_ops.cu -- launch of the tree operators, FP64: the tiles (k_tileops.cu), then
// the loop-closure segment on the level-parallel driver (ops_device.cuh).
#include "abi_device.cuh"
#include "ops_device.cuh"

namespace sbg {

cudaError_t launchTreeOp(const DevTables& T, const LaunchPlan& P, const TileSet& S, const OpIO& io, const double* y,
                         double* scratchLoop, int32_t* status, cudaStream_t s) {
    treeOpTiles(T, S, io, y, status, s);
    if (P.nLoopGroupBlocks > 0)
        treeOpKernel<<<P.nLoopGroupBlocks, 32, 0, s>>>(T, P.loopGroupFirst, y, scratchLoop, io, status);
    return cudaGetLastError();
}

}  // namespace sbg
