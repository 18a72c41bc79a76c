// k_tilerkmixed.cu -- FP64 steps of mixed batches on the tile driver: those of
// the instances that a mixed integration has in FP64 mode, and all of them once
// it has switched to FP64.
#include "tilerk_device.cuh"

namespace sbg {

void rkTilesMixed(const KArgs& a, const TileSet& S, cudaStream_t s) { rkTilesWith<0>(a, S, s); }

namespace {

// The instances in FP64 mode at this launch (T.fbList), one at a time per
// block on the block's own records (TT: one tile per instance).
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    rkTileListKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, double* __restrict__ recs,
                     int64_t recStride, double* y, double* __restrict__ time, double* fbuf, int64_t fplane,
                     int32_t* __restrict__ status, double h, StepCtl sc, double accuracy, double consTol, int pes) {
    __shared__ TileShare<4> sh;
    const int32_t* list = T.fbList + (int64_t)(sc.launch & 1) * T.ninst;
    const int n = T.fbCount[sc.launch & 1];
    for (int g = blockIdx.x; g < n; g += gridDim.x) {
        const TileCtx c = tileCtxOne<TileOne>(TT, list[g], recs + recStride * blockIdx.x);
        rkTile<TileOne, true>(T, TT, c, sh, y, time, fbuf, fplane, status, h, sc, accuracy, consTol, pes != 0);
        __syncthreads();
    }
}

}  // namespace

void rkTilesList(const KArgs& a, const TileSet& S, cudaStream_t s) {
    const int blocks = a.T->ninst < S.blocks ? a.T->ninst : S.blocks;
    if (blocks <= 0) return;
    rkTileListKernel<<<blocks, 32 * S.tt.W, 0, s>>>(*a.T, S.tt, S.recs, S.recStride, a.ystate, a.time, a.T->fbuf64, a.fplane,
                                                    a.status, a.h, a.step, a.accuracy, a.consTol, a.projectEveryStep);
}

}  // namespace sbg
