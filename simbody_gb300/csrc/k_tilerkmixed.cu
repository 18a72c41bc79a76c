// k_tilerkmixed.cu -- FP64 steps of mixed batches on the tile driver: those of
// the instances that a mixed integration has in FP64 mode, and all of them once
// it has switched to FP64.
#include "tilerk_device.cuh"

namespace sbg {

void rkTilesMixed(const KArgs& a, const TileSet& S, cudaStream_t s) { rkTilesWith<0>(a, S, s); }

namespace {

// The instances in FP64 mode at this launch on the batch's tiles, where the list
// is longer than `few` (fullTiles).
template <class CF>
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    rkTileListedKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int ntiles, int few,
                       double* __restrict__ recs, double* y, double* __restrict__ time, double* fbuf, int64_t fplane,
                       int32_t* __restrict__ status, double h, StepCtl sc, double accuracy, double consTol, int pes) {
    __shared__ TileShare<4> sh;
    if (T.fbCount[sc.launch & 1] <= few) return;
    forTiles<CF>(T, TT, 0, ntiles, recs, [&](TileCtx c) {
        c.on = c.on && T.fbMode[(int64_t)(sc.launch & 1) * T.ninst + c.inst];
        rkTile<CF, true>(T, TT, c, sh, y, time, fbuf, fplane, status, h, sc, accuracy, consTol, pes != 0);
    });
}

// The instances of a list (T.fbList) of up to `few`, one at a time per block on
// the block's own records (TT: one tile per instance).
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    rkTileListKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int few,
                     double* __restrict__ recs, double* y, double* __restrict__ time, double* fbuf,
                     int64_t fplane, int32_t* __restrict__ status, double h, StepCtl sc, double accuracy, double consTol,
                     int pes) {
    __shared__ TileShare<4> sh;
    const int32_t* list = T.fbList + (int64_t)(sc.launch & 1) * T.ninst;
    const int n = T.fbCount[sc.launch & 1];
    if (n > few) return;
    for (int g = blockIdx.x; g < n; g += gridDim.x) {
        const TileCtx c = tileCtxOne<TileOne>(TT, list[g], recs + TT.recStride * blockIdx.x);
        rkTile<TileOne, true>(T, TT, c, sh, y, time, fbuf, fplane, status, h, sc, accuracy, consTol, pes != 0);
        __syncthreads();
    }
}

}  // namespace

void rkTilesList(const KArgs& a, const TileSet& S, const TileSet& ones, cudaStream_t s) {
    const int blocks = a.T->ninst < ones.blocks ? a.T->ninst : ones.blocks;
    if (blocks <= 0) return;
    const bool full = fullTiles(S, a.T->ninst);
    if (full)
        tileDispatch<0>(S, [&](auto cf) {
            const TileLaunch L(S, S.ntiles);
            rkTileListedKernel<decltype(cf)><<<L.grid, L.block, 0, s>>>(
                *a.T, S.tt, S.ntiles, fewInstances(S), S.recs, a.ystate, a.time, a.T->fbuf64, a.fplane, a.status, a.h, a.step,
                a.accuracy, a.consTol, a.projectEveryStep);
        });
    rkTileListKernel<<<blocks, 32 * ones.tt.W, 0, s>>>(*a.T, ones.tt, full ? fewInstances(S) : a.T->ninst, ones.recs, a.ystate, a.time, a.T->fbuf64, a.fplane, a.status,
                                                       a.h, a.step, a.accuracy, a.consTol, a.projectEveryStep);
}

}  // namespace sbg
