// k_tile.cu -- FP64 realize(Acceleration) and M^-1 f on the tile driver, and
// the FP64 recomputation of a mixed realize's ill-conditioned instances.
#include "tile_device.cuh"

namespace sbg {

namespace {

// FLAGGED: the FP64 recomputation of a mixed realize's instances that reported
// an ill-conditioned M, where there are more than `few` of them (fullTiles); the
// other lanes stay idle. T.fallbacks counts them.
template <class CF, bool FLAGGED>
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    realizeTileKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int tile0, int ntiles,
                      const double* __restrict__ y, double* __restrict__ ydot, double* __restrict__ recs,
                      int32_t* __restrict__ status, int few) {
    __shared__ TileShare<0> sh;
    if (FLAGGED && *T.flagged <= few) return;
    forTiles<CF>(T, TT, tile0, ntiles, recs, [&](TileCtx c) {
        if constexpr (FLAGGED) {
            c.on = c.on && (status[c.inst] & SBG_INST_ILL_CONDITIONED);
            const int n = __popc(__ballot_sync(0xffffffffu, c.on));
            if (n == 0) return;  // every warp of the tile counts the same
            if (c.w == 0 && c.lane == 0) atomicAdd(T.fallbacks, (unsigned long long)n);
        }
        const TileYSrc<CF::YS> src{{T, c.inst}, y};
        TileOut<CF::YS> out(src.c, ydot);
        int st = tileRhs<CF, false>(T, TT, c, src, out, true);
        if (!out.finite) st |= SBG_INST_NONFINITE;
        st = tileReduce(TT, c, sh, st);
        if (c.on && c.w == 0) status[c.inst] = st;
    });
}

template <class CF>
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    minvTileKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int ntiles,
                   const double* __restrict__ y,
                   const double* __restrict__ f, double* __restrict__ o, double* __restrict__ recs,
                   int32_t* __restrict__ status) {
    __shared__ TileShare<0> sh;
    forTiles<CF>(T, TT, 0, ntiles, recs, [&](const TileCtx& c) {
        const TileFSrc<CF::YS> src{{T, c.inst}, y, f};
        TileUOut<CF::YS> out(src.c, o);
        int st = tileRhs<CF, true>(T, TT, c, src, out, true);
        if (!out.finite) st |= SBG_INST_NONFINITE;
        st = tileReduce(TT, c, sh, st);
        if (c.on && c.w == 0) status[c.inst] = st;
    });
}

// The instances at order positions [first, first + count) whose mixed realize
// reported an ill-conditioned M and that are still flagged, one at a time per
// block on the block's own records (TT: one tile per instance). A block takes
// every gridDim-th position, so that neighbours (instances of one topology lie
// side by side and are often flagged together) go to different blocks.
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    realizeFallbackTileKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int first,
                              int count, const double* __restrict__ y, double* __restrict__ ydot,
                              double* __restrict__ recs, int32_t* __restrict__ status) {
    __shared__ TileShare<0> sh;
    __shared__ int list[32 * kTileMaxWarps], n;
    for (int64_t k0 = 0; blockIdx.x + k0 * gridDim.x < count; k0 += blockDim.x) {
        if (threadIdx.x == 0) n = 0;
        __syncthreads();
        const int64_t p = blockIdx.x + (k0 + threadIdx.x) * gridDim.x;
        if (p < count) {
            const int inst = T.order[first + p];
            if (status[inst] & SBG_INST_ILL_CONDITIONED) list[atomicAdd(&n, 1)] = inst;
        }
        __syncthreads();
        for (int k = 0; k < n; ++k) {
            const TileCtx c = tileCtxOne<TileOne>(TT, list[k], recs + TT.recStride * blockIdx.x);
            const TileYSrc<0> src{{T, c.inst}, y};
            TileOut<0> out(src.c, ydot);
            int st = tileRhs<TileOne, false>(T, TT, c, src, out, true);
            if (!out.finite) st |= SBG_INST_NONFINITE;
            st = tileReduce(TT, c, sh, st);
            if (c.on && c.w == 0) {
                status[c.inst] = st;
                atomicAdd(T.fallbacks, 1ULL);
            }
        }
        __syncthreads();  // the list is written again
    }
}

}  // namespace

void realizeTiles(const KArgs& a, const TileSet& S, int tile0, int ntiles, cudaStream_t s) {
    if (ntiles <= 0) return;
    const TileLaunch L(S, ntiles);
    tileDispatch<kTile>(S, [&](auto cf) {
        realizeTileKernel<decltype(cf), false><<<L.grid, L.block, 0, s>>>(*a.T, S.tt, tile0, ntiles, a.y, a.ydot, S.recs,
                                                                         a.status, 0);
    });
}
void minvTiles(const KArgs& a, const TileSet& S, cudaStream_t s) {
    if (S.ntiles <= 0) return;
    const TileLaunch L(S, S.ntiles);
    tileDispatch<kTile>(S, [&](auto cf) {
        minvTileKernel<decltype(cf)><<<L.grid, L.block, 0, s>>>(*a.T, S.tt, S.ntiles, a.y, a.f, a.ydot, S.recs, a.status);
    });
}
void realizeFallbackTiles(const KArgs& a, const TileSet& S, int tile0, int ntiles, const TileSet& ones, int first, int count,
                          int block0, int blocks, cudaStream_t s) {
    if (count <= 0) return;
    if (fullTiles(S, count))
        tileDispatch<0>(S, [&](auto cf) {
            const TileLaunch L(S, ntiles);
            realizeTileKernel<decltype(cf), true><<<L.grid, L.block, 0, s>>>(*a.T, S.tt, tile0, ntiles, a.y, a.ydot, S.recs,
                                                                             a.status, fewInstances(S));
        });
    realizeFallbackTileKernel<<<count < blocks ? count : blocks, 32 * ones.tt.W, 0, s>>>(
        *a.T, ones.tt, first, count, a.y, a.ydot, ones.recs + ones.tt.recStride * block0, a.status);
}

}  // namespace sbg
