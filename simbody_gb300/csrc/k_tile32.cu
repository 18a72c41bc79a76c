// k_tile32.cu -- realize(Acceleration), mixed and FP32 forms, on the tile
// driver (kernel variant 9).
#include "tile32_device.cuh"

namespace sbg {

namespace {

template <class CF, int NM, bool REF>
__global__ void __launch_bounds__(32 * kTileMaxWarps, 1)
    realizeTile32Kernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int tile0, int ntiles,
                        const double* __restrict__ y, double* __restrict__ ydot, float* __restrict__ recs,
                        int32_t* __restrict__ status) {
    __shared__ TileShare<0> sh;
    __shared__ TileMax mx;
    const int id = tileId(TT, tile0, ntiles);
    if (id < 0) return;
    const TileCtx c = tileCtx<CF>(T, TT, id, nullptr);
    const YSrc src{y, T.ybase[c.inst], T.ystride[c.inst], T.inq[c.inst]};
    YdOut out{ydot, T.ybase[c.inst], T.ystride[c.inst], T.inq[c.inst]};
    int st = tileRhs32<CF, NM, REF>(T, TT, c, recs, tileStage<NM>(), src, out, true);
    if (!out.finite) st |= SBG_INST_NONFINITE;
    st = tileReduce(TT, c, sh, st);
    if constexpr (REF) st |= tileIll(T, TT, c, mx, out);
    if (c.on && c.w == 0) {
        status[c.inst] = st;
        if constexpr (REF) countFlagged(T, st);
    }
}

template <int NM, bool REF> void go(const KArgs& a, const TileSet& S, int tile0, int ntiles, cudaStream_t s) {
    const TileLaunch L(S, ntiles);
    float* recs = reinterpret_cast<float*>(S.recs);
    auto launch = [&](auto cf) {
        auto* const kernel = realizeTile32Kernel<decltype(cf), NM, REF>;
        kernel<<<L.grid, L.block, tileStageBytes<NM>(kernel, L.block), s>>>(*a.T, S.tt, tile0, ntiles, a.y, a.ydot, recs,
                                                                            a.status);
    };
    if (S.tt.shared) launch(TileCfg<32, true, 0>());
    else launch(TileCfg<32, false, 0>());
}

}  // namespace

void realizeTiles32(const KArgs& a, const TileSet& S, bool refine, int tile0, int ntiles, cudaStream_t s) {
    if (ntiles <= 0) return;
    if (a.P->nm == 1) {
        if (refine) go<1, true>(a, S, tile0, ntiles, s); else go<1, false>(a, S, tile0, ntiles, s);
    } else {
        if (refine) go<3, true>(a, S, tile0, ntiles, s); else go<3, false>(a, S, tile0, ntiles, s);
    }
}

}  // namespace sbg
