// tile32_device.cuh -- the mixed and FP32 forms on the tile driver: the chain
// driver's per-body routines (abi_device.cuh), taken in the order of a tile's
// schedule by the warps of a block instead of one thread's row by row.
//
// The one-thread driver is bound by latency: a few warps per SM, each walking
// its 32 trees' rows one after another through five passes of dependent loads
// and FP32 chains, lanes apart on mobilizers. Here up to eight warps share the
// 32 trees, a body of each a step, so a pass has as many steps as the trees are
// deep or an eighth of their rows, whichever is more. Every routine and the
// order in which a parent's children add to it (falling rows, kept by the
// schedule) are the chain driver's, so the results are the same bit for bit.
#pragma once
#include "abi_device.cuh"
#include "tile_device.cuh"

namespace sbg {

// One RHS of the tile's instances for which `active` holds. A slot's record is
// at slot * TT.rsTotal in the tile's interleaved records.
template <class CF, int NM, bool REF, class Src, class Out>
__device__ __forceinline__ int tileRhs32(const DevTables& T, const TileTables& TT, const TileCtx& c, float* recs,
                                         const Src& src, Out& out, bool active) {
    const int body0 = T.ibody[c.inst], rs = TT.rsTotal;
    const V3<float> g = mk3(float(T.grav[3 * c.inst]), float(T.grav[3 * c.inst + 1]), float(T.grav[3 * c.inst + 2]));
    const ScrTiled<float> S{recs + c.d.rec0 + c.lane};
    const bool run = c.on && active;
    bool ok = true;
    tileSweep<CF, true>(TT, c, run, [&](int, int slot, const tile::SlotRow& r, auto) {
        const int rec = slot * rs;
        const Kin<float> P = r.parent < 0 ? groundKin<float>() : loadKin<float>(S, r.parent * rs);
        const Kin<float> K = body1<float, NM>(T, body0 + r.row, rec, S, src, out, g, P);
        storeKin(S, rec, K);
        storeC2(S, rec, zeroC2<float>());
    });
    tileSweep<CF, false>(TT, c, run, [&](int cl, int slot, const tile::SlotRow& r, auto) {
        const int rec = slot * rs, row = body0 + r.row;
        const float m = T.par32[(int64_t)row * kParamStride];
        const C2<float> in = loadC2<float>(S, rec);
        C2<float> outC;
        if (cl == tile::CL_FREE) ok &= body2Free<float>(T, row, rec, S, m, in, outC);
        else ok &= body2<float, NM>(T, row, rec, (r.info >> 4) & 15, S, m, in, outC);
        if (r.parent >= 0) pushC2(S, r.parent * rs, outC);
    });
    tileSweep<CF, true>(TT, c, run, [&](int cl, int slot, const tile::SlotRow& r, auto) {
        const int rec = slot * rs, row = body0 + r.row;
        const A3<float> Ap = r.parent < 0 ? A3<float>{} : loadA3<float>(S, r.parent * rs, REF);
        A3<float> A;
        if (cl == tile::CL_FREE) body3Free<float, REF>(T, row, rec, S, out, Ap, r.parent >= 0, A);
        else A = body3<float, NM, REF>(T, row, rec, (r.info >> 4) & 15, S, out, Ap, r.parent >= 0);
        storeA3(S, rec, A, REF);
        if constexpr (REF)
            for (int i = 0; i < 6; ++i) S(rec, kRecZ2acc + i) = 0.f;
    });
    if constexpr (REF) {
        tileSweep<CF, false>(TT, c, run, [&](int cl, int slot, const tile::SlotRow& r, auto) {
            const int rec = slot * rs, row = body0 + r.row;
            const C4 own = loadC4(S, rec);
            C4 outC;
            if (cl == tile::CL_FREE) body4Free(T, row, rec, S, own, zeroC4(), outC);
            else outC = body4<NM>(T, row, rec, (r.info >> 4) & 15, S, own, zeroC4());
            if (r.parent >= 0) {
                C4 a = loadC4(S, r.parent * rs);
                addC4(a, outC);
                storeC4(S, r.parent * rs, a);
            }
        });
        tileSweep<CF, true>(TT, c, run, [&](int cl, int slot, const tile::SlotRow& r, auto) {
            const int rec = slot * rs, row = body0 + r.row;
            const A3<float> Ap = r.parent < 0 ? A3<float>{} : loadA3<float>(S, r.parent * rs, false);
            A3<float> A;
            if (cl == tile::CL_FREE) body5Free(T, row, rec, S, out, Ap, r.parent >= 0, A);
            else A = body5<NM>(T, row, rec, (r.info >> 4) & 15, S, out, Ap, r.parent >= 0);
            storeA3(S, rec, A, false);
        });
    }
    return ok ? 0 : SBG_INST_SINGULAR_D;
}

// The largest |udot0| and correction over the tile's warps, per lane.
struct TileMax {
    float u[kTileMaxWarps][32], d[kTileMaxWarps][32];
};
// illConditioned() of abi_device.cuh over the warps of a tile; contact: the
// lane has a body with contact spheres in this warp.
template <class Out>
__device__ __forceinline__ int tileIll(const DevTables& T, const TileTables& TT, const TileCtx& c, TileMax& sh,
                                       const Out& out) {
    float um = out.umax, dm = out.dmax;
    if (TT.W > 1) {
        sh.u[c.sub * TT.W + c.w][c.lane] = um;
        sh.d[c.sub * TT.W + c.w][c.lane] = dm;
        tileSync(TT.W, c);
        for (int w = 0; w < TT.W; ++w) {
            um = fmaxf(um, sh.u[c.sub * TT.W + w][c.lane]);
            dm = fmaxf(dm, sh.d[c.sub * TT.W + w][c.lane]);
        }
        tileSync(TT.W, c);
    }
    return illConditionedBy(T, c.inst, um, dm);
}

}  // namespace sbg
