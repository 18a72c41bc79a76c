// tile32_device.cuh -- the mixed and FP32 forms on the tile driver: the chain
// driver's per-body routines (abi_device.cuh), taken in the order of a tile's
// schedule by the warps of a block instead of one thread's row by row.
//
// The one-thread driver is bound by latency: a few warps per SM, each walking
// its 32 trees' rows one after another through five passes of dependent loads
// and FP32 chains, lanes apart on mobilizers. Here up to four warps share the
// 32 trees, a body of each a step, so a pass has as many steps as the trees are
// deep or a quarter of their rows, whichever is more. Every routine and the
// order in which a parent's children add to it (falling rows, kept by the
// schedule) are the chain driver's, so the results are the same bit for bit.
#pragma once
#include "stage_device.cuh"
#include "tile_device.cuh"

namespace sbg {

// Fields that passes 2 to 5 of the tile driver read of a body's own record and
// that its own thread wrote in an earlier pass; what children add to (P, z and
// the inverse dynamics' force) is read where it lies.
template <int N> struct TileSets {
    using S = Sets<N>;
    using P2 = typename S::P2;
    using P3 = StageSet<kRecPc, kRecBF + 6, kRecH, S::eU0, 0, 0, 0, 0>;
    using P4 = StageSet<kRecL, kRecL + 3, kRecH, S::eDI, S::eG, S::eEps, 0, 0>;
    using P5 = typename S::P5;
    static constexpr int most = P3::size > P5::size ? P3::size : P5::size;
    static_assert(P2::size <= most && P4::size <= most, "buffer of a step");
    static constexpr int warpFloats = 2 * most * kTile;  // of a warp: this step's fields and the next one's
};

// tileSweep with the fields SET of a body's record copied to the warp's buffer
// in shared memory while it works on the step before; f gets the record's
// accessor. Free bodies, whose records are wider, are read where they lie.
// With every field loaded where it was used, 43 % of the mixed kernel's issue
// slots waited for a load and 29 % at the barrier for a warp that did.
template <class CF, class SET, bool FORWARD, class F>
__device__ __forceinline__ void tileStagedSweep(const TileTables& TT, const TileCtx& c, bool run, float* recs, float* buf, F f) {
    const int n = c.d.nsteps, W = TT.W;
    const int first = FORWARD ? 0 : n - 1, inc = FORWARD ? 1 : -1;
    float* const tile = recs + c.d.rec0;
    const int64_t recSize = (int64_t)TT.rsTotal * kTile;
    const uint32_t sb0 = (uint32_t)__cvta_generic_to_shared(buf);
    constexpr int bufFloats = SET::size * kTile;
    auto classAt = [&](int k) { return TT.cls[c.d.cls0 + (first + inc * (k < n ? k : n - 1)) * W + c.w]; };
    auto staged = [](int cl) { return cl >= 0 && cl != tile::CL_FREE; };
    auto copy = [&](int step, int k) {
        stage<SET>(tile + (step * W + c.w) * recSize, sb0 + (uint32_t)((k & 1) * bufFloats * sizeof(float)), c.lane);
    };
    TileSlot t = tileSlot<CF>(TT, c, first);
    int cl1 = classAt(1);
    if (staged(t.cl)) copy(first, 0);
    cpAsyncCommit();
    for (int k = 0; k < n; ++k) {
        const int step = first + inc * k;
        const TileSlot next = tileSlot<CF>(TT, c, k + 1 < n ? step + inc : step);
        const int cl2 = classAt(k + 2);
        if (k + 1 < n && staged(cl1)) copy(step + inc, k + 1);
        cpAsyncCommit();
        cpAsyncWait<1>();  // this lane's copies for the step have landed
        __syncwarp();      // ... and every other lane's
        if (t.cl >= 0 && run && t.some()) {
            const int slot = step * W + c.w;
            if (t.cl == tile::CL_FREE) f(std::true_type(), slot, t.row(), ScrTiled<float>{tile + c.lane});
            else f(std::false_type(), slot, t.row(), ScrStaged<SET>{tile + c.lane, buf + (k & 1) * bufFloats + c.lane});
        }
        tileSync(W, c);  // also: the buffer is refilled at the next step
        t = next;
        cl1 = cl2;
    }
    cpAsyncWait<0>();
    __threadfence_block();  // this pass's record writes, before the next one's copies of them
    tileSync(W, c);
}

// One RHS of the tile's instances for which `active` holds. A slot's record is
// at slot * TT.rsTotal in the tile's interleaved records.
template <class CF, int NM, bool REF, class Src, class Out>
__device__ __forceinline__ int tileRhs32(const DevTables& T, const TileTables& TT, const TileCtx& c, float* recs, float* buf,
                                         const Src& src, Out& out, bool active) {
    using TS = TileSets<NM>;
    const int body0 = T.ibody[c.inst], rs = TT.rsTotal;
    const V3<float> g = mk3(float(T.grav[3 * c.inst]), float(T.grav[3 * c.inst + 1]), float(T.grav[3 * c.inst + 2]));
    const ScrTiled<float> R{recs + c.d.rec0 + c.lane};
    const bool run = c.on && active;
    bool ok = true;
    tileSweep<CF, true>(TT, c, run, [&](int, int slot, const tile::SlotRow& r, auto) {
        const int rec = slot * rs;
        const Kin<float> P = r.parent < 0 ? groundKin<float>() : loadKin<float>(R, r.parent * rs);
        const Kin<float> K = body1<float, NM>(T, body0 + r.row, rec, R, src, out, g, P);
        storeKin(R, rec, K);
        storeC2(R, rec, zeroC2<float>());
    });
    __threadfence_block();  // the records, before pass 2 copies them
    tileSync(TT.W, c);
    tileStagedSweep<CF, typename TS::P2, false>(TT, c, run, recs, buf, [&](auto six, int slot, const tile::SlotRow& r, const auto& S) {
        const int rec = slot * rs, row = body0 + r.row;
        const float m = T.par32[(int64_t)row * kParamStride];
        const C2<float> in = loadC2<float>(R, rec);
        C2<float> outC;
        if constexpr (decltype(six)::value) ok &= body2Free<float>(T, row, rec, S, m, in, outC);
        else ok &= body2<float, NM>(T, row, rec, (r.info >> 4) & 15, S, m, in, outC);
        if (r.parent >= 0) pushC2(R, r.parent * rs, outC);
    });
    tileStagedSweep<CF, typename TS::P3, true>(TT, c, run, recs, buf, [&](auto six, int slot, const tile::SlotRow& r, const auto& S) {
        const int rec = slot * rs, row = body0 + r.row;
        const A3<float> Ap = r.parent < 0 ? A3<float>{} : loadA3<float>(R, r.parent * rs, REF);
        A3<float> A;
        if constexpr (decltype(six)::value) body3Free<float, REF>(T, row, rec, S, out, Ap, r.parent >= 0, A);
        else A = body3<float, NM, REF>(T, row, rec, (r.info >> 4) & 15, S, out, Ap, r.parent >= 0);
        storeA3(R, rec, A, REF);
        if constexpr (REF)
            for (int i = 0; i < 6; ++i) R(rec, kRecZ2acc + i) = 0.f;
    });
    if constexpr (REF) {
        tileStagedSweep<CF, typename TS::P4, false>(TT, c, run, recs, buf, [&](auto six, int slot, const tile::SlotRow& r, const auto& S) {
            const int rec = slot * rs, row = body0 + r.row;
            const C4 own = loadC4(R, rec);
            C4 outC;
            if constexpr (decltype(six)::value) body4Free(T, row, rec, S, own, zeroC4(), outC);
            else outC = body4<NM>(T, row, rec, (r.info >> 4) & 15, S, own, zeroC4());
            if (r.parent >= 0) {
                C4 a = loadC4(R, r.parent * rs);
                addC4(a, outC);
                storeC4(R, r.parent * rs, a);
            }
        });
        tileStagedSweep<CF, typename TS::P5, true>(TT, c, run, recs, buf, [&](auto six, int slot, const tile::SlotRow& r, const auto& S) {
            const int rec = slot * rs, row = body0 + r.row;
            const A3<float> Ap = r.parent < 0 ? A3<float>{} : loadA3<float>(R, r.parent * rs, false);
            A3<float> A;
            if constexpr (decltype(six)::value) body5Free(T, row, rec, S, out, Ap, r.parent >= 0, A);
            else A = body5<NM>(T, row, rec, (r.info >> 4) & 15, S, out, Ap, r.parent >= 0);
            storeA3(R, rec, A, false);
        });
    }
    return ok ? 0 : SBG_INST_SINGULAR_D;
}

// The warp's staging buffer in the block's dynamic shared memory, and the
// launch's size of it.
template <int NM> __device__ __forceinline__ float* tileStage() {
    extern __shared__ float4 stageRaw[];
    return reinterpret_cast<float*>(stageRaw) + (threadIdx.x >> 5) * TileSets<NM>::warpFloats;
}
template <int NM, class K> inline size_t tileStageBytes(K kernel, int block) {
    constexpr size_t warpBytes = TileSets<NM>::warpFloats * sizeof(float);
    // The limit is the kernel's in the whole process, whichever batch launches it
    // on whichever thread: always the widest block's. An error is left for the
    // launch's cudaGetLastError.
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kTileMaxWarps * warpBytes));
    return (block / 32) * warpBytes;
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
