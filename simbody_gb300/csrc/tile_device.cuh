// tile_device.cuh -- the FP64 driver: tiles of instances, one per lane, whose
// trees W warps sweep together, body by body in the order of the tile's
// schedule (tile_program.h), with the per-body arithmetic of tile_core.cuh.
//
// An FP64 warp instruction holds its SM sub-partition's FP64 pipe for 64
// cycles however many lanes are active (measured: 64.0 cycles for 1 to 32
// lanes, one to four warps per SM, any instruction-level parallelism), so
// what counts is the number of warp instructions on the busiest sub-partition.
// The schedule gives every lane of a step the same mobilizer (no divergence),
// and W warps on W sub-partitions share a tile when there are fewer tiles than
// sub-partitions. Records live in global memory, field by field across the
// lanes; their loads are short beside a step's FP64 instructions.
#pragma once
#include <algorithm>

#include "kernels.h"
#include "tile_program.h"

namespace sbg {

// LS: lane stride of the records (the widest a tile can be); SH: the tables
// have no lanes (one topology per tile); YS: stride of the state columns, 0 =
// the instance's own.
template <int LS_, bool SH_, int YS_> struct TileCfg {
    static constexpr int LS = LS_, YS = YS_;
    static constexpr bool SH = SH_;
};

struct TileCtx {
    TileDesc d;
    double* rec;     // the lane's column of the tile's records
    const int4* slots;  // the lane's column of the slot integers, parameters
    const double* par;
    int lane, w;     // lane and warp of the tile
    int sub;         // tile of the block
    bool on;         // the lane holds an instance
    int inst;
};

// Tiles of fewer than four warps share a block where there are more of them
// than SMs, so that the block's warps take the SM's sub-partitions in turn:
// single-warp blocks landed two on one sub-partition beside an empty one when
// other kernels' blocks came and went (20,000 FP64 chains in two chunks 1.64
// ms, 1.27 ms so); while there are SMs for all, each its own (1,024 pendulums
// 9.3 ms, four to a block 10.1 ms).
inline int tilesPerBlock(const TileSet& S, int sms) {
    return S.tt.W >= 4 || S.tt.recStride ? 1 : std::max(1, std::min(4 / S.tt.W, (S.ntiles + sms - 1) / sms));
}
__device__ __forceinline__ void tileSync(int W, const TileCtx& c) {
    if (W == 1) __syncwarp();
    else if (W == 2) asm volatile("bar.sync %0, 64;" ::"r"(1 + c.sub) : "memory");
    else __syncthreads();
}

template <class CF> __device__ __forceinline__ void tileTables(const TileTables& TT, TileCtx& c) {
    c.lane = threadIdx.x & 31;
    c.sub = (threadIdx.x >> 5) / TT.W;
    c.w = (threadIdx.x >> 5) - c.sub * TT.W;
    const int l = CF::SH || c.lane >= CF::LS ? 0 : c.lane;
    c.slots = reinterpret_cast<const int4*>(TT.slots + c.d.slot0) + 2 * l;
    c.par = TT.par + c.d.par0 + l;
}
// Tile `id` of a batch.
template <class CF>
__device__ __forceinline__ TileCtx tileCtx(const DevTables& T, const TileTables& TT, int id, double* recs) {
    TileCtx c;
    c.d = TT.desc[id];
    tileTables<CF>(TT, c);
    c.on = c.lane < c.d.lanes;
    c.rec = recs + c.d.rec0 + (c.on ? c.lane : 0);
    c.inst = c.on ? T.order[c.d.pos0 + c.lane] : T.order[c.d.pos0];
    return c;
}
// The warp's tile among [tile0, tile0 + count), -1 past the end.
__device__ __forceinline__ int tileId(const TileTables& TT, int tile0, int count) {
    const int k = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) / TT.W;
    return k < count ? tile0 + k : -1;
}
// f(tile) for the warp's tile among [tile0, tile0 + count), if any; where blocks
// share records (TT.recStride), for every gridDim-th tile from the block's on.
template <class CF, class F>
__device__ __forceinline__ void forTiles(const DevTables& T, const TileTables& TT, int tile0, int count, double* recs, F f) {
    int id = tileId(TT, tile0, count);
    if (id < 0) return;
    if constexpr (CF::LS == 1) {
        for (const int end = tile0 + count; id < end; id += TT.recStride ? gridDim.x : count) {
            TileCtx c = tileCtx<CF>(T, TT, id, recs);
            if (TT.recStride) c.rec = recs + TT.recStride * blockIdx.x;
            f(c);
            tileSync(TT.W, c);
        }
    } else {
        f(tileCtx<CF>(T, TT, id, recs));
    }
}
// The tile of one instance, in a tile set with one tile per instance, on the
// block's own records.
template <class CF> __device__ __forceinline__ TileCtx tileCtxOne(const TileTables& TT, int inst, double* recs) {
    TileCtx c;
    c.d = TT.desc[inst];
    tileTables<CF>(TT, c);
    c.on = c.lane == 0;
    c.rec = recs;
    c.inst = inst;
    return c;
}

// The warp's slot at a step: its class (-1: none) and the lane's integers.
struct TileSlot {
    int cl;
    int4 a, b;
    __device__ __forceinline__ bool some() const { return a.x >= 0; }  // a body on this lane
    __device__ __forceinline__ tile::SlotRow row() const { return tile::SlotRow{a.x, a.y, a.z, a.w, b.x, b.y, b.z}; }
};
template <class CF> __device__ __forceinline__ TileSlot tileSlot(const TileTables& TT, const TileCtx& c, int step) {
    const int slot = step * TT.W + c.w;
    const int4* s = c.slots + (int64_t)slot * (2 * (CF::SH ? 1 : CF::LS));
    TileSlot t;
    t.cl = TT.cls[c.d.cls0 + slot];
    t.a = s[0];
    t.b = s[1];
    return t;
}

// f(slot, row, parameters) for the warp's bodies in the order of the steps (or
// back), the next step's integers loaded ahead; f runs on the lanes of `run`
// that have a body at the step.
template <class CF, bool FORWARD, class F>
__device__ __forceinline__ void tileSweep(const TileTables& TT, const TileCtx& c, bool run, F f) {
    constexpr int LN = CF::SH ? 1 : CF::LS;
    const int n = c.d.nsteps, W = TT.W;
    const int first = FORWARD ? 0 : n - 1, inc = FORWARD ? 1 : -1;
    TileSlot t = tileSlot<CF>(TT, c, first);
    for (int k = 0; k < n; ++k) {
        const int step = first + inc * k;
        const TileSlot next = tileSlot<CF>(TT, c, k + 1 < n ? step + inc : step);
        if (t.cl >= 0 && run && t.some()) {
            const int slot = step * W + c.w;
            f(t.cl, slot, t.row(), tile::Par<LN>{c.par + (int64_t)slot * (tile::PR_COUNT * LN)});
        }
        tileSync(W, c);
        t = next;
    }
}

// One RHS of the tile's instances for which `active` holds; SINGULAR_D is
// reported to the thread whose body met it. All warps of the block call it.
template <class CF, bool MINV, class Src, class Out>
__device__ __forceinline__ int tileRhs(const DevTables& T, const TileTables& TT, const TileCtx& c, const Src& src,
                                       Out& out, bool active) {
    using namespace tile;
    constexpr int LN = CF::SH ? 1 : CF::LS;
    typedef Rec<CF::LS> RC;
    typedef Par<LN> PA;
    Model md;
    md.kpar = T.kpar64;
    md.rs = TT.rs;
    md.pose = !MINV && TT.pose;
    md.g = Vec{T.grav[3 * c.inst], T.grav[3 * c.inst + 1], T.grav[3 * c.inst + 2]};
    const int body0 = T.ibody[c.inst];
    md.bodyPar = T.par64 + (int64_t)body0 * kParamStride;
    const bool run = c.on && active;
    bool ok = true;
    const int64_t recSize = (int64_t)TT.rsTotal * CF::LS;
    auto recOf = [&](int slot) { return RC{c.rec + slot * recSize}; };
    tileSweep<CF, true>(TT, c, run, [&](int cl, int slot, SlotRow r, PA par) {
        const RC rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
        // contact spheres are grouped by body row of the batch's body table
        if (md.pose && r.kcnt > 0) r.kbeg = T.kbeg[body0 + r.row];
        switch (cl) {
        case CL_PIN: pass1<CL_PIN, MINV>(md, r, par, rec, recP, src, out); break;
        case CL_SLIDER: pass1<CL_SLIDER, MINV>(md, r, par, rec, recP, src, out); break;
        case CL_UNIV: pass1<CL_UNIV, MINV>(md, r, par, rec, recP, src, out); break;
        case CL_BALL: pass1<CL_BALL, MINV>(md, r, par, rec, recP, src, out); break;
        case CL_FREE: pass1<CL_FREE, MINV>(md, r, par, rec, recP, src, out); break;
        default: pass1<CL_GEN, MINV>(md, r, par, rec, recP, src, out); break;
        }
    });
    tileSweep<CF, false>(TT, c, run, [&](int cl, int slot, SlotRow r, PA par) {
        const RC rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
        switch (cl) {
        case CL_PIN: ok &= pass2<CL_PIN, MINV>(r, par, rec, recP); break;
        case CL_SLIDER: ok &= pass2<CL_SLIDER, MINV>(r, par, rec, recP); break;
        case CL_UNIV: ok &= pass2<CL_UNIV, MINV>(r, par, rec, recP); break;
        case CL_BALL: ok &= pass2<CL_BALL, MINV>(r, par, rec, recP); break;
        case CL_FREE: ok &= pass2<CL_FREE, MINV>(r, par, rec, recP); break;
        default: ok &= pass2<CL_GEN, MINV>(r, par, rec, recP); break;
        }
    });
    tileSweep<CF, true>(TT, c, run, [&](int cl, int slot, SlotRow r, PA par) {
        const RC rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
        switch (cl) {
        case CL_PIN: pass3<CL_PIN, MINV>(md, r, par, rec, recP, out); break;
        case CL_SLIDER: pass3<CL_SLIDER, MINV>(md, r, par, rec, recP, out); break;
        case CL_UNIV: pass3<CL_UNIV, MINV>(md, r, par, rec, recP, out); break;
        case CL_BALL: pass3<CL_BALL, MINV>(md, r, par, rec, recP, out); break;
        case CL_FREE: pass3<CL_FREE, MINV>(md, r, par, rec, recP, out); break;
        default: pass3<CL_GEN, MINV>(md, r, par, rec, recP, out); break;
        }
    });
    return ok ? 0 : SBG_INST_SINGULAR_D;
}

// Calls f(row) for the lane's bodies that this warp owns.
template <class CF, class F>
__device__ __forceinline__ void tileBodies(const TileTables& TT, const TileCtx& c, bool run, F f) {
    for (int step = 0; step < c.d.nsteps; ++step) {
        const TileSlot t = tileSlot<CF>(TT, c, step);
        if (t.cl >= 0 && run && t.some()) f(t.row());
    }
}

// Per-lane status bits over the tile's warps, the same on every warp.
constexpr int kTileMaxWarps = 8;
template <int N> struct TileShare {
    double v[N > 0 ? N : 1][kTileMaxWarps][32];  // tileSums: per sum, tile of the block and lane
    int bits[kTileMaxWarps][32];
};
template <int N>
__device__ __forceinline__ int tileReduce(const TileTables& TT, const TileCtx& c, TileShare<N>& sh, int bits) {
    if (TT.W == 1) return bits;
    sh.bits[c.sub * TT.W + c.w][c.lane] = bits;
    tileSync(TT.W, c);
    int b = 0;
    for (int w = 0; w < TT.W; ++w) b |= sh.bits[c.sub * TT.W + w][c.lane];
    tileSync(TT.W, c);  // the array may be written again
    return b;
}

// Sums over an instance's bodies of the error norms and projection gates, in
// the order of its rows whatever the tile's schedule: added up by the warps
// that the schedule deals the bodies to, an instance's step sizes would depend
// on the other instances of its tile. Each body has left its parts in the
// column plane `part` (tileReduce after it makes them visible to every warp): at
// its first u slot the u error; at its first q slot the q error, and for a
// quaternion at the next two the error of its length and the q error after
// normalization. v: q error, u error, length errors, number of quaternions, q
// error after normalization (N = 5). A warp takes every W-th sum: all of them
// on one warp would be four chains of FP64 additions over the rows, with the
// others waiting (3,000 contact trees, four steps: 12.43 ms with partial sums per
// warp, 12.49 so).
template <int N, class Col>
__device__ __forceinline__ void tileSums(const DevTables& T, const TileTables& TT, const TileCtx& c, TileShare<N>& sh,
                                         const Col& col, const double* part, bool run, double* v) {
    const int body0 = T.ibody[c.inst], nb = run ? T.inb[c.inst] : 0;
    // f(info, q slot, u slot) of the rows with mobilities
    auto sum = [&](auto f) {
        double s = 0;
#pragma unroll 4
        for (int r = body0; r < body0 + nb; ++r) {
            const int info = T.info[r];
            if ((info >> 4) & 15) s += f(info, T.qoff[r], T.uoff[r]);
        }
        return s;
    };
    auto one = [&](int k) -> double {
        if (k == 0) return sum([&](int, int q, int) { return part[col.at(q)]; });
        if (k == 1) return sum([&](int, int, int u) { return part[col.atU(u)]; });
        if (k == 2) return sum([&](int info, int q, int) { return info & F_QUAT ? part[col.at(q + 1)] : 0.0; });
        if (k == 3) {
            int n = 0;
            for (int r = body0; r < body0 + nb; ++r) n += (T.info[r] & F_QUAT) != 0;
            return n;
        }
        return sum([&](int info, int q, int) { return part[col.at(info & F_QUAT ? q + 2 : q)]; });
    };
    const int W = TT.W;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        if (W == 1) v[k] = one(k);
        else if (k % W == c.w) sh.v[k][c.sub][c.lane] = one(k);
    }
    if (W == 1) return;
    tileSync(W, c);
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = sh.v[k][c.sub][c.lane];
    tileSync(W, c);  // the arrays and the plane may be written again
}

// ----------------------------------------------------------- sources, sinks
// An instance's column: element k at k * YS from its base.
template <int YS> struct TileCol {
    int64_t base;
    int stride, nq;
    __device__ __forceinline__ TileCol(const DevTables& T, int inst)
        : base(T.ybase[inst]), stride(YS ? YS : (int)T.ystride[inst]), nq(T.inq[inst]) {}
    __device__ __forceinline__ int64_t at(int k) const { return base + (int64_t)k * (YS ? YS : stride); }
    __device__ __forceinline__ int64_t atU(int k) const { return at(nq + k); }
};
template <int YS> struct TileYSrc {
    TileCol<YS> c;
    const double* y;
    __device__ __forceinline__ double q(int k) const { return y[c.at(k)]; }
    __device__ __forceinline__ double u(int k) const { return y[c.atU(k)]; }
    __device__ __forceinline__ double fext(int) const { return 0.0; }
};
template <int YS> struct TileFSrc {  // M^-1 f: q and the given forces
    TileCol<YS> c;
    const double *y, *f;
    __device__ __forceinline__ double q(int k) const { return y[c.at(k)]; }
    __device__ __forceinline__ double u(int) const { return 0.0; }
    __device__ __forceinline__ double fext(int k) const { return f[c.atU(k)]; }
};
// Stage input y0 + c * combo(f) of RK-Merson (RungeKuttaMersonIntegrator.cpp:
// 108-126) into the plane yt, element by element over the block's warps. Formed
// in the bodies' loads instead, its five cases made up most of the kernel's
// code, which then ran from beyond the instruction cache.
template <class CF, class F>
__device__ __forceinline__ void tileStageInput(const TileTables& TT, const TileCtx& c, const TileCol<CF::YS>& col, int ny,
                                               bool run, int stage, double h, const double* y, const F* f0, const F* fa,
                                               const F* fb, double* yt) {
    const int W = TT.W;
    auto all = [&](auto f) {
        if (run) {
#pragma unroll 4
            for (int k = c.w; k < ny; k += W) {
                const int64_t e = col.at(k);
                yt[e] = f(e);
            }
        }
    };
    if (stage == 0) all([&](int64_t e) { return y[e]; });
    else if (stage == 1) all([&](int64_t e) { return y[e] + h * double(f0[e]); });                          // h/3 f0
    else if (stage == 2) all([&](int64_t e) { return y[e] + h * (double(f0[e]) + double(fa[e])); });                // h/6 (f0+f1)
    else if (stage == 3) all([&](int64_t e) { return y[e] + h * (double(f0[e]) + 3.0 * double(fa[e])); });          // h/8 (f0+3f2)
    else all([&](int64_t e) {                                                                       // h/2 (f0-3f2+4f3)
        return y[e] + h * ((double(f0[e]) - 3.0 * double(fa[e])) + 4.0 * double(fb[e]));
    });
    tileSync(W, c);
}
template <int YS> struct TileOut {
    TileCol<YS> c;
    double* f;
    bool finite = true;
    __device__ __forceinline__ TileOut(TileCol<YS> col, double* p) : c(col), f(p) {}
    __device__ __forceinline__ void position(double v) { finite &= tile::finiteBits(v); }
    __device__ __forceinline__ void qdot(int k, double v) { f[c.at(k)] = v; finite &= tile::finiteBits(v); }
    __device__ __forceinline__ void udot(int k, double v) { f[c.atU(k)] = v; finite &= tile::finiteBits(v); }
};
template <int YS> struct TileUOut {  // M^-1 f: u slots only
    TileCol<YS> c;
    double* f;
    bool finite = true;
    __device__ __forceinline__ TileUOut(TileCol<YS> col, double* p) : c(col), f(p) {}
    __device__ __forceinline__ void position(double) {}
    __device__ __forceinline__ void qdot(int, double) {}
    __device__ __forceinline__ void udot(int k, double v) { f[c.atU(k)] = v; finite &= tile::finiteBits(v); }
};

// |q|^2 dq - q (q . dq): N N^-1 dq of the unnormalised quaternion q with unit
// weights (Rotation.h:712-748), squared.
__device__ __forceinline__ double tileQuatErrSq(const double* q, const double* dq) {
    const double n2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
    const double d = q[0] * dq[0] + q[1] * dq[1] + q[2] * dq[2] + q[3] * dq[3];
    double s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double o = n2 * dq[k] - d * q[k];
        s += o * o;
    }
    return s;
}

// Calls f(TileCfg) for the kind of the tiles of a batch whose state columns
// have stride YS (0: each its own).
template <int YS, class F> inline void tileDispatch(const TileSet& S, F f) {
    if (S.tt.ls == 1) f(TileCfg<1, true, YS>());
    else if (S.tt.ls == 8 && !S.tt.shared) f(TileCfg<8, false, YS>());
    else if (S.tt.shared) f(TileCfg<32, true, YS>());
    else f(TileCfg<32, false, YS>());
}
// Grid and block of a launch over `ntiles` of the set's tiles.
struct TileLaunch {
    int grid, block;
    TileLaunch(const TileSet& S, int ntiles) {
        const int per = tilesPerBlock(S, S.sms);
        grid = S.tt.recStride ? std::min(ntiles, S.blocks) : (ntiles + per - 1) / per;
        block = 32 * S.tt.W * per;
    }
};
typedef TileCfg<1, true, 0> TileOne;  // one tile per instance

}  // namespace sbg
