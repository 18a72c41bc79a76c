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
#include "kernels.h"
#include "tile_program.h"

namespace sbg {

struct TileCtx {
    TileDesc d;
    double* rec;     // the lane's column of the tile's records
    int lane, w;     // lane of the tile, warp of the block
    bool on;         // the lane holds an instance
    int inst;
};

__device__ __forceinline__ void tileSync(int W) {
    if (W == 1) __syncwarp(); else __syncthreads();
}

// Tile `id` of a batch.
__device__ __forceinline__ TileCtx tileCtx(const DevTables& T, const TileTables& TT, int id, double* recs) {
    TileCtx c;
    c.d = TT.desc[id];
    c.lane = threadIdx.x & 31;
    c.w = threadIdx.x >> 5;
    c.on = c.lane < c.d.lanes;
    c.rec = recs + c.d.rec0 + c.lane;
    c.inst = c.on ? T.order[c.d.pos0 + c.lane] : 0;
    return c;
}
// The tile of one instance, in a tile set with one tile per instance, on the
// block's own records.
__device__ __forceinline__ TileCtx tileCtxOne(const TileTables& TT, int inst, double* recs) {
    TileCtx c;
    c.d = TT.desc[inst];
    c.lane = threadIdx.x & 31;
    c.w = threadIdx.x >> 5;
    c.on = c.lane == 0;
    c.rec = recs;
    c.inst = inst;
    return c;
}

// Class of the warp's body at a step (-1: none), and the lane's row of it
// (false: none on this lane).
__device__ __forceinline__ int tileClass(const TileTables& TT, const TileCtx& c, int step) {
    return TT.cls[c.d.cls0 + step * TT.W + c.w];
}
__device__ __forceinline__ bool tileRow(const TileTables& TT, const TileCtx& c, int slot, tile::SlotRow& r, tile::Par& par) {
    const int64_t st = c.d.shared ? 1 : c.d.ls, l = c.d.shared ? 0 : c.lane;
    const int32_t* s = TT.slots + c.d.slot0 + (int64_t)slot * tile::SI_COUNT * st + l;
    r.qo = s[tile::SI_Q * st];
    r.uo = s[tile::SI_U * st];
    r.parent = s[tile::SI_PARENT * st];
    r.info = s[tile::SI_INFO * st];
    r.row = s[tile::SI_ROW * st];
    r.kbeg = s[tile::SI_KBEG * st];
    r.kcnt = s[tile::SI_KCNT * st];
    par.p = TT.par + c.d.par0 + (int64_t)slot * tile::PR_COUNT * st + l;
    par.ls = st;
    return r.qo >= 0;
}

// One RHS of the tile's instances for which `active` holds; SINGULAR_D is
// reported to the thread whose body met it. All warps of the block call it.
template <bool MINV, class Src, class Out>
__device__ __forceinline__ int tileRhs(const DevTables& T, const TileTables& TT, const TileCtx& c, const Src& src,
                                       Out& out, bool active) {
    using namespace tile;
    const int W = TT.W, nsteps = c.d.nsteps;
    const int64_t ls = c.d.ls, rs = TT.rsTotal;
    Model md;
    md.kpar = T.kpar64;
    md.rs = TT.rs;
    md.pose = !MINV && TT.pose;
    md.bodyPar = nullptr;
    md.g = zero();
    int body0 = 0;
    if (c.on) {
        md.g = Vec{T.grav[3 * c.inst], T.grav[3 * c.inst + 1], T.grav[3 * c.inst + 2]};
        body0 = T.ibody[c.inst];
        md.bodyPar = T.par64 + (int64_t)body0 * kParamStride;
    }
    const bool run = c.on && active;
    bool ok = true;
    auto recOf = [&](int slot) { return Rec{c.rec + (int64_t)slot * rs * ls, ls}; };
    for (int step = 0; step < nsteps; ++step) {
        const int cl = tileClass(TT, c, step), slot = step * W + c.w;
        SlotRow r;
        Par par;
        if (cl >= 0 && run && tileRow(TT, c, slot, r, par)) {
            const Rec rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
            // contact spheres are grouped by body row of the batch's body table
            if (r.kcnt > 0 && md.pose) r.kbeg = T.kbeg[body0 + r.row];
            switch (cl) {
            case CL_PIN: pass1<CL_PIN, MINV>(md, r, par, rec, recP, src, out); break;
            case CL_SLIDER: pass1<CL_SLIDER, MINV>(md, r, par, rec, recP, src, out); break;
            case CL_UNIV: pass1<CL_UNIV, MINV>(md, r, par, rec, recP, src, out); break;
            case CL_BALL: pass1<CL_BALL, MINV>(md, r, par, rec, recP, src, out); break;
            case CL_FREE: pass1<CL_FREE, MINV>(md, r, par, rec, recP, src, out); break;
            default: pass1<CL_GEN, MINV>(md, r, par, rec, recP, src, out); break;
            }
        }
        tileSync(W);
    }
    for (int step = nsteps - 1; step >= 0; --step) {
        const int cl = tileClass(TT, c, step), slot = step * W + c.w;
        SlotRow r;
        Par par;
        if (cl >= 0 && run && tileRow(TT, c, slot, r, par)) {
            const Rec rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
            switch (cl) {
            case CL_PIN: ok &= pass2<CL_PIN, MINV>(r, par, rec, recP); break;
            case CL_SLIDER: ok &= pass2<CL_SLIDER, MINV>(r, par, rec, recP); break;
            case CL_UNIV: ok &= pass2<CL_UNIV, MINV>(r, par, rec, recP); break;
            case CL_BALL: ok &= pass2<CL_BALL, MINV>(r, par, rec, recP); break;
            case CL_FREE: ok &= pass2<CL_FREE, MINV>(r, par, rec, recP); break;
            default: ok &= pass2<CL_GEN, MINV>(r, par, rec, recP); break;
            }
        }
        tileSync(W);
    }
    for (int step = 0; step < nsteps; ++step) {
        const int cl = tileClass(TT, c, step), slot = step * W + c.w;
        SlotRow r;
        Par par;
        if (cl >= 0 && run && tileRow(TT, c, slot, r, par)) {
            const Rec rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
            switch (cl) {
            case CL_PIN: pass3<CL_PIN, MINV>(md, r, par, rec, recP, out); break;
            case CL_SLIDER: pass3<CL_SLIDER, MINV>(md, r, par, rec, recP, out); break;
            case CL_UNIV: pass3<CL_UNIV, MINV>(md, r, par, rec, recP, out); break;
            case CL_BALL: pass3<CL_BALL, MINV>(md, r, par, rec, recP, out); break;
            case CL_FREE: pass3<CL_FREE, MINV>(md, r, par, rec, recP, out); break;
            default: pass3<CL_GEN, MINV>(md, r, par, rec, recP, out); break;
            }
        }
        tileSync(W);
    }
    return ok ? 0 : SBG_INST_SINGULAR_D;
}

// Calls f(row) for the lane's bodies that this warp owns.
template <class F>
__device__ __forceinline__ void tileBodies(const TileTables& TT, const TileCtx& c, F f) {
    for (int step = 0; step < c.d.nsteps; ++step) {
        tile::SlotRow r;
        tile::Par par;
        if (tileClass(TT, c, step) >= 0 && c.on && tileRow(TT, c, step * TT.W + c.w, r, par)) f(r);
    }
}

// Per-lane sums and status bits over the block's warps, the same on every
// warp (warps in order).
constexpr int kTileMaxWarps = 8;
template <int N> struct TileShare {
    double v[N > 0 ? N : 1][kTileMaxWarps][32];
    int bits[kTileMaxWarps][32];
};
template <int N>
__device__ __forceinline__ int tileReduce(const TileTables& TT, const TileCtx& c, TileShare<N>& sh, double* v, int bits) {
    if (TT.W == 1) return bits;
#pragma unroll
    for (int k = 0; k < N; ++k) sh.v[k][c.w][c.lane] = v[k];
    sh.bits[c.w][c.lane] = bits;
    __syncthreads();
    int b = 0;
    double s[N > 0 ? N : 1] = {};
    for (int w = 0; w < TT.W; ++w) {
#pragma unroll
        for (int k = 0; k < N; ++k) s[k] = w == 0 ? sh.v[k][0][c.lane] : s[k] + sh.v[k][w][c.lane];
        b |= sh.bits[w][c.lane];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = s[k];
    __syncthreads();  // the arrays may be written again
    return b;
}

// ----------------------------------------------------------- sources, sinks
struct TileYSrc {
    const double* y;
    int64_t base, stride;
    int nq;
    __device__ __forceinline__ double q(int k) const { return y[base + (int64_t)k * stride]; }
    __device__ __forceinline__ double u(int k) const { return y[base + (int64_t)(nq + k) * stride]; }
    __device__ __forceinline__ double fext(int) const { return 0.0; }
};
struct TileFSrc {  // M^-1 f: q and the given forces
    const double* y;
    const double* f;
    int64_t base, stride;
    int nq;
    __device__ __forceinline__ double q(int k) const { return y[base + (int64_t)k * stride]; }
    __device__ __forceinline__ double u(int) const { return 0.0; }
    __device__ __forceinline__ double fext(int k) const { return f[base + (int64_t)(nq + k) * stride]; }
};
// Stage input y0 + c * combo(f) of RK-Merson, formed while pass 1 loads it
// (RungeKuttaMersonIntegrator.cpp:108-126).
struct TileStageSrc {
    const double* y;
    const double *f0, *fa, *fb;
    int64_t base, stride;
    int nq, stage;
    double c;
    __device__ __forceinline__ double at(int k) const {
        const int64_t e = base + (int64_t)k * stride;
        const double y0 = y[e];
        switch (stage) {
        case 0: return y0;
        case 1: return y0 + c * f0[e];                                    // h/3 f0
        case 2: return y0 + c * (f0[e] + fa[e]);                          // h/6 (f0+f1)
        case 3: return y0 + c * (f0[e] + 3.0 * fa[e]);                    // h/8 (f0+3f2)
        default: return y0 + c * ((f0[e] - 3.0 * fa[e]) + 4.0 * fb[e]);   // h/2 (f0-3f2+4f3)
        }
    }
    __device__ __forceinline__ double q(int k) const { return at(k); }
    __device__ __forceinline__ double u(int k) const { return at(nq + k); }
    __device__ __forceinline__ double fext(int) const { return 0.0; }
};
struct TileOut {
    double* f;
    int64_t base, stride;
    int nq;
    bool finite = true;
    __device__ __forceinline__ void qdot(int k, double v) { f[base + (int64_t)k * stride] = v; finite &= tile::finiteBits(v); }
    __device__ __forceinline__ void udot(int k, double v) { f[base + (int64_t)(nq + k) * stride] = v; finite &= tile::finiteBits(v); }
};
struct TileUOut {  // M^-1 f: u slots only
    double* f;
    int64_t base, stride;
    int nq;
    bool finite = true;
    __device__ __forceinline__ void qdot(int, double) {}
    __device__ __forceinline__ void udot(int k, double v) { f[base + (int64_t)(nq + k) * stride] = v; finite &= tile::finiteBits(v); }
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

}  // namespace sbg
