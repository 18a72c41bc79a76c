// tilerk_device.cuh -- FP64 fixed-step RK-Merson on the tile driver, shared by
// the translation units of the FP64 batches (k_tilerk.cu) and of the mixed
// ones (k_tilerkmixed.cu), which compile in parallel.
#pragma once
#include "tile_device.cuh"
#include "steps_device.cuh"

namespace sbg {

template <class Col> __device__ __forceinline__ void tileNormalize(double* y, const Col& col, int qo) {
    double qq[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) qq[j] = y[col.at(qo + j)];
    const double len = sqrt(qq[0] * qq[0] + qq[1] * qq[1] + qq[2] * qq[2] + qq[3] * qq[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) y[col.at(qo + j)] = qq[j] / len;
}

// The steps of one tile (rkMersonKernel of abi_device.cuh in tiles). Every
// warp of the block follows its lanes' times and step counts, so all of them
// take the same decisions. LIST: one step of one instance in FP64 mode.
template <class CF, bool LIST>
__device__ __forceinline__ void rkTile(const DevTables& T, const TileTables& TT, const TileCtx& c, TileShare<4>& sh,
                                       double* y, double* time, double* fbuf, int64_t fplane, int32_t* status, double h,
                                       const StepCtl& sc, double accuracy, double consTol, bool pes) {
    const TileCol<CF::YS> col(T, c.inst);
    const int nq = col.nq, nu = T.inu[c.inst];
    double *f0 = fbuf, *fA = fbuf + fplane, *fB = fbuf + 2 * fplane, *fC = fbuf + 3 * fplane, *yt = fbuf + 4 * fplane;
    int st = c.on ? status[c.inst] : 0;
    double tc = c.on ? time[c.inst] : 0.0;
    const double tStop = sc.tStop;
    const int nst = sc.nsteps, maxSteps = sc.maxSteps > 0 ? sc.maxSteps : kMaxStepsPerCall;
    int left = T.stepsLeft && c.on ? T.stepsLeft[c.inst] : kMaxStepsPerCall;
    const double projLimit = fmax(2 * consTol, sqrt(consTol));
    bool going = c.on;
    int taken = 0;
    for (int step = 0;; ++step) {
        double t1 = tc;
        if (going) {
            if (step >= maxSteps || left <= 0) going = false;
            else if (nst >= 0) {
                if (step >= nst) going = false;
                else t1 = tc + h;
            } else if (!stepToTarget(tc, h, tStop, &t1) || step >= kMaxStepsPerCall) {
                if (tc < tStop) st |= SBG_INST_TIMEOUT;  // time no longer advances
                going = false;
            }
        }
        if (!__any_sync(0xffffffffu, going)) break;
        const double hs = t1 - tc;
        int bits = 0;
        // f0 = f(y0); f1 -> fA; f2 -> fB (input f1 in fA); f3 -> fC (input f2
        // in fB); f4 -> fA (input f2, f3)
#pragma unroll 1
        for (int stg = 0; stg < 5; ++stg) {
            const double cc = stg == 0 ? 0.0 : stg == 1 ? hs / 3 : stg == 2 ? hs / 6 : stg == 3 ? hs / 8 : hs / 2;
            tileStageInput<CF>(TT, c, col, nq + nu, going, stg, cc, y, f0, stg >= 3 ? fB : fA, fC, yt);
            const TileYSrc<CF::YS> src{col, yt};
            TileOut<CF::YS> out(col, stg == 0 ? f0 : stg == 2 ? fB : stg == 3 ? fC : fA);
            bits |= tileRhs<CF, false>(T, TT, c, src, out, going);
            if (!out.finite) bits |= SBG_INST_NONFINITE;
        }
        // y1 = y0 + h/6 (f0 + 4 f3 + f4); yerr = 0.2 |y1 - ysave|; error norm
        // (RungeKuttaMersonIntegrator.cpp:124-139, IntegratorRep.h:454-523)
        const double h6 = hs / 6, h2 = hs / 2;
        tileBodies<CF>(TT, c, going, [&](const tile::SlotRow& r) {
                const int nqb = slotQ(r.info), n = (r.info >> 4) & 15;
                double q1[4], dq[4], sq = 0, extra = 0, su = 0;
#pragma unroll
                for (int j = 0; j < 7; ++j)
                    if (j < nqb) {
                        const int64_t e = col.at(r.qo + j);
                        const double y0 = y[e], a0 = f0[e], aB = fB[e], aC = fC[e], aA = fA[e];
                        const double ys = y0 + h2 * ((a0 - 3.0 * aB) + 4.0 * aC);
                        const double y1v = y0 + h6 * ((a0 + 4.0 * aC) + aA);
                        const double dj = 0.2 * fabs(y1v - ys);
                        y[e] = y1v;
                        if (!tile::finiteBits(y1v)) bits |= SBG_INST_NONFINITE;
                        if (j < 4) { q1[j] = y1v; dq[j] = dj; }
                        if (j >= 4 || !(r.info & F_QUAT)) extra += dj * dj;
                    }
                if (r.info & F_QUAT) {
                    sq = tileQuatErrSq(q1, dq);
                    const double len = sqrt(q1[0] * q1[0] + q1[1] * q1[1] + q1[2] * q1[2] + q1[3] * q1[3]);
                    yt[col.at(r.qo + 1)] = (len - 1) * (len - 1);
                }
                for (int j = 0; j < n; ++j) {
                    const int64_t e = col.atU(r.uo + j);
                    const double y0 = y[e], a0 = f0[e], aB = fB[e], aC = fC[e], aA = fA[e];
                    const double ys = y0 + h2 * ((a0 - 3.0 * aB) + 4.0 * aC);
                    const double y1v = y0 + h6 * ((a0 + 4.0 * aC) + aA);
                    const double vi = fabs(y0);
                    double d = 0.2 * fabs(y1v - ys);
                    if (vi > 1) d = d / vi;  // calcRelativeScaling, frozen at step start
                    su += d * d;
                    y[e] = y1v;
                    if (!tile::finiteBits(y1v)) bits |= SBG_INST_NONFINITE;
                }
                if (n > 0) {  // tileSums
                    yt[col.at(r.qo)] = sq + extra;
                    yt[col.atU(r.uo)] = su;
                }
            });
        bits = tileReduce(TT, c, sh, bits);
        double v[4];  // sq, su, squat, nquat
        tileSums(T, TT, c, sh, col, yt, going, v);
        bool renorm = false;
        if (going) {
            st |= bits;
            const double qn = nq ? sqrt(v[0] / nq) : 0.0, un = nu ? sqrt(v[1] / nu) : 0.0;
            const double errNorm = qn >= un ? qn : un;
            // projection gate and quaternion normalization
            // (AbstractIntegratorRep.cpp:158-190, SimbodyMatterSubsystemRep.cpp:4096-4183)
            if (errNorm <= 16 * accuracy && v[3] > 0) {
                const double quatNorm = sqrt(v[2] / v[3]);
                if (quatNorm > projLimit) st |= SBG_INST_PROJECTION_FAILED;
                else if (quatNorm > consTol || pes)
                    renorm = true;
            }
            tc = t1;
            --left;
            ++taken;
        }
        if (__any_sync(0xffffffffu, renorm))
            tileBodies<CF>(TT, c, renorm, [&](const tile::SlotRow& r) {
                if (r.info & F_QUAT) tileNormalize(y, col, r.qo);
            });
        tileSync(TT.W, c);
    }
    if (c.on && c.w == 0) {
        if (T.stepsLeft) T.stepsLeft[c.inst] = left;
        if constexpr (LIST) {
            T.fbLeft[c.inst] -= taken;
            atomicAdd(T.fbSteps, (unsigned long long)taken);
            fbNext(T, sc.launch, c.inst, T.fbLeft[c.inst] > 0);
        }
        time[c.inst] = tc;
        status[c.inst] = st;
    }
}

template <class CF>
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    rkTileKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int ntiles,
                 double* __restrict__ recs, double* y, double* __restrict__ time, double* fbuf, int64_t fplane, int32_t* __restrict__ status,
                 double h, StepCtl sc, double accuracy, double consTol, int pes) {
    __shared__ TileShare<4> sh;
    forTiles<CF>(T, TT, 0, ntiles, recs, [&](const TileCtx& c) {
        rkTile<CF, false>(T, TT, c, sh, y, time, fbuf, fplane, status, h, sc, accuracy, consTol, pes != 0);
    });
}

template <int YS> void rkTilesWith(const KArgs& a, const TileSet& S, cudaStream_t s) {
    if (S.ntiles <= 0) return;
    const TileLaunch L(S, S.ntiles);
    tileDispatch<YS>(S, [&](auto cf) {
        rkTileKernel<decltype(cf)><<<L.grid, L.block, 0, s>>>(*a.T, S.tt, S.ntiles, S.recs, a.ystate, a.time,
                                                                    static_cast<double*>(a.fbuf), a.fplane, a.status, a.h,
                                                                    a.step, a.accuracy, a.consTol, a.projectEveryStep);
    });
}
void rkTilesMixed(const KArgs& a, const TileSet& S, cudaStream_t s);  // k_tilerkmixed.cu

}  // namespace sbg
