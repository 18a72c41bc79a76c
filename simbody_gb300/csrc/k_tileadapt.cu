// k_tileadapt.cu -- error-controlled (variable-step) Runge-Kutta-Merson over a
// batch, FP64: Integrator::setFinalTime(tFinal), initialize(state) and
// stepTo(tFinal) of a RungeKuttaMersonIntegrator with error control
// (AbstractIntegratorRep.cpp:341-577), every instance with its own step size,
// accept/reject decisions and time, inside one persistent kernel on
// the tile driver; an instance that has reached tFinal leaves its lane idle.
//
// Each attempt takes the five stages of the fixed-step kernel
// (RungeKuttaMersonIntegrator.cpp:86-140; f0 is kept across rejected
// attempts, as the reference keeps the derivatives saved at the start of the
// step), then, without touching y:
//   - the error norm of 0.2 |y1 - ysave| (IntegratorRep.h:454-523), with the
//     scaling of u frozen at the start of the step;
//   - the projection test of attemptDAEStep (AbstractIntegratorRep.cpp:158-199):
//     when the norm is within 2^4 accuracy, quaternions whose RMS error passes
//     max(2 consTol, sqrt(consTol)) fail the attempt (norm = infinity), and
//     quaternions are normalized when it passes consTol (or every step), the
//     radial part of their error estimate removed and the norm recomputed
//     (RigidBodyNodeSpec_Ball.h:417-434);
//   - adjustStepSize (:448-502) picks the next step size and accepts the
//     step when it did not shrink.
// An accepted step writes y1 (with its normalized quaternions); a rejected one
// leaves y and retries with the smaller step. Each step's t1 follows
// takeOneStep's rule against tMax = tFinal (:536-544), which marks a step
// shortened to reach tFinal as artificially limited.
#include "steps_device.cuh"
#include "tile_device.cuh"

namespace sbg {

// AbstractIntegratorRep::adjustStepSize (AbstractIntegratorRep.cpp:448-502):
// returns whether the step succeeded (the new size is not smaller); hMin /
// hMax <= 0: no user limit.
__device__ __forceinline__ bool adjustStepSizeDev(double err, int errOrder, bool limited, double accuracy, double hMin,
                                                  double hMax, double& h) {
    const double Safety = 0.9, MinShrink = 0.1, MaxGrow = 5, HysteresisLow = 0.9, HysteresisHigh = 1.2;
    double hNew;
    if (!isfinite(err)) hNew = MinShrink * h;
    else if (err == 0) hNew = MaxGrow * h;
    else hNew = Safety * h * pow(accuracy / err, 1.0 / double(errOrder));
    if (hNew > h && (limited || hNew < HysteresisHigh * h)) hNew = h;
    if (hNew < h) {
        if (err <= accuracy) hNew = h;
        else hNew = fmin(hNew, HysteresisLow * h);
    }
    hNew = fmin(hNew, MaxGrow * h);
    hNew = fmax(hNew, MinShrink * h);
    if (hMin > 0) hNew = fmax(hNew, hMin);
    if (hMax > 0) hNew = fmin(hNew, hMax);
    const bool success = hNew >= h;
    h = hNew;
    return success;
}

namespace {

template <class CF>
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    rkAdaptiveTileKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT,
                         int ntiles, double* __restrict__ recs, double* y, double* __restrict__ time, double* fbuf, int64_t fplane,
                         int32_t* __restrict__ status, const __grid_constant__ AdaptCtl ac) {
    __shared__ TileShare<5> sh;
    forTiles<CF>(T, TT, 0, ntiles, recs, [&](const TileCtx& c) {
        const TileCol<CF::YS> col(T, c.inst);
        const int nq = col.nq, nu = T.inu[c.inst];
        double *f0 = fbuf, *fA = fbuf + fplane, *fB = fbuf + 2 * fplane, *fC = fbuf + 3 * fplane, *yt = fbuf + 4 * fplane;
        int st = 0;
        double tc = c.on ? time[c.inst] : 0.0;
        const double tFinal = ac.tFinal;
        double h = ac.hInit > 0 ? ac.hInit : 0.01;  // the system timescale / 10 (AbstractIntegratorRep.cpp:41-49)
        if (ac.hMin > 0) h = fmax(h, ac.hMin);
        if (ac.hMax > 0) h = fmin(h, ac.hMax);
        const double acc = ac.accuracy, consTol = ac.consTol;
        const double projLimit = fmax(2 * consTol, sqrt(consTol));
        long long nAcc = 0, nRej = 0;
        bool haveF0 = false, going = c.on;
        for (;;) {
            if (going && !(tc < tFinal)) going = false;
            if (going && nAcc >= ac.maxSteps) {
                st |= SBG_INST_TIMEOUT;
                going = false;
            }
            bool limited = false;
            double t1 = tc;
            if (going) {
                if (tFinal < tc + 0.95 * h) { limited = true; t1 = tFinal; }
                else if (tFinal > tc + 1.001 * h) t1 = tc + h;
                else t1 = tFinal;
            }
            // f0 = f(y0), kept across rejected attempts (the time-out below leaves
            // it formed, as it does in takeOneStep)
            const bool needF0 = going && !haveF0;
            if (going && !(t1 > tc)) {
                st |= SBG_INST_TIMEOUT;
                going = false;
            }
            if (!__any_sync(0xffffffffu, going || needF0)) break;
            const double hs = t1 - tc;
            int bits = 0;
    #pragma unroll 1
            for (int stg = __any_sync(0xffffffffu, needF0) ? 0 : 1; stg < 5; ++stg) {
                const double cc = stg == 0 ? 0.0 : stg == 1 ? hs / 3 : stg == 2 ? hs / 6 : stg == 3 ? hs / 8 : hs / 2;
                tileStageInput<CF>(TT, c, col, nq + nu, stg == 0 ? needF0 : going, stg, cc, y, f0, stg >= 3 ? fB : fA, fC, yt);
                const TileYSrc<CF::YS> src{col, yt};
                TileOut<CF::YS> out(col, stg == 0 ? f0 : stg == 2 ? fB : stg == 3 ? fC : fA);
                bits |= tileRhs<CF, false>(T, TT, c, src, out, stg == 0 ? needF0 : going);
                if (!out.finite) bits |= SBG_INST_NONFINITE;
            }
            const double h6 = hs / 6, h2 = hs / 2;
            auto y1At = [&](int64_t e, double* ysv) {
                const double y0 = y[e];
                const double a0 = f0[e], aB = fB[e], aC = fC[e], aA = fA[e];
                *ysv = y0 + h2 * ((a0 - 3.0 * aB) + 4.0 * aC);
                return y0 + h6 * ((a0 + 4.0 * aC) + aA);
            };
            // error norm and quaternion errors of y1, y untouched
            tileBodies<CF>(TT, c, going, [&](const tile::SlotRow& r) {
                    const int nqb = slotQ(r.info), n = (r.info >> 4) & 15;
                    double q1[4], dq[4], sq = 0, sqP = 0, extra = 0, su = 0;
    #pragma unroll
                    for (int j = 0; j < 7; ++j)
                        if (j < nqb) {
                            double ysv;
                            const double y1v = y1At(col.at(r.qo + j), &ysv);
                            const double dj = 0.2 * fabs(y1v - ysv);
                            if (j < 4) { q1[j] = y1v; dq[j] = dj; }
                            if (j >= 4 || !(r.info & F_QUAT)) extra += dj * dj;
                        }
                    if (r.info & F_QUAT) {
                        sq = tileQuatErrSq(q1, dq);
                        const double len = sqrt(q1[0] * q1[0] + q1[1] * q1[1] + q1[2] * q1[2] + q1[3] * q1[3]);
                        yt[col.at(r.qo + 1)] = (len - 1) * (len - 1);
                        // the same after normalization, the radial part of dq removed
                        double qn[4], dqn[4];
    #pragma unroll
                        for (int k = 0; k < 4; ++k) qn[k] = q1[k] / len;
                        const double d = dq[0] * qn[0] + dq[1] * qn[1] + dq[2] * qn[2] + dq[3] * qn[3];
    #pragma unroll
                        for (int k = 0; k < 4; ++k) dqn[k] = dq[k] - d * qn[k];
                        sqP = tileQuatErrSq(qn, dqn);
                    }
                    for (int j = 0; j < n; ++j) {
                        const int64_t e = col.atU(r.uo + j);
                        double ysv;
                        const double y1v = y1At(e, &ysv);
                        const double vi = fabs(y[e]);
                        double d = 0.2 * fabs(y1v - ysv);
                        if (vi > 1) d = d / vi;  // calcRelativeScaling, frozen at step start
                        su += d * d;
                    }
                    if (n > 0) {  // tileSums
                        yt[col.at(r.qo)] = sq + extra;
                        if (r.info & F_QUAT) yt[col.at(r.qo + 2)] = sqP + extra;
                        yt[col.atU(r.uo)] = su;
                    }
                });
            bits = tileReduce(TT, c, sh, bits);
            double v[5];  // sq, su, squat, nquat, sq after the projection
            tileSums(T, TT, c, sh, col, yt, going, v);
            bool take = false, proj = false;
            if (going) {
                st |= bits;
                haveF0 = true;
                const double un = nu ? sqrt(v[1] / nu) : 0.0;
                double qnorm = nq ? sqrt(v[0] / nq) : 0.0;
                double errNorm = qnorm >= un ? qnorm : un;
                if (errNorm <= 16 * acc) {  // attemptDAEStep's projection (AbstractIntegratorRep.cpp:158-199)
                    const double quatNorm = v[3] > 0 ? sqrt(v[2] / v[3]) : 0.0;
                    if (quatNorm > projLimit) {
                        errNorm = INFINITY;  // the step did not converge
                    } else if (quatNorm > consTol || ac.projectEveryStep) {
                        proj = true;
                        qnorm = nq ? sqrt(v[4] / nq) : 0.0;
                        errNorm = qnorm >= un ? qnorm : un;
                    }
                }
                take = adjustStepSizeDev(errNorm, 4, limited, acc, ac.hMin, ac.hMax, h);
                if (!take) {
                    ++nRej;
                    if (nRej > 64LL * ac.maxSteps) {
                        st |= SBG_INST_TIMEOUT;
                        going = false;
                    }
                }
            } else {
                st |= needF0 ? bits : 0;
            }
            int fin = 0;
            tileBodies<CF>(TT, c, take, [&](const tile::SlotRow& r) {
                    const int nqb = slotQ(r.info), n = (r.info >> 4) & 15;
                    double q1[4];
    #pragma unroll
                    for (int j = 0; j < 7; ++j)
                        if (j < nqb) {
                            double ysv;
                            const int64_t e = col.at(r.qo + j);
                            const double y1v = y1At(e, &ysv);
                            if (j < 4) q1[j] = y1v;
                            if (j >= 4 || !(proj && (r.info & F_QUAT))) {
                                y[e] = y1v;
                                if (!tile::finiteBits(y1v)) fin |= SBG_INST_NONFINITE;
                            }
                        }
                    if (proj && (r.info & F_QUAT)) {
                        const double len = sqrt(q1[0] * q1[0] + q1[1] * q1[1] + q1[2] * q1[2] + q1[3] * q1[3]);
    #pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const double qk = q1[k] / len;
                            y[col.at(r.qo + k)] = qk;
                            if (!tile::finiteBits(qk)) fin |= SBG_INST_NONFINITE;
                        }
                    }
                    for (int j = 0; j < n; ++j) {
                        double ysv;
                        const int64_t e = col.atU(r.uo + j);
                        const double y1v = y1At(e, &ysv);
                        y[e] = y1v;
                        if (!tile::finiteBits(y1v)) fin |= SBG_INST_NONFINITE;
                    }
                });
            fin = tileReduce(TT, c, sh, fin);
            if (take) {
                st |= fin;
                tc = t1;
                ++nAcc;
                haveF0 = false;
            }
        }
        if (c.on && c.w == 0) {
            time[c.inst] = tc;
            status[c.inst] = st;
            if (ac.stats) {
                ac.stats[2 * (int64_t)c.inst] = nAcc;
                ac.stats[2 * (int64_t)c.inst + 1] = nRej;
            }
        }
    });
}

}  // namespace

void rkAdaptiveTiles(const KArgs& a, const TileSet& S, const AdaptCtl& ac, cudaStream_t s) {
    if (S.ntiles <= 0) return;
    const TileLaunch L(S, S.ntiles);
    tileDispatch<kTile>(S, [&](auto cf) {
        rkAdaptiveTileKernel<decltype(cf)><<<L.grid, L.block, 0, s>>>(*a.T, S.tt, S.ntiles, S.recs, a.ystate, a.time,
                                                                            static_cast<double*>(a.fbuf), a.fplane,
                                                                            a.status, ac);
    });
}

}  // namespace sbg
