// k_tilerk32.cu -- fixed-step RK-Merson, mixed and FP32 forms, on the tile driver
// (kernel variant 9): rkMersonKernel of abi_device.cuh in tiles.
#include "tile32_device.cuh"

namespace sbg {

namespace {

template <class CF, int NM, bool REF>
__global__ void __launch_bounds__(32 * kTileMaxWarps, 1)
    rkTile32Kernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int ntiles,
                   float* __restrict__ recs, double* y, double* yt, double* __restrict__ time, float* fbuf, int64_t fplane,
                   int32_t* __restrict__ status, double h, StepCtl sc, double accuracy, double consTol, int pes) {
    __shared__ TileShare<4> sh;
    __shared__ TileMax mx;
    const int id = tileId(TT, 0, ntiles);
    if (id < 0) return;
    const TileCtx c = tileCtx<CF>(T, TT, id, nullptr);
    const int inst = c.inst;
    const TileCol<CF::YS> col(T, inst);
    const int nq = col.nq, nu = T.inu[inst];
    float *f0 = fbuf, *fA = fbuf + fplane, *fB = fbuf + 2 * fplane, *fC = fbuf + 3 * fplane;
    // One-step launches of a mixed batch integration: an instance in FP64 mode
    // is the list kernel's at this launch.
    const bool split = REF && T.fbList != nullptr;
    const bool mine = c.on && !(split && T.fbMode[(int64_t)(sc.launch & 1) * T.ninst + inst]);
    bool toFp64 = false;  // split: this launch's mixed step met an ill-conditioned M
    int st = mine ? status[inst] : 0;
    double tc = mine ? time[inst] : 0.0;
    const double tStop = sc.tStop;
    const int nst = sc.nsteps, maxSteps = sc.maxSteps > 0 ? sc.maxSteps : kMaxStepsPerCall;
    int left = T.stepsLeft && mine ? T.stepsLeft[inst] : kMaxStepsPerCall;
    const double projLimit = fmax(2 * consTol, sqrt(consTol));
    bool going = mine;
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
        int bits = 0, ill = 0;
#pragma unroll 1
        for (int stg = 0; stg < 5; ++stg) {
            const double cc = stg == 0 ? 0.0 : stg == 1 ? hs / 3 : stg == 2 ? hs / 6 : stg == 3 ? hs / 8 : hs / 2;
            tileStageInput<CF>(TT, c, col, nq + nu, going, stg, cc, y, f0, stg >= 3 ? fB : fA, fC, yt);
            const YSrc src{yt, col.base, col.stride, nq};
            FOut<float> out{stg == 0 ? f0 : stg == 2 ? fB : stg == 3 ? fC : fA, col.base, col.stride, nq};
            bits |= tileRhs32<CF, NM, REF>(T, TT, c, recs, tileStage<NM>(), src, out, going);
            if (!out.finite) bits |= SBG_INST_NONFINITE;
            if constexpr (REF) ill |= tileIll(T, TT, c, mx, out);
        }
        if (going && split && ill) {
            // Leave y and t as they were; the FP64 list kernel takes this step
            // at the next launch, and the next few.
            toFp64 = true;
        }
        const bool take = going && !toFp64;
        const double h6 = hs / 6, h2 = hs / 2;
        tileBodies<CF>(TT, c, take, [&](const tile::SlotRow& r) {
            const int nqb = slotQ(r.info), n = (r.info >> 4) & 15;
            double q1[4], dq[4], sq = 0, extra = 0, su = 0;
#pragma unroll
            for (int j = 0; j < 7; ++j)
                if (j < nqb) {
                    const int64_t e = col.at(r.qo + j);
                    const double y0 = y[e];
                    const double a0 = double(f0[e]), aB = double(fB[e]), aC = double(fC[e]), aA = double(fA[e]);
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
                const double y0 = y[e];
                const double a0 = double(f0[e]), aB = double(fB[e]), aC = double(fC[e]), aA = double(fA[e]);
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
        tileSums(T, TT, c, sh, col, yt, take, v);
        bool renorm = false;
        if (going) {
            st |= bits;
            if (!split) st |= ill;
            if (toFp64) {
                if (c.w == 0) T.fbLeft[inst] = kFp64Steps;
                going = false;
            }
        }
        if (take) {
            const double qn = nq ? sqrt(v[0] / nq) : 0.0, un = nu ? sqrt(v[1] / nu) : 0.0;
            const double errNorm = qn >= un ? qn : un;
            if (errNorm <= 16 * accuracy && v[3] > 0) {
                const double quatNorm = sqrt(v[2] / v[3]);
                if (quatNorm > projLimit) st |= SBG_INST_PROJECTION_FAILED;
                else if (quatNorm > consTol || pes) renorm = true;
            }
            tc = t1;
            --left;
        }
        if (__any_sync(0xffffffffu, renorm))
            tileBodies<CF>(TT, c, renorm, [&](const tile::SlotRow& r) {
                if (r.info & F_QUAT) normalizeQuatAt(y, col.base, col.stride, r.qo);
            });
        tileSync(TT.W, c);
    }
    if (mine && c.w == 0) {
        if (T.stepsLeft) T.stepsLeft[inst] = left;
        if (split) fbNext(T, sc.launch, inst, toFp64);
        time[inst] = tc;
        status[inst] = st;
    }
}

template <int NM, bool REF> void go(const KArgs& a, const TileSet& S, cudaStream_t s) {
    const TileLaunch L(S, S.ntiles);
    float *fb = static_cast<float*>(a.fbuf), *recs = reinterpret_cast<float*>(S.recs);
    auto launch = [&](auto cf) {
        auto* const kernel = rkTile32Kernel<decltype(cf), NM, REF>;
        kernel<<<L.grid, L.block, tileStageBytes<NM>(kernel, L.block), s>>>(
            *a.T, S.tt, S.ntiles, recs, a.ystate, S.yt, a.time, fb, a.fplane, a.status, a.h, a.step, a.accuracy, a.consTol,
            a.projectEveryStep);
    };
    if (S.tt.shared) launch(TileCfg<32, true, 0>());
    else launch(TileCfg<32, false, 0>());
}

}  // namespace

void rkTiles32(const KArgs& a, const TileSet& S, bool refine, cudaStream_t s) {
    if (S.ntiles <= 0) return;
    if (a.P->nm == 1) {
        if (refine) go<1, true>(a, S, s); else go<1, false>(a, S, s);
    } else {
        if (refine) go<3, true>(a, S, s); else go<3, false>(a, S, s);
    }
}

}  // namespace sbg
