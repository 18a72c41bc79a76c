// k_util.cu -- state packing kernels, quaternion normalization and the
// precision dispatch of the launchers.
#include "abi_device.cuh"
#include "tile_core.cuh"

#include <algorithm>

namespace sbg {

// Integrator::initialize forces a projection: quaternions are normalized
// (Integrator.cpp:376-377, RigidBodyNodeSpec_Ball.h:417-434).
// One warp per instance, its lanes over the bodies: one thread per instance
// took 0.67 ms for 1,500 trees of up to 256 bodies, a chain of FP64 square roots
// and divisions per thread.
__global__ void __launch_bounds__(128) normalizeQuatKernel(const __grid_constant__ DevTables T, double* __restrict__ y) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= T.ninst) return;
    const int inst = T.order[t];
    if (T.incons[inst] > 0) return;  // loop closures: the RK kernel's initialization projects and normalizes
    const int64_t base = T.ybase[inst], stride = T.ystride[inst];
    const int body0 = T.ibody[inst], nb = T.inb[inst];
    for (int lb = threadIdx.x & 31; lb < nb; lb += 32) {
        const int row = body0 + lb;
        if (T.info[row] & F_QUAT) normalizeQuatAt(y, base, stride, T.qoff[row]);
    }
}

// State::getQDotDot() at Stage::Acceleration from the resident state and the
// last realize's udot, into the host packing (nq values per instance from
// qHost[inst]): qdotdot = udot for Pin/Slider/Universal; for the quaternion
// of a Ball or Free body N(q) udot_w - |w|^2/4 q with the unnormalized q
// (Rotation.h:1006-1013: convertAngVelDotToQuaternionDotDot), then the Free
// body's translational udot (RigidBodyNodeSpec_Ball.h:355-390,
// RigidBodyNodeSpec_Free.h:418-455). One thread per instance.
__global__ void qdotdotKernel(DevTables T, const int64_t* __restrict__ qHost, const double* __restrict__ y,
                              const double* __restrict__ ydot, double* __restrict__ out) {
    const int inst = blockIdx.x * blockDim.x + threadIdx.x;
    if (inst >= T.ninst) return;
    const int64_t base = T.ybase[inst], stride = T.ystride[inst];
    const int nq = T.inq[inst], body0 = T.ibody[inst], nb = T.inb[inst];
    double* o = out + qHost[inst];
    auto Y = [&](int k) { return y[base + (int64_t)k * stride]; };
    auto UD = [&](int k) { return ydot[base + (int64_t)(nq + k) * stride]; };
    for (int lb = 0; lb < nb; ++lb) {
        const int row = body0 + lb;
        const int type = T.info[row] & 15, n = (T.info[row] >> 4) & 15;
        const int qo = T.qoff[row], uo = T.uoff[row];
        if (type == T_BALL || type == T_FREE) {
            if (!(T.info[row] & F_QUAT)) {
                // body-fixed X-Y-Z angles: Rotation::convertAngAccInParentToBodyXYZDotDot
                // (Rotation.h:1041-1060) with qdot = N_P(q) w (Rotation.h:395-406)
                double c0, s0, c1, s1;
                sincos(Y(qo), &s0, &c0);
                sincos(Y(qo + 1), &s1, &c1);
                const double ooc1 = 1.0 / c1;
                const double w0 = Y(nq + uo), w1 = Y(nq + uo + 1), w2 = Y(nq + uo + 2);
                const double b0 = UD(uo), b1 = UD(uo + 1), b2 = UD(uo + 2);
                const double tw = (s0 * w1 - c0 * w2) * ooc1, tb = (s0 * b1 - c0 * b2) * ooc1;
                const double qd0 = w0 + tw * s1, qd2 = -tw;
                const double qd1 = c0 * w1 + s0 * w2;
                const double q1oc1 = qd1 * ooc1;
                o[qo + 0] = (b0 + tb * s1) + (qd0 * s1 - qd2) * q1oc1;
                o[qo + 1] = (c0 * b1 + s0 * b2) + qd0 * qd2 * c1;
                o[qo + 2] = -tb + (qd2 * s1 - qd0) * q1oc1;
                if (type == T_FREE) {
                    for (int k = 0; k < 3; ++k) o[qo + 3 + k] = UD(uo + 3 + k);
                    o[qo + 6] = 0.0;
                } else {
                    o[qo + 3] = 0.0;  // the unused slot
                }
                continue;
            }
        } else {  // u = qdot
            for (int k = 0; k < n; ++k) o[qo + k] = UD(uo + k);
            continue;
        }
        const double q0 = Y(qo), q1 = Y(qo + 1), q2 = Y(qo + 2), q3 = Y(qo + 3);
        const double w0 = Y(nq + uo), w1 = Y(nq + uo + 1), w2 = Y(nq + uo + 2);
        const double b0 = UD(uo), b1 = UD(uo + 1), b2 = UD(uo + 2);
        const double e0 = 0.5 * q0, e1 = 0.5 * q1, e2 = 0.5 * q2, e3 = 0.5 * q3;
        const double s = -0.25 * (w0 * w0 + w1 * w1 + w2 * w2);
        o[qo + 0] = (-e1 * b0 + -e2 * b1 + -e3 * b2) + s * q0;
        o[qo + 1] = (e0 * b0 + e3 * b1 + -e2 * b2) + s * q1;
        o[qo + 2] = (-e3 * b0 + e0 * b1 + e1 * b2) + s * q2;
        o[qo + 3] = (e2 * b0 + -e1 * b1 + e0 * b2) + s * q3;
        if (type == T_FREE)
            for (int k = 0; k < 3; ++k) o[qo + 4 + k] = UD(uo + 3 + k);
    }
}

cudaError_t launchQDotDot(const DevTables& T, const int64_t* qHost, const double* y, const double* ydot, double* out,
                          cudaStream_t s) {
    const int threads = 128, blocks = (T.ninst + threads - 1) / threads;
    if (blocks == 0) return cudaSuccess;
    qdotdotKernel<<<blocks, threads, 0, s>>>(T, qHost, y, ydot, out);
    return cudaGetLastError();
}

// Pack/unpack between the host's per-instance packing and the columns.
// part 0: all of [q,u]; part 1: the u slots only (nu values per instance).
// Contiguous columns: one block per instance.
template <bool SCATTER>
__global__ void __launch_bounds__(128) packKernel(const __grid_constant__ DevTables T, const int64_t* __restrict__ hostOff,
                                                  const double* __restrict__ src, double* __restrict__ dst, int part,
                                                  int pos0) {
    const int inst = T.order[pos0 + blockIdx.x];
    const int nq = T.inq[inst];
    const int cnt = part == 0 ? nq + T.inu[inst] : T.inu[inst];
    const int64_t base = T.ybase[inst] + (part == 0 ? 0 : nq), off = hostOff[inst];
    for (int k = threadIdx.x; k < cnt; k += blockDim.x) {
        if (SCATTER) dst[base + k] = src[off + k];
        else dst[off + k] = src[base + k];
    }
}
// Interleaved columns: the 32 instances of a tile by 32 elements at a time
// through shared memory, so that both sides move whole 256-byte rows. Bound by
// DRAM: 65,536 columns of 224 elements up in 50 us and down in 49 us, against
// 92 and 83 us with each instance's elements written 256 bytes apart.
template <bool SCATTER>
__global__ void __launch_bounds__(256) packTileKernel(const __grid_constant__ DevTables T,
                                                      const int64_t* __restrict__ hostOff,
                                                      const double* __restrict__ src, double* __restrict__ dst, int part,
                                                      int pos0, int count) {
    __shared__ double sm[32][33];
    __shared__ int64_t off[32], col[32];
    __shared__ int cnt[32], most;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w == 0) {
        const int p = blockIdx.x * kTile + lane;
        int n = 0;
        if (p < count) {
            const int inst = T.order[pos0 + p], nq = T.inq[inst], nu = T.inu[inst];
            n = part == 0 ? nq + nu : nu;
            off[lane] = hostOff[inst];
            col[lane] = T.ybase[inst] + (part == 0 ? 0 : (int64_t)nq * kTile);
        }
        cnt[lane] = n;
        n = __reduce_max_sync(0xffffffffu, n);
        if (lane == 0) most = n;
    }
    __syncthreads();
    for (int k0 = 32 * blockIdx.y; k0 < most; k0 += 32 * gridDim.y) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = w + 8 * r;
            if (SCATTER) {  // row of instance i
                if (k0 + lane < cnt[i]) sm[i][lane] = src[off[i] + k0 + lane];
            } else {        // element k0 + i of all
                if (k0 + i < cnt[lane]) sm[i][lane] = src[col[lane] + (int64_t)(k0 + i) * kTile];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = w + 8 * r;
            if (SCATTER) {
                if (k0 + i < cnt[lane]) dst[col[lane] + (int64_t)(k0 + i) * kTile] = sm[lane][i];
            } else {
                if (k0 + lane < cnt[i]) dst[off[i] + k0 + lane] = sm[lane][i];
            }
        }
        __syncthreads();
    }
}

template <bool SCATTER>
static cudaError_t launchPack(const Packing& P, const int64_t* hostOff, const double* src, double* dst, int part,
                              cudaStream_t s, int pos0, int count) {
    auto tiles = [&](int p0, int n) {
        if (n <= 0) return;
        const int nt = (n + kTile - 1) / kTile, rows = (P.maxCol + 31) / 32;
        const int split = std::max(1, std::min(rows, 1024 / nt));  // few tiles: their elements over several blocks
        packTileKernel<SCATTER><<<dim3(nt, split), 256, 0, s>>>(*P.T, hostOff, src, dst, part, p0, n);
    };
    if (count >= 0) {
        tiles(pos0, count);
    } else {
        tiles(0, P.tiles0);
        if (P.tiles1 > P.tiles0)
            packKernel<SCATTER><<<P.tiles1 - P.tiles0, 128, 0, s>>>(*P.T, hostOff, src, dst, part, P.tiles0);
        tiles(P.tiles1, P.ninst - P.tiles1);
    }
    return cudaGetLastError();
}
cudaError_t launchScatter(const Packing& P, const int64_t* hostOff, const double* packed, double* cols, int part,
                          cudaStream_t s, int pos0, int count) {
    return launchPack<true>(P, hostOff, packed, cols, part, s, pos0, count);
}
cudaError_t launchGather(const Packing& P, const int64_t* hostOff, const double* cols, double* packed, int part,
                         cudaStream_t s, int pos0, int count) {
    return launchPack<false>(P, hostOff, cols, packed, part, s, pos0, count);
}

// Run the chain segment, then the loop-closure segment, on the main stream
// and the level-parallel segment on the side stream, forked from and joined
// back into the main stream.
template <class FC, class FL, class FG>
static cudaError_t forkJoin(const LaunchPlan& P, const Streams& s, FC chain, FL loops, FG group) {
    const bool c = P.nChain > 0 || P.nLoop > 0, g = P.nGroupBlocks > 0;
    auto mainWork = [&](cudaStream_t st) {
        if (P.nChain > 0) chain(st);
        if (P.nLoop > 0) loops(st);
    };
    if (c && g) {
        cudaError_t e = cudaEventRecord(s.fork, s.main);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s.side, s.fork, 0);
        if (e != cudaSuccess) return e;
        group(s.side);
        mainWork(s.main);
        e = cudaEventRecord(s.join, s.side);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s.main, s.join, 0);
        if (e != cudaSuccess) return e;
    } else if (c) {
        mainWork(s.main);
    } else if (g) {
        group(s.main);
    }
    return cudaGetLastError();
}

static KArgs baseArgs(const DevTables& T, const LaunchPlan& P, const BatchBufs& B, int32_t* status) {
    KArgs a{};
    a.T = &T; a.P = &P; a.scratch = B.scratch; a.scratchLoop = B.scratchLoop; a.fbuf = B.fbuf;
    a.fbufLoop = B.fbufLoop; a.fplane = B.fplane; a.status = status; a.tiles32 = B.tiles32;
    return a;
}
// FP64: the tiles on the main stream and the loop-closure segment beside them
// on the side stream.
template <class FT, class FL>
static cudaError_t tilesAndLoops(const LaunchPlan& P, const TileSet& S, const Streams& s, FT tiles, FL loops) {
    if (P.nLoop == 0 || S.ntiles == 0) {
        if (P.nLoop > 0) loops(s.main); else tiles(s.main);
        return cudaGetLastError();
    }
    cudaError_t e = cudaEventRecord(s.fork, s.main);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.side, s.fork, 0);
    if (e != cudaSuccess) return e;
    loops(s.side);
    tiles(s.main);
    e = cudaEventRecord(s.join, s.side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.main, s.join, 0);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launchRealize(const DevTables& T, const LaunchPlan& P, int precision, const double* y, double* ydot,
                          const BatchBufs& B, int32_t* status, const Streams& s) {
    KArgs a = baseArgs(T, P, B, status);
    a.y = y; a.ydot = ydot;
    auto loops = [&](cudaStream_t st) { realizeLoopGroup(a, 32, st); };
    if (precision == SBG_PRECISION_FP64)
        return tilesAndLoops(P, *B.tiles, s, [&](cudaStream_t st) { realizeTiles(a, *B.tiles, 0, B.tiles->ntiles, st); }, loops);
    const bool ref = precision == SBG_PRECISION_MIXED;
    cudaError_t e = cudaSuccess;
    if (ref && fullTiles(*B.tiles, T.ninst)) e = cudaMemsetAsync(T.flagged, 0, sizeof(int32_t), s.main);
    if (e == cudaSuccess)
        e = forkJoin(P, s, [&](cudaStream_t st) { realize32Chain(a, ref, st); }, loops,
                     [&](cudaStream_t st) { realize32Group(a, ref, st); });
    if (e != cudaSuccess || !ref) return e;
    const TileSet& S = *B.tiles;  // the chain segment's tiles, then the group segment's
    const int group0 = P.nChain + P.nLoop, chainTiles = S.ntiles ? (P.nChain + S.tt.ls - 1) / S.tt.ls : 0;
    realizeFallbackTiles(a, S, 0, chainTiles, *B.ones, 0, P.nChain, 0, B.ones->blocks, s.main);
    realizeFallbackTiles(a, S, chainTiles, S.ntiles - chainTiles, *B.ones, group0, T.ninst - group0, 0, B.ones->blocks,
                         s.main);
    return cudaGetLastError();
}

cudaError_t launchMInv(const DevTables& T, const LaunchPlan& P, int precision, const double* y, const double* f,
                       double* out, const BatchBufs& B, int32_t* status, const Streams& s) {
    KArgs a = baseArgs(T, P, B, status);
    a.y = y; a.f = f; a.ydot = out;
    auto loops = [&](cudaStream_t st) { minvLoopGroup(a, 32, st); };
    if (precision == SBG_PRECISION_FP64)
        return tilesAndLoops(P, *B.tiles, s, [&](cudaStream_t st) { minvTiles(a, *B.tiles, st); }, loops);
    return forkJoin(P, s, [&](cudaStream_t st) { minv32Chain(a, st); }, loops,
                    [&](cudaStream_t st) { minv32Group(a, st); });
}

cudaError_t launchRKMerson(const DevTables& T, const LaunchPlan& P, int precision, double* y, double* time,
                           const BatchBufs& B, int32_t* status, double h, StepCtl step, double accuracy,
                           double consTol, int projectEveryStep, const Streams& s) {
    KArgs a = baseArgs(T, P, B, status);
    a.ystate = y; a.time = time; a.h = h; a.step = step; a.accuracy = accuracy; a.consTol = consTol;
    a.projectEveryStep = projectEveryStep;
    auto loops = [&](cudaStream_t st) { rkLoopGroup(a, 32, st); };
    if (precision == SBG_PRECISION_FP64)
        return tilesAndLoops(P, *B.tiles, s, [&](cudaStream_t st) { rkTiles(a, *B.tiles, st); }, loops);
    const bool ref = precision == SBG_PRECISION_MIXED;
    return forkJoin(P, s, [&](cudaStream_t st) { rk32Chain(a, ref, st); }, loops,
                    [&](cudaStream_t st) { rk32Group(a, ref, st); });
}

cudaError_t launchRKFp64List(const DevTables& T, const TileSet& S, const TileSet& ones, double* y, double* time, int32_t* status, double h,
                             StepCtl step, double accuracy, double consTol, int projectEveryStep, int64_t fplane,
                             cudaStream_t s) {
    KArgs a{};
    a.T = &T; a.ystate = y; a.time = time; a.status = status; a.h = h; a.step = step;
    a.accuracy = accuracy; a.consTol = consTol; a.projectEveryStep = projectEveryStep; a.fplane = fplane;
    rkTilesList(a, S, ones, s);
    return cudaGetLastError();
}

// Parameters of the tiles' slots (tile_core.cuh) from the body table: entry k
// is lane k % ls of slot k / ls, parRow[k] its row and kParIdentity (-1: none).
__global__ void __launch_bounds__(128) tileParKernel(const __grid_constant__ DevTables T,
                                                     const int32_t* __restrict__ parRow, int64_t n, int ls,
                                                     double* __restrict__ par) {
    using namespace tile;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        if (parRow[k] < 0) continue;
        const int row = parRow[k] & ~kParIdentity;
        double* o = par + (k / ls) * PR_COUNT * ls + k % ls;
        auto put = [&](int f, double v) { o[(int64_t)f * ls] = v; };
        const double* b = T.par64 + (int64_t)row * kParamStride;
        const int parent = T.parent[row];
        M3<double> RMB, PR = ident3<double>(), RPF;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            RMB.a[i] = b[22 + i];
            RPF.a[i] = b[10 + i];
        }
        const V3<double> com = mk3(b[1], b[2], b[3]), pMB = mk3(b[31], b[32], b[33]), pPF = mk3(b[19], b[20], b[21]);
        V3<double> pP = z3<double>();
        if (parent >= 0) {
            const double* p = T.par64 + (int64_t)(T.row0[row] + parent) * kParamStride;
#pragma unroll
            for (int i = 0; i < 9; ++i) PR.a[i] = p[22 + i];
            pP = mk3(p[31], p[32], p[33]);
        }
        const double m = b[0];
        const V3<double> c = mul(RMB, com) + pMB;
        // unit inertia about the mass centre in body axes, turned to M axes, then about M's origin
        const S3<double> G{b[4], b[5], b[6], b[7], b[8], b[9]};
        const S3<double> J = m * (reexpress(RMB, G - pointMassUnit(com)) + pointMassUnit(c));
        // The identity where the host's product is, whatever this one rounds to: a
        // lane applies C or leaves it out by what the other lanes of its step do.
        const M3<double> C = (parRow[k] & kParIdentity) ? ident3<double>() : mul(PR, RPF);
        const V3<double> d = mul(PR, pPF) + pP;
        put(PR_M, m);
        put(PR_MC, m * c.x); put(PR_MC + 1, m * c.y); put(PR_MC + 2, m * c.z);
        put(PR_J, J.xx); put(PR_J + 1, J.yy); put(PR_J + 2, J.zz);
        put(PR_J + 3, J.xy); put(PR_J + 4, J.xz); put(PR_J + 5, J.yz);
#pragma unroll
        for (int i = 0; i < 9; ++i) put(PR_C + i, C.a[i]);
        put(PR_D, d.x); put(PR_D + 1, d.y); put(PR_D + 2, d.z);
        put(PR_PITCH, b[34]);
        put(PR_PMB, pMB.x); put(PR_PMB + 1, pMB.y); put(PR_PMB + 2, pMB.z);
        // Q0: the rest position of the mobility's stiffest spring
        double K[6] = {}, S[6] = {}, B[6] = {}, Q0[6] = {}, stiff[6] = {};
        auto forces = [&](auto use) {
            for (int f = T.fbeg[row]; f < T.fbeg[row] + T.fcnt[row]; ++f) {
                const int which = T.fkind_which[f] & 255;
                const bool damper = (T.fkind_which[f] >> 8) != 0;
#pragma unroll
                for (int j = 0; j < 6; ++j)
                    if (j == which) use(j, damper, T.fcoef64[f], T.fq064[f]);
            }
        };
        forces([&](int j, bool damper, double v, double q0) {
            if (!damper && fabs(v) > stiff[j]) { stiff[j] = fabs(v); Q0[j] = q0; }
        });
        forces([&](int j, bool damper, double v, double q0) {
            if (damper) B[j] += v;
            else { K[j] += v; S[j] += v * (q0 - Q0[j]); }
        });
#pragma unroll
        for (int j = 0; j < 6; ++j) { put(PR_K + j, K[j]); put(PR_S + j, S[j]); put(PR_B + j, B[j]); put(PR_Q0 + j, Q0[j]); }
    }
}
cudaError_t launchTilePar(const DevTables& T, const int32_t* parRow, int64_t n, int ls, double* par, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    tileParKernel<<<(int)std::min<int64_t>((n + 127) / 128, 16384), 128, 0, s>>>(T, parRow, n, ls, par);
    return cudaGetLastError();
}

__global__ void fillIntKernel(int32_t* __restrict__ p, int n, int v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}
cudaError_t launchFillInt(int32_t* p, int n, int v, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    fillIntKernel<<<(n + 255) / 256, 256, 0, s>>>(p, n, v);
    return cudaGetLastError();
}

// Instances of a one-step integration call that have steps left (stepsLeft
// > 0; with stepsLeft null: time < tStop and no TIMEOUT status).
__global__ void countUnfinishedKernel(int n, const int32_t* __restrict__ stepsLeft, const double* __restrict__ time,
                                      const int32_t* __restrict__ status, double tStop, int32_t* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool left = false;
    if (i < n) left = stepsLeft ? stepsLeft[i] > 0 : (time[i] < tStop && !(status[i] & SBG_INST_TIMEOUT));
    const unsigned b = __ballot_sync(0xffffffffu, left);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(out, __popc(b));
}
cudaError_t launchCountUnfinished(int n, const int32_t* stepsLeft, const double* time, const int32_t* status,
                                  double tStop, int32_t* out, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(int32_t), s);
    if (e != cudaSuccess || n <= 0) return e;
    countUnfinishedKernel<<<(n + 255) / 256, 256, 0, s>>>(n, stepsLeft, time, status, tStop, out);
    return cudaGetLastError();
}

cudaError_t launchNormalizeQuat(const DevTables& T, double* y, cudaStream_t s) {
    const int blocks = (T.ninst + 3) / 4;
    if (blocks == 0) return cudaSuccess;
    normalizeQuatKernel<<<blocks, 128, 0, s>>>(T, y);
    return cudaGetLastError();
}

}  // namespace sbg
