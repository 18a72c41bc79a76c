// k_tileops.cu -- the O(n) tree operators of ops_device.cuh on the tile driver,
// in FP64 whatever the batch's precision, for the instances without loop
// closures (those keep the level-parallel kernel).
//
// Like the forward dynamics (tile_core.cuh) the sweeps keep each body in its
// mobilizer frame M: the body's inertia and the offsets are constants there,
// nothing but R_FM is formed per body, and Ground axes are carried along only
// where an operand or a result is in them. FP64 instructions bound them; a
// body takes about 150 (M x) to 300 (composite inertias), the sweeps in Ground
// axes about 400 to 700, and mobilizers don't diverge. 6,000 trees of 20 to 40
// bodies, inverse dynamics: 2.07 ms for the kernel before, 0.39 ms now.
#include "tile_device.cuh"

namespace sbg {

namespace {

using tile::Vec;
using tile::get3;
using tile::get9;
using tile::put3;
using tile::zero;

// Record of a body: E = R_FM, l, A = (alpha, a) of the origin of M, w and w.w,
// wrench about that origin, R_GM, composite m, m c, J. Below the columns and
// forces that a GEN joint keeps.
enum : int { OR_E = 0, OR_L = 9, OR_A = 12, OR_W = 18, OR_F = 22, OR_R = 28, OR_C = 37 };
static_assert(OR_C + 10 <= tile::RC_X, "operator records overlap the joint's");

struct OpCoords {
    TileCol<0> c;
    const double* y;
    bool withU;
    __device__ __forceinline__ double q(int k) const { return y[c.at(k)]; }
    __device__ __forceinline__ double u(int k) const { return withU ? y[c.atU(k)] : 0.0; }
    __device__ __forceinline__ double fext(int) const { return 0.0; }
};
struct OpNull {
    __device__ __forceinline__ void qdot(int, double) {}
};

// A joint's E = R_FM, p_FM, its columns times x (M axes), and the velocity
// terms sum u h_w, sum u h_v, sum u hdot_w (F axes).
struct OpJoint {
    M3<double> E;
    Vec p, xw, xv, wrel, vrel, hd;
};

template <int CL, class PA, class RC>
__device__ __forceinline__ void opJoint(const tile::SlotRow& r, const PA& par, const RC& rec, const OpCoords& src,
                                        const double* x, OpJoint& j) {
    j.E = ident3<double>();
    j.p = j.xw = j.xv = j.wrel = j.vrel = j.hd = zero();
    auto X = [&](int k) { return x ? x[r.uo + k] : 0.0; };
    if (CL == tile::CL_PIN) {
        double s, c;
        sincos(src.q(r.qo), &s, &c);
        j.E.a[0] = c; j.E.a[1] = -s; j.E.a[3] = s; j.E.a[4] = c;
        j.xw.z = X(0);
        j.wrel.z = src.u(r.uo);
    } else if (CL == tile::CL_SLIDER) {
        j.p.x = src.q(r.qo);
        j.xv.x = X(0);
        j.vrel.x = src.u(r.uo);
    } else if (CL == tile::CL_UNIV) {
        double s1, c1, s2, c2;
        sincos(src.q(r.qo), &s1, &c1);
        sincos(src.q(r.qo + 1), &s2, &c2);
        j.E = M3<double>{{c2, 0, s2, s2 * s1, c1, -(s1 * c2), -(s2 * c1), s1, c1 * c2}};
        j.xw = tile::rotT<1>(c2, s2, Vec{X(0), X(1), 0});
        const double u0 = src.u(r.uo), u1 = src.u(r.uo + 1);
        j.wrel = Vec{u0, u1 * c1, u1 * s1};
        j.hd = (u0 * u1) * Vec{0, -s1, c1};
    } else if (CL == tile::CL_BALL || CL == tile::CL_FREE) {
        double q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = src.q(r.qo + k);
        j.E = tile::quatMatrix(q);
        j.xw = mulT(j.E, Vec{X(0), X(1), X(2)});
        j.wrel = Vec{src.u(r.uo), src.u(r.uo + 1), src.u(r.uo + 2)};
        if (CL == tile::CL_FREE) {
            j.p = Vec{src.q(r.qo + 4), src.q(r.qo + 5), src.q(r.qo + 6)};
            j.xv = mulT(j.E, Vec{X(3), X(4), X(5)});
            j.vrel = Vec{src.u(r.uo + 3), src.u(r.uo + 4), src.u(r.uo + 5)};
        }
    } else {
        OpNull sink;
        tile::GenJoint g;
        tile::pass1Gen<false>(r, par, rec, src, sink, g);
        j.E = g.E;
        j.p = g.p;
        j.wrel = g.wrel;
        j.vrel = g.vrel;
        j.hd = g.hd;
        for (int k = 0; k < g.n; ++k) {
            j.xw = axpy(j.xw, X(k), get3(rec, tile::RC_H + 6 * k));
            j.xv = axpy(j.xv, X(k), get3(rec, tile::RC_H + 6 * k + 3));
        }
    }
}

template <class CF>
__global__ void __launch_bounds__(32 * kTileMaxWarps)
    tileOpKernel(const __grid_constant__ DevTables T, const __grid_constant__ TileTables TT, int ntiles,
                 const double* __restrict__ y, double* __restrict__ recs, const __grid_constant__ OpIO io,
                 int32_t* __restrict__ status) {
    using namespace tile;
    __shared__ TileShare<0> sh;
    forTiles<CF>(T, TT, 0, ntiles, recs, [&](const TileCtx& c) {
        typedef Rec<CF::LS> RC;
        typedef Par<(CF::SH ? 1 : CF::LS)> PA;
        const int64_t recSize = (int64_t)TT.rsTotal * CF::LS;
        auto recOf = [&](int slot) { return RC{c.rec + slot * recSize}; };
        const int kind = io.kind;
        const bool accel = kind == OP_RESIDUAL || kind == OP_MV || kind == OP_JV;
        const bool ground = kind == OP_JV || kind == OP_JTF || kind == OP_COMPOSITE || (kind == OP_RESIDUAL && io.fbody);
        const OpCoords src{{T, c.inst}, y, kind == OP_RESIDUAL};
        const int64_t u0 = io.uoff[c.inst], b0 = io.boff[c.inst];
        const int body0 = T.ibody[c.inst];
        const double* x = accel && io.x ? io.x + u0 : nullptr;
        bool finite = true;

        tileSweep<CF, true>(TT, c, c.on, [&](int cl, int slot, SlotRow r, PA par) {
            const RC rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
            const bool hasP = r.parent >= 0, ci = (r.info & F_CI) != 0;
            OpJoint j;
            switch (cl) {
            case CL_PIN: opJoint<CL_PIN>(r, par, rec, src, x, j); break;
            case CL_SLIDER: opJoint<CL_SLIDER>(r, par, rec, src, x, j); break;
            case CL_UNIV: opJoint<CL_UNIV>(r, par, rec, src, x, j); break;
            case CL_BALL: opJoint<CL_BALL>(r, par, rec, src, x, j); break;
            case CL_FREE: opJoint<CL_FREE>(r, par, rec, src, x, j); break;
            default: opJoint<CL_GEN>(r, par, rec, src, x, j); break;
            }
            // on Ground a position enters nothing; a state that is not finite is reported
            finite &= finiteBits(j.p.x) & finiteBits(j.p.y) & finiteBits(j.p.z);
            const M3<double> C = ci ? ident3<double>() : get9(par, PR_C);
            const M3<double> RL = ci ? j.E : mul(C, j.E);  // parent's axes <- these
            const Vec l = get3(par, PR_D) + (ci ? j.p : mul(C, j.p));
    #pragma unroll
            for (int k = 0; k < 9; ++k) rec[OR_E + k] = RL.a[k];
            put3(rec, OR_L, l);
            M3<double> RG = RL;
            if (ground) {
                if (hasP) RG = mul(get9(recP, OR_R), RL);
    #pragma unroll
                for (int k = 0; k < 9; ++k) rec[OR_R + k] = RG.a[k];
            }
            const double m = par[PR_M];
            const Vec mc = get3(par, PR_MC);
            const S3<double> J{par[PR_J], par[PR_J + 1], par[PR_J + 2], par[PR_J + 3], par[PR_J + 4], par[PR_J + 5]};
            if (kind == OP_COMPOSITE) {
                rec[OR_C] = m;
                put3(rec, OR_C + 1, mc);
                rec[OR_C + 4] = J.xx; rec[OR_C + 5] = J.yy; rec[OR_C + 6] = J.zz;
                rec[OR_C + 7] = J.xy; rec[OR_C + 8] = J.xz; rec[OR_C + 9] = J.yz;
                return;
            }
            Vec N = zero(), F = zero();
            if (accel) {
                // A = ~Phi A_parent + H x (+ a) (RigidBodyNodeSpec.cpp:566-582, 658-669, 762-775)
                Vec aw = j.xw, av = j.xv;
                if (hasP) {
                    const Vec pw = get3(recP, OR_A), pv = get3(recP, OR_A + 3);
                    aw = aw + mulT(RL, pw);
                    av = av + mulT(RL, pv + cross(pw, l));
                }
                if (kind == OP_RESIDUAL) {
                    const Vec wP = hasP ? get3(recP, OR_W) : zero();
                    const Vec wF = ci ? wP : mulT(C, wP);
                    const Vec w = mulT(j.E, wF + j.wrel);
                    aw = aw + mulT(j.E, cross(wF, j.wrel) + j.hd);
                    if (hasP) {
                        const Vec t = cross2(wP, recP[OR_W + 3], l);
                        av = av + mulT(j.E, (ci ? t : mulT(C, t)) + cross(wF + wF, j.vrel));
                    }
                    const double w2 = dot(w, w);
                    put3(rec, OR_W, w);
                    rec[OR_W + 3] = w2;
                    N = cross(w, mul(J, w));  // gyroscopic force (RigidBodyNode.cpp:98-174)
                    F = cross2(w, w2, mc);
                }
                put3(rec, OR_A, aw);
                put3(rec, OR_A + 3, av);
                if (kind == OP_JV) {  // velocity of the body's origin
                    const Vec ow = mul(RG, aw), ov = mul(RG, av + cross(aw, get3(par, PR_PMB)));
                    double* o = io.out + 6 * (b0 + T.bidx[body0 + r.row]);
                    o[0] = ow.x; o[1] = ow.y; o[2] = ow.z; o[3] = ov.x; o[4] = ov.y; o[5] = ov.z;
                    finite &= finiteBits(ow.x) & finiteBits(ow.y) & finiteBits(ow.z) & finiteBits(ov.x) & finiteBits(ov.y) &
                              finiteBits(ov.z);
                    return;
                }
                N = N + mul(J, aw) + cross(mc, av);
                F = F + m * av + cross(aw, mc);
            }
            if (io.fbody && kind != OP_MV) {
                const double* fb = io.fbody + 6 * (b0 + T.bidx[body0 + r.row]);
                const Vec fv = mulT(RG, Vec{fb[3], fb[4], fb[5]});
                const Vec fw = mulT(RG, Vec{fb[0], fb[1], fb[2]}) + cross(get3(par, PR_PMB), fv);
                if (kind == OP_JTF) { N = fw; F = fv; }
                else { N = N - fw; F = F - fv; }
            }
            put3(rec, OR_F, N);
            put3(rec, OR_F + 3, F);
        });

        if (kind != OP_JV)
            tileSweep<CF, false>(TT, c, c.on, [&](int cl, int slot, SlotRow r, PA par) {
                const RC rec = recOf(slot), recP = recOf(r.parent < 0 ? slot : r.parent);
                const bool hasP = r.parent >= 0;
                const M3<double> RL = get9(rec, OR_E);
                const Vec l = get3(rec, OR_L);
                if (kind == OP_COMPOSITE) {
                    // R = Mk + sum R_c (RigidBodyNode.cpp:232-243), about M's origin;
                    // the result about the body's origin
                    const double m = rec[OR_C];
                    const Vec mc = get3(rec, OR_C + 1);
                    const S3<double> J{rec[OR_C + 4], rec[OR_C + 5], rec[OR_C + 6], rec[OR_C + 7], rec[OR_C + 8], rec[OR_C + 9]};
                    const double oom = 1.0 / m;
                    const M3<double> RG = get9(rec, OR_R);
                    const Vec cM = oom * mc, p = get3(par, PR_PMB), cB = cM - p;
                    // unit inertia about the body's origin: G_M - point(cM) + point(cB)
                    S3<double> G = oom * J;
                    G = (G - pointMassUnit(cM)) + pointMassUnit(cB);
                    const Vec oc = mul(RG, cB);
                    const S3<double> oG = reexpress(RG, G);
                    double* o = io.out + 10 * (b0 + T.bidx[body0 + r.row]);
                    o[0] = m; o[1] = oc.x; o[2] = oc.y; o[3] = oc.z;
                    o[4] = oG.xx; o[5] = oG.yy; o[6] = oG.zz; o[7] = oG.xy; o[8] = oG.xz; o[9] = oG.yz;
                    finite &= finiteBits(m) & finiteBits(oc.x) & finiteBits(oc.y) & finiteBits(oc.z) & finiteBits(oG.xx) &
                              finiteBits(oG.yy) & finiteBits(oG.zz) & finiteBits(oG.xy) & finiteBits(oG.xz) & finiteBits(oG.yz);
                    if (hasP) {
                        // about the parent's M origin: J + 2 (l . mc) - (l mc~ + mc l~) + m (l.l - l l~)
                        const Vec k = mul(RL, mc), h = k + (0.5 * m) * l;  // so that l and h carry both terms
                        const S3<double> Jp = reexpress(RL, J);
                        const double lh = 2.0 * dot(l, h);
                        recP[OR_C] = recP[OR_C] + m;
                        put3(recP, OR_C + 1, get3(recP, OR_C + 1) + k + m * l);
                        recP[OR_C + 4] = recP[OR_C + 4] + Jp.xx + (lh - 2.0 * (l.x * h.x));
                        recP[OR_C + 5] = recP[OR_C + 5] + Jp.yy + (lh - 2.0 * (l.y * h.y));
                        recP[OR_C + 6] = recP[OR_C + 6] + Jp.zz + (lh - 2.0 * (l.z * h.z));
                        recP[OR_C + 7] = recP[OR_C + 7] + Jp.xy - (l.x * h.y + l.y * h.x);
                        recP[OR_C + 8] = recP[OR_C + 8] + Jp.xz - (l.x * h.z + l.z * h.x);
                        recP[OR_C + 9] = recP[OR_C + 9] + Jp.yz - (l.y * h.z + l.z * h.y);
                    }
                    return;
                }
                const Vec N = get3(rec, OR_F), F = get3(rec, OR_F + 3);
                const Vec Np = mul(RL, N), Fp = mul(RL, F);  // parent's axes
                if (hasP) {  // Phi F = (F_w + l x F_v, F_v)
                    put3(recP, OR_F, get3(recP, OR_F) + Np + cross(l, Fp));
                    put3(recP, OR_F + 3, get3(recP, OR_F + 3) + Fp);
                }
                // tau = ~H F (- f)
                auto put = [&](int k, double t) {
                    if (kind == OP_RESIDUAL && io.fmob) t = t - io.fmob[u0 + r.uo + k];
                    io.out[u0 + r.uo + k] = t;
                    finite &= finiteBits(t);
                };
                if (cl == CL_PIN) {
                    put(0, N.z);
                } else if (cl == CL_SLIDER) {
                    put(0, F.x);
                } else if (cl == CL_GEN) {
                    const int n = (r.info >> 4) & 15;
                    for (int k = 0; k < n; ++k)
                        put(k, dot(get3(rec, RC_H + 6 * k), N) + dot(get3(rec, RC_H + 6 * k + 3), F));
                } else {
                    // F axes: back by C where it is not the identity
                    const bool ci = (r.info & F_CI) != 0;
                    const Vec Nf = ci ? Np : mulT(get9(par, PR_C), Np);
                    put(0, Nf.x);
                    if (cl == CL_UNIV) {
                        put(1, N.y);
                    } else {
                        put(1, Nf.y);
                        put(2, Nf.z);
                        if (cl == CL_FREE) {
                            const Vec Ff = ci ? Fp : mulT(get9(par, PR_C), Fp);
                            put(3, Ff.x);
                            put(4, Ff.y);
                            put(5, Ff.z);
                        }
                    }
                }
            });
        int st = finite ? 0 : SBG_INST_NONFINITE;
        st = tileReduce(TT, c, sh, st);
        if (c.on && c.w == 0) status[c.inst] = st;
    });
}

}  // namespace

void treeOpTiles(const DevTables& T, const TileSet& S, const OpIO& io, const double* y, int32_t* status, cudaStream_t s) {
    if (S.ntiles <= 0) return;
    const TileLaunch L(S, S.ntiles);
    tileDispatch<0>(S, [&](auto cf) {
        tileOpKernel<decltype(cf)><<<L.grid, L.block, 0, s>>>(T, S.tt, S.ntiles, y, S.recs, io, status);
    });
}

}  // namespace sbg
