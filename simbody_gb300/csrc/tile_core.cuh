// tile_core.cuh -- FP64 articulated-body forward dynamics in joint frames: the
// per-body arithmetic of the tile driver (tile_device.cuh).
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition,
// whether one lane or 32 are active and whatever else the warp does, so an
// FP64 sweep costs its FP64 instructions and hardly anything else. The
// recursion here is the one of RigidBodyNodeSpec.cpp:249-446 written for the
// fewest of them. Everything of a body is kept in the axes and about the
// origin of its mobilizer frame M (fixed in the body):
//   - the joint's axes are then coordinate axes (of M, or of the frame between
//     the two axes of a Universal), so P H, D and G are rows of P, and what a
//     rotational joint transmits has zero rows that are neither computed nor
//     rotated: a Ball passes on six numbers of P+ instead of 21;
//   - the body's own inertia and the offset to its children are constants;
//   - no position or linear velocity is needed: velocities enter through
//     w x J w, w x (w x m c) and w x (w x l) alone, and gravity is an
//     acceleration of the base (contact spheres carry the Ground pose along).
// FP64 instructions of one RHS per body: Pin about 300, Slider 200, Universal
// 500, Ball 390; the sweeps in Ground axes about body origins that they
// replace take about 950 with three columns.
//
// Host-compilable (no intrinsics).
#pragma once
#include <cmath>
#include <cstdint>

#include "engine.h"
#include "spatial.cuh"

namespace sbg {
namespace tile {

// What a slot of the tile's schedule runs (uniform over the lanes).
enum : int { CL_PIN = 0, CL_SLIDER, CL_UNIV, CL_BALL, CL_FREE, CL_GEN, CL_COUNT };

// Parameters of a body (doubles), in M axes about the origin of M.
//   C = R of the inboard frame F in the parent's M axes, d = its origin there
//   mobility forces folded per mobility: f_j = S_j - K_j (q_j - Q0_j) - B_j u_j,
//   S_j zero unless springs of several rest positions act on j
//   p_MB, the body's origin
enum : int { PR_M = 0, PR_MC = 1, PR_J = 4, PR_C = 10, PR_D = 19, PR_PITCH = 22, PR_K = 23, PR_S = 29, PR_B = 35,
             PR_Q0 = 41, PR_PMB = 47, PR_COUNT = 50 };
// Integers of a body: q and u slots, slot of the parent (-1 = Ground), info
// word (body table), body row, contacts.
enum : int { SI_Q = 0, SI_U, SI_PARENT, SI_INFO, SI_ROW, SI_KBEG, SI_KCNT, SI_COUNT = 8 };
// Info word of a slot, on every lane alike: C is the identity; no mobility
// force acts on the body; a spring and a damper act on every mobility.
constexpr int F_CI = 1 << 20, F_FREELY = 1 << 21, F_FORCES = 1 << 22;

// Record of a body (doubles).
//   P (J F M) and z: own inertia and force, then the children's on top
//   w and w.w, then A = (alpha, a of the origin of M)
//   l: parent's M origin to this one's, parent axes; E = R_FM (or c s c s)
//   gamma: velocity part of the acceleration; X: f, then the factorisation
// In a batch with contact spheres the Ground pose and velocity follow.
enum : int { RC_J = 0, RC_F = 6, RC_M = 15, RC_Z = 21, RC_W = 27, RC_W2 = 30, RC_L = 33, RC_E = 36, RC_GAM = 45, RC_X = 51,
             RC_SMALL = 63, RC_H = 63, RC_G = 99, RC_GEN = 135, RC_POSE = 15 };

typedef double D;
typedef V3<double> Vec;

// A body's record and parameters, field by field across LS lanes: LS is known
// at compile time, so a field is an offset in its load or store.
template <int LS> struct Rec {
    D* p;
    __host__ __device__ __forceinline__ D& operator[](int f) const { return p[f * LS]; }
};
template <int LS> struct Par {
    const D* p;
    __host__ __device__ __forceinline__ D operator[](int f) const { return p[f * LS]; }
};

#define TILE_FN __host__ __device__ __forceinline__
#ifdef __CUDACC__
#define TILE_CALL __host__ __device__ __noinline__ inline  // a call, not inlined
#else
#define TILE_CALL inline
#endif

template <class A> TILE_FN Vec get3(const A& a, int f) { return Vec{a[f], a[f + 1], a[f + 2]}; }
template <class A> TILE_FN void put3(const A& r, int f, Vec v) { r[f] = v.x; r[f + 1] = v.y; r[f + 2] = v.z; }
template <class A> TILE_FN S3<D> get6(const A& r, int f) { return S3<D>{r[f], r[f + 1], r[f + 2], r[f + 3], r[f + 4], r[f + 5]}; }
template <class A> TILE_FN M3<D> get9(const A& a, int f) {
    M3<D> m;
#pragma unroll
    for (int i = 0; i < 9; ++i) m.a[i] = a[f + i];
    return m;
}
TILE_FN Vec zero() { return Vec{0, 0, 0}; }
// Tests of the bits: an FP64 comparison would take the FP64 pipe.
TILE_FN uint64_t bitsOf(D v) {
    union { D d; uint64_t u; } b;
    b.d = v;
    return b.u;
}
TILE_FN bool finiteBits(D v) { return (bitsOf(v) & 0x7ff0000000000000ull) != 0x7ff0000000000000ull; }
TILE_FN bool nonzero(D v) { return (bitsOf(v) << 1) != 0; }

// Rotations about one axis: v in the rotated frame -> v in the fixed one
// (rot) and back (rotT).
template <int AX> TILE_FN Vec rot(D c, D s, Vec v) {
    if (AX == 0) return Vec{v.x, c * v.y - s * v.z, s * v.y + c * v.z};
    if (AX == 1) return Vec{c * v.x + s * v.z, v.y, c * v.z - s * v.x};
    return Vec{c * v.x - s * v.y, s * v.x + c * v.y, v.z};
}
template <int AX> TILE_FN Vec rotT(D c, D s, Vec v) { return rot<AX>(c, -s, v); }
// 2x2 symmetric block (a b; b d) rotated by (c, s): six operations by way of
// the double angle.
TILE_FN void rotBlock(D c, D s, D& a, D& b, D& d) {
    const D m = s * (a - d) + (c + c) * b;
    const D b2 = c * m - b;
    a = a - s * m;
    d = d + s * m;
    b = b2;
}
template <int AX> TILE_FN void rotSym(D c, D s, S3<D>& m) {
    if (AX == 0) {
        rotBlock(c, s, m.yy, m.yz, m.zz);
        const D t = c * m.xy - s * m.xz;
        m.xz = s * m.xy + c * m.xz;
        m.xy = t;
    } else if (AX == 1) {  // (z, x) is the rotated pair
        rotBlock(c, s, m.zz, m.xz, m.xx);
        const D t = c * m.yz - s * m.xy;
        m.xy = s * m.yz + c * m.xy;
        m.yz = t;
    } else {
        rotBlock(c, s, m.xx, m.xy, m.yy);
        const D t = c * m.xz - s * m.yz;
        m.yz = s * m.xz + c * m.yz;
        m.xz = t;
    }
}
// R F R^T about AX for an F whose row AX is zero (and stays so).
template <int AX> TILE_FN void rotMat(D c, D s, M3<D>& f) {
    constexpr int i = (AX + 1) % 3, j = (AX + 2) % 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const D t = c * f.a[3 * i + k] - s * f.a[3 * j + k];
        f.a[3 * j + k] = s * f.a[3 * i + k] + c * f.a[3 * j + k];
        f.a[3 * i + k] = t;
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        D* row = f.a + 3 * (m == 0 ? i : j);
        const D t = c * row[i] - s * row[j];
        row[j] = s * row[i] + c * row[j];
        row[i] = t;
    }
}
TILE_FN M3<D> mulABt(const M3<D>& A, const M3<D>& B) {
    M3<D> C;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            C.a[3 * i + j] = A.a[3 * i] * B.a[3 * j] + A.a[3 * i + 1] * B.a[3 * j + 1] + A.a[3 * i + 2] * B.a[3 * j + 2];
    return C;
}

// The same for a symmetric matrix whose row and column AX are zero.
template <int AX> TILE_FN void rotSym2(D c, D s, S3<D>& m) {
    if (AX == 0) rotBlock(c, s, m.yy, m.yz, m.zz);
    else if (AX == 1) rotBlock(c, s, m.zz, m.xz, m.xx);
    else rotBlock(c, s, m.xx, m.xy, m.yy);
}
// A zero that adding leaves out at compile time: x + (-0.0) is x.
#define TILE_NIL (-0.0)

TILE_FN D rsqrtD(D x) {
#ifdef __CUDA_ARCH__
    return rsqrt(x);
#else
    return D(1) / sqrt(x);
#endif
}
// Quaternion (normalised here) -> R_FM (RigidBodyNodeSpec_Ball.h:134-214).
TILE_FN M3<D> quatMatrix(const D* q) {
    D oo = rsqrtD(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    if (!nonzero(oo)) oo = D(NAN);  // |q|^2 overflows: no rotation, not the identity that 1 - 0 would make
    const D e0 = q[0] * oo, e1 = q[1] * oo, e2 = q[2] * oo, e3 = q[3] * oo;
    const D f1 = e1 + e1, f2 = e2 + e2, f3 = e3 + e3;
    const D p01 = e0 * f1, p02 = e0 * f2, p03 = e0 * f3;
    const D t1 = D(1) - e1 * f1;
    M3<D> R;
    R.a[0] = (D(1) - e2 * f2) - e3 * f3;
    R.a[4] = t1 - e3 * f3;
    R.a[8] = t1 - e2 * f2;
    R.a[1] = e1 * f2 - p03;
    R.a[3] = e1 * f2 + p03;
    R.a[2] = e1 * f3 + p02;
    R.a[6] = e1 * f3 - p02;
    R.a[5] = e2 * f3 - p01;
    R.a[7] = e2 * f3 + p01;
    return R;
}
// w x (w x v), w2 = w . w
TILE_FN Vec cross2(Vec w, D w2, Vec v) {
    const D t = dot(w, v);
    return Vec{t * w.x - w2 * v.x, t * w.y - w2 * v.y, t * w.z - w2 * v.z};
}

// Inverse of a symmetric 3x3; false when its determinant is zero.
TILE_FN bool invSym(const S3<D>& J, S3<D>& o) {
    const D c00 = J.yy * J.zz - J.yz * J.yz, c01 = J.xz * J.yz - J.xy * J.zz, c02 = J.xy * J.yz - J.xz * J.yy;
    const D det = J.xx * c00 + J.xy * c01 + J.xz * c02;
    const D r = D(1) / det;
    o.xx = r * c00;
    o.xy = r * c01;
    o.xz = r * c02;
    o.yy = r * (J.xx * J.zz - J.xz * J.xz);
    o.yz = r * (J.xy * J.xz - J.xx * J.yz);
    o.zz = r * (J.xx * J.yy - J.xy * J.xy);
    return nonzero(det);
}

struct SlotRow {
    int qo, uo, parent, info, row, kbeg, kcnt;
};

// ---------------------------------------------------------------- contacts
// SmoothSphereHalfSpaceForce (SmoothSphereHalfSpaceForce.cpp:252-336) of the
// spheres of one body, as contactForces of abi_device.cuh: moment about the
// body-fixed point with pose (R, p), whose velocity and spin in Ground are v
// and w; the station is the body's, taken through R_MB and p_MB of its
// parameters. Out of line: the other rows do not pay for its registers.
struct ContactWrench { Vec w, v; };
TILE_CALL ContactWrench contactWrench(const D* KP, int kb, int kc, const D* bodyPar,
                                                                    M3<D> R, Vec p, Vec w, Vec v) {
    Vec Mw = zero(), Fv = zero();
    M3<D> RMB;
    for (int i = 0; i < 9; ++i) RMB.a[i] = bodyPar[22 + i];
    const Vec pMB = Vec{bodyPar[31], bodyPar[32], bodyPar[33]};
    for (int k = 0; k < kc; ++k) {
        const D* c = KP + (int64_t)kb + (int64_t)k * kContactStride;
        const Vec n = Vec{c[4], c[5], c[6]};
        const Vec centre = mul(R, mul(RMB, Vec{c[0], c[1], c[2]}) + pMB) + p;
        const D ind = dot(centre - Vec{c[7], c[8], c[9]}, n) + c[3];
        const Vec r = (centre + (c[3] - D(0.5) * ind) * n) - p;
        const Vec vp = v + cross(w, r);
        const D vn = dot(vp, n);
        const Vec vt = vp - vn * n;
        // Hertz, smoothed about zero indentation (s^1.5 = s sqrt(s)), then Hunt-Crossley
        const D s = sqrt(ind * ind + c[16]);
        const D fh = c[10] * (s * sqrt(s)) * (D(0.5) + D(0.5) * tanh(c[17] * ind));
        const D fn = fh * (D(1) + D(1.5) * c[11] * vn) * (D(0.5) + D(0.5) * tanh(c[18] * (vn + c[19])));
        // smoothed static / dynamic / viscous friction along the slip
        const D vs = sqrt(dot(vt, vt) + c[16]);
        const D vr = vs / c[15];
        const D ff = fn * ((vr < D(1) ? vr : D(1)) * (c[13] + D(2) * (c[12] - c[13]) / (D(1) + vr * vr)) + c[14] * vs);
        const Vec force = fn * n + (ff / vs) * vt;
        Mw = Mw - cross(r, force);
        Fv = Fv - force;
    }
    return ContactWrench{Mw, Fv};
}

// Mobility force j. The difference from the rest position comes first: K q
// against a stored K q0 would lose what the two have in common. Where some lane
// of the step has a mobility without a spring or a damper, an element that is
// not there is left out, so that a body's force does not depend on its
// neighbours at an infinite coordinate either; out of line, the usual bodies
// (a spring and a damper each, or nothing) do not pay for the tests (8,192
// trees, four steps: 11.64 ms with K q0 folded, 12.0 with the tests inline, 11.9
// so).
TILE_CALL D mobForceSome(D S, D K, D d, D B, D u) {
    if (nonzero(K)) S = S - K * d;
    if (nonzero(B)) S = S - B * u;
    return S;
}
template <class PA> TILE_FN D mobForce(const PA& par, int info, int j, D q, D u) {
    const D S = par[PR_S + j], K = par[PR_K + j], d = q - par[PR_Q0 + j], B = par[PR_B + j];
    return (info & F_FORCES) ? (S - K * d) - B * u : mobForceSome(S, K, d, B, u);
}

// ------------------------------------------------------------------ pass 1
// Base to tip: joint rotation, spin, velocity terms, own inertia and force,
// mobility forces, qdot. MINV: rest, the forces given by the source. out also gets
// the positions: on Ground they enter nothing here, and a state that is not
// finite is still reported.
struct Model {
    const D* kpar;     // contact parameters
    const D* bodyPar;  // kParamStride per body row (contacts only)
    Vec g;             // gravity
    int rs;            // record size without the pose
    bool pose;         // the batch has contact spheres
};

// The coordinates of a GEN joint: E = R_FM, p_FM, and its columns in F.
struct GenJoint {
    M3<D> E;
    Vec p, wrel, vrel, hd;  // sum u h_w, sum u h_v, sum u hdot_w
    int n;
};

template <bool MINV, class PA, class RC, class Src, class Out>
TILE_FN void pass1Gen(const SlotRow& r, const PA& par, const RC& rec, const Src& src, Out& out, GenJoint& j) {
    const int type = r.info & 15, n = (r.info >> 4) & 15;
    D q[6], u[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        q[k] = k < n ? src.q(r.qo + k) : D(0);
        u[k] = k < n ? (MINV ? D(0) : src.u(r.uo + k)) : D(0);
    }
    j.E = ident3<D>();
    j.p = j.wrel = j.vrel = j.hd = zero();
    j.n = n;
    const bool ball = type == 3, freeJ = type == 4;             // Euler-angle form
    const bool xyz = ball || freeJ || type == 5 || type == 9;   // Gimbal, Bushing
    Vec h[3];  // rotational columns
    h[0] = Vec{1, 0, 0}; h[1] = Vec{0, 1, 0}; h[2] = Vec{0, 0, 1};
    if (xyz) {
        D c0, s0, c1, s1, c2, s2;
        sincos(q[0], &s0, &c0);
        sincos(q[1], &s1, &c1);
        sincos(q[2], &s2, &c2);
        const D s0s1 = s0 * s1, s2c0 = s2 * c0, c0c2 = c0 * c2;
        j.E.a[0] = c1 * c2;              j.E.a[1] = -(s2 * c1);            j.E.a[2] = s1;
        j.E.a[3] = s2c0 + s0s1 * c2;     j.E.a[4] = c0c2 - s0s1 * s2;      j.E.a[5] = -(s0 * c1);
        j.E.a[6] = s0 * s2 - s1 * c0c2;  j.E.a[7] = s0 * c2 + s1 * s2c0;   j.E.a[8] = c0 * c1;
        if (ball || freeJ) {
            // qdot = N_P(q) w_FM (Rotation.h:395-406); the last q slot is unused
            const D t = (s0 * u[1] - c0 * u[2]) / c1;
            out.qdot(r.qo + 0, u[0] + t * s1);
            out.qdot(r.qo + 1, c0 * u[1] + s0 * u[2]);
            out.qdot(r.qo + 2, -t);
            if (freeJ)
                for (int k = 3; k < 6; ++k) out.qdot(r.qo + k, u[k]);
            out.qdot(r.qo + (ball ? 3 : 6), D(0));
        } else {
            h[1] = Vec{0, c0, s0};
            h[2] = Vec{s1, -(s0 * c1), c0 * c1};
            const D dc0 = -s0 * u[0], dc1 = -s1 * u[1], ds0 = c0 * u[0], ds1 = c1 * u[1];
            j.hd = u[1] * Vec{0, dc0, ds0} + u[2] * Vec{ds1, -ds0 * c1 - s0 * dc1, dc0 * c1 + c0 * dc1};
        }
        if (freeJ || type == 9) j.p = Vec{q[3], q[4], q[5]};
        j.wrel = u[0] * h[0] + u[1] * h[1] + u[2] * h[2];
        if (freeJ || type == 9) j.vrel = Vec{u[3], u[4], u[5]};
    } else if (type == 6) {  // Translation
        j.p = Vec{q[0], q[1], q[2]};
        j.vrel = Vec{u[0], u[1], u[2]};
    } else if (type == 7 || type == 8 || type == 11) {  // Cylinder, Planar, Screw: about Fz
        D c, s;
        sincos(q[0], &s, &c);
        j.E.a[0] = c; j.E.a[1] = -s; j.E.a[3] = s; j.E.a[4] = c;
        j.wrel = Vec{0, 0, u[0]};
        if (type == 7) { j.p = Vec{0, 0, q[1]}; j.vrel = Vec{0, 0, u[1]}; }
        if (type == 8) { j.p = Vec{q[1], q[2], 0}; j.vrel = Vec{u[1], u[2], 0}; }
        if (type == 11) { j.p = Vec{0, 0, q[0] * par[PR_PITCH]}; j.vrel = Vec{0, 0, u[0] * par[PR_PITCH]}; }
    }
    if (!(ball || freeJ))
        for (int k = 0; k < n; ++k) out.qdot(r.qo + k, u[k]);
    // columns in M axes
    for (int k = 0; k < n; ++k) {
        Vec hw = zero(), hv = zero();
        if (xyz) {
            if (k < 3) hw = k == 0 ? h[0] : k == 1 ? h[1] : h[2];
            else hv = Vec{D(k == 3), D(k == 4), D(k == 5)};
        } else if (type == 6) {
            hv = Vec{D(k == 0), D(k == 1), D(k == 2)};
        } else if (k == 0) {
            hw = Vec{0, 0, 1};
            if (type == 11) hv = Vec{0, 0, par[PR_PITCH]};
        } else {
            hv = type == 7 ? Vec{0, 0, 1} : Vec{D(k == 1), D(k == 2), 0};
        }
        put3(rec, RC_H + 6 * k, mulT(j.E, hw));
        put3(rec, RC_H + 6 * k + 3, mulT(j.E, hv));
    }
    for (int k = 0; k < n; ++k) {
        if (MINV) rec[RC_X + k] = src.fext(r.uo + k);
        else {
            const D qk = (ball || freeJ) && k >= n ? D(0) : src.q(r.qo + k);
            rec[RC_X + k] = mobForce(par, r.info, k, qk, src.u(r.uo + k));
        }
    }
}

template <int CL, bool MINV, class PA, class RC, class Src, class Out>
TILE_FN void pass1(const Model& md, const SlotRow& r, const PA& par, const RC& rec, const RC& recP, const Src& src,
                   Out& out) {
    const bool hasP = r.parent >= 0, ci = (r.info & F_CI) != 0, freely = !MINV && (r.info & F_FREELY) != 0;
    const Vec d = get3(par, PR_D);
    const Vec wP = (!MINV && hasP) ? get3(recP, RC_W) : zero();
    const D wP2 = (!MINV && hasP) ? recP[RC_W2] : D(0);
    Vec l = d, w = zero(), gw = zero(), gv = zero();
    // rotates by C^T (into F) where C is not the identity
    auto toF = [&](Vec v) { return ci ? v : mulT(get9(par, PR_C), v); };
    const Vec wF = MINV ? zero() : toF(wP);
    M3<D> E;
    Vec vrelL = zero();  // velocity of M's origin relative to F, M axes (pose only)
    D c1 = 1, s1 = 0, c2 = 1, s2 = 0;
    if (CL == CL_PIN) {
        const D q0 = src.q(r.qo), u0 = MINV ? D(0) : src.u(r.uo);
        sincos(q0, &s1, &c1);
        rec[RC_E] = c1;
        rec[RC_E + 1] = s1;
        out.qdot(r.qo, u0);
        if (MINV) rec[RC_X] = src.fext(r.uo);
        else {
            rec[RC_X] = freely ? D(0) : mobForce(par, r.info, 0, q0, u0);
            w.z = u0;
            if (hasP) {
                const Vec t = rotT<2>(c1, s1, wF);
                w = Vec{t.x, t.y, t.z + u0};
                gw = Vec{u0 * t.y, -(u0 * t.x), 0};
                gv = rotT<2>(c1, s1, toF(cross2(wP, wP2, l)));
            }
        }
    } else if (CL == CL_SLIDER) {
        const D q0 = src.q(r.qo), u0 = MINV ? D(0) : src.u(r.uo);
        out.position(q0);
        if (ci) l.x = l.x + q0;
        else l = l + q0 * Vec{par[PR_C], par[PR_C + 3], par[PR_C + 6]};
        out.qdot(r.qo, u0);
        if (MINV) rec[RC_X] = src.fext(r.uo);
        else {
            rec[RC_X] = freely ? D(0) : mobForce(par, r.info, 0, q0, u0);
            w = wF;
            if (hasP) {
                gv = toF(cross2(wP, wP2, l));
                const D t = u0 + u0;
                gv.y = gv.y + t * wF.z;
                gv.z = gv.z - t * wF.y;
            }
            vrelL.x = u0;
        }
    } else if (CL == CL_UNIV) {
        const D q0 = src.q(r.qo), q1 = src.q(r.qo + 1);
        const D u0 = MINV ? D(0) : src.u(r.uo), u1 = MINV ? D(0) : src.u(r.uo + 1);
        sincos(q0, &s1, &c1);
        sincos(q1, &s2, &c2);
        rec[RC_E] = c1; rec[RC_E + 1] = s1; rec[RC_E + 2] = c2; rec[RC_E + 3] = s2;
        out.qdot(r.qo, u0);
        out.qdot(r.qo + 1, u1);
        if (MINV) { rec[RC_X] = src.fext(r.uo); rec[RC_X + 1] = src.fext(r.uo + 1); }
        else {
            rec[RC_X] = freely ? D(0) : mobForce(par, r.info, 0, q0, u0);
            rec[RC_X + 1] = freely ? D(0) : mobForce(par, r.info, 1, q1, u1);
            const Vec t = rotT<0>(c1, s1, wF);  // between the axes
            gw = Vec{-(t.z * u1), t.z * u0, (t.x * u1 - t.y * u0) + u0 * u1};
            if (hasP) gv = rotT<0>(c1, s1, toF(cross2(wP, wP2, l)));
            w = rotT<1>(c2, s2, Vec{t.x + u0, t.y + u1, t.z});
        }
    } else if (CL == CL_BALL || CL == CL_FREE) {
        D q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = src.q(r.qo + k);
        E = quatMatrix(q);
#pragma unroll
        for (int k = 0; k < 9; ++k) rec[RC_E + k] = E.a[k];
        Vec pf = zero(), uv = zero();
        if (CL == CL_FREE) {
            pf = Vec{src.q(r.qo + 4), src.q(r.qo + 5), src.q(r.qo + 6)};
            out.position(pf.x);
            out.position(pf.y);
            out.position(pf.z);
            l = l + (ci ? pf : mul(get9(par, PR_C), pf));
        }
        constexpr int n = CL == CL_FREE ? 6 : 3;
        if (MINV) {
#pragma unroll
            for (int k = 0; k < n; ++k) rec[RC_X + k] = src.fext(r.uo + k);
        } else {
            const Vec uw = Vec{src.u(r.uo), src.u(r.uo + 1), src.u(r.uo + 2)};
            if (CL == CL_FREE) uv = Vec{src.u(r.uo + 3), src.u(r.uo + 4), src.u(r.uo + 5)};
            // qdot = N(q) w with e = q/2 (Rotation.h:712-719, 990-992)
            const Vec hu = D(0.5) * uw;
            out.qdot(r.qo + 0, -q[1] * hu.x - q[2] * hu.y - q[3] * hu.z);
            out.qdot(r.qo + 1, q[0] * hu.x + q[3] * hu.y - q[2] * hu.z);
            out.qdot(r.qo + 2, -q[3] * hu.x + q[0] * hu.y + q[1] * hu.z);
            out.qdot(r.qo + 3, q[2] * hu.x - q[1] * hu.y + q[0] * hu.z);
            if (CL == CL_FREE) {
                out.qdot(r.qo + 4, uv.x);
                out.qdot(r.qo + 5, uv.y);
                out.qdot(r.qo + 6, uv.z);
            }
            const D uu[6] = {uw.x, uw.y, uw.z, uv.x, uv.y, uv.z};
            // a spring on mobility j reads q slot j, the quaternion's slots among them (Force.cpp:347-350)
            const D qq[6] = {q[0], q[1], q[2], q[3], pf.x, pf.y};
#pragma unroll
            for (int k = 0; k < n; ++k)
                rec[RC_X + k] = freely ? D(0) : mobForce(par, r.info, k, qq[k], uu[k]);
            w = mulT(E, wF + uw);
            if (hasP) {
                gw = mulT(E, cross(wF, uw));
                Vec t = toF(cross2(wP, wP2, l));
                if (CL == CL_FREE) t = t + cross(wF + wF, uv);
                gv = mulT(E, t);
            }
            if (md.pose) vrelL = mulT(E, uv);
        }
    } else {
        GenJoint j;
        pass1Gen<MINV>(r, par, rec, src, out, j);
        E = j.E;
        out.position(j.p.x);
        out.position(j.p.y);
        out.position(j.p.z);
#pragma unroll
        for (int k = 0; k < 9; ++k) rec[RC_E + k] = E.a[k];
        l = l + (ci ? j.p : mul(get9(par, PR_C), j.p));
        if (!MINV) {
            w = mulT(E, wF + j.wrel);
            gw = mulT(E, cross(wF, j.wrel) + j.hd);
            gv = mulT(E, toF(cross2(wP, wP2, l)) + cross(wF + wF, j.vrel));
            vrelL = mulT(E, j.vrel);
        }
    }
    put3(rec, RC_L, l);
    // own inertia about M's origin and velocity force
    const D m = par[PR_M];
    const Vec mc = get3(par, PR_MC);
    S3<D> J{par[PR_J], par[PR_J + 1], par[PR_J + 2], par[PR_J + 3], par[PR_J + 4], par[PR_J + 5]};
    Vec zw = zero(), zv = zero();
    if (!MINV) {
        const D w2 = dot(w, w);
        put3(rec, RC_W, w);
        rec[RC_W2] = w2;
        put3(rec, RC_GAM, gw);
        put3(rec, RC_GAM + 3, gv);
        zw = cross(w, mul(J, w));
        zv = cross2(w, w2, mc);
        if (md.pose) {
            // Ground pose, velocity of M's origin (M axes) and contacts
            M3<D> RP = ident3<D>();
            Vec pP = zero(), vP = zero();
            if (hasP) {
                RP = get9(recP, md.rs);
                pP = get3(recP, md.rs + 9);
                vP = get3(recP, md.rs + 12);
            }
            M3<D> EE;
            if (CL == CL_PIN) EE = M3<D>{{c1, -s1, 0, s1, c1, 0, 0, 0, 1}};
            else if (CL == CL_SLIDER) EE = ident3<D>();
            else if (CL == CL_UNIV)
                EE = M3<D>{{c2, 0, s2, s2 * s1, c1, -(s1 * c2), -(s2 * c1), s1, c1 * c2}};
            else EE = E;
            const M3<D> RL = ci ? EE : mul(get9(par, PR_C), EE);
            const M3<D> RG = mul(RP, RL);
            const Vec pG = pP + mul(RP, l);
            const Vec vL = mulT(RL, vP + cross(wP, l)) + vrelL;
#pragma unroll
            for (int k = 0; k < 9; ++k) rec[md.rs + k] = RG.a[k];
            put3(rec, md.rs + 9, pG);
            put3(rec, md.rs + 12, vL);
            if (r.kcnt > 0) {
                const ContactWrench W = contactWrench(md.kpar, r.kbeg, r.kcnt,
                                                      md.bodyPar + (int64_t)r.row * kParamStride, RG, pG, mul(RG, w),
                                                      mul(RG, vL));
                zw = zw - mulT(RG, W.w);
                zv = zv - mulT(RG, W.v);
            }
        }
    }
    rec[RC_J] = J.xx; rec[RC_J + 1] = J.yy; rec[RC_J + 2] = J.zz;
    rec[RC_J + 3] = J.xy; rec[RC_J + 4] = J.xz; rec[RC_J + 5] = J.yz;
    rec[RC_F] = 0; rec[RC_F + 1] = -mc.z; rec[RC_F + 2] = mc.y;
    rec[RC_F + 3] = mc.z; rec[RC_F + 4] = 0; rec[RC_F + 5] = -mc.x;
    rec[RC_F + 6] = -mc.y; rec[RC_F + 7] = mc.x; rec[RC_F + 8] = 0;
    rec[RC_M] = m; rec[RC_M + 1] = m; rec[RC_M + 2] = m;
    rec[RC_M + 3] = 0; rec[RC_M + 4] = 0; rec[RC_M + 5] = 0;
    put3(rec, RC_Z, zw);
    put3(rec, RC_Z + 3, zv);
}

// ------------------------------------------------------------------ pass 2
// Adds P+ (in F axes about the origin of M, rotated here by C) and z+ to the
// parent's record: P+ shifted by l, z+ by l.
template <class RC> TILE_FN void pushShift(const RC& recP, Vec l, const S3<D>& J, const M3<D>& F, const S3<D>& M, Vec zw, Vec zv) {
    const D x = l.x, y = l.y, z = l.z;
    const D* f = F.a;
    D g[9];
    g[0] = f[0] + (y * M.xz - z * M.xy);
    g[1] = f[1] + (y * M.yz - z * M.yy);
    g[2] = f[2] + (y * M.zz - z * M.yz);
    g[3] = f[3] + (z * M.xx - x * M.xz);
    g[4] = f[4] + (z * M.xy - x * M.yz);
    g[5] = f[5] + (z * M.xz - x * M.zz);
    g[6] = f[6] + (x * M.xy - y * M.xx);
    g[7] = f[7] + (x * M.yy - y * M.xy);
    g[8] = f[8] + (x * M.yz - y * M.xz);
    recP[RC_J + 0] = (recP[RC_J + 0] + J.xx) + y * (f[2] + g[2]) - z * (f[1] + g[1]);
    recP[RC_J + 1] = (recP[RC_J + 1] + J.yy) + z * (f[3] + g[3]) - x * (f[5] + g[5]);
    recP[RC_J + 2] = (recP[RC_J + 2] + J.zz) + x * (f[7] + g[7]) - y * (f[6] + g[6]);
    recP[RC_J + 3] = (recP[RC_J + 3] + J.xy) + z * (f[0] - g[4]) - x * f[2] + y * g[5];
    recP[RC_J + 4] = (recP[RC_J + 4] + J.xz) + x * f[1] - z * g[7] - y * (f[0] - g[8]);
    recP[RC_J + 5] = (recP[RC_J + 5] + J.yz) + x * (f[4] - g[8]) - y * f[3] + z * g[6];
#pragma unroll
    for (int k = 0; k < 9; ++k) recP[RC_F + k] = recP[RC_F + k] + g[k];
    recP[RC_M + 0] = recP[RC_M + 0] + M.xx;
    recP[RC_M + 1] = recP[RC_M + 1] + M.yy;
    recP[RC_M + 2] = recP[RC_M + 2] + M.zz;
    recP[RC_M + 3] = recP[RC_M + 3] + M.xy;
    recP[RC_M + 4] = recP[RC_M + 4] + M.xz;
    recP[RC_M + 5] = recP[RC_M + 5] + M.yz;
    put3(recP, RC_Z, (get3(recP, RC_Z) + zw) + cross(l, zv));
    put3(recP, RC_Z + 3, get3(recP, RC_Z + 3) + zv);
}
template <class PA, class RC> TILE_FN void pushFull(const SlotRow& r, const PA& par, const RC& recP, Vec l, const S3<D>& J, const M3<D>& F,
                      const S3<D>& M, Vec zw, Vec zv) {
    if (r.info & F_CI) {
        pushShift(recP, l, J, F, M, zw, zv);
    } else {
        const M3<D> C = get9(par, PR_C);
        pushShift(recP, l, reexpress(C, J), mulABt(mul(C, F), C), reexpress(C, M), mul(C, zw), mul(C, zv));
    }
}
// The same for P+ = (0, 0, M): what a rotational joint with three axes passes
// on. force: zw (the joint's own torque) is not zero.
template <class PA, class RC> TILE_FN void pushMass(const SlotRow& r, const PA& par, const RC& recP, Vec l, S3<D> M, Vec zw, bool force,
                                                   Vec zv) {
    if (!(r.info & F_CI)) {
        const M3<D> C = get9(par, PR_C);
        M = reexpress(C, M);
        if (force) zw = mul(C, zw);
        zv = mul(C, zv);
    }
    const D x = l.x, y = l.y, z = l.z;
    D g[9];
    g[0] = y * M.xz - z * M.xy;
    g[1] = y * M.yz - z * M.yy;
    g[2] = y * M.zz - z * M.yz;
    g[3] = z * M.xx - x * M.xz;
    g[4] = z * M.xy - x * M.yz;
    g[5] = z * M.xz - x * M.zz;
    g[6] = x * M.xy - y * M.xx;
    g[7] = x * M.yy - y * M.xy;
    g[8] = x * M.yz - y * M.xz;
    recP[RC_J + 0] = recP[RC_J + 0] + y * g[2] - z * g[1];
    recP[RC_J + 1] = recP[RC_J + 1] + z * g[3] - x * g[5];
    recP[RC_J + 2] = recP[RC_J + 2] + x * g[7] - y * g[6];
    recP[RC_J + 3] = recP[RC_J + 3] - z * g[4] + y * g[5];
    recP[RC_J + 4] = recP[RC_J + 4] - z * g[7] + y * g[8];
    recP[RC_J + 5] = recP[RC_J + 5] - x * g[8] + z * g[6];
#pragma unroll
    for (int k = 0; k < 9; ++k) recP[RC_F + k] = recP[RC_F + k] + g[k];
    recP[RC_M + 0] = recP[RC_M + 0] + M.xx;
    recP[RC_M + 1] = recP[RC_M + 1] + M.yy;
    recP[RC_M + 2] = recP[RC_M + 2] + M.zz;
    recP[RC_M + 3] = recP[RC_M + 3] + M.xy;
    recP[RC_M + 4] = recP[RC_M + 4] + M.xz;
    recP[RC_M + 5] = recP[RC_M + 5] + M.yz;
    Vec t = get3(recP, RC_Z) + cross(l, zv);
    if (force) t = t + zw;
    put3(recP, RC_Z, t);
    put3(recP, RC_Z + 3, get3(recP, RC_Z + 3) + zv);
}

// P - g (P h)^T for the unit rotation about AX, whose row and column become
// zero: g = P h / D without the AX entry (the two other angular ones in
// cyclic order, then the linear ones). Returns D.
template <int AX> TILE_FN D eliminate(S3<D>& J, M3<D>& F, S3<D>& M, Vec& zw, Vec& zv, D f, D g[5], D& e) {
    D p0, p1, d;  // P h, angular
    if (AX == 0) { d = J.xx; p0 = J.xy; p1 = J.xz; }
    else if (AX == 1) { d = J.yy; p0 = J.yz; p1 = J.xy; }
    else { d = J.zz; p0 = J.xz; p1 = J.yz; }
    constexpr int i = (AX + 1) % 3, k = (AX + 2) % 3;
    const D f0 = F.a[3 * AX], f1 = F.a[3 * AX + 1], f2 = F.a[3 * AX + 2];
    const D rd = D(1) / d;
    g[0] = p0 * rd; g[1] = p1 * rd; g[2] = f0 * rd; g[3] = f1 * rd; g[4] = f2 * rd;
    // the 2x2 angular block left over: (i,i), (i,k), (k,k)
    if (AX == 0) { J.yy -= g[0] * p0; J.yz -= g[0] * p1; J.zz -= g[1] * p1; J.xx = J.xy = J.xz = TILE_NIL; }
    else if (AX == 1) { J.zz -= g[0] * p0; J.xz -= g[0] * p1; J.xx -= g[1] * p1; J.yy = J.yz = J.xy = TILE_NIL; }
    else { J.xx -= g[0] * p0; J.xy -= g[0] * p1; J.yy -= g[1] * p1; J.zz = J.xz = J.yz = TILE_NIL; }
    F.a[3 * i] -= g[0] * f0; F.a[3 * i + 1] -= g[0] * f1; F.a[3 * i + 2] -= g[0] * f2;
    F.a[3 * k] -= g[1] * f0; F.a[3 * k + 1] -= g[1] * f1; F.a[3 * k + 2] -= g[1] * f2;
    F.a[3 * AX] = F.a[3 * AX + 1] = F.a[3 * AX + 2] = TILE_NIL;
    M.xx -= g[2] * f0; M.xy -= g[2] * f1; M.xz -= g[2] * f2;
    M.yy -= g[3] * f1; M.yz -= g[3] * f2; M.zz -= g[4] * f2;
    D* w = &zw.x;
    const D eps = f - w[AX];
    w[i] += g[0] * eps;
    w[k] += g[1] * eps;
    w[AX] = f;
    zv.x += g[2] * eps; zv.y += g[3] * eps; zv.z += g[4] * eps;
    e = eps * rd;
    return d;
}

template <int CL, bool MINV, class PA, class RC>
TILE_FN bool pass2(const SlotRow& r, const PA& par, const RC& rec, const RC& recP) {
    const bool hasP = r.parent >= 0;
    S3<D> J = get6(rec, RC_J), M = get6(rec, RC_M);
    M3<D> F = get9(rec, RC_F);
    Vec zw = get3(rec, RC_Z), zv = get3(rec, RC_Z + 3);
    const Vec l = get3(rec, RC_L);
    Vec gw = zero(), gv = zero();
    if (!MINV) {
        gw = get3(rec, RC_GAM);
        gv = get3(rec, RC_GAM + 3);
    }
    bool ok = true;
    if (CL == CL_PIN) {
        D g[5], e;
        ok = nonzero(eliminate<2>(J, F, M, zw, zv, rec[RC_X], g, e));
        rec[RC_X] = e;
#pragma unroll
        for (int k = 0; k < 5; ++k) rec[RC_X + 1 + k] = g[k];
        if (hasP) {
            if (!MINV) {  // + P+ gamma; the z row of J and F and gamma_w.z are zero
                zw.x += J.xx * gw.x + J.xy * gw.y + (F.a[0] * gv.x + F.a[1] * gv.y + F.a[2] * gv.z);
                zw.y += J.xy * gw.x + J.yy * gw.y + (F.a[3] * gv.x + F.a[4] * gv.y + F.a[5] * gv.z);
                zv = zv + mul(M, gv) + Vec{F.a[0] * gw.x + F.a[3] * gw.y, F.a[1] * gw.x + F.a[4] * gw.y, F.a[2] * gw.x + F.a[5] * gw.y};
            }
            const D c = rec[RC_E], s = rec[RC_E + 1];
            rotSym2<2>(c, s, J);
            rotMat<2>(c, s, F);
            rotSym<2>(c, s, M);
            pushFull(r, par, recP, l, J, F, M, rot<2>(c, s, zw), rot<2>(c, s, zv));
        }
    } else if (CL == CL_SLIDER) {
        const D d = M.xx, rd = D(1) / d;
        ok = nonzero(d);
        const D f0 = F.a[0], f1 = F.a[3], f2 = F.a[6];
        const D g0 = f0 * rd, g1 = f1 * rd, g2 = f2 * rd, g3 = M.xy * rd, g4 = M.xz * rd;
        const D eps = rec[RC_X] - zv.x;
        J.xx -= g0 * f0; J.xy -= g0 * f1; J.xz -= g0 * f2; J.yy -= g1 * f1; J.yz -= g1 * f2; J.zz -= g2 * f2;
        F.a[1] -= g0 * M.xy; F.a[2] -= g0 * M.xz;
        F.a[4] -= g1 * M.xy; F.a[5] -= g1 * M.xz;
        F.a[7] -= g2 * M.xy; F.a[8] -= g2 * M.xz;
        F.a[0] = F.a[3] = F.a[6] = TILE_NIL;
        M.yy -= g3 * M.xy; M.yz -= g3 * M.xz; M.zz -= g4 * M.xz;
        M.xx = M.xy = M.xz = TILE_NIL;
        zw = zw + Vec{g0 * eps, g1 * eps, g2 * eps};
        zv.y += g3 * eps;
        zv.z += g4 * eps;
        zv.x = rec[RC_X];
        rec[RC_X] = eps * rd;
        rec[RC_X + 1] = g0; rec[RC_X + 2] = g1; rec[RC_X + 3] = g2; rec[RC_X + 4] = g3; rec[RC_X + 5] = g4;
        if (hasP) {
            if (!MINV) {  // gamma_w = 0, and the x column of F and M
                zw = zw + Vec{F.a[1] * gv.y + F.a[2] * gv.z, F.a[4] * gv.y + F.a[5] * gv.z, F.a[7] * gv.y + F.a[8] * gv.z};
                zv.y += M.yy * gv.y + M.yz * gv.z;
                zv.z += M.yz * gv.y + M.zz * gv.z;
            }
            pushFull(r, par, recP, l, J, F, M, zw, zv);
        }
    } else if (CL == CL_UNIV) {
        const D c1 = rec[RC_E], s1 = rec[RC_E + 1], c2 = rec[RC_E + 2], s2 = rec[RC_E + 3];
        D g[5], e;
        ok = nonzero(eliminate<1>(J, F, M, zw, zv, rec[RC_X + 1], g, e));
        rec[RC_X + 1] = e;
#pragma unroll
        for (int k = 0; k < 5; ++k) rec[RC_X + 2 + k] = g[k];
        rotSym2<1>(c2, s2, J);
        rotMat<1>(c2, s2, F);
        rotSym<1>(c2, s2, M);
        zw = rot<1>(c2, s2, zw);
        zv = rot<1>(c2, s2, zv);
        // the x axis, between the two: the y rows of J and F are zero
        const D d = J.xx, p1 = J.xz, rd = D(1) / d;
        ok &= nonzero(d);
        const D f0 = F.a[0], f1 = F.a[1], f2 = F.a[2];
        const D g1 = p1 * rd, g2 = f0 * rd, g3 = f1 * rd, g4 = f2 * rd;
        const D eps = rec[RC_X] - zw.x;
        rec[RC_X + 7] = g1; rec[RC_X + 8] = g2; rec[RC_X + 9] = g3; rec[RC_X + 10] = g4;
        zw.x = rec[RC_X];
        rec[RC_X] = eps * rd;
        if (hasP) {
            const D jzz = J.zz - g1 * p1;
            D fz[3] = {F.a[6] - g1 * f0, F.a[7] - g1 * f1, F.a[8] - g1 * f2};
            M.xx -= g2 * f0; M.xy -= g2 * f1; M.xz -= g2 * f2;
            M.yy -= g3 * f1; M.yz -= g3 * f2; M.zz -= g4 * f2;
            zw.z += g1 * eps;
            zv = zv + Vec{g2 * eps, g3 * eps, g4 * eps};
            if (!MINV) {  // only (z, z) of J and the z row of F are left
                zw.z += jzz * gw.z + (fz[0] * gv.x + fz[1] * gv.y + fz[2] * gv.z);
                zv = zv + mul(M, gv) + gw.z * Vec{fz[0], fz[1], fz[2]};
            }
            const D t = s1 * jzz;
            J = S3<D>{TILE_NIL, s1 * t, c1 * (c1 * jzz), TILE_NIL, TILE_NIL, -(c1 * t)};
            const D h1 = c1 * fz[1] - s1 * fz[2], h2 = s1 * fz[1] + c1 * fz[2];
            F = M3<D>{{TILE_NIL, TILE_NIL, TILE_NIL, -(s1 * fz[0]), -(s1 * h1), -(s1 * h2), c1 * fz[0], c1 * h1, c1 * h2}};
            rotSym<0>(c1, s1, M);
            pushFull(r, par, recP, l, J, F, M, rot<0>(c1, s1, zw), rot<0>(c1, s1, zv));
        }
    } else if (CL == CL_BALL) {
        const M3<D> E = get9(rec, RC_E);
        const Vec f = get3(rec, RC_X);
        S3<D> Ji;
        ok = invSym(J, Ji);
        const bool freely = !MINV && (r.info & F_FREELY) != 0;
        const Vec e = freely ? mul(Ji, -zw) : mul(Ji, mulT(E, f) - zw);
        M3<D> Y;  // J^-1 F
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Y.a[k] = Ji.xx * F.a[k] + Ji.xy * F.a[3 + k] + Ji.xz * F.a[6 + k];
            Y.a[3 + k] = Ji.xy * F.a[k] + Ji.yy * F.a[3 + k] + Ji.yz * F.a[6 + k];
            Y.a[6 + k] = Ji.xz * F.a[k] + Ji.yz * F.a[3 + k] + Ji.zz * F.a[6 + k];
        }
        put3(rec, RC_X, e);
#pragma unroll
        for (int k = 0; k < 9; ++k) rec[RC_X + 3 + k] = Y.a[k];
        if (hasP) {
            M.xx -= F.a[0] * Y.a[0] + F.a[3] * Y.a[3] + F.a[6] * Y.a[6];
            M.xy -= F.a[0] * Y.a[1] + F.a[3] * Y.a[4] + F.a[6] * Y.a[7];
            M.xz -= F.a[0] * Y.a[2] + F.a[3] * Y.a[5] + F.a[6] * Y.a[8];
            M.yy -= F.a[1] * Y.a[1] + F.a[4] * Y.a[4] + F.a[7] * Y.a[7];
            M.yz -= F.a[1] * Y.a[2] + F.a[4] * Y.a[5] + F.a[7] * Y.a[8];
            M.zz -= F.a[2] * Y.a[2] + F.a[5] * Y.a[5] + F.a[8] * Y.a[8];
            zv = zv + mulT(F, e);
            if (!MINV) zv = zv + mul(M, gv);
            pushMass(r, par, recP, l, reexpress(E, M), f, !freely, mul(E, zv));
        }
    } else if (CL == CL_FREE) {
        // P+ = 0: the body's acceleration follows from its own balance
        const M3<D> E = get9(rec, RC_E);
        const Vec fw = get3(rec, RC_X), fv = get3(rec, RC_X + 3);
        const Vec rw = mulT(E, fw) - zw, rv = mulT(E, fv) - zv;
        S3<D> Ji, Si;
        ok = invSym(J, Ji);
        M3<D> Y;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Y.a[k] = Ji.xx * F.a[k] + Ji.xy * F.a[3 + k] + Ji.xz * F.a[6 + k];
            Y.a[3 + k] = Ji.xy * F.a[k] + Ji.yy * F.a[3 + k] + Ji.yz * F.a[6 + k];
            Y.a[6 + k] = Ji.xz * F.a[k] + Ji.yz * F.a[3 + k] + Ji.zz * F.a[6 + k];
        }
        M.xx -= F.a[0] * Y.a[0] + F.a[3] * Y.a[3] + F.a[6] * Y.a[6];
        M.xy -= F.a[0] * Y.a[1] + F.a[3] * Y.a[4] + F.a[6] * Y.a[7];
        M.xz -= F.a[0] * Y.a[2] + F.a[3] * Y.a[5] + F.a[6] * Y.a[8];
        M.yy -= F.a[1] * Y.a[1] + F.a[4] * Y.a[4] + F.a[7] * Y.a[7];
        M.yz -= F.a[1] * Y.a[2] + F.a[4] * Y.a[5] + F.a[7] * Y.a[8];
        M.zz -= F.a[2] * Y.a[2] + F.a[5] * Y.a[5] + F.a[8] * Y.a[8];
        ok &= invSym(M, Si);
        const Vec e = mul(Ji, rw);
        const Vec a = mul(Si, rv - mulT(F, e));
        put3(rec, RC_X, e - mul(Y, a));
        put3(rec, RC_X + 3, a);
        if (hasP) {
            const S3<D> none{0, 0, 0, 0, 0, 0};
            pushMass(r, par, recP, l, none, fw, true, fv);
        }
    } else {
        // one column after another, the outermost last: a joint of n mobilities
        // is n joints of one with massless bodies between them
        const int n = (r.info >> 4) & 15;
        AB<D> P;
        P.J = J; P.F = F; P.M = M;
        for (int j = n - 1; j >= 0; --j) {
            const Vec hw = get3(rec, RC_H + 6 * j), hv = get3(rec, RC_H + 6 * j + 3);
            Vec pw, pv;
            abmul(P, hw, hv, pw, pv);
            const D d = dot(hw, pw) + dot(hv, pv), rd = D(1) / d;
            ok &= nonzero(d);
            const Vec ow = rd * pw, ov = rd * pv;
            const D eps = rec[RC_X + j] - (dot(hw, zw) + dot(hv, zv));
            P.J.xx -= ow.x * pw.x; P.J.xy -= ow.x * pw.y; P.J.xz -= ow.x * pw.z;
            P.J.yy -= ow.y * pw.y; P.J.yz -= ow.y * pw.z; P.J.zz -= ow.z * pw.z;
            P.M.xx -= ov.x * pv.x; P.M.xy -= ov.x * pv.y; P.M.xz -= ov.x * pv.z;
            P.M.yy -= ov.y * pv.y; P.M.yz -= ov.y * pv.z; P.M.zz -= ov.z * pv.z;
            P.F.a[0] -= ow.x * pv.x; P.F.a[1] -= ow.x * pv.y; P.F.a[2] -= ow.x * pv.z;
            P.F.a[3] -= ow.y * pv.x; P.F.a[4] -= ow.y * pv.y; P.F.a[5] -= ow.y * pv.z;
            P.F.a[6] -= ow.z * pv.x; P.F.a[7] -= ow.z * pv.y; P.F.a[8] -= ow.z * pv.z;
            zw = axpy(zw, eps, ow);
            zv = axpy(zv, eps, ov);
            rec[RC_X + j] = eps * rd;
            put3(rec, RC_G + 6 * j, ow);
            put3(rec, RC_G + 6 * j + 3, ov);
        }
        if (hasP) {
            if (!MINV) {
                Vec pw, pv;
                abmul(P, gw, gv, pw, pv);
                zw = zw + pw;
                zv = zv + pv;
            }
            const M3<D> E = get9(rec, RC_E);
            pushFull(r, par, recP, l, reexpress(E, P.J), mulABt(mul(E, P.F), E), reexpress(E, P.M), mul(E, zw),
                     mul(E, zv));
        }
    }
    return ok;
}

// ------------------------------------------------------------------ pass 3
// Base to tip: udot and the body's acceleration.
template <int CL, bool MINV, class PA, class RC, class Out>
TILE_FN void pass3(const Model& md, const SlotRow& r, const PA& par, const RC& rec, const RC& recP, Out& out) {
    const bool ci = (r.info & F_CI) != 0;
    Vec aw = zero(), av = MINV ? zero() : -md.g;
    if (r.parent >= 0) {
        aw = get3(recP, RC_W);
        av = get3(recP, RC_W + 3) + cross(aw, get3(rec, RC_L));
    }
    if (!ci) {
        const M3<D> C = get9(par, PR_C);
        aw = mulT(C, aw);
        av = mulT(C, av);
    }
    Vec gw = zero(), gv = zero();
    if (!MINV) {
        gw = get3(rec, RC_GAM);
        gv = get3(rec, RC_GAM + 3);
    }
    if (CL == CL_PIN) {
        const D c = rec[RC_E], s = rec[RC_E + 1];
        aw = rotT<2>(c, s, aw);
        av = rotT<2>(c, s, av) + gv;
        aw.x += gw.x;
        aw.y += gw.y;
        const D ud = rec[RC_X] - (aw.z + rec[RC_X + 1] * aw.x + rec[RC_X + 2] * aw.y + rec[RC_X + 3] * av.x +
                                  rec[RC_X + 4] * av.y + rec[RC_X + 5] * av.z);
        out.udot(r.uo, ud);
        aw.z += ud;
    } else if (CL == CL_SLIDER) {
        av = av + gv;
        const D ud = rec[RC_X] - (av.x + rec[RC_X + 1] * aw.x + rec[RC_X + 2] * aw.y + rec[RC_X + 3] * aw.z +
                                  rec[RC_X + 4] * av.y + rec[RC_X + 5] * av.z);
        out.udot(r.uo, ud);
        av.x += ud;
    } else if (CL == CL_UNIV) {
        const D c1 = rec[RC_E], s1 = rec[RC_E + 1], c2 = rec[RC_E + 2], s2 = rec[RC_E + 3];
        aw = rotT<0>(c1, s1, aw) + gw;
        av = rotT<0>(c1, s1, av) + gv;
        const D u0 = rec[RC_X] - (aw.x + rec[RC_X + 7] * aw.z + rec[RC_X + 8] * av.x + rec[RC_X + 9] * av.y +
                                  rec[RC_X + 10] * av.z);
        out.udot(r.uo, u0);
        aw.x += u0;
        aw = rotT<1>(c2, s2, aw);
        av = rotT<1>(c2, s2, av);
        const D u1 = rec[RC_X + 1] - (aw.y + rec[RC_X + 2] * aw.z + rec[RC_X + 3] * aw.x + rec[RC_X + 4] * av.x +
                                      rec[RC_X + 5] * av.y + rec[RC_X + 6] * av.z);
        out.udot(r.uo + 1, u1);
        aw.y += u1;
    } else if (CL == CL_BALL || CL == CL_FREE) {
        const M3<D> E = get9(rec, RC_E);
        const Vec a0w = mulT(E, aw) + gw, a0v = mulT(E, av) + gv;
        if (CL == CL_BALL) {
            aw = get3(rec, RC_X) - mul(get9(rec, RC_X + 3), a0v);
            av = a0v;
        } else {
            aw = get3(rec, RC_X);
            av = get3(rec, RC_X + 3);
        }
        const Vec x = mul(E, aw - a0w);
        out.udot(r.uo, x.x);
        out.udot(r.uo + 1, x.y);
        out.udot(r.uo + 2, x.z);
        if (CL == CL_FREE) {
            const Vec t = mul(E, av - a0v);
            out.udot(r.uo + 3, t.x);
            out.udot(r.uo + 4, t.y);
            out.udot(r.uo + 5, t.z);
        }
    } else {
        const M3<D> E = get9(rec, RC_E);
        aw = mulT(E, aw) + gw;
        av = mulT(E, av) + gv;
        const int n = (r.info >> 4) & 15;
        for (int j = 0; j < n; ++j) {
            const D ud = rec[RC_X + j] - (dot(get3(rec, RC_G + 6 * j), aw) + dot(get3(rec, RC_G + 6 * j + 3), av));
            out.udot(r.uo + j, ud);
            aw = axpy(aw, ud, get3(rec, RC_H + 6 * j));
            av = axpy(av, ud, get3(rec, RC_H + 6 * j + 3));
        }
    }
    put3(rec, RC_W, aw);
    put3(rec, RC_W + 3, av);
}

}  // namespace tile
}  // namespace sbg
