// Solver rows of one contact point (SequentialImpulseConstraintSolver.java:418-786), shared by the solver's
// kernels.
#pragma once
#include "jbgpu_internal.cuh"

namespace jbg {
using namespace jbd;

struct BodyV { V lin, ang, com; float im; M iw; };

JBD BodyV load_body(const DevWorld& w, int b) {
    BodyV r;
    r.lin = mk4(w.linvel[b]);
    r.ang = mk4(w.angvel[b]);
    r.com = mk(w.xr0[b].w, w.xr1[b].w, w.xr2[b].w);
    r.im = w.iloc[b].w;
    r.iw = load_iw(w, b);
    return r;
}

// The rows of a point as 15 float4 planes: the normal row's contactNormal | jacDiagABInv,
// relpos1CrossNormal | positional error, relpos2CrossNormal | restitution, angularComponentA |
// friction, angularComponentB | appliedImpulse, then per friction row its direction |
// jacDiagABInv, relpos1CrossNormal | appliedImpulse, relpos2CrossNormal, angularComponentA,
// angularComponentB.
constexpr int ROW_PLANES = 15;
enum { RP_N = 0, RP_N1, RP_N2, RP_NA, RP_NB, RP_F = 5 };

template <class E>
JBD void friction_planes(E&& emit, int plane, V dir, V rp1, V rp2, const BodyV& A, const BodyV& B, float impulse) {
    V t1 = crs(rp1, dir), t2 = crs(rp2, dir);
    V angA = mulMv(t1, A.iw), angB = mulMv(t2, B.iw);
    float d0 = __fadd_rn(A.im, dot(dir, crs(angA, rp1)));
    float d1 = __fadd_rn(B.im, dot(dir, crs(angB, rp2)));
    float jac = jdiv(1.0f, __fadd_rn(d0, d1));
    emit(plane + 0, f4(dir, jac));
    emit(plane + 1, f4(t1, impulse));
    emit(plane + 2, f4(t2, 0.0f));
    emit(plane + 3, f4(angA, 0.0f));
    emit(plane + 4, f4(angB, 0.0f));
}

// The rows of manifold point k (an index into the point arrays of P), handed to emit(plane, value);
// a point without friction directions gets them here (solveGroupCacheFriendlySetup, java:600-760).
template <class E>
JBD void point_rows(const DevWorld& w, const DevPairs& P, int k, const BodyV& A, const BodyV& B, bool warm, float dt,
                    E&& emit) {
    float4 pa = P.pA[k];
    float dist = pa.w;
    float4 wa = P.wA[k], wb = P.wB[k], nr = P.nrm[k], im = P.imp[k];
    V nrm = mk(nr.x, nr.y, nr.z);
    V rp1 = sub(mk(wa.x, wa.y, wa.z), A.com), rp2 = sub(mk(wb.x, wb.y, wb.z), B.com);
    V angA = mulMv(crs(rp1, nrm), A.iw);
    V angB = mulMv(crs(rp2, nrm), B.iw);
    float d0 = __fadd_rn(A.im, dot(nrm, crs(angA, rp1)));
    float d1 = __fadd_rn(B.im, dot(nrm, crs(angB, rp2)));
    float jac = jdiv(1.0f, __fadd_rn(d0, d1));
    V rp1xn = crs(rp1, nrm), rp2xn = crs(rp2, nrm);
    V vel1 = add(crs(A.ang, rp1), A.lin);
    V vel2 = add(crs(B.ang, rp2), B.lin);
    V vel = sub(vel1, vel2);
    float rel_vel = dot(nrm, vel);
    float pen = jmin(__fadd_rn(dist, w.slop), 0.0f);
    float rest = __fmul_rn(wb.w, -rel_vel);
    if (rest <= 0.0f) rest = 0.0f;
    float penVel = jdiv(-pen, dt);
    if (rest > penVel) pen = 0.0f;
    float imp = warm ? __fmul_rn(nr.w, w.warm) : 0.0f;
    emit(RP_N, f4(nrm, jac));
    emit(RP_N1, f4(rp1xn, jdiv(__fmul_rn(-pen, w.erp), dt)));   // positionalError (java:248)
    emit(RP_N2, f4(rp2xn, rest));
    emit(RP_NA, f4(angA, wa.w));                                // friction coefficient
    emit(RP_NB, f4(angB, imp));
    V dir1, dir2;
    if (im.z == 0.0f) {
        dir1 = sub(vel, scl(nrm, rel_vel));
        float lat = len2(dir1);
        if (lat > FLT_EPS) {
            dir1 = scl(dir1, jdiv(1.0f, jsqrt(lat)));
            dir2 = nor(crs(dir1, nrm));
        } else {
            plane_space1(nrm, dir1, dir2);
        }
        P.d1[k] = f4(dir1, 0.0f);
        P.d2[k] = f4(dir2, 0.0f);
        P.imp[k] = make_float4(im.x, im.y, 1.0f, 0.0f);
    } else {
        dir1 = mk4(P.d1[k]);
        dir2 = mk4(P.d2[k]);
    }
    friction_planes(emit, RP_F, dir1, rp1, rp2, A, B, warm ? __fmul_rn(im.x, w.warm) : 0.0f);
    friction_planes(emit, RP_F + 5, dir2, rp1, rp2, A, B, warm ? __fmul_rn(im.y, w.warm) : 0.0f);
}

JBD void apply_imp(V& lin, V& ang, V n, float im, V angc, float imp) {   // SolverBody.internalApplyImpulse
    if (im != 0.0f) {
        V lc = scl(n, im);
        lin.x = __fadd_rn(lin.x, __fmul_rn(imp, lc.x));
        lin.y = __fadd_rn(lin.y, __fmul_rn(imp, lc.y));
        lin.z = __fadd_rn(lin.z, __fmul_rn(imp, lc.z));
        ang.x = __fadd_rn(ang.x, __fmul_rn(imp, angc.x));
        ang.y = __fadd_rn(ang.y, __fmul_rn(imp, angc.y));
        ang.z = __fadd_rn(ang.z, __fmul_rn(imp, angc.z));
    }
}

enum { PH_WARM = 0, PH_NORMAL = 1, PH_FRICTION = 2 };

}  // namespace jbg
