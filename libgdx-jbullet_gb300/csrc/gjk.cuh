// GJK closest points (collision/narrowphase/GjkPairDetector.java:73-316) with the Voronoi
// sub-simplex solver (collision/narrowphase/VoronoiSimplexSolver.java) on the device, one
// thread per convex pair.  The penetration fallback (GjkEpaSolver) lives in epa.cuh and
// runs in a second kernel over the pairs that need it.
#pragma once
#include "shapes.cuh"

namespace jbg {
using namespace jbd;

// The sub-simplex solver.  What bounds it is instruction issue with few lanes active: the warp runs
// every region of every face some lane is in, and its code does not stay in the instruction cache
// when each face has a copy.  So the vertices are in registers (selects by the vertex count, no
// indexed arrays), a vertex's difference W = P - Q is formed again instead of kept, the triangle's
// regions are chosen by selects around one division, and the tetrahedron's faces and the triangle
// run through one copy of it in a loop over the faces a lane needs.
// k_narrow at 600,000 pairs of 100,000 mixed bodies 558 -> 475 us, 0.8 million ray casts 2.75 -> 1.35 ms
// against indexed arrays in local memory and a copy of the code per face.
struct Simplex {
    int nv;
    V P[4], Q[4];
    V cP1, cP2, cV, lastW;
    bool valid, needsUpdate;
};

JBD void sx_reset(Simplex& s) {
    s.valid = false;
    s.nv = 0;
    s.needsUpdate = true;
    s.lastW = mk(1e30f, 1e30f, 1e30f);
    s.cP1 = s.cP2 = s.cV = mk(0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 4; i++) s.P[i] = s.Q[i] = mk(0.0f, 0.0f, 0.0f);
}
JBD V vsel(bool c, V a, V b) { return mk(c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z); }
JBD V sx_w(const Simplex& s, int i) { return sub(s.P[i], s.Q[i]); }
// addVertex (w == p - q); a simplex of four has ended the caller's loop
JBD void sx_add(Simplex& s, V w, V p, V q) {
    s.lastW = w;
    s.needsUpdate = true;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        s.P[i] = vsel(s.nv == i, p, s.P[i]);
        s.Q[i] = vsel(s.nv == i, q, s.Q[i]);
    }
    s.nv++;
}
// reduceVertices: an unused vertex gives its place to the last one.
JBD void sx_reduce(Simplex& s, int used) {
#pragma unroll
    for (int i = 3; i >= 0; i--) {
        const bool drop = s.nv > i && !(used & (1 << i));
        s.nv -= drop ? 1 : 0;
#pragma unroll
        for (int k = i + 1; k < 4; k++) {
            s.P[i] = vsel(drop && s.nv == k, s.P[k], s.P[i]);
            s.Q[i] = vsel(drop && s.nv == k, s.Q[k], s.Q[i]);
        }
    }
}
JBD bool sx_in(const Simplex& s, V w) {
    bool found = vequals(w, s.lastW);
#pragma unroll
    for (int i = 0; i < 4; i++) found = found || (i < s.nv && vequals(sx_w(s, i), w));
    return found;
}

// VoronoiSimplexSolver.closestPtPointTriangle (java:267-370) for the origin: the barycentric
// coordinates, the vertices used (bits 0 to 2) and the squared length of the closest point.
struct TriPoint {
    int used;
    float b0, b1, b2, sq;
};
JBD TriPoint closest_pt_triangle(V a, V b, V c) {
    const V p = mk(0.0f, 0.0f, 0.0f);
    const V ab = sub(b, a), ac = sub(c, a), ap = sub(p, a), bp = sub(p, b), cp = sub(p, c);
    const float d1 = dot(ab, ap), d2 = dot(ac, ap), d3 = dot(ab, bp), d4 = dot(ac, bp), d5 = dot(ab, cp), d6 = dot(ac, cp);
    const float vc = __fsub_rn(__fmul_rn(d1, d4), __fmul_rn(d3, d2));
    const float vb = __fsub_rn(__fmul_rn(d5, d2), __fmul_rn(d1, d6));
    const float va = __fsub_rn(__fmul_rn(d3, d6), __fmul_rn(d5, d4));
    const float d43 = __fsub_rn(d4, d3), d56 = __fsub_rn(d5, d6);
    const bool inA = d1 <= 0.0f && d2 <= 0.0f;
    const bool inB = !inA && d3 >= 0.0f && d4 <= d3;
    const bool onAB = !inA && !inB && vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f;
    const bool ab3 = inA || inB || onAB;
    const bool inC = !ab3 && d6 >= 0.0f && d5 <= d6;
    const bool onAC = !ab3 && !inC && vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f;
    const bool onBC = !ab3 && !inC && !onAC && va <= 0.0f && d43 >= 0.0f && d56 >= 0.0f;
    const bool vertex = inA || inB || inC, edge = onAB || onAC || onBC;
    const float num = vertex ? 0.0f : onAB ? d1 : onAC ? d2 : onBC ? d43 : 1.0f;
    const float den = vertex ? 1.0f : onAB ? __fsub_rn(d1, d3) : onAC ? __fsub_rn(d2, d6) : onBC ? __fadd_rn(d43, d56)
                                    : __fadd_rn(__fadd_rn(va, vb), vc);
    const float q = jdiv(num, den);
    const float v = __fmul_rn(vb, q), u = __fmul_rn(vc, q), rest = __fsub_rn(1.0f, q);
    TriPoint r;
    r.used = inA ? 1 : inB ? 2 : inC ? 4 : onAB ? 3 : onAC ? 5 : onBC ? 6 : 7;
    r.b0 = inA ? 1.0f : inB || inC || onBC ? 0.0f : edge ? rest : __fsub_rn(__fsub_rn(1.0f, v), u);
    r.b1 = inB ? 1.0f : inA || inC || onAC ? 0.0f : onAB ? q : onBC ? rest : v;
    r.b2 = inC ? 1.0f : inA || inB || onAB ? 0.0f : edge ? q : u;
    const V base = vsel(inB || onBC, b, vsel(inC, c, a));
    const V along = vsel(onAC, ac, vsel(onBC, sub(c, b), ab));
    V t = add(base, scl(along, edge ? q : v));
    t = vsel(vertex, base, t);
    t = vsel(vertex || edge, t, add(t, scl(ac, u)));
    r.sq = dot(t, t);
    return r;
}

// VoronoiSimplexSolver.pointOutsideOfPlane (java:373-403) for the origin
JBD int origin_outside_plane(V a, V b, V c, V d) {
    V normal = crs(sub(b, a), sub(c, a));
    float signp = dot(sub(mk(0.0f, 0.0f, 0.0f), a), normal);
    float signd = dot(sub(d, a), normal);
    if (__fmul_rn(signd, signd) < __fmul_rn(1e-4f, 1e-4f)) return -1;
    return (__fmul_rn(signp, signd) < 0.0f) ? 1 : 0;
}

JBD V wsum3(V a, float x, V b, float y, V c, float z) {
    V t1 = scl(a, x), t2 = scl(b, y), t3 = scl(c, z);
    return mk(__fadd_rn(__fadd_rn(t1.x, t2.x), t3.x), __fadd_rn(__fadd_rn(t1.y, t2.y), t3.y), __fadd_rn(__fadd_rn(t1.z, t2.z), t3.z));
}

// VoronoiSimplexSolver.updateClosestVectorAndPoints (java:98-265), closestPtPointTetrahedron
// (java:405-535): the tetrahedron's faces in the order ABC, ACD, ADB, BDC.
JBD bool sx_update(Simplex& s) {
    if (!s.needsUpdate) return s.valid;
    s.needsUpdate = false;
    if (s.nv == 0) {
        s.valid = false;
    } else if (s.nv == 1) {
        s.cP1 = s.P[0];
        s.cP2 = s.Q[0];
        s.cV = sub(s.cP1, s.cP2);
        s.valid = true;
    } else if (s.nv == 2) {
        const V from = sx_w(s, 0);
        const V diff = sub(mk(0.0f, 0.0f, 0.0f), from);
        const V v = sub(sx_w(s, 1), from);
        float t = dot(v, diff);
        int used = 1;
        if (t > 0.0f) {
            const float dotVV = dot(v, v);
            used = t < dotVV ? 3 : 2;
            t = t < dotVV ? jdiv(t, dotVV) : 1.0f;
        } else {
            t = 0.0f;
        }
        s.cP1 = add(s.P[0], scl(sub(s.P[1], s.P[0]), t));
        s.cP2 = add(s.Q[0], scl(sub(s.Q[1], s.Q[0]), t));
        s.cV = sub(s.cP1, s.cP2);
        s.valid = __fsub_rn(1.0f, t) >= 0.0f && t >= 0.0f;
        sx_reduce(s, used);
    } else {
        const V A = sx_w(s, 0), B = sx_w(s, 1), C = sx_w(s, 2), D = sx_w(s, 3);
        const bool tetra = s.nv == 4;
        int todo = 1;   // faces to look at
        if (tetra) {
            const int o0 = origin_outside_plane(A, B, C, D), o1 = origin_outside_plane(A, C, D, B);
            const int o2 = origin_outside_plane(A, D, B, C), o3 = origin_outside_plane(B, D, C, A);
            if (o0 < 0 || o1 < 0 || o2 < 0 || o3 < 0) {   // degenerate
                s.valid = false;
                return false;
            }
            todo = o0 | (o1 << 1) | (o2 << 2) | (o3 << 3);
            if (todo == 0) {                              // the origin is inside
                s.cV = mk(0.0f, 0.0f, 0.0f);
                s.valid = true;
                return true;
            }
        }
        float best = 3.40282347e+38f;
        float b0 = 0.0f, b1 = 0.0f, b2 = 0.0f, b3 = 0.0f;
        int used = 15;
        while (todo) {
            const int f = __ffs(todo) - 1;
            todo &= todo - 1;
            const TriPoint t = closest_pt_triangle(vsel(f == 3, B, A), vsel(f == 0, B, vsel(f == 1, C, D)),
                                                   vsel(f == 1, D, vsel(f == 2, B, C)));
            if (!tetra || t.sq < best) {
                best = t.sq;
                b0 = f == 3 ? 0.0f : t.b0;
                b1 = f == 0 ? t.b1 : f == 1 ? 0.0f : f == 2 ? t.b2 : t.b0;
                b2 = f == 0 ? t.b2 : f == 1 ? t.b1 : f == 2 ? 0.0f : t.b2;
                b3 = f == 0 ? 0.0f : f == 1 ? t.b2 : t.b1;
                const int u0 = t.used & 1, u1 = (t.used >> 1) & 1, u2 = t.used >> 2;
                used = f == 0 ? t.used : f == 1 ? (u0 | (u1 << 2) | (u2 << 3)) : f == 2 ? (u0 | (u2 << 1) | (u1 << 3))
                                                                                        : ((u0 << 1) | (u2 << 2) | (u1 << 3));
            }
        }
        const V p3 = wsum3(s.P[0], b0, s.P[1], b1, s.P[2], b2), q3 = wsum3(s.Q[0], b0, s.Q[1], b1, s.Q[2], b2);
        s.cP1 = vsel(tetra, add(p3, scl(s.P[3], b3)), p3);
        s.cP2 = vsel(tetra, add(q3, scl(s.Q[3], b3)), q3);
        s.cV = sub(s.cP1, s.cP2);
        s.valid = b0 >= 0.0f && b1 >= 0.0f && b2 >= 0.0f && b3 >= 0.0f;
        sx_reduce(s, used);
    }
    return s.valid;
}

// Result of the GJK part of GjkPairDetector.getClosestPoints, before the EPA fallback.
struct GjkPart {
    bool isValid;
    bool needEpa;    // checkPenetration && (!isValid || catchDegeneratePenetrationCase)
    float distance;
    V pointOnA, pointOnB, normalInB;
    V offset;        // positionOffset
};

// support_without_margin with a hull's vertex scan split across the G lanes of a pair (gl: lane in
// the group, gmask: the group's lanes): each lane keeps the first strictly larger dot of its
// vertices, the group then the larger dot and, on equal dots, the lower vertex - the vertex the
// scan in order selects.
template <int G>
JBD V support_lanes(const ShapeRef& s, V vec, int gl, unsigned gmask) {
    if (G == 1 || s.type != SHAPE_HULL) return support_without_margin(s, vec);
    const V v = normalize_dir(vec);
    float maxDot = -1e30f;
    int idx = 0x7fffffff;
    for (int i = gl; i < s.npts; i += G) {
        const float4 p = s.pts[i];
        const float nd = dot(v, mk(p.x, p.y, p.z));
        if (nd > maxDot) { maxDot = nd; idx = i; }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        const float od = __shfl_xor_sync(gmask, maxDot, o);
        const int oi = __shfl_xor_sync(gmask, idx, o);
        if (od > maxDot || (od == maxDot && oi < idx)) { maxDot = od; idx = oi; }
    }
    if (idx == 0x7fffffff) return mk(0.0f, 0.0f, 0.0f);
    const float4 p = s.pts[idx];
    return mk(p.x, p.y, p.z);
}

// GjkPairDetector.getClosestPoints up to the penetration fallback (java:73-257), a step of its loop
// at a time.  lA, lB: the transforms with the middle of their origins taken off.
struct GjkRun {
    float sqd;
    int curIter, degenerate;
    bool check, penetration;
    Simplex s;   // its cV is the separating direction
};
JBD void gjk_begin(GjkRun& r) {
    r.sqd = SIMD_INFINITY;
    r.curIter = r.degenerate = 0;
    r.check = false;
    r.penetration = true;
    sx_reset(r.s);
    r.s.cV = mk(0.0f, 1.0f, 0.0f);
}
template <int G>
JBD bool gjk_step(GjkRun& r, const ShapeRef& sa, const Xf& lA, const ShapeRef& sb, const Xf& lB, float maxDist2, int gl,
                  unsigned gmask) {   // true: the loop has ended
    const float REL_ERROR2 = 1.0e-6f;
    const V pW = xf_apply(lA, support_lanes<G>(sa, mulMTv(scl(r.s.cV, -1.0f), lA.b), gl, gmask));
    const V qW = xf_apply(lB, support_lanes<G>(sb, mulMTv(r.s.cV, lB.b), gl, gmask));
    const V w = sub(pW, qW);
    const float delta = dot(r.s.cV, w);
    if ((delta > 0.0f) && (__fmul_rn(delta, delta) > __fmul_rn(r.sqd, maxDist2))) { r.penetration = false; return true; }
    if (sx_in(r.s, w)) { r.degenerate = 1; r.check = true; return true; }
    const float f0 = __fsub_rn(r.sqd, delta);
    const float f1 = __fmul_rn(r.sqd, REL_ERROR2);
    if (f0 <= f1) { if (f0 <= 0.0f) r.degenerate = 2; r.check = true; return true; }
    sx_add(r.s, w, pW, qW);
    const bool ok = sx_update(r.s);                  // closest(v)
    if (!ok) { r.degenerate = 3; r.check = true; return true; }
    if (len2(r.s.cV) < REL_ERROR2) { r.degenerate = 6; r.check = true; return true; }
    const float previous = r.sqd;
    r.sqd = len2(r.s.cV);
    if (__fsub_rn(previous, r.sqd) <= __fmul_rn(FLT_EPS, previous)) { r.check = true; return true; }
    if (r.curIter++ > 1000) return true;
    return r.s.nv == 4;
}
JBD GjkPart gjk_end(GjkRun& g, float marginA, float marginB, V offset) {
    GjkPart r;
    r.distance = 0.0f;
    r.normalInB = mk(0.0f, 0.0f, 0.0f);
    r.pointOnA = r.pointOnB = mk(0.0f, 0.0f, 0.0f);
    r.offset = offset;
    const float margin = __fadd_rn(marginA, marginB);
    bool isValid = false;
    if (g.check) {
        sx_update(g.s);                              // compute_points
        r.pointOnA = g.s.cP1;
        r.pointOnB = g.s.cP2;
        r.normalInB = sub(r.pointOnA, r.pointOnB);
        float lenSqr = len2(g.s.cV);
        if (lenSqr < 0.0001f) g.degenerate = 5;
        if (lenSqr > __fmul_rn(FLT_EPS, FLT_EPS)) {
            float rlen = jdiv(1.0f, jsqrt(lenSqr));
            r.normalInB = scl(r.normalInB, rlen);
            float sq = jsqrt(g.sqd);
            r.pointOnA = sub(r.pointOnA, scl(g.s.cV, jdiv(marginA, sq)));
            r.pointOnB = add(r.pointOnB, scl(g.s.cV, jdiv(marginB, sq)));
            r.distance = __fsub_rn(jdiv(1.0f, rlen), margin);
            isValid = true;
        }
    }
    bool catchDegen = (g.degenerate != 0 && (__fadd_rn(r.distance, margin) < 0.01f));
    r.isValid = isValid;
    r.needEpa = g.penetration && (!isValid || catchDegen);
    return r;
}
template <int G = 1>
JBD GjkPart gjk_part(const ShapeRef& sa, const Xf& tA, const ShapeRef& sb, const Xf& tB, float maxDist2, int gl = 0,
                     unsigned gmask = 0u, int* steps = nullptr) {
    const V offset = scl(add(tA.o, tB.o), 0.5f);
    Xf lA = tA, lB = tB;
    lA.o = sub(lA.o, offset);
    lB.o = sub(lB.o, offset);
    GjkRun r;
    gjk_begin(r);
    int n = 1;
    while (!gjk_step<G>(r, sa, lA, sb, lB, maxDist2, gl, gmask)) n++;
    if (steps) *steps = n;
    return gjk_end(r, sa.margin, sb.margin, offset);
}

}  // namespace jbg
