// The flow solver: the contact rows' warm start and Gauss-Seidel iterations as a dataflow between
// the bodies' velocities, for solves with a fixed number of iterations and no joints.
//
// Gauss-Seidel gives the same floats for any schedule in which the manifolds of each dynamic body
// are solved in the same order.  That order is the colouring's (solver.cu): within a phase (warm
// start, then normal rows and friction rows per iteration) a body's manifolds follow by local
// colour, then by cut colour - its links (prevLink, nextLink).  Every velocity carries a tag, the
// phase and colour of the manifold that wrote it; the next manifold of the body waits for exactly
// that tag, so no barrier stands between colours, and a row waits only for the rows it reads.
//
// What bounds it: the chain of manifolds through one body, colours x phases long, each link a
// handful of dependent binary32 operations per row.  So the links are made short.  The bodies are
// split into flow blocks (a part of the colouring, or a piece of a large batch world); a block
// holds its bodies' velocities and the rows of its manifolds in shared memory for all phases -
// rows are formed there, straight from the manifolds, and only what does not fit goes to memory.
// A body whose next manifold lies in another block travels through a 32-byte record in L2, each
// 16-byte half written and read whole (.b128) with its tag, so one poll brings tag and data.
#include <algorithm>
#include <vector>
#include "../../include/jbgpu.h"
#include "gridsync.cuh"
#include "prims.cuh"
#include "rows.cuh"
#include "solver.cuh"

namespace jbg {
using namespace jbd;

namespace {
constexpr int FLOW_TAG_SHIFT = 11;
constexpr int FLOW_STEPS = MAX_LOCAL + MAX_COLOURS;   // colours of a phase: local, then cut
static_assert(FLOW_STEPS + 1 < (1 << FLOW_TAG_SHIFT), "a tag holds phase and colour");
constexpr int FLOW_BINS = 4 * FLOW_STEPS;             // a step's candidates by points, so that a group's have as many
constexpr size_t FLOW_HIST_BYTES = sizeof(int) * FLOW_BINS;
constexpr int FLOW_QUADS = 8;                         // manifolds of a group: four lanes each
// 256 threads and two blocks an SM.  With 384 or 512 threads the registers spill (an earlier form of
// this kernel, setup and solve: 100k pile 1193 / 1226 / 1276 us, 1,000 boxes in pieces of 128
// 364 / 374 / 412 us); three blocks leave each a third less room for rows (1341 and 447 us).
constexpr int FLOW_THREADS = 256, FLOW_BLOCKS = 2;
// Polls of a wait, about half a microsecond each, for every FLOW_SPIN_ITERATIONS iterations or part of
// them: a world's first piece can wait for another world's whole solve before a block is free for its second.
constexpr int FLOW_SPIN_LIMIT = 1 << 21, FLOW_SPIN_ITERATIONS = 512;
static_assert((long long)FLOW_SPIN_LIMIT * (FLOW_MAX_ITERATIONS / FLOW_SPIN_ITERATIONS + 1) < 0x7fffffff, "an int counts them");
}

// 16 bytes written and read whole, between blocks (global memory) and within one (shared memory),
// by the lanes whose `on` holds: predicated, because a divergent branch costs a lone warp more than
// the access.
#define FLOW_B128_LD(space, cons, v, p, on)                                                                                \
    asm volatile("{ .reg .pred q; .reg .b128 t; .reg .b64 lo, hi; setp.ne.u32 q, %5, 0; mov.b64 lo, {%0, %1}; "           \
                 "mov.b64 hi, {%2, %3}; mov.b128 t, {lo, hi}; @q ld.relaxed." space ".b128 t, [%4]; "                       \
                 "mov.b128 {lo, hi}, t; mov.b64 {%0, %1}, lo; mov.b64 {%2, %3}, hi; }"                                      \
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : cons(p), "r"((unsigned)(on)) : "memory")
#define FLOW_B128_ST(space, cons, p, v, on)                                                                                \
    asm volatile("{ .reg .pred q; .reg .b128 t; .reg .b64 lo, hi; setp.ne.u32 q, %5, 0; mov.b64 lo, {%1, %2}; "           \
                 "mov.b64 hi, {%3, %4}; mov.b128 t, {lo, hi}; @q st.relaxed." space ".b128 [%0], t; }"                      \
                 :: cons(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"((unsigned)(on)) : "memory")
JBD void ld_whole_gpu(float4& v, const float4* p, bool on) { FLOW_B128_LD("gpu.global", "l", v, p, on); }
JBD void st_whole_gpu(float4* p, float4 v, bool on) { FLOW_B128_ST("gpu.global", "l", p, v, on); }
JBD void ld_whole_cta(float4& v, unsigned p, bool on) { FLOW_B128_LD("cta.shared", "r", v, p, on); }
JBD void st_whole_cta(unsigned p, float4 v, bool on) { FLOW_B128_ST("cta.shared", "r", p, v, on); }
JBD void ld_still(float4& v, const float4* p, bool on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.v4.f32 {%0, %1, %2, %3}, [%4]; }"
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "l"(p), "r"((unsigned)on) : "memory");
}
// Plain shared memory by address (the rows' near and far copies are told apart by branches; as
// pointers the compiler would merge them into generic accesses, which take twice as long).
JBD float4 lds4(unsigned p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p) : "memory");
    return v;
}
JBD float lds1(unsigned p) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
    return v;
}
JBD void sts4(unsigned p, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
JBD void sts1(unsigned p, float v, bool on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q st.shared.f32 [%0], %1; }" :: "r"(p), "f"(v), "r"((unsigned)on)
                 : "memory");
}

// A side's flags in the top byte of its body word (bodies stay below 2^24).
enum { FS_READ_EXCH = 1, FS_WRITE_EXCH = 2, FS_FIRST = 4, FS_LAST = 8, FS_DYN = 16 };   // bits 5-6: points - 1
constexpr unsigned FS_OFF = 128;   // a lane beyond its group's slots (bit 31)

// What the solver needs of a candidate, gathered for its block: side words (body | flags), the body's
// place in its home block | colour step of the manifold before it, inverse masses, the pair, and the
// candidate's own step << 4 | point mask.
struct FlowCand {
    unsigned word[2], place[2];
    float im[2];
    int pair, stepMask;
};
static_assert(sizeof(FlowCand) == 32, "two 16-byte loads");

JBD int flow_step(const SolverBuffers& sb, int k) { return sb.colourOf[k] + (sb.bucket[k] < sb.nParts ? 0 : MAX_LOCAL); }

// How side `side` of candidate k meets its body: where its velocity comes from and goes to, and
// the colour step of the manifold before it (over the turn of a phase for the body's first).
JBD void flow_side(const DevWorld& w, const SolverBuffers& sb, int k, int side, int b, int block, FlowCand& r) {
    r.word[side] = (unsigned)b;
    r.place[side] = 0;
    r.im[side] = w.iloc[b].w;
    if (w.island[b] < 0) return;                      // static or kinematic: its velocity never changes
    unsigned f = FS_DYN;
    const int pos = sb.posOf[b], start = sb.flowBody[block], end = sb.flowBody[block + 1];
    const bool home = pos >= start && pos < end;
    bool prevHome, nextHome;   // the manifold before (after) it on this body is solved in the body's home block
    int prevStep;
    if (w.ctr[C_COL_FAIL]) {   // coloured by claim passes: by its links
        const int self = 2 * k + side;
        int prev = sb.prevLink[self], next = sb.nextLink[self];
        if (prev < 0) { f |= FS_FIRST; prev = sb.lastLink[b]; }
        if (next < 0) { f |= FS_LAST; next = sb.firstLink[b]; }
        prevHome = sb.execOf[prev >> 1] == block;
        nextHome = sb.execOf[next >> 1] == block;
        prevStep = flow_step(sb, prev >> 1);
    } else {                   // by the colours its body holds: internal ones in order, then cut ones
        const uint4 lm = sb.localMask[b];
        unsigned long long m[2] = {(unsigned long long)lm.y << 32 | lm.x, 0}, h[2] = {(unsigned long long)lm.w << 32 | lm.z, 0};
        if (!sb.worldParts) {
            const uint4 ct = sb.cutToken[b];
            m[1] = (unsigned long long)ct.y << 32 | ct.x;
            h[1] = (unsigned long long)sb.cutHome[2 * b + 1] << 32 | sb.cutHome[2 * b];
        }
        const int cls = sb.bucket[k] < sb.nParts ? 0 : 1, c = sb.colourOf[k];
        const unsigned long long below = m[cls] & ((1ull << c) - 1), above = (m[cls] >> c) >> 1 << c << 1;
        int pc = cls, nc = cls, p, q;   // class and colour of the neighbours
        if (below) p = 63 - __clzll((long long)below);
        else if (cls == 1 && m[0]) { pc = 0; p = 63 - __clzll((long long)m[0]); }
        else { f |= FS_FIRST; pc = m[1] ? 1 : 0; p = 63 - __clzll((long long)m[pc]); }
        if (above) q = __ffsll((long long)above) - 1;
        else if (cls == 0 && m[1]) { nc = 1; q = __ffsll((long long)m[1]) - 1; }
        else { f |= FS_LAST; nc = m[0] ? 0 : 1; q = __ffsll((long long)m[nc]) - 1; }
        prevHome = h[pc] >> p & 1;
        nextHome = h[nc] >> q & 1;
        prevStep = p + (pc ? MAX_LOCAL : 0);
    }
    if (!home || !prevHome) f |= FS_READ_EXCH;
    if (!home || !nextHome) f |= FS_WRITE_EXCH;
    r.place[side] = (unsigned)(home ? pos - start : 0) | (unsigned)prevStep << 16;
    r.word[side] |= f << 24;
}

// A thread per candidate: its FlowCand into its block's list (candidates that got no colour - out of
// colours, reported as an error - are left out and never solved).
__global__ void k_flow_gather(DevWorld w, DevPairs P, SolverBuffers sb) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, nCand = *sb.nCand;
    if (k >= nCand || sb.colourOf[k] < 0) return;
    const int e = sb.execOf[k], p = sb.cand[k];
    if (e < 0) return;
    const int b0 = P.b0[p], b1 = P.b1[p], m = P.n[p];
    int mask = 0;
    for (int j = 0; j < m; j++)
        if (P.pA[p * 4 + j].w <= 0.0f) mask |= 1 << j;
    FlowCand c;
    flow_side(w, sb, k, 0, b0, e, c);
    flow_side(w, sb, k, 1, b1, e, c);
    const unsigned more = (unsigned)(__popc(mask) - 1) << 29;
    c.word[0] |= more;
    c.word[1] |= more;
    c.pair = p;
    c.stepMask = flow_step(sb, k) << 4 | mask;
    const unsigned same = __match_any_sync(__activemask(), e);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&sb.flowFill[e], __popc(same));
    base = __shfl_sync(same, base, leader) + __popc(same & ((1u << lane) - 1u));
    float4* out = (float4*)(sb.flowCand + (size_t)(sb.flowStart[e] - nCand + base) * 8);
    out[0] = make_float4(__uint_as_float(c.word[0]), __uint_as_float(c.word[1]), __uint_as_float(c.place[0]),
                         __uint_as_float(c.place[1]));
    out[1] = make_float4(c.im[0], c.im[1], __int_as_float(c.pair), __int_as_float(c.stepMask));
}

// A point's rows as the solver keeps them: 15 float4 (the planes of rows.cuh) side by side, the .w
// fields rearranged - a row's three direction vectors all carry jacDiagABInv, the angular vectors
// the point's scalars.
enum { FW_C1 = RP_NA, FW_REST = RP_NB, FW_FRIC = RP_F + 3, FW_IMP = RP_F + 4, FW_IMP1 = RP_F + 8, FW_IMP2 = RP_F + 9 };
constexpr unsigned REC_BYTES = ROW_PLANES * 16;

// A lane's part of a row: the vector its velocity is dotted with (.w: jacDiagABInv) and the one its
// velocity moves along.
struct RowPart { float4 v, a; };

// Where a block keeps its rows: points below recCap in shared memory, the others in global memory.
struct FlowRows {
    unsigned near;         // shared address of point 0
    float4* far;           // global address of point 0 (points from recCap on)
    int recCap;
    unsigned offV, offA;   // this lane's vectors within a row, bytes
};
// NEAR: every point of the block is in shared memory.
template <bool NEAR> JBD RowPart row_part(const FlowRows& F, int idx, int row) {
    RowPart r;
    if (NEAR || idx < F.recCap) {
        const unsigned a = F.near + REC_BYTES * (unsigned)idx + 80u * row;
        r.v = lds4(a + F.offV);
        r.a = lds4(a + F.offA);
    } else {
        const char* a = (const char*)(F.far + (size_t)ROW_PLANES * idx) + 80 * row;
        r.v = *(const float4*)(a + F.offV);
        r.a = *(const float4*)(a + F.offA);
    }
    return r;
}
template <bool NEAR> JBD float row_scalar(const FlowRows& F, int idx, int plane) {
    if (NEAR || idx < F.recCap) return lds1(F.near + REC_BYTES * (unsigned)idx + 16u * plane + 12u);
    return F.far[(size_t)ROW_PLANES * idx + plane].w;
}
template <bool NEAR> JBD void row_keep(const FlowRows& F, int idx, int plane, float x, bool on) {
    if (NEAR) sts1(F.near + REC_BYTES * (unsigned)idx + 16u * plane + 12u, x, on);
    else if (on) {
        if (idx < F.recCap) sts1(F.near + REC_BYTES * (unsigned)idx + 16u * plane + 12u, x, true);
        else F.far[(size_t)ROW_PLANES * idx + plane].w = x;
    }
}

// The lane of a manifold that holds velocity v of one side, and its row arithmetic.
struct FlowLane {
    V v;
    float along;       // linear velocities move along direction * inverse mass
    bool moves;        // inverse mass not 0
    bool side1, first; // its side; the first of the manifold's four lanes
    // SolverBody.internalApplyImpulse of +imp to body0, -imp to body1, where `on` holds
    JBD void apply(const RowPart& r, float imp, bool on) {
        const float i2 = side1 ? -imp : imp;
        const float x = __fadd_rn(v.x, __fmul_rn(i2, __fmul_rn(r.a.x, along)));
        const float y = __fadd_rn(v.y, __fmul_rn(i2, __fmul_rn(r.a.y, along)));
        const float z = __fadd_rn(v.z, __fmul_rn(i2, __fmul_rn(r.a.z, along)));
        const bool go = on && moves;
        v.x = go ? x : v.x;
        v.y = go ? y : v.y;
        v.z = go ? z : v.z;
    }
    // relative velocity along a row: (dir.lin0 + r1.ang0) - (dir.lin1 + r2.ang1)
    JBD float rel_vel(const RowPart& r) const {
        const float d = dot(mk4(r.v), v);
        const float mine = __fadd_rn(d, __shfl_xor_sync(0xffffffffu, d, 1));
        const float other = __shfl_xor_sync(0xffffffffu, mine, 2);
        return __fsub_rn(side1 ? other : mine, side1 ? mine : other);
    }
};
// resolveSingleFrictionCacheFriendly's clamp (java:286-346)
JBD float clamp_friction(float acc, float limit) {
    const float lo = acc < -limit ? -limit : acc;
    return limit < acc ? limit : lo;
}

// The rows of a warp's manifolds in one phase, four lanes each: the warp runs `most` points, a lane
// whose manifold has fewer repeats its last one without effect (no lane leaves the path).  r: row 0
// (normal, warm start) or 1 (friction) of the first point, loaded ahead, as the next point's is
// while one is solved.  The arithmetic is that of the reference's rows (java:234-346).
template <bool NEAR, int KIND>
JBD void flow_solve(const FlowRows& F, int idx, int npt, int most, RowPart r, FlowLane& L) {
    const int last = idx + max(npt, 1) - 1;
#pragma unroll 1
    for (int j = 0; j < most; j++) {
        const bool on = j < npt;
        const int next = min(idx + 1, last);
        if (KIND == PH_NORMAL) {
            const float c1 = row_scalar<NEAR>(F, idx, FW_C1), rest = row_scalar<NEAR>(F, idx, FW_REST),
                        old = row_scalar<NEAR>(F, idx, FW_IMP);
            const RowPart rn = row_part<NEAR>(F, next, 0);
            const float velErr = __fsub_rn(rest, L.rel_vel(r));
            const float sum = __fadd_rn(old, __fadd_rn(c1, __fmul_rn(velErr, r.v.w)));
            const float acc = 0.0f > sum ? 0.0f : sum;
            L.apply(r, __fsub_rn(acc, old), on);
            row_keep<NEAR>(F, idx, FW_IMP, acc, on && L.first);
            r = rn;
        } else if (KIND == PH_FRICTION) {
            const float total = __fadd_rn(row_scalar<NEAR>(F, idx, FW_IMP), 0.0f);   // + appliedPushImpulse
            const float limit = __fmul_rn(total, row_scalar<NEAR>(F, idx, FW_FRIC));
            const float old1 = row_scalar<NEAR>(F, idx, FW_IMP1), old2 = row_scalar<NEAR>(F, idx, FW_IMP2);
            const RowPart r2 = row_part<NEAR>(F, idx, 2), rn = row_part<NEAR>(F, next, 1);
            const bool push = on && total > 0.0f;
            const float acc1 = clamp_friction(__fadd_rn(old1, __fmul_rn(-L.rel_vel(r), r.v.w)), limit);
            L.apply(r, __fsub_rn(acc1, old1), push);
            const float acc2 = clamp_friction(__fadd_rn(old2, __fmul_rn(-L.rel_vel(r2), r2.v.w)), limit);
            L.apply(r2, __fsub_rn(acc2, old2), push);
            row_keep<NEAR>(F, idx, FW_IMP1, acc1, push && L.first);
            row_keep<NEAR>(F, idx, FW_IMP2, acc2, push && L.first);
            r = rn;
        } else {   // warm start: the normal impulse, then both friction impulses (java:680-760)
            L.apply(r, row_scalar<NEAR>(F, idx, FW_IMP), on);
            L.apply(row_part<NEAR>(F, idx, 1), row_scalar<NEAR>(F, idx, FW_IMP1), on);
            L.apply(row_part<NEAR>(F, idx, 2), row_scalar<NEAR>(F, idx, FW_IMP2), on);
            r = row_part<NEAR>(F, next, 0);
        }
        idx = next;
    }
}

// What the lanes of one side of a slot read each phase (one 16-byte load): body | flags | points - 1,
// the body's place in its home block | step of the manifold before << 16, the slot's first
// point | its step << 21, the inverse mass.
constexpr int FLOW_IDX_BITS = 21;   // points of a block (a block with more would need 2 M contact points)

template <bool NEAR>
JBD void flow_phases(const DevWorld& w, const SolverBuffers& sb, const FlowRows& F, unsigned smem0, bool descIn,
                     unsigned descAt, const int4* descFar, int n, int nGroups, int np, bool& dead) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    const int side = lane >> 1 & 1;
    const bool odd = lane & 1;
    const float4* const still = odd ? w.angvel : w.linvel;
    const int nPhases = 1 + 2 * w.numIter;
    const int spinLimit = FLOW_SPIN_LIMIT * (w.numIter / FLOW_SPIN_ITERATIONS + 1);
    const int* const groupFar = (const int*)(descFar + 2 * (size_t)n);
    const unsigned half = odd ? 16u * (unsigned)np : 0u;
    // lanes beyond a group's slots take its last slot's words with nothing to read, solve or write
    auto load_desc = [&](int g) {
        const int gw = descIn ? __float_as_int(lds1(descAt + 32u * (unsigned)n + 4u * (unsigned)g)) : groupFar[g];
        const int in = (gw & 15) - 1, at = 2 * ((gw >> 4) + min(lane >> 2, in)) + side;
        int4 d;
        if (descIn) {
            const float4 q = lds4(descAt + 16u * (unsigned)at);
            d = make_int4(__float_as_int(q.x), __float_as_int(q.y), __float_as_int(q.z), __float_as_int(q.w));
        } else {
            d = descFar[at];
        }
        if ((lane >> 2) > in) d.x = (d.x & ~(0x7f << 24)) | (int)(FS_OFF << 24);
        return d;
    };
    if (warp >= nGroups) return;
    int4 d = load_desc(warp);
    for (int ph = 0; ph < nPhases; ph++) {
        const unsigned tagBase = ((unsigned)ph << FLOW_TAG_SHIFT) + 1u;
        const bool lastPh = ph + 1 == nPhases, friction = ph > 0 && !(ph & 1);
        for (int g = warp; g < nGroups; g += nWarps) {
            const unsigned word = (unsigned)d.x;
            const bool off = (word & FS_OFF << 24) != 0, changes = (word & FS_DYN << 24) != 0;
            const int npt = off ? 0 : (int)(word >> 29 & 3u) + 1;
            const int idx = (int)((unsigned)d.z & ((1u << FLOW_IDX_BITS) - 1u));
            const unsigned tag = tagBase + ((unsigned)d.z >> FLOW_IDX_BITS);
            const unsigned home = smem0 + 16u * ((unsigned)d.y & 0xffffu) + half;
            const int body = (int)(word & 0xffffffu);
            float4* const ex = sb.exch + 2 * (size_t)body + (odd ? 1 : 0);
            const RowPart r0 = row_part<NEAR>(F, idx, friction ? 1 : 0);
            // this lane's half of its body's velocity: read at once when it never changes or nothing
            // wrote it yet, else from where the manifold before leaves it
            float4 v4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const bool first = (word & FS_FIRST << 24) != 0, now = !changes || (ph == 0 && first);
            ld_still(v4, still + body, now && !off);
            const unsigned want = tagBase + ((unsigned)d.y >> 16) - (first ? 1u << FLOW_TAG_SHIFT : 0u);
            bool waitOut = !now && (word & FS_READ_EXCH << 24) != 0, waitIn = !now && !waitOut;
            // the wait: bounded; on giving up the status flag ends every other wait too
            for (int spins = 0; !dead; ) {
                ld_whole_cta(v4, home, waitIn);
                ld_whole_gpu(v4, ex, waitOut);
                const bool there = __float_as_uint(v4.w) == want;
                waitIn = waitIn && !there;
                waitOut = waitOut && !there;
                if (!__any_sync(0xffffffffu, waitIn || waitOut)) break;
                if ((++spins & 1023) == 0) {
                    const bool give = spins >= spinLimit;
                    if (give && lane == 0) atomicOr(&w.ctr[C_STATUS], ST_TIMEOUT);
                    dead = __any_sync(0xffffffffu, give || (ld_acquire(&w.ctr[C_STATUS]) & ST_TIMEOUT) != 0);
                }
            }
            FlowLane L;
            L.v = mk4(v4);
            const float im = __int_as_float(d.w);
            L.along = odd ? 1.0f : im;
            L.moves = im != 0.0f;
            L.side1 = side != 0;
            L.first = (lane & 3) == 0;
            const int most = __reduce_max_sync(0xffffffffu, npt);
            d = load_desc(g + nWarps < nGroups ? g + nWarps : warp);   // this warp's next group
            if (ph == 0) flow_solve<NEAR, PH_WARM>(F, idx, npt, most, r0, L);
            else if (friction) flow_solve<NEAR, PH_FRICTION>(F, idx, npt, most, r0, L);
            else flow_solve<NEAR, PH_NORMAL>(F, idx, npt, most, r0, L);
            const bool ends = lastPh && (word & FS_LAST << 24) != 0, out = (word & FS_WRITE_EXCH << 24) != 0;
            const float4 res = f4(L.v, __uint_as_float(tag));
            st_whole_gpu(ex, res, changes && !ends && out);
            st_whole_cta(home, res, changes && !ends && !out);
            if (lastPh && changes && ends && L.moves) (odd ? w.angvel : w.linvel)[body] = f4(L.v, 0.0f);
            __syncwarp();   // the impulses kept by a manifold's first lane are read by all four next
        }
    }
}

JBD int nth_bit(int mask, int j) {
    for (int q = 0; q < j; q++) mask &= mask - 1;
    return __ffs(mask) - 1;
}
// A warp's contact points, count per lane: they are numbered lane after lane.
struct WarpPoints {
    int start, end, total;   // this lane's points; the warp's
    JBD WarpPoints(int count) {
        const int lane = threadIdx.x & 31;
        end = count;
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += q;
        }
        start = end - count;
        total = __shfl_sync(0xffffffffu, end, 31);
    }
    // the lane that holds point q (any lane past the last), j: its place among that lane's
    JBD int owner(int q, int& j) const {
        int lo = 0;   // the first lane whose end is above q
        for (int o = 16; o > 0; o >>= 1)
            if (__shfl_sync(0xffffffffu, end, lo + o - 1) <= q) lo += o;
        lo = min(lo, 31);
        j = q - __shfl_sync(0xffffffffu, start, lo);
        return lo;
    }
};

__global__ void __launch_bounds__(FLOW_THREADS, FLOW_BLOCKS) k_flow(DevWorld w, DevPairs P, DevRows R, SolverBuffers sb, float dt) {
    extern __shared__ __align__(16) unsigned char fsm[];
    __shared__ int shBlock, shTop, shRows, shOvf;
    __shared__ int2 shScan[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    const int nCand = *sb.nCand;
    if (nCand == 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicMax(&w.ctr[C_PGS_ITERS], w.numIter);
    const bool warm = (w.solverMode & 4) != 0;
    const unsigned smem0 = (unsigned)__cvta_generic_to_shared(fsm);
    bool dead = false;   // a wait gave up: later waits return at once
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) shBlock = atomicAdd(sb.flowTop, 1);
        __syncthreads();
        if (shBlock >= sb.nFlow) break;
        const int block = sb.flowOrder[shBlock];
        const int x0 = sb.flowStart[block] - nCand, n = sb.flowFill[block];   // its candidates
        if (n == 0) continue;
        const int bodyStart = sb.flowBody[block], np = sb.flowBody[block + 1] - bodyStart;
        float4* const vel = (float4*)fsm;                     // lin of body i at i, ang at np + i
        for (int i = threadIdx.x; i < 2 * np; i += blockDim.x) vel[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        // ---- the block's candidates sorted by colour step --------------------------------------
        int* const hist = (int*)(fsm + sb.flowSmem) - FLOW_BINS;   // counts, then fill positions
        for (int i = threadIdx.x; i < FLOW_BINS; i += blockDim.x) hist[i] = 0;
        if (threadIdx.x == 0) shTop = shRows = 0;
        __syncthreads();
        float4* const cands = (float4*)sb.flowCand + 2 * (size_t)x0;
        int rowsMine = 0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int sm = __float_as_int(cands[2 * i + 1].w);
            atomicAdd(&hist[(sm >> 4) * 4 + __popc(sm & 15) - 1], 1);
            rowsMine += __popc(sm & 15);
        }
        rowsMine = __reduce_add_sync(0xffffffffu, rowsMine);
        if (lane == 0 && rowsMine) { atomicAdd(&w.ctr[C_ROWS], rowsMine); atomicAdd(&shRows, rowsMine); }
        __syncthreads();
        const int rows = shRows;
        const int per = (FLOW_STEPS + blockDim.x - 1) / blockDim.x;
        int cnt = 0, grp = 0;
        for (int e = 0; e < per; e++) {
            const int st = threadIdx.x * per + e;
            if (st >= FLOW_STEPS) break;
            const int c = hist[4 * st] + hist[4 * st + 1] + hist[4 * st + 2] + hist[4 * st + 3];
            cnt += c;
            grp += (c + FLOW_QUADS - 1) / FLOW_QUADS;
        }
        int c0 = cnt, g0 = grp;   // inclusive scans over the block's threads
        for (int o = 1; o < 32; o <<= 1) {
            const int tc = __shfl_up_sync(0xffffffffu, c0, o), tg = __shfl_up_sync(0xffffffffu, g0, o);
            if (lane >= o) { c0 += tc; g0 += tg; }
        }
        if (lane == 31) shScan[warp] = make_int2(c0, g0);
        __syncthreads();
        int nGroups = 0;
        for (int q = 0; q < nWarps; q++) {
            if (q < warp) { c0 += shScan[q].x; g0 += shScan[q].y; }
            nGroups += shScan[q].y;
        }
        c0 -= cnt;
        g0 -= grp;
        // Slots (32 bytes, by step) and groups of up to eight slots of one step (first slot << 4 |
        // slots) in shared memory, after the bodies; a block with too many keeps them in global memory.
        const unsigned velBytes = 32u * (unsigned)np;
        const size_t descBytes = (32 * (size_t)n + 4 * (size_t)nGroups + 15) & ~(size_t)15;
        const bool descIn = velBytes + descBytes + FLOW_HIST_BYTES <= (size_t)sb.flowSmem;
        int4* const desc = descIn ? (int4*)(fsm + velBytes) : (int4*)(sb.flowDesc + FLOW_DESC_INTS * (size_t)x0);
        int* const group = (int*)(desc + 2 * (size_t)n);
        const unsigned recOff = velBytes + (descIn ? (unsigned)descBytes : 0u);
        FlowRows F;
        F.recCap = (int)(((unsigned)sb.flowSmem - recOff) / REC_BYTES);
        F.near = smem0 + recOff;
        F.offV = 16u * ((lane & 1) ? RP_N1 + (lane >> 1 & 1) : RP_N);
        F.offA = 16u * ((lane & 1) ? RP_NA + (lane >> 1 & 1) : RP_N);
        for (int e = 0; e < per; e++) {
            const int st = threadIdx.x * per + e;
            if (st >= FLOW_STEPS) break;
            int c = 0;
            for (int q = 0; q < 4; q++) {
                const int h = hist[4 * st + q];
                hist[4 * st + q] = c0 + c;
                c += h;
            }
            for (int q = 0; q < c; q += FLOW_QUADS) group[g0++] = (c0 + q) << 4 | min(FLOW_QUADS, c - q);
            c0 += c;
        }
        if (threadIdx.x == 0) {
            shOvf = rows > F.recCap ? atomicAdd(sb.flowTop + 1, rows - F.recCap) - F.recCap : 0;
            if (rows > 1 << FLOW_IDX_BITS) atomicOr(&w.ctr[C_STATUS], ST_CAPACITY);
        }
        __syncthreads();
        F.far = R.planes + (long long)ROW_PLANES * shOvf;
        // ---- slots, a lane per candidate; the points of a warp's candidates take consecutive places ----
        for (int i0 = 32 * warp; i0 < n; i0 += 32 * nWarps) {
            const int i = i0 + lane;
            float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f), t = u;
            if (i < n) {
                u = cands[2 * i];
                t = cands[2 * i + 1];
            }
            const int mask = __float_as_int(t.w) & 15, st = __float_as_int(t.w) >> 4;
            const WarpPoints wp(__popc(mask));
            int base = 0;
            if (lane == 31) base = atomicAdd(&shTop, wp.end);
            base = __shfl_sync(0xffffffffu, base, 31);
            if (i < n) {
                const int idx = base + wp.start, s = atomicAdd(&hist[4 * st + __popc(mask) - 1], 1), z = idx | st << FLOW_IDX_BITS;
                desc[2 * s] = make_int4(__float_as_int(u.x), __float_as_int(u.z), z, __float_as_int(t.x));
                desc[2 * s + 1] = make_int4(__float_as_int(u.y), __float_as_int(u.w), z, __float_as_int(t.y));
                cands[2 * i + 1].w = __int_as_float(idx << 4 | mask);
            }
        }
        __syncthreads();   // the step positions lie where rows go next
        // ---- rows, a lane per point -------------------------------------------------------------------
        for (int i0 = 32 * warp; i0 < n; i0 += 32 * nWarps) {
            const int i = i0 + lane;
            float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f), t = u;
            if (i < n) {
                u = cands[2 * i];
                t = cands[2 * i + 1];
            }
            const int first = __float_as_int(t.w) >> 4, mask = __float_as_int(t.w) & 15;
            const WarpPoints wp(__popc(mask));
            for (int q0 = 0; q0 < wp.total; q0 += 32) {
                int j;
                const int own = wp.owner(q0 + lane, j);
                const int p = __shfl_sync(0xffffffffu, __float_as_int(t.z), own);
                const int mk = __shfl_sync(0xffffffffu, mask, own);
                const unsigned w0 = __shfl_sync(0xffffffffu, __float_as_uint(u.x), own);
                const unsigned w1 = __shfl_sync(0xffffffffu, __float_as_uint(u.y), own);
                const int idx = __shfl_sync(0xffffffffu, first, own) + j;
                if (q0 + lane >= wp.total) continue;
                const BodyV A = load_body(w, w0 & 0xffffff), B = load_body(w, w1 & 0xffffff);
                const bool near = idx < F.recCap;
                const unsigned nearAt = F.near + REC_BYTES * (unsigned)idx;
                float4* const farAt = F.far + (size_t)ROW_PLANES * idx;
                float jac = 0.0f, c1 = 0.0f, rest = 0.0f, fric = 0.0f, imp = 0.0f, imp1 = 0.0f, imp2 = 0.0f;
                point_rows(w, P, p * 4 + nth_bit(mk, j), A, B, warm, dt, [&](int plane, float4 v) {
                    switch (plane) {   // planes come in order; each takes its scalar here and carries another's
                    case RP_N: case RP_F: case RP_F + 5: jac = v.w; break;
                    case RP_N1: c1 = __fmul_rn(v.w, jac); v.w = jac; break;   // positionalError * jacDiagABInv
                    case RP_N2: rest = v.w; v.w = jac; break;
                    case RP_NA: fric = v.w; v.w = c1; break;
                    case RP_NB: imp = v.w; v.w = rest; break;
                    case RP_F + 1: imp1 = v.w; v.w = jac; break;
                    case RP_F + 6: imp2 = v.w; v.w = jac; break;
                    case RP_F + 2: case RP_F + 7: v.w = jac; break;
                    case FW_FRIC: v.w = fric; break;
                    case FW_IMP: v.w = imp; break;
                    case FW_IMP1: v.w = imp1; break;
                    case FW_IMP2: v.w = imp2; break;
                    }
                    if (near) sts4(nearAt + 16u * plane, v);
                    else farAt[plane] = v;
                });
            }
        }
        __syncthreads();   // rows written, velocity tags clear
        if (rows <= F.recCap) flow_phases<true>(w, sb, F, smem0, descIn, smem0 + velBytes, desc, n, nGroups, np, dead);
        else flow_phases<false>(w, sb, F, smem0, descIn, smem0 + velBytes, desc, n, nGroups, np, dead);
        __syncthreads();
        // ---- write-back (java:901-912), a lane per point ---------------------------------------------
        for (int i0 = 32 * warp; i0 < n; i0 += 32 * nWarps) {
            const float4 t = i0 + lane < n ? cands[2 * (i0 + lane) + 1] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const WarpPoints wp(__popc(__float_as_int(t.w) & 15));
            for (int q0 = 0; q0 < wp.total; q0 += 32) {
                int j;
                const int own = wp.owner(q0 + lane, j);
                const int p = __shfl_sync(0xffffffffu, __float_as_int(t.z), own);
                const int im = __shfl_sync(0xffffffffu, __float_as_int(t.w), own);
                if (q0 + lane >= wp.total) continue;
                const int k = p * 4 + nth_bit(im & 15, j), idx = (im >> 4) + j;
                P.nrm[k].w = row_scalar<false>(F, idx, FW_IMP);
                P.imp[k].x = row_scalar<false>(F, idx, FW_IMP2);   // appliedImpulseLateral1 ends as friction row 2's
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------------------
template <class T> static cudaError_t falloc(T** p, size_t n) { return cudaMalloc((void**)p, sizeof(T) * (n ? n : 1)); }
template <class T> static void ffree(T*& p) { if (p) cudaFree((void*)p); p = nullptr; }

int flow_plan(SolverBuffers& sb, const std::vector<int>& start, int sms, cudaStream_t s) {
    const int parts = (int)start.size() - 1;
    std::vector<int2> part(parts);
    std::vector<int> body, size(parts), order;
    // Bodies of a block of a batch world.  Small pieces shorten a large world's critical path while
    // the SMs have room for them (setup and solve of one 1,000-box world: 416 us at 256 bodies, 234 at
    // 128, 197 at 64, 658 + 37 us colour by colour); with more bodies than that, the exchange between
    // pieces costs more than it gives (64 worlds of up to 1,500: 247 us at 96, 309 at 128, 459 at 256,
    // 807 colour by colour; 512 worlds of up to 512: 729 at 64, 505 at 128, 494 at 256, 567; 1,000
    // worlds of up to 300: 765 at 64, 529 at 128, 454 at 256, 780).
    const int finite = start[parts], seats = FLOW_BLOCKS * sms;
    const int T = finite <= 64 * seats ? 96 : finite <= 256 * seats ? 128 : 256;
    for (int p = 0; p < parts; p++) {
        const int n = start[p + 1] - start[p];
        const int pieces = sb.worldParts ? std::max(1, (n + T - 1) / T) : 1;
        const int each = std::max(1, (n + pieces - 1) / pieces);
        part[p] = make_int2((int)body.size(), each);
        size[p] = n;
        for (int at = 0; at == 0 || at < n; at += each) body.push_back(start[p] + at);
    }
    const int nFlow = (int)body.size();
    body.push_back(start[parts]);
    // larger parts first; a part's blocks follow each other, so that the blocks of a part are
    // taken before any later part's (the lowest part unfinished always finds free blocks)
    std::vector<int> by(parts);
    for (int p = 0; p < parts; p++) by[p] = p;
    std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return size[a] > size[b]; });
    int most = 0;
    for (int p : by) {
        const int first = part[p].x, end = p + 1 < parts ? part[p + 1].x : nFlow;
        most = std::max(most, end - first);
        for (int q = first; q < end; q++) order.push_back(q);
    }
    const int buckets = parts + 2 + nFlow + 1;
    if (buckets > sb.flowCap) {
        flow_free(sb);
        if (falloc(&sb.bucketCount, buckets) || falloc(&sb.bucketFill, buckets) || falloc(&sb.bucketStart, buckets) ||
            falloc(&sb.flowPart, buckets) || falloc(&sb.flowBody, buckets) || falloc(&sb.flowOrder, buckets) ||
            falloc(&sb.flowTop, 2) || cudaMalloc(&sb.flowScan, scan_scratch_bytes(buckets)))
            return 1;
        sb.flowCap = buckets;
    }
    sb.flowCount = sb.bucketCount + parts + 2;
    sb.flowFill = sb.bucketFill + parts + 2;
    sb.flowStart = sb.bucketStart + parts + 2;
    sb.nFlow = nFlow;
    sb.flowExch = !sb.worldParts || nFlow > parts;
    sb.gridFlow = sb.worldParts ? most : nFlow;   // blocks that wait on one another; flow_configure adds the rest
    return cudaMemcpyAsync(sb.flowPart, part.data(), sizeof(int2) * parts, cudaMemcpyHostToDevice, s) != cudaSuccess ||
           cudaMemcpyAsync(sb.flowBody, body.data(), sizeof(int) * (nFlow + 1), cudaMemcpyHostToDevice, s) != cudaSuccess ||
           cudaMemcpyAsync(sb.flowOrder, order.data(), sizeof(int) * nFlow, cudaMemcpyHostToDevice, s) != cudaSuccess ||
           cudaStreamSynchronize(s) != cudaSuccess;
}

static int flow_threads(const SolverBuffers& sb) { return sb.threads < SOLVER_THREADS ? sb.threads : FLOW_THREADS; }

int flow_configure(SolverBuffers& sb, int sms, int smemBodies) {
    int dev = 0, perSm = 0, perBlock = 0, most = sb.gridFlow, blocks = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&perSm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&perBlock, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncSetAttribute(k_flow, cudaFuncAttributeMaxDynamicSharedMemorySize, perBlock - 2048) != cudaSuccess)
        return 1;
    // two blocks an SM: half of its shared memory each, less the 1 KB a block reserves and the
    // kernel's static arrays
    sb.flowSmem = (perSm / FLOW_BLOCKS - 2048) & ~127;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_flow, flow_threads(sb), sb.flowSmem) != cudaSuccess) return 1;
    sb.gridFlow = std::min(sb.nFlow, blocks * sms);
    // Past about 512 bodies a resident block the blocks come in so many rounds, each as long as the
    // longest chain of its manifolds, that the colour-by-colour solver's wider blocks win.  Flow / by colour
    // with its setup, us: 57k bodies in 1,024 worlds 345 / 685, 128k in 256 larger ones 1032 / 1240, 152k in
    // 1,024 854 / 1013; 444k in 1,024 3094 / 1891.
    const bool wide = sb.worldParts && sb.nFinite > 512 * blocks * sms;
    sb.flowOk = !wide && most <= sb.gridFlow && !sb.movingStatic && (smemBodies <= 0 || sb.partMax <= smemBodies) &&
                (size_t)sb.partMax * 32 + FLOW_HIST_BYTES <= (size_t)sb.flowSmem;
    return 0;
}

void flow_free(SolverBuffers& sb) {
    ffree(sb.bucketCount); ffree(sb.bucketFill); ffree(sb.bucketStart); ffree(sb.flowPart); ffree(sb.flowBody);
    ffree(sb.flowOrder); ffree(sb.flowTop);
    if (sb.flowScan) cudaFree(sb.flowScan);
    sb.flowScan = nullptr;
    sb.flowCap = 0;
}

void flow_launch(const DevWorld& w, DevPairs& P, int nPairs, DevRows& R, SolverBuffers& sb, float dt, cudaStream_t s) {
    k_flow_gather<<<(nPairs + 255) / 256, 256, 0, s>>>(w, P, sb); note_launch();
    DevWorld wc = w;
    DevPairs pc = P;
    DevRows rc = R;
    SolverBuffers sc = sb;
    float dtc = dt;
    void* args[] = {&wc, &pc, &rc, &sc, &dtc};
    cudaLaunchCooperativeKernel((void*)k_flow, sb.gridFlow, flow_threads(sb), args, sb.flowSmem, s); note_launch();
}

}  // namespace jbg
