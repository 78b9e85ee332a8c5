// Broadphase: the overlapping-pair set of the reference's DbvtBroadphase, rebuilt each step.
//
// The reference keeps an incremental dynamic AABB tree and, after collide(), its pair cache
// holds exactly the filter-passing pairs whose proxy aabbs intersect inclusively
// (collision/broadphase/DbvtBroadphase.java:89-150, DbvtTreeCollider.java:36-51,
// DbvtAabbMm.java:209-212, HashedOverlappingPairCache.java:179-188).  Here:
//   1. 30-bit Morton codes of finite proxy aabb centres, world index in the high key bits;
//   2. stable radix sort; 3. Karras radix tree over the sorted leaves (one root per world);
//   4. bottom-up refit; 5. a counting traversal (pair owner = the lower body index, or the
//   finite body of a pair with a static plane), exclusive scan -> per-owner CSR;
//   6. a filling traversal, per-owner partner sort -> keys sorted ascending;
//   7. persistence: each new key is looked up among last step's sorted keys and its
//   manifold (the reference's algorithm lifetime, HashedOverlappingPairCache.java:222-228) is
//   carried over.
// Static planes (infinite aabb, StaticPlaneShape.java:124-128) stay out of the tree; each
// finite body tests the planes of its world directly.  Small worlds test all their bodies so
// (direct pairs, below) and keep of these steps the order, 1 and 2, for the solver's parts.
#include <utility>

#include "broadphase.cuh"
#include "dispatch.cuh"
#include "prims.cuh"

namespace jbg {
using namespace jbd;

__device__ __forceinline__ unsigned f2ord(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Scene bounds of finite aabb centres (ordered-int atomics, one a warp).  By whole warps; i >= nBodies:
// none.
JBD void box_centre_bounds(const DevWorld& w, int i, unsigned* s) {
    unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
    if (i < w.nBodies && !(w.flags[i] & CF_LISTED)) {
        float4 a = w.amin[i], b = w.amax[i];
        float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
        for (int k = 0; k < 3; k++) lo[k] = hi[k] = f2ord(c[k]);
    }
    for (int k = 0; k < 3; k++) {
        const unsigned mn = __reduce_min_sync(0xffffffffu, lo[k]), mx = __reduce_max_sync(0xffffffffu, hi[k]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s[k], mn);
            atomicMax(&s[3 + k], mx);
        }
    }
}
__global__ void k_bounds(DevWorld w, unsigned* bnd) {
    __shared__ unsigned s[6];
    if (threadIdx.x < 6) s[threadIdx.x] = (threadIdx.x < 3) ? 0xffffffffu : 0u;
    __syncthreads();
    box_centre_bounds(w, blockIdx.x * blockDim.x + threadIdx.x, s);
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&bnd[threadIdx.x], s[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&bnd[threadIdx.x], s[threadIdx.x]);
}

__device__ __forceinline__ unsigned expand_bits(unsigned v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// key = world << 32 | morton30 for finite bodies; planes get the all-ones key (sorted last).
JBD uint64_t morton_key(const DevWorld& w, const unsigned* bnd, int i) {
    if (w.flags[i] & CF_LISTED) return ~0ull;
    float lo[3], hi[3];
    for (int k = 0; k < 3; k++) { lo[k] = ord2f(bnd[k]); hi[k] = ord2f(bnd[3 + k]); }
    float4 a = w.amin[i], b = w.amax[i];
    float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
    unsigned q[3];
    for (int k = 0; k < 3; k++) {
        float ext = hi[k] - lo[k];
        float t = ext > 0.0f ? (c[k] - lo[k]) / ext : 0.5f;
        t = fminf(fmaxf(t, 0.0f), 1.0f);
        q[k] = min((unsigned)(t * 1024.0f), 1023u);
    }
    unsigned m = (expand_bits(q[0]) << 2) | (expand_bits(q[1]) << 1) | expand_bits(q[2]);
    return ((uint64_t)(unsigned)w.world[i] << 32) | m;
}
__global__ void k_morton(DevWorld w, const unsigned* bnd, uint64_t* keys, int* vals) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w.nBodies) return;
    vals[i] = i;
    keys[i] = morton_key(w, bnd, i);
}

// Bounds, keys and the stable sort by key in one block, for up to ORDER_SMALL bodies: a bitonic
// network over key and body in one word (the world above ORDER_WORLD_BITS would not fit), R words a
// thread in registers, exchanged by shuffles within a warp and through shared memory beyond it.  The
// general path is 15 launches and more (four or five radix passes), some 2.5 us each however few the
// bodies.
constexpr int ORDER_SMALL = 4096, ORDER_THREADS = 1024, ORDER_WORLD_BITS = 21;
template <int R>
__global__ void __launch_bounds__(ORDER_THREADS) k_order_small(DevWorld w, uint64_t* keys, int* vals) {
    __shared__ uint64_t sx[ORDER_SMALL];
    __shared__ unsigned bnd[6];
    const int n = w.nBodies, tid = threadIdx.x, threads = blockDim.x, size = R * threads;
    if (tid < 6) bnd[tid] = tid < 3 ? 0xffffffffu : 0u;
    __syncthreads();
    for (int r = 0; r < R; r++) box_centre_bounds(w, r * threads + tid, bnd);
    __syncthreads();
    uint64_t x[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = tid * R + r;
        uint64_t m = ~0ull << 12;   // listed bodies and the padding behind them last
        if (i < n && !(w.flags[i] & CF_LISTED)) {
            const uint64_t key = morton_key(w, bnd, i);
            m = ((key >> 32) << 42) | ((key & 0x3fffffffu) << 12);
        }
        x[r] = m | (unsigned)i;
    }
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32 * R) {
                __syncthreads();
#pragma unroll
                for (int r = 0; r < R; r++) sx[tid * R + r] = x[r];
                __syncthreads();
            }
            uint64_t y[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (j >= 32 * R) y[r] = sx[(tid * R + r) ^ j];
                else if (j >= R) y[r] = __shfl_xor_sync(0xffffffffu, x[r], j / R);
                else y[r] = R > 2 && j == 2 ? x[(r ^ 2) & (R - 1)] : x[(r ^ 1) & (R - 1)];
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int e = tid * R + r;
                const bool least = ((e & j) == 0) == ((e & k) == 0);
                x[r] = least == (x[r] < y[r]) ? x[r] : y[r];
            }
        }
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int e = tid * R + r;
        if (e >= n) continue;
        const int i = (int)(x[r] & 0xfffu);
        vals[e] = i;
        keys[e] = w.flags[i] & CF_LISTED ? ~0ull : ((x[r] >> 42) << 32) | ((x[r] >> 12) & 0x3fffffffu);
    }
}

__device__ __forceinline__ int delta(const uint64_t* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    uint64_t a = k[i], b = k[j];
    if (a == b) return 64 + __clz(i ^ j);
    return __clzll(a ^ b);
}

// World leaf ranges in the sorted leaf order; single-leaf worlds get the leaf as root.
__global__ void k_world_ranges(const uint64_t* keys, int nf, int* wstart, int* wend, int* wroot) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nf) return;
    int wi = (int)(keys[i] >> 32);
    if (i == 0 || (int)(keys[i - 1] >> 32) != wi) wstart[wi] = i;
    if (i == nf - 1 || (int)(keys[i + 1] >> 32) != wi) {
        wend[wi] = i + 1;
        int s = (i == 0 || (int)(keys[i - 1] >> 32) != wi) ? i : -1;
        if (s == i) wroot[wi] = LEAF_FLAG | i;
    }
}

// Karras 2012 radix-tree construction over nf sorted leaves.
__global__ void k_karras(const uint64_t* keys, int nf, Bvh t, const int* wstart, const int* wend, int* wroot) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nf - 1) return;
    int d = (delta(keys, nf, i, i + 1) - delta(keys, nf, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, nf, i, i - d);
    int lmax = 2;
    while (delta(keys, nf, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int s = lmax >> 1; s >= 1; s >>= 1)
        if (delta(keys, nf, i, i + (l + s) * d) > dmin) l += s;
    int j = i + l * d;
    int dnode = delta(keys, nf, i, j);
    int s = 0, tt = l;
    do {
        tt = (tt + 1) >> 1;
        if (delta(keys, nf, i, i + (s + tt) * d) > dnode) s += tt;
    } while (tt > 1);
    int gamma = i + s * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    int left = (lo == gamma) ? (LEAF_FLAG | gamma) : gamma;
    int right = (hi == gamma + 1) ? (LEAF_FLAG | (gamma + 1)) : (gamma + 1);
    t.left[i] = left;
    t.right[i] = right;
    t.lo[i] = lo;
    t.hi[i] = hi;
    if (left & LEAF_FLAG) t.leafParent[gamma] = i; else t.parent[gamma] = i;
    if (right & LEAF_FLAG) t.leafParent[gamma + 1] = i; else t.parent[gamma + 1] = i;
    int wi = (int)(keys[lo] >> 32);
    if (wstart[wi] == lo && wend[wi] == hi + 1) wroot[wi] = i;
}

// Bottom-up refit into the parents' child records: a leaf writes its box into its parent's
// record; the second child to arrive at a node merges the node's two child boxes and writes the
// union into the node's slot in its own parent (roots have parent -1).
__global__ void k_refit(DevWorld w, const int* sortedBody, int nf, Bvh t) {
    int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= nf) return;
    const int b = sortedBody[leaf];
    float4 mn = w.amin[b], mx = w.amax[b];
    int child = LEAF_FLAG | leaf, last = leaf;
    int node = t.leafParent[leaf];
    while (node >= 0) {
        const int side = t.left[node] == child ? 0 : 2;
        __stcg(&t.node[4 * node + side], make_float4(mn.x, mn.y, mn.z, __int_as_float(child)));
        __stcg(&t.node[4 * node + side + 1], make_float4(mx.x, mx.y, mx.z, __int_as_float(last)));
        // release: this child's record; acquire: the sibling's (the second arrival goes on)
        int prev;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(prev) : "l"(t.visit + node) : "memory");
        if (prev == 0) return;
        const float4 l0 = __ldcg(&t.node[4 * node]), l1 = __ldcg(&t.node[4 * node + 1]);
        const float4 r0 = __ldcg(&t.node[4 * node + 2]), r1 = __ldcg(&t.node[4 * node + 3]);
        mn = make_float4(fminf(l0.x, r0.x), fminf(l0.y, r0.y), fminf(l0.z, r0.z), 0.0f);
        mx = make_float4(fmaxf(l1.x, r1.x), fmaxf(l1.y, r1.y), fmaxf(l1.z, r1.z), 0.0f);
        child = node;
        last = t.hi[node];
        node = t.parent[node];
    }
}

__device__ __forceinline__ bool ovl(float4 a0, float4 a1, float4 b0, float4 b1) {
    return (a0.x <= b1.x) && (a1.x >= b0.x) && (a0.y <= b1.y) && (a1.y >= b0.y) && (a0.z <= b1.z) && (a1.z >= b0.z);
}
__device__ __forceinline__ bool filt(const DevWorld& w, int a, int b) {
    return (w.group[a] & w.mask[b]) != 0 && (w.group[b] & w.mask[a]) != 0;
}

constexpr int STACK = 96;

// One leaf's traversal: pairs (s, t) with t > s in sorted order.  FILL == false counts
// pairs per owner and keeps up to TRAV_CACHE of leaf s's partners; FILL == true writes partners
// into the owner's CSR segment, from that cache when it holds all of them, else by traversing
// again.
template <bool FILL>
__global__ void k_traverse(DevWorld w, const int* sortedBody, int nf, Bvh t, const int* wroot, int* cnt, const int* off,
                           int* cursor, int* partners, int capacity, int* tcount, int* tcache) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nf) return;
    int bi = sortedBody[s];
    auto emit = [&](int bj) {
        int owner = bi < bj ? bi : bj, partner = bi < bj ? bj : bi;
        const int subs = w.hasCompound ? pair_subs(w.sh, w.shape[owner], w.shape[partner]) : 1;
        if (!FILL) {
            atomicAdd(&cnt[owner], subs);
        } else {
            int pos = off[owner] + atomicAdd(&cursor[owner], subs);
            for (int k = 0; k < subs; k++)
                if (pos + k < capacity) partners[pos + k] = partner | (k << 24);
        }
    };
    if (FILL) {
        const int found = tcount[s];
        if (found <= TRAV_CACHE) {
            for (int i = 0; i < found; i++) emit(sortedBody[tcache[(size_t)s * TRAV_CACHE + i]]);
            return;
        }
    }
    int root = wroot[w.world[bi]];
    if (root & LEAF_FLAG) {   // single-leaf world
        if (!FILL) tcount[s] = 0;
        return;
    }
    float4 a0 = w.amin[bi], a1 = w.amax[bi];
    int found = 0;
    int stack[STACK];
    int sp = 0;
    stack[sp++] = root;
    while (sp > 0) {
        const float4* nd = t.node + 4 * stack[--sp];
        const float4 rec[4] = {nd[0], nd[1], nd[2], nd[3]};
        for (int c = 0; c < 2; c++) {
            const float4 mn = rec[2 * c], mx = rec[2 * c + 1];
            if (__float_as_int(mx.w) <= s) continue;   // the child's leaves all precede s
            if (!ovl(a0, a1, mn, mx)) continue;
            const int x = __float_as_int(mn.w);
            if (x & LEAF_FLAG) {
                const int tl = x & ~LEAF_FLAG;
                const int bj = sortedBody[tl];
                if (!filt(w, bi, bj)) continue;
                emit(bj);
                if (!FILL && found < TRAV_CACHE) tcache[(size_t)s * TRAV_CACHE + found] = tl;
                ++found;
            } else {
                if (sp < STACK) stack[sp++] = x;
                else atomicOr(&w.ctr[C_STATUS], ST_CAPACITY);
            }
        }
    }
    if (!FILL) tcount[s] = found;
}

// Pairs of each body in the tree with the listed bodies (static planes, triangle meshes) of its
// world, owned by the former.
// The counting pass also sums, into candBound, the triangle candidates the concave pass will
// list for the body's mesh pairs (an upper bound: pairs whose bodies are both inactive list none).
template <bool FILL>
__global__ void k_plane_pairs(DevWorld w, const int* planeList, const int* planeStart, int* cnt, const int* off,
                              int* cursor, int* partners, int capacity, int* candBound) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w.nBodies || (w.flags[i] & CF_LISTED)) return;
    int wi = w.world[i];
    float4 a0 = w.amin[i], a1 = w.amax[i];
    for (int k = planeStart[wi]; k < planeStart[wi + 1]; k++) {
        int p = planeList[k];
        if (!ovl(a0, a1, w.amin[p], w.amax[p]) || !filt(w, i, p)) continue;
        const int subs = w.hasCompound ? pair_subs(w.sh, w.shape[i], w.shape[p]) : 1;
        if (!FILL && candBound) {
            const int c = mesh_candidates(w, i, p, [&](const Leaf& l, const Leaf& t) { return mesh_walk(w, l, t); });
            if (c) atomicAdd(candBound, c);
        }
        if (!FILL) atomicAdd(&cnt[i], subs);
        else {
            int pos = off[i] + atomicAdd(&cursor[i], subs);
            for (int k = 0; k < subs; k++)
                if (pos + k < capacity) partners[pos + k] = p | (k << 24);
        }
    }
}

// Ascending sort of c words in place: in registers up to 32, else a Shell sort in memory.
JBD void sort_words(unsigned* p, int c) {
    if (c <= 32) {
        unsigned v[32];
        for (int k = 0; k < c; k++) v[k] = p[k];
        for (int k = 1; k < c; k++) {
            unsigned x = v[k];
            int j = k - 1;
            while (j >= 0 && v[j] > x) { v[j + 1] = v[j]; j--; }
            v[j + 1] = x;
        }
        for (int k = 0; k < c; k++) p[k] = v[k];
        return;
    }
    for (int gap = c / 2; gap > 0; gap /= 2)
        for (int k = gap; k < c; k++) {
            unsigned x = p[k];
            int j = k;
            while (j >= gap && p[j - gap] > x) { p[j] = p[j - gap]; j -= gap; }
            p[j] = x;
        }
}

// Sort each owner's partner words (sub << 24 | partner, compared unsigned) ascending and emit the
// canonical keys.  With compounds a partner's child combinations are written together, so the
// owner's distinct partners (the words with sub 0) are sorted alone and the keys generated sub
// by sub - the same ascending order without sorting every combination.
__global__ void k_segment_sort(DevWorld w, int n, const int* off, const int* cnt, int* partners, uint64_t* keys,
                               int capacity) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int o = off[i], c = cnt[i];
    if (o + c > capacity) return;
    unsigned* p = (unsigned*)partners + o;
    if (w.hasCompound) {
        int np = 0;
        for (int k = 0; k < c; k++)
            if ((p[k] >> 24) == 0) p[np++] = p[k];   // in place: np <= k
        sort_words(p, np);
        const uint64_t hi = (uint64_t)(unsigned)i << 32;
        int at = 0, more = 1;
        for (unsigned sub = 0; more && at < c; sub++) {
            more = 0;
            for (int k = 0; k < np; k++) {
                const int subs = pair_subs(w.sh, w.shape[i], w.shape[p[k]]);
                if ((int)sub < subs) {
                    keys[o + at++] = hi | (sub << 24) | p[k];
                    more |= (int)sub + 1 < subs;
                }
            }
        }
        return;
    }
    if (c <= 32) {
        unsigned v[32];
        for (int k = 0; k < c; k++) v[k] = p[k];
        for (int k = 1; k < c; k++) {
            unsigned x = v[k];
            int j = k - 1;
            while (j >= 0 && v[j] > x) { v[j + 1] = v[j]; j--; }
            v[j + 1] = x;
        }
        for (int k = 0; k < c; k++) keys[o + k] = ((uint64_t)(unsigned)i << 32) | v[k];
    } else {
        for (int gap = c / 2; gap > 0; gap /= 2)          // Shell sort for rare crowded owners
            for (int k = gap; k < c; k++) {
                unsigned x = p[k];
                int j = k;
                while (j >= gap && p[j - gap] > x) { p[j] = p[j - gap]; j -= gap; }
                p[j] = x;
            }
        for (int k = 0; k < c; k++) keys[o + k] = ((uint64_t)(unsigned)i << 32) | p[k];
    }
}

// The same for worlds without compounds, in two passes.  A thread per owner sorts a segment of up
// to SEG_REG partner words in registers (a bitonic network over 8, padding words 0xffffffff
// sorting last) and lists the owners of longer segments; then a warp per listed owner sorts up
// to 32 words across the lanes by a bitonic network, a crowded segment in place by one lane.
constexpr int SEG_REG = 8;
__global__ void k_segment_sort_short(int n, const int* off, const int* cnt, const int* partners, uint64_t* keys,
                                     int capacity, int* longList, int* longCount) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;   // the grid covers whole warps
    int o = 0, c = 0;
    if (i < n) {
        o = off[i];
        c = cnt[i];
        if (o + c > capacity) c = 0;
    }
    if (c > 0 && c <= SEG_REG) {
        const unsigned* p = (const unsigned*)partners + o;
        unsigned r[SEG_REG];
#pragma unroll
        for (int k = 0; k < SEG_REG; k++) r[k] = k < c ? p[k] : 0xffffffffu;
#pragma unroll
        for (int k = 2; k <= SEG_REG; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
                for (int a = 0; a < SEG_REG; a++) {
                    const int b = a ^ j;
                    if (b > a) {
                        const unsigned x = r[a], y = r[b];
                        if ((x > y) == ((a & k) == 0)) { r[a] = y; r[b] = x; }
                    }
                }
        const uint64_t hi = (uint64_t)(unsigned)i << 32;
#pragma unroll
        for (int k = 0; k < SEG_REG; k++)
            if (k < c) keys[o + k] = hi | r[k];
    }
    const bool lng = c > SEG_REG;
    const unsigned m = __ballot_sync(0xffffffffu, lng);
    if (m) {
        const int leader = __ffs(m) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(longCount, __popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (lng) longList[base + __popc(m & ((1u << lane) - 1u))] = i;
    }
}
__global__ void k_segment_sort_long(const int* off, const int* cnt, int* partners, uint64_t* keys, const int* longList,
                                    const int* longCount) {
    const int lane = threadIdx.x & 31;
    const int nl = *longCount, nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); q < nl; q += nw) {   // uniform per warp
        const int i = longList[q], o = off[i], c = cnt[i];
        const uint64_t hi = (uint64_t)(unsigned)i << 32;
        unsigned* p = (unsigned*)partners + o;
        if (c <= 32) {
            unsigned v = lane < c ? p[lane] : 0xffffffffu;
            for (int k = 2; k <= 32; k <<= 1)
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const unsigned u = __shfl_xor_sync(0xffffffffu, v, j);
                    v = (((lane & j) == 0) == ((lane & k) == 0)) ? min(v, u) : max(v, u);
                }
            if (lane < c) keys[o + lane] = hi | v;
        } else {
            if (lane == 0)
                for (int gap = c / 2; gap > 0; gap /= 2)   // Shell sort for rare crowded owners
                    for (int k = gap; k < c; k++) {
                        const unsigned x = p[k];
                        int j = k;
                        while (j >= gap && p[j - gap] > x) { p[j] = p[j - gap]; j -= gap; }
                        p[j] = x;
                    }
            __syncwarp();
            for (int k = lane; k < c; k += 32) keys[o + k] = hi | p[k];
            __syncwarp();
        }
    }
}

// Carry the manifold of the lane's pair p over when it persists: its key is searched in
// old.keys[lo .. hi].  The warp then copies its pairs' points together, a lane a point (four lanes
// read a pair's 64 bytes of each array): a lane a pair, every lane on lines of its own, took 347 us
// for 1.9 million pairs, 257 us so.  By whole warps.
JBD void persist_warp(const DevWorld& w, DevPairs& nw, const DevPairs& old, bool valid, int p, uint64_t key, int lo, int hi) {
    const int lane = threadIdx.x & 31;
    int found = -1, n = 0;
    if (valid) {
        while (lo <= hi) {
            int mid = (lo + hi) >> 1;
            uint64_t k = old.keys[mid];
            if (k == key) { found = mid; break; }
            if (k < key) lo = mid + 1; else hi = mid - 1;
        }
        int mb0, mb1;
        const int has = found >= 0 && old.has[found] ? 1 : 0;
        if (has) {
            n = old.n[found];
            mb0 = old.b0[found];
            mb1 = old.b1[found];
        } else {
            const int a = key_owner(key), b = key_partner(key);
            manifold_bodies(a, b, w.sh.type[w.shape[min(a, b)]], w.sh.type[w.shape[max(a, b)]], mb0, mb1);
        }
        nw.has[p] = has;
        nw.steps[p] = has ? old.steps[found] : 0;
        nw.n[p] = n;
        nw.b0[p] = mb0;
        nw.b1[p] = mb1;
    }
    unsigned left = __ballot_sync(0xffffffffu, n > 0);
    while (left) {   // eight pairs with points at a time
        unsigned m = left;
        int src = -1;
        for (int q = 0; q < 8 && m; q++, m &= m - 1)
            if (q == lane >> 2) src = __ffs(m) - 1;
        left = m;
        const int from = max(src, 0);
        const int so = __shfl_sync(0xffffffffu, found, from), d0 = __shfl_sync(0xffffffffu, p, from);
        const int cnt = __shfl_sync(0xffffffffu, n, from);
        if (src >= 0 && (lane & 3) < cnt) {
            const size_t s = (size_t)so * 4 + (lane & 3), d = (size_t)d0 * 4 + (lane & 3);
            const float4 x0 = old.pA[s], x1 = old.pB[s], x2 = old.wA[s], x3 = old.wB[s];
            const float4 x4 = old.nrm[s], x5 = old.imp[s], x6 = old.d1[s], x7 = old.d2[s];
            nw.pA[d] = x0; nw.pB[d] = x1; nw.wA[d] = x2; nw.wB[d] = x3;
            nw.nrm[d] = x4; nw.imp[d] = x5; nw.d1[d] = x6; nw.d2[d] = x7;
        }
    }
}

// The range of old.keys that can hold a key of owner o: its segment of last step's per-owner offsets
// when they are at hand, else all of them.
JBD void persist_range(const int* offPrev, int nOld, int o, int& lo, int& hi) {
    lo = offPrev ? offPrev[o] : 0;
    hi = (offPrev ? min(offPrev[o + 1], nOld) : nOld) - 1;
}

__global__ void k_persist(DevWorld w, DevPairs nw, DevPairs old, int nNew, int nOld, const int* offPrev, const int* newCnt,
                          const int* oldCnt) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (newCnt) nNew = min(nNew, *newCnt);
    if (oldCnt) nOld = min(nOld, *oldCnt);
    if ((p & ~31) >= nNew) return;   // whole warps
    const bool valid = p < nNew;
    const uint64_t key = valid ? nw.keys[p] : 0;
    int lo = 0, hi = -1;
    if (valid) persist_range(offPrev, nOld, key_owner(key), lo, hi);
    persist_warp(w, nw, old, valid, p, key, lo, hi);
}

// ---- direct pairs ----------------------------------------------------------------------------
// Small worlds without the tree: a warp per owner tests the bodies of its world that can be its
// partners - listed bodies (planes, meshes) and finite bodies of a higher index - 32 at a time in
// index order, so that its keys come out sorted.  What the tree costs instead, however small the
// world: a chain of dependent launches (sort, topology, refit, two traversals, two segment sorts),
// a refit that climbs the tree one node at a time and a walk by a single lane.
// The eight owners of a block are neighbours in the list and share its boxes, DIRECT_TILE at a time
// in shared memory with the next tile's on their way: with every warp reading its own from L2 the
// count of 4,000 hulls took 69 us, 40 us so.
constexpr int DIRECT_THREADS = 256, DIRECT_TILE = 256;
struct DirectTile {
    float mn[3][DIRECT_TILE], mx[3][DIRECT_TILE];
    int body[DIRECT_TILE];
    int end;
};

// f(j, hit) by all lanes of the owner's warp for 32 candidates j (hit: overlapping, filter passed) at a
// time, ascending.  q: the owner's place in the list; called by whole blocks, `active` per warp.
template <class F>
JBD void direct_partners(const DevWorld& w, const DirectList& dl, const int* planeList, const int* planeStart, int q,
                         bool active, DirectTile& t, F&& f) {
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    const int first = q - (tid >> 5) + 1;   // the block's first owner + 1
    int i = 0, end = 0;
    float4 a0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), a1 = a0;
    if (tid == 0) t.end = 0;
    __syncthreads();
    if (active) {
        i = dl.body[q];
        const int wi = w.world[i];
        end = dl.end[wi];
        a0 = w.amin[i];
        a1 = w.amax[i];
        if (lane == 0) atomicMax(&t.end, end);
        for (int k = planeStart[wi]; k < planeStart[wi + 1]; k += 32) {   // listed bodies before i
            const int j = k + lane < planeStart[wi + 1] ? planeList[k + lane] : i;
            f(j, j < i && ovl(a0, a1, w.amin[j], w.amax[j]) && filt(w, i, j));
        }
    }
    __syncthreads();
    const int last = t.end;
    int j = 0;
    float4 b0, b1;
    auto load = [&](int base) {
        if (base + tid >= last) return;
        j = dl.body[base + tid];
        b0 = w.amin[j];
        b1 = w.amax[j];
    };
    load(first);
    for (int base = first; base < last; base += DIRECT_TILE) {            // every body after i
        if (base + tid < last) {
            t.mn[0][tid] = b0.x; t.mn[1][tid] = b0.y; t.mn[2][tid] = b0.z;
            t.mx[0][tid] = b1.x; t.mx[1][tid] = b1.y; t.mx[2][tid] = b1.z;
            t.body[tid] = j;
        }
        __syncthreads();
        load(base + DIRECT_TILE);
        if (base < end) {
            unsigned hits = 0;   // of the lane, a bit per 32 boxes; no branch between the loads
#pragma unroll
            for (int c = 0; c < DIRECT_TILE / 32; c++) {
                const int e = 32 * c + lane, k = base + e;
                const bool hit = (k > q) & (k < end) & (a0.x <= t.mx[0][e]) & (a1.x >= t.mn[0][e]) & (a0.y <= t.mx[1][e]) &
                                 (a1.y >= t.mn[1][e]) & (a0.z <= t.mx[2][e]) & (a1.z >= t.mn[2][e]);
                hits |= hit ? 1u << c : 0u;
            }
            for (unsigned any = __reduce_or_sync(0xffffffffu, hits); any; any &= any - 1) {
                const int c = __ffs(any) - 1, other = t.body[32 * c + lane];
                f(other, ((hits >> c) & 1) && filt(w, i, other));
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(DIRECT_THREADS) k_direct_count(DevWorld w, DirectList dl, const int* planeList,
                                                                 const int* planeStart, int* cnt, int* tcount, int* kept) {
    __shared__ DirectTile t;
    const int lane = threadIdx.x & 31;
    const int q = (blockIdx.x * DIRECT_THREADS + threadIdx.x) >> 5;
    const int i = q < w.nBodies ? dl.body[q] : w.nBodies;   // the entry past the bodies counts none
    const bool active = q < w.nBodies && !(w.flags[i] & CF_LISTED);
    int c = 0, found = 0;
    direct_partners(w, dl, planeList, planeStart, q, active, t, [&](int j, bool hit) {
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        const int d = found + __popc(m & ((1u << lane) - 1u));
        if (hit && d < DIRECT_CACHE) kept[(size_t)i * DIRECT_CACHE + d] = j;
        found += __popc(m);
        if (hit && w.hasCompound) c += pair_subs(w.sh, w.shape[i], w.shape[j]);
    });
    if (w.hasCompound) c = __reduce_add_sync(0xffffffffu, c);
    else c = found;
    if (lane == 0 && q <= w.nBodies) {
        cnt[i] = c;
        if (q < w.nBodies) tcount[i] = found;
    }
}

// The concave pass's candidates, bounded (see k_plane_pairs), by a warp a body: 55 us by a thread each for
// 4,000 bodies on a triangle-mesh landscape, 36 us so.
__global__ void __launch_bounds__(128) k_mesh_bound(DevWorld w, const int* planeList, const int* planeStart, int* candBound) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= w.nBodies || (w.flags[i] & CF_LISTED)) return;
    const int wi = w.world[i];
    int total = 0;
    for (int k = planeStart[wi]; k < planeStart[wi + 1]; k++) {
        const int p = planeList[k];
        if (!ovl(w.amin[i], w.amax[i], w.amin[p], w.amax[p]) || !filt(w, i, p)) continue;
        total += mesh_candidates(w, i, p, [&](const Leaf& l, const Leaf& t) { return mesh_walk_warp(w, l, t, 0, nullptr); });
    }
    if ((threadIdx.x & 31) == 0 && total) atomicAdd(candBound, total);
}

// Keys and persistence of an owner's pairs: the partners the count kept, or tested again when there
// were more.  With compounds the keys go by child combination, then by partner.
__global__ void __launch_bounds__(DIRECT_THREADS) k_direct_fill(DevWorld w, DirectList dl, const int* planeList,
                                                                const int* planeStart, const int* off, const int* tcount,
                                                                const int* kept, int* partners, DevPairs nw, DevPairs old,
                                                                int capacity, int nOld, const int* offPrev,
                                                                const int* oldCnt) {
    __shared__ DirectTile t;
    const int lane = threadIdx.x & 31;
    const int q = (blockIdx.x * DIRECT_THREADS + threadIdx.x) >> 5;
    const int i = q < w.nBodies ? dl.body[q] : 0;
    int o = 0, c = 0, found = 0;
    if (q < w.nBodies && !(w.flags[i] & CF_LISTED)) {
        o = off[i];
        c = off[i + 1] - o;
        found = tcount[i];
        if (o + c > capacity) c = 0;
    }
    const uint64_t owner = (uint64_t)(unsigned)i << 32;
    const bool again = c > 0 && found > DIRECT_CACHE;
    const int* list = again ? partners + o : kept + (size_t)i * DIRECT_CACHE;
    if (__syncthreads_or(again)) {
        int at = o;
        direct_partners(w, dl, planeList, planeStart, q, again, t, [&](int j, bool hit) {
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (hit) partners[at + __popc(m & ((1u << lane) - 1u))] = j;
            at += __popc(m);
        });
        __syncwarp();
    }
    if (c == 0) return;
    if (oldCnt) nOld = min(nOld, *oldCnt);
    int lo, hi;
    persist_range(offPrev, nOld, i, lo, hi);
    int at = o;
    for (int sub = 0; at < o + c; sub++) {
        const int before = at;
        for (int k = 0; k < found; k += 32) {
            const int j = k + lane < found ? list[k + lane] : -1;
            const bool put = j >= 0 && (sub == 0 || sub < pair_subs(w.sh, w.shape[i], w.shape[j]));
            const unsigned m = __ballot_sync(0xffffffffu, put);
            const int p = at + __popc(m & ((1u << lane) - 1u));
            const uint64_t key = owner | ((unsigned)sub << 24) | (unsigned)j;
            if (put) nw.keys[p] = key;
            persist_warp(w, nw, old, put, p, key, lo, hi);
            at += __popc(m);
        }
        if (at == before) break;
    }
}

static inline int gridn(int n, int b) { return (n + b - 1) / b; }

// The bodies' Morton order is renewed every rebuildInterval steps, and with it the tree's topology;
// in between the tree is only refitted to the new AABBs: a refitted tree bounds every body exactly,
// so the traversal finds the same pair set whatever the tree's shape; only its cost depends on how
// stale the order is.
// The order: Morton keys of the current w.amin/w.amax centres (the batch world in the high bits),
// sorted.
void broadphase_order(const DevWorld& w, BroadphaseBuffers& bb, cudaStream_t s) {
    const int n = w.nBodies;
    bb.built = true;
    bb.treeBuilt = false;
    bb.sinceBuild = 0;
    if (n <= ORDER_SMALL && bb.worldBits <= ORDER_WORLD_BITS) {
        int size = 32;
        while (size < n) size <<= 1;
        auto k = size <= ORDER_THREADS ? k_order_small<1> : size == 2 * ORDER_THREADS ? k_order_small<2> : k_order_small<4>;
        k<<<1, std::min(size, ORDER_THREADS), 0, s>>>(w, bb.mkeys, bb.sortedBody); note_launch();
        return;
    }
    cudaMemsetAsync(bb.bounds, 0, sizeof(unsigned) * 6, s);
    cudaMemsetAsync(bb.bounds, 0xff, sizeof(unsigned) * 3, s);
    k_bounds<<<gridn(n, 256), 256, 0, s>>>(w, bb.bounds); note_launch();
    k_morton<<<gridn(n, 256), 256, 0, s>>>(w, bb.bounds, bb.mkeys, bb.sortedBody); note_launch();
    radix_sort_pairs(bb.mkeys, bb.sortedBody, bb.mkeys_alt, bb.vals_alt, n, 32 + bb.worldBits, bb.sortScratch, s);
}

// The tree over the current order: world leaf ranges, Karras topology.  Boxes are written by a refit.
void broadphase_topology(BroadphaseBuffers& bb, cudaStream_t s) {
    const int nf = bb.nFinite;
    bb.treeBuilt = true;
    cudaMemsetAsync(bb.wroot, 0xff, sizeof(int) * bb.nWorlds, s);   // no root: worlds of listed bodies alone
    if (nf > 0) {
        cudaMemsetAsync(bb.wstart, 0xff, sizeof(int) * bb.nWorlds, s);
        cudaMemsetAsync(bb.wend, 0xff, sizeof(int) * bb.nWorlds, s);
        k_world_ranges<<<gridn(nf, 256), 256, 0, s>>>(bb.mkeys, nf, bb.wstart, bb.wend, bb.wroot); note_launch();
        if (nf > 1) {
            cudaMemsetAsync(bb.bvh.parent, 0xff, sizeof(int) * (nf - 1), s);
            cudaMemsetAsync(bb.bvh.leafParent, 0xff, sizeof(int) * nf, s);   // single-leaf worlds keep -1
            k_karras<<<gridn(nf - 1, 256), 256, 0, s>>>(bb.mkeys, nf, bb.bvh, bb.wstart, bb.wend, bb.wroot); note_launch();
        }
    }
}

// Refit of the current tree topology over the boxes in wq.amin / wq.amax into another node
// record array (the broadphase's own records are left as they are).
void broadphase_refit_into(const DevWorld& wq, const BroadphaseBuffers& bb, float4* node, int* visit, cudaStream_t s) {
    const int nf = bb.nFinite;
    if (nf < 2) return;
    Bvh t = bb.bvh;
    t.node = node;
    t.visit = visit;
    cudaMemsetAsync(visit, 0, sizeof(int) * (nf - 1), s);
    k_refit<<<gridn(nf, 256), 256, 0, s>>>(wq, bb.sortedBody, nf, t); note_launch();
}

bool broadphase_rebuilds(const BroadphaseBuffers& bb) { return !(bb.built && bb.sinceBuild + 1 < bb.rebuildInterval); }

// A query on bodies changed since the last step makes the order and, when it needs none, leaves the tree.
bool broadphase_makes_tree(const BroadphaseBuffers& bb) {
    return !bb.direct && (!bb.treeBuilt || broadphase_rebuilds(bb));
}

void broadphase_run_count(const DevWorld& w, BroadphaseBuffers& bb, cudaStream_t s) {
    const int n = w.nBodies, nf = bb.nFinite;
    const bool tree = broadphase_makes_tree(bb);
    if (broadphase_rebuilds(bb)) broadphase_order(w, bb, s);
    else bb.sinceBuild++;
    if (tree) broadphase_topology(bb, s);
    if (bb.meshes) cudaMemsetAsync(bb.candBound, 0, sizeof(int), s);   // else it stays 0
    if (bb.direct) {
        k_direct_count<<<gridn(n + 1, DIRECT_THREADS / 32), DIRECT_THREADS, 0, s>>>(w, bb.list, bb.planeList, bb.planeStart,
                                                                                    bb.cnt, bb.tcount, bb.kept);
        note_launch();
        if (bb.meshes) {
            k_mesh_bound<<<gridn(n, 4), 128, 0, s>>>(w, bb.planeList, bb.planeStart, bb.candBound); note_launch();
        }
    } else {
        cudaMemsetAsync(bb.cnt, 0, sizeof(int) * (n + 1), s);
        if (nf > 1) {
            cudaMemsetAsync(bb.bvh.visit, 0, sizeof(int) * (nf - 1), s);
            k_refit<<<gridn(nf, 256), 256, 0, s>>>(w, bb.sortedBody, nf, bb.bvh); note_launch();
            k_traverse<false><<<gridn(nf, 128), 128, 0, s>>>(w, bb.sortedBody, nf, bb.bvh, bb.wroot, bb.cnt, nullptr,
                                                              nullptr, nullptr, 0, bb.tcount, bb.tcache); note_launch();
        }
        if (bb.nPlanes > 0)
            k_plane_pairs<false><<<gridn(n, 256), 256, 0, s>>>(w, bb.planeList, bb.planeStart, bb.cnt, nullptr, nullptr,
                                                                nullptr, 0, bb.candBound); note_launch();
    }
    exclusive_scan(bb.cnt, bb.off, bb.total, n + 1, bb.scanScratch, s);
}

// Count and fill, us, tree / direct: 60 bodies 85 / 30, 1,000 131 / 40, 4,000 hulls 287 / 100, 256
// worlds of 17 bodies 169 / 85; 20,000 252 / 312; 1,024 worlds of 433 bodies 710 / 1184 - the count
// pays for 32 tests at a time (steps) and the fill for a warp an owner.
bool broadphase_direct(const std::vector<int>& bodies, const std::vector<int>& finite) {
    double steps = 0.0, owners = 0.0;
    for (size_t k = 0; k < bodies.size(); k++) {
        steps += finite[k] * (1.0 + bodies[k] / 64.0);
        owners += finite[k];
    }
    return owners <= 32768.0 && steps <= 1.0e6;
}

static void tree_fill(const DevWorld& w, BroadphaseBuffers& bb, DevPairs& nw, int capacity, cudaStream_t s) {
    int n = w.nBodies, nf = bb.nFinite;
    cudaMemsetAsync(bb.cursor, 0, sizeof(int) * (n + 1), s);
    // counts are recovered from the offsets: cnt[i] = off[i+1] - off[i]
    if (nf > 1)
        k_traverse<true><<<gridn(nf, 128), 128, 0, s>>>(w, bb.sortedBody, nf, bb.bvh, bb.wroot, nullptr, bb.off,
                                                         bb.cursor, bb.partners, capacity, bb.tcount, bb.tcache); note_launch();
    if (bb.nPlanes > 0)
        k_plane_pairs<true><<<gridn(n, 256), 256, 0, s>>>(w, bb.planeList, bb.planeStart, nullptr, bb.off, bb.cursor,
                                                           bb.partners, capacity, nullptr); note_launch();
    if (w.hasCompound) {
        k_segment_sort<<<gridn(n, 128), 128, 0, s>>>(w, n, bb.off, bb.cursor, bb.partners, nw.keys, capacity);
    } else {
        // the long segments' owners are listed in tcount, which the filling traversal has read
        cudaMemsetAsync(bb.segLong, 0, sizeof(int), s);
        k_segment_sort_short<<<gridn(n, 128), 128, 0, s>>>(n, bb.off, bb.cursor, bb.partners, nw.keys, capacity,
                                                            bb.tcount, bb.segLong);
        note_launch();
        k_segment_sort_long<<<std::min(gridn(n, 4), 1024), 128, 0, s>>>(bb.off, bb.cursor, bb.partners, nw.keys,
                                                                        bb.tcount, bb.segLong);
    }
    note_launch();
}

void broadphase_fill(const DevWorld& w, BroadphaseBuffers& bb, DevPairs& nw, const DevPairs& old, int capacity, int nNew,
                     int nOld, cudaStream_t s, const int* newCnt, const int* oldCnt) {
    const int* offPrev = bb.offPrevValid ? bb.offPrev : nullptr;
    if (bb.direct) {
        k_direct_fill<<<gridn(w.nBodies, DIRECT_THREADS / 32), DIRECT_THREADS, 0, s>>>(
            w, bb.list, bb.planeList, bb.planeStart, bb.off, bb.tcount, bb.kept, bb.partners, nw, old, capacity, nOld,
            offPrev, oldCnt);
        note_launch();
    } else {
        tree_fill(w, bb, nw, capacity, s);
        if (nNew > 0) {
            k_persist<<<gridn(nNew, 256), 256, 0, s>>>(w, nw, old, nNew, nOld, offPrev, newCnt, oldCnt);
            note_launch();
        }
    }
    std::swap(bb.off, bb.offPrev);   // this step's offsets index the pair array the next step persists from
    bb.offPrevValid = true;
}

}  // namespace jbg
