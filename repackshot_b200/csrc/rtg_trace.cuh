// Ray queries on the device: the watertight triangle test, the quantised 8-wide slab test and
// the two-level closest-hit / any-hit traversal (engine/crates/rt-core/src/geometry/
// triangle.rs:60-160, traverse.rs:47-802), and the hit details of geometry/mod.rs:682-808.
//
// The answer of a nearest-hit query is the smallest (t, instance, triangle) in lexicographic
// order over the triangles the ray meets in [t_min, t_max] whose enclosing boxes pass the
// reference's slab test. Those boxes are not always conservative: a computed t may lie inside the
// interval while its triangle's flat box begins past t_max or ends before t_min, and the reference
// drops that hit. So the tree is walked with a cheaper slab test that passes every box the
// reference's passes (and a few more), and a leaf's first hit puts the leaf's exact box to the
// reference's own test (box_kept); an instance's world box is put to it before its tree is walked.
// Boxes further up contain these, and rounding is monotonic, so they pass when these pass.
#pragma once
#include "rtg_dev.h"

namespace rtg {

constexpr int STACK_CAP = 96;
constexpr uint32_t STACK_RETURN = 0xfffffffeu;
#define RTG_ROBUST 1.00000047683715820312f  // 1 + 4 f32::EPSILON (Ize 2013)

struct PRay {
    float org[3], inv[3];
    bool neg[3];
    int kx, ky, kz;
    float sx, sy, sz;
    float tmin, tmax;
};

RTG_D PRay prepare_ray(V3 o, V3 d, float tmin, float tmax) {  // triangle.rs:60
    PRay r;
    float dd[3] = {d.x, d.y, d.z};
    r.inv[0] = __frcp_rn(d.x);  // 1 / d, correctly rounded (the division's IEEE result)
    r.inv[1] = __frcp_rn(d.y);
    r.inv[2] = __frcp_rn(d.z);
    float a0 = absf(d.x), a1 = absf(d.y), a2 = absf(d.z);
    int kz = (a0 >= a1 && a0 >= a2) ? 0 : (a1 >= a2 ? 1 : 2);
    int kx = (kz + 1) % 3, ky = (kz + 2) % 3;
    if (dd[kz] < 0.0f) { int t = kx; kx = ky; ky = t; }
    float sz = r.inv[kz];
    r.org[0] = o.x; r.org[1] = o.y; r.org[2] = o.z;
    r.neg[0] = signbitf(r.inv[0]);
    r.neg[1] = signbitf(r.inv[1]);
    r.neg[2] = signbitf(r.inv[2]);
    r.kx = kx; r.ky = ky; r.kz = kz;
    r.sx = dd[kx] * sz;
    r.sy = dd[ky] * sz;
    r.sz = sz;
    r.tmin = tmin;
    r.tmax = rmin(tmax, F_MAX);
    return r;
}
RTG_D float pick3(const float* v, int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); }

// The scalar watertight test (triangle.rs:123), the reference's operations in its order.
RTG_D bool watertight(const PRay& r, const float* v0, const float* v1, const float* v2, float tmax, bool cull_back,
                      float& t, float& u, float& v, float& w, float& det) {
    float ox = r.org[r.kx], oy = r.org[r.ky], oz = r.org[r.kz];
    float a_x = pick3(v0, r.kx) - ox, a_y = pick3(v0, r.ky) - oy, a_z = pick3(v0, r.kz) - oz;
    float b_x = pick3(v1, r.kx) - ox, b_y = pick3(v1, r.ky) - oy, b_z = pick3(v1, r.kz) - oz;
    float c_x = pick3(v2, r.kx) - ox, c_y = pick3(v2, r.ky) - oy, c_z = pick3(v2, r.kz) - oz;
    float ax = a_x - r.sx * a_z, ay = a_y - r.sy * a_z;
    float bx = b_x - r.sx * b_z, by = b_y - r.sy * b_z;
    float cx = c_x - r.sx * c_z, cy = c_y - r.sy * c_z;
    u = cx * by - cy * bx;
    v = ax * cy - ay * cx;
    w = bx * ay - by * ax;
    bool negative = u < 0.0f || v < 0.0f || w < 0.0f;
    bool positive = u > 0.0f || v > 0.0f || w > 0.0f;
    bool rejected = cull_back ? negative : (negative && positive);
    det = u + v + w;
    if (rejected || det == 0.0f) return false;
    float az = r.sz * a_z, bz = r.sz * b_z, cz = r.sz * c_z;
    t = (u * az + v * bz + w * cz) / det;
    return t >= r.tmin && t <= tmax;
}

RTG_D float smax_(float a, float b) { return a > b ? a : b; }
RTG_D float smin_(float a, float b) { return a < b ? a : b; }

RTG_D uint64_t stack_key(float t, uint32_t ref) { return ((uint64_t)__float_as_uint(t) << 32) | (uint64_t)ref; }

RTG_D V3 xf_point(const float* m, V3 p) {
    return v3(m[0] * p.x + m[1] * p.y + m[2] * p.z + m[3], m[4] * p.x + m[5] * p.y + m[6] * p.z + m[7],
              m[8] * p.x + m[9] * p.y + m[10] * p.z + m[11]);
}
RTG_D V3 xf_vector(const float* m, V3 v) {
    return v3(m[0] * v.x + m[1] * v.y + m[2] * v.z, m[4] * v.x + m[5] * v.y + m[6] * v.z, m[8] * v.x + m[9] * v.y + m[10] * v.z);
}
RTG_D V3 xf_transpose(const float* m, V3 v) {
    return v3(m[0] * v.x + m[4] * v.y + m[8] * v.z, m[1] * v.x + m[5] * v.y + m[9] * v.z, m[2] * v.x + m[6] * v.y + m[10] * v.z);
}

struct TraceResult { uint32_t inst, tri; float t; };  // tri: the leaf triangle (SceneDev::tris)

// A traversal stack whose first SHORT_STACK entries sit in shared memory, interleaved by thread
// (entry k of thread i at sm[k * stride + i]), and the deeper ones in a per-thread array. Almost
// every ray stays within the shared part.
// A build may set RTG_SHORT_STACK to trade shared memory (8 bytes x 128 threads per entry and
// block) against spills to the deeper part. 16 entries (16 KB a block) leave 128 KB of the SM's
// shared memory to L1 at 8 blocks per SM, where the node fetches hit; 10, 16 and 24 entries measured
// 193.1, 192.7 and 193.4 ms on the 1080p product frame.
#ifndef RTG_SHORT_STACK
#define RTG_SHORT_STACK 16
#endif
constexpr int SHORT_STACK = RTG_SHORT_STACK;
struct SplitStack {
    uint64_t* sm;   // this thread's column of the shared block
    uint64_t* deep; // STACK_CAP - SHORT_STACK entries
    int stride;
    RTG_D void put(int k, uint64_t v) {
        if (k < SHORT_STACK) sm[k * stride] = v;
        else deep[k - SHORT_STACK] = v;
    }
    RTG_D uint64_t get(int k) const { return k < SHORT_STACK ? sm[k * stride] : deep[k - SHORT_STACK]; }
};

// The traversal state of one ray, advanced one step (trav_node, trav_leaf) at a time. A kernel can then give
// a lane whose ray has finished a new ray while the rest of its warp keeps traversing. The state
// is kept small (the traversal kernels run at 64 registers): the world ray is read again from
// where the query came from (`src`) on the rare ways into and out of a transformed instance.
constexpr uint32_t TLAS_LEVEL = 0xffffffffu;
struct Trav {
    float org[3], inv[3];  // the ray in the space of the tree being walked; inv is clamped (trav_ray)
    float sx, sy, sz;      // the watertight test's shear
    int kz;                // its major axis; the other two follow in cyclic order
    bool flip;             // the direction runs down the major axis: the reference swaps the other two
    bool camera;
    bool any;              // TRACE_EITHER: this ray's query is any-hit
    float best_t;          // nearest hit so far (any-hit queries: t_max)
    uint32_t best_i, best_k, cur;  // its instance and leaf triangle
    uint32_t blas;         // the BLAS being walked: index << 3 | moved << 2 | flags; TLAS_LEVEL: none
    int sp;
};
constexpr uint32_t BLAS_MOVED = 4u;  // its ray is in a transformed instance's object space

constexpr float INV_MOST = 1.152921504606847e18f;  // 2^60
// Sets the state's ray. The slab test's reciprocals are clamped to 2^60 times the major axis's, so
// that a zero component gives no 0 x inf: such an axis then bounds t by planes 2^60 times as far as
// the ray's major axis goes, which only a box the origin's coordinate lies outside of can fail.
RTG_D void trav_ray(Trav& T, V3 o, V3 d) {
    const float i0 = __frcp_rn(d.x), i1 = __frcp_rn(d.y), i2 = __frcp_rn(d.z);  // 1 / d, correctly rounded
    const float a0 = absf(d.x), a1 = absf(d.y), a2 = absf(d.z);
    const int kz = (a0 >= a1 && a0 >= a2) ? 0 : (a1 >= a2 ? 1 : 2);  // triangle.rs:60
    const float dk = kz == 0 ? d.x : (kz == 1 ? d.y : d.z), dx = kz == 0 ? d.y : (kz == 1 ? d.z : d.x),
                dy = kz == 0 ? d.z : (kz == 1 ? d.x : d.y);
    const float sz = kz == 0 ? i0 : (kz == 1 ? i1 : i2);
    T.org[0] = o.x; T.org[1] = o.y; T.org[2] = o.z;
    const float most = absf(sz) * INV_MOST;
    T.inv[0] = copysign_(smin_(absf(i0), most), i0);
    T.inv[1] = copysign_(smin_(absf(i1), most), i1);
    T.inv[2] = copysign_(smin_(absf(i2), most), i2);
    T.kz = kz;
    T.flip = dk < 0.0f;
    T.sx = dx * sz;
    T.sy = dy * sz;
    T.sz = sz;
}

// Sets up a query. False when the ray can meet nothing (non-finite or zero direction, empty
// interval): a miss.
RTG_D bool trav_init(const SceneDev& S, Trav& T, V3 o, V3 d, float tmin, float tmax, bool camera) {
    if (!(vfinite(o) && vfinite(d) && !veq(d, v3(0, 0, 0)))) return false;
    T.best_t = rmin(tmax, F_MAX);
    if (!(tmin <= T.best_t)) return false;
    trav_ray(T, o, d);
    T.best_i = 0xffffffffu;
    T.best_k = 0xffffffffu;
    T.sp = 0;
    T.camera = camera;
    T.cur = S.tlas_root;
    T.blas = S.single_blas;  // 0 (BLAS 0 unmoved, no flags) when the scene is one world-space tree
    return true;
}

// 32 bytes, a whole sector, in one load.
RTG_D void load32(const void* p, uint32_t v[8]) {
#ifdef __CUDA_ARCH__
    uint64_t d[4];
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(d[0]), "=l"(d[1]), "=l"(d[2]), "=l"(d[3]) : "l"(p));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[2 * k] = (uint32_t)d[k];
        v[2 * k + 1] = (uint32_t)(d[k] >> 32);
    }
#else
    std::memcpy(v, p, 32);
#endif
}
// The reference's slab test of the box [lo, hi] over [tmin, tmax], its operations in its order
// (traverse.rs:184).
RTG_D bool slab_passes(V3 lo, V3 hi, V3 org, V3 inv, float tmin, float tmax) {
    float n = tmin, f = tmax;
    const auto axis = [&](float l, float h, float o, float i) {
        const bool neg = signbitf(i);
        n = smax_(((neg ? h : l) - o) * i, n);
        f = smin_(((neg ? l : h) - o) * i, f);
    };
    axis(lo.x, hi.x, org.x, inv.x);
    axis(lo.y, hi.y, org.y, inv.y);
    axis(lo.z, hi.z, org.z, inv.z);
    return n <= f * RTG_ROBUST;
}
// The same for a ray with a clamped reciprocal (trav_ray), from its direction: the query's, `d`,
// taken into the tree of `blas`. Out of line: such rays run almost along a plane of the axes.
RTG_D_NI bool slab_passes_axial(const BlasInst* __restrict__ blases, V3 lo, V3 hi, V3 org, V3 d, uint32_t blas, float tmin, float tmax) {
    if (blas != TLAS_LEVEL && (blas & BLAS_MOVED)) {
        float m[12];
        for (int k = 0; k < 12; ++k) m[k] = __ldg(&blases[blas >> 3].to_local[k]);
        d = xf_vector(m, d);
    }
    return slab_passes(lo, hi, org, v3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z)), tmin, tmax);
}
// Whether the reference's slab test passes the box at `at` (lower corner in [0, 3), upper in [4, 7))
// for the ray of the tree being walked. A load and some forty instructions a leaf with a hit, and the same
// an instance entered: against a test of hits near t_min only, which let hits past t_max through, the
// 1080p product frame went from 151.3 to 155.8 ms, the instanced frame from 31.8 to 33.8 ms. The test with
// min and max in place of the sign's selects, or put off to the end of the leaf, took as long.
template <class Src>
RTG_D bool box_kept(const SceneDev& S, const Trav& T, const float* at, float tmin, float tmax, const Src& src) {
    uint32_t v[8];
    load32(at, v);
    const V3 lo = v3(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]));
    const V3 hi = v3(__uint_as_float(v[4]), __uint_as_float(v[5]), __uint_as_float(v[6]));
    const V3 org = v3(T.org[0], T.org[1], T.org[2]), inv = v3(T.inv[0], T.inv[1], T.inv[2]);
    if (!(fmaxf(fmaxf(absf(inv.x), absf(inv.y)), absf(inv.z)) < absf(T.sz) * INV_MOST)) {
        V3 o, d;
        src(o, d);
        return slab_passes_axial(S.blas, lo, hi, org, d, T.blas, tmin, tmax);
    }
    return slab_passes(lo, hi, org, inv, tmin, tmax);
}

// Child `c` of a node whose first `inner` children are nodes: their index, or a leaf reference.
RTG_D uint32_t child_ref(uint32_t inner, uint32_t node_base, uint32_t leaf_base, uint32_t off_lo, uint32_t off_hi, uint32_t c) {
    return (__byte_perm(off_lo, off_hi, c) & 0xffu) + (c < inner ? node_base : leaf_base);
}

// A node in three 32-byte loads (one sector each) and a top-level leaf's record in one 16-byte load.
struct NodeHead {
    float p[3], scale[3];
    uint32_t node_base, leaf_base;
};
struct NodePlanes {
    uint32_t w[12], off_lo, off_hi, inner;
};
RTG_D NodeHead load_head(const QNode* node) {
    uint32_t v[8];
    load32(node, v);
    NodeHead h;
    for (int a = 0; a < 3; ++a) {
        h.p[a] = __uint_as_float(v[a]);
        h.scale[a] = __uint_as_float(v[3 + a]);
    }
    h.node_base = v[6];
    h.leaf_base = v[7];
    return h;
}
RTG_D NodePlanes load_planes(const QNode* node) {
    uint32_t v[16];
    load32(reinterpret_cast<const uint8_t*>(node) + 32, v);
    load32(reinterpret_cast<const uint8_t*>(node) + 64, v + 8);
    NodePlanes q;
    for (int k = 0; k < 12; ++k) q.w[k] = v[k];
    q.off_lo = v[12];
    q.off_hi = v[13];
    q.inner = v[14];
    return q;
}
RTG_D uint4 load_blas(const BlasInst* bi) { return __ldg(reinterpret_cast<const uint4*>(&bi->root)); }

// Slab planes of one axis for a node: t of the plane of byte q is fma(1 + q 2^-15, a, b). The byte
// becomes 1 + q 2^-15 by one permute into the second-lowest byte of 1.0f's pattern, so a plane
// costs two instructions. The near planes take `b_near` and the far ones `b_far`, moved apart by
// 2^-19 |m| + 2^-21 |a|, so that every box the reference's test passes, this one passes: with u =
// 2^-24, the roundings here are at most 5u |m| + 2.1u |a| (two in m, one each in b, in the pad's sum and
// in the plane's), those of the reference's plane 2u |t|, and its factor 1 + 4 eps with its own
// rounding moves a far plane by 9u |t| more, where |t| <= |m| + |a| / 128: 16u |m| + 2.2u |a| in all, of a
// pad of 32u |m| + 8u |a|. (Of half the |m| term random planes needed up to 0.82.)
struct AxisPlanes {
    float a, b_near, b_far;
    uint32_t n0, n1, f0, f1;  // the near and far planes' bytes
};
RTG_D AxisPlanes axis_planes(float p, float scale, float org, float inv, uint32_t lo0, uint32_t lo1, uint32_t hi0, uint32_t hi1) {
    AxisPlanes x;
    const float m = (p - org) * inv;
    x.a = scale * inv;
    const float b = m - x.a;
    const float pad = __fmaf_rn(absf(x.a), 4.76837158203125e-7f, absf(m) * 1.9073486328125e-6f);
    x.b_near = b - pad;
    x.b_far = b + pad;
    const bool neg = inv < 0.0f;
    x.n0 = neg ? hi0 : lo0;
    x.n1 = neg ? hi1 : lo1;
    x.f0 = neg ? lo0 : hi0;
    x.f1 = neg ? lo1 : hi1;
    return x;
}
RTG_D float plane_t(uint32_t word, uint32_t k, float a, float b) {
    return __fmaf_rn(__uint_as_float(__byte_perm(word, 0x3f800000u, 0x7604u | (k << 4))), a, b);
}

// A hit child's key: its entry distance's bits as an unsigned number with the slot in the three lowest
// bits. That is the reference's order (traverse.rs:47), in which entries before the origin come last, the
// farthest of them at the end. Back from a key the distance is rounded down, as it only orders children
// and culls them later.
RTG_D uint32_t child_key(float n, uint32_t slot) { return (__float_as_uint(n) & ~7u) | slot; }
template <bool POS>
RTG_D uint32_t key_distance(uint32_t k) { return !POS && (k & 0x80000000u) ? k | 7u : k & ~7u; }

// Sorts eight keys, ascending: a network of 19 exchanges.
RTG_D void exchange(uint32_t& a, uint32_t& b) {
    const uint32_t lo = a < b ? a : b, hi = a < b ? b : a;
    a = lo;
    b = hi;
}
RTG_D void sort8(uint32_t k[8]) {
    exchange(k[0], k[2]); exchange(k[1], k[3]); exchange(k[4], k[6]); exchange(k[5], k[7]);
    exchange(k[0], k[4]); exchange(k[1], k[5]); exchange(k[2], k[6]); exchange(k[3], k[7]);
    exchange(k[0], k[1]); exchange(k[2], k[3]); exchange(k[4], k[5]); exchange(k[6], k[7]);
    exchange(k[2], k[4]); exchange(k[3], k[5]);
    exchange(k[1], k[4]); exchange(k[3], k[6]);
    exchange(k[1], k[2]); exchange(k[3], k[4]); exchange(k[5], k[6]);
}

enum TraceMode { TRACE_NEAREST, TRACE_ANY, TRACE_EITHER };
// The next node or leaf from the stack: its nearest entry still in range. False when the query is
// over; `hit` then says whether it found one.
template <TraceMode MODE, class Stack, class Src>
RTG_D bool trav_pop(const SceneDev& S, Trav& T, Stack& stack, bool& hit, const Src& src) {
    for (;;) {
        if (T.sp == 0) {
            hit = MODE != TRACE_ANY && T.best_i != 0xffffffffu;  // no any-hit query sets it
            return false;
        }
        const uint64_t e = stack.get(--T.sp);
        const uint32_t ref = (uint32_t)e;
        if (ref == STACK_RETURN) {
            if (T.blas & BLAS_MOVED) {  // an identity instance's tree was walked with the world ray itself
                V3 o, d;
                src(o, d);
                trav_ray(T, o, d);
            }
            T.blas = TLAS_LEVEL;
            continue;
        }
        if (MODE == TRACE_ANY || __uint_as_float((uint32_t)(e >> 32)) <= T.best_t * RTG_ROBUST) { T.cur = ref; return true; }
    }
}

// One step of the two-level traversal is a node part (the slab test of one node) for a ray at a node
// and then a leaf part (the triangles of one leaf) for a ray at a leaf, the one it has just come to
// included; each ends at the next node or leaf (a child, or the nearest entry of the stack that is
// still in range). `MODE`: the nearest hit with the reference's tie-break, children nearest first; or
// any hit in [t_min, t_max], which ends the query (children in slot order, leaves first); or either,
// as T.any says, children nearest first. `POS`: t_min is known to be positive. `src(o, d)` gives the
// query's world ray. Both return true when the query is over; `hit` then says whether it found one
// (nearest: in T.best_*). A stack that would overflow sets *err bit 0 and ends the query as a miss.
//
// A warp goes through both parts whenever some of its rays are at nodes and some at leaves, so a ray
// that takes both in one step wastes neither: against one part a step, the 1080p product frame went
// from 158.6 to 150.6 ms, the instanced frame from 34.7 to 31.8 ms. The parts are functions of their
// own so that a warp meets again between them (as one function with early returns the leaf part ran
// once for each way into it: 168 ms). Holding the leaf part back until 4, 8, 12 or 16 rays are at
// leaves: 150.2, 149.9, 151.0 and 154.4 ms.
// A leaf is the builder's whole one. Its triangles in runs of two with boxes of their own took 155.8
// instead of 156.9 ms (instanced frame 33.8 and 36.8), but a ray that grazes a triangle can hit it where
// its run's box does not reach, and no growth of the boxes bounds how far off.
// What bounds it is instruction issue (and, in thin rounds, the chain of one ray's steps), not
// memory: the tree stays in L2. So a node step is kept short: two instructions a plane, 32-bit keys
// sorted once, child references computed instead of loaded, full nodes (Flattener). Against exact
// planes (five instructions each), a 64-bit selection per pushed child and a greedy collapse, the
// 1080p product frame went from 312.7 to 229.0 ms, the instanced frame (10 M triangles, 4 spp) from
// 66.4 to 46.1 ms, a 64 x 64 tile from 1.35 to 0.88 ms; films bit-equal.
RTG_D bool trav_at_leaf(const Trav& T) { return (T.cur & NODE_LEAF) != 0; }
template <TraceMode MODE, bool POS, class Stack, class Src>
RTG_D bool trav_node(const SceneDev& S, Trav& T, float tmin, Stack& stack, uint32_t* err, bool& hit, const Src& src) {
    const QNode* node = S.nodes + T.cur;
    const NodeHead h = load_head(node);
    const NodePlanes q = load_planes(node);
    const AxisPlanes X = axis_planes(h.p[0], h.scale[0], T.org[0], T.inv[0], q.w[0], q.w[1], q.w[6], q.w[7]);
    const AxisPlanes Y = axis_planes(h.p[1], h.scale[1], T.org[1], T.inv[1], q.w[2], q.w[3], q.w[8], q.w[9]);
    const AxisPlanes Z = axis_planes(h.p[2], h.scale[2], T.org[2], T.inv[2], q.w[4], q.w[5], q.w[10], q.w[11]);
    const uint32_t off_lo = q.off_lo, off_hi = q.off_hi, inner = q.inner, leaf_base = h.leaf_base | NODE_LEAF;
    const float tmax = T.best_t * RTG_ROBUST;
    if (T.sp + 7 > STACK_CAP) { *err |= 1u; hit = false; return true; }
    // The hit children's keys. Every array index is a constant after unrolling, so the keys stay in
    // registers.
    uint32_t key[8];
    uint32_t next = 0xffffffffu;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
        const uint32_t k = c & 3u;
        const float n = fmaxf(fmaxf(fmaxf(plane_t(c < 4 ? X.n0 : X.n1, k, X.a, X.b_near), plane_t(c < 4 ? Y.n0 : Y.n1, k, Y.a, Y.b_near)),
                                    plane_t(c < 4 ? Z.n0 : Z.n1, k, Z.a, Z.b_near)), tmin);
        const float f = fminf(fminf(fminf(plane_t(c < 4 ? X.f0 : X.f1, k, X.a, X.b_far), plane_t(c < 4 ? Y.f0 : Y.f1, k, Y.a, Y.b_far)),
                                    plane_t(c < 4 ? Z.f0 : Z.f1, k, Z.a, Z.b_far)), tmax);
        if (MODE == TRACE_ANY) {
            // Slot order, the highest slot (leaves come last) next, the others pushed.
            if (n <= f) {
                if (next != 0xffffffffu) stack.put(T.sp++, (uint64_t)next);
                next = child_ref(inner, h.node_base, leaf_base, off_lo, off_hi, c);
            }
        } else {
            key[c] = n <= f ? child_key(n, c) : 0xffffffffu;
        }
    }
    if (MODE != TRACE_ANY) {
        // Nearest next, the others pushed farthest first: a sorting network of 19 exchanges.
        sort8(key);
        if (key[0] != 0xffffffffu) {
#pragma unroll
            for (int j = 7; j >= 1; --j)
                if (key[j] != 0xffffffffu)
                    stack.put(T.sp++, ((uint64_t)key_distance<POS>(key[j]) << 32) | child_ref(inner, h.node_base, leaf_base, off_lo, off_hi, key[j] & 7u));
            next = child_ref(inner, h.node_base, leaf_base, off_lo, off_hi, key[0] & 7u);
        }
    }
    T.cur = next;
    return next == 0xffffffffu && !trav_pop<MODE>(S, T, stack, hit, src);
}
template <TraceMode MODE, bool POS, class Stack, class Src>
RTG_D bool trav_leaf(const SceneDev& S, Trav& T, float tmin, Stack& stack, uint32_t* err, bool& hit, const Src& src) {
    const bool any = MODE == TRACE_ANY || (MODE == TRACE_EITHER && T.any);
    if (T.cur != NODE_EMPTY) {
        uint32_t k = T.cur & ~NODE_LEAF;
        if (T.blas == TLAS_LEVEL) {
            const BlasInst* bi = S.blas + k;
            const uint4 b = load_blas(bi);  // root, identity, instance, flags
            if (!(T.camera && (b.w & 2u)) && (b.y || box_kept(S, T, bi->box, tmin, T.best_t, src))) {
                if (T.sp + 1 > STACK_CAP) { *err |= 1u; hit = false; return true; }
                stack.put(T.sp++, stack_key(0.0f, STACK_RETURN));
                T.blas = (k << 3) | (b.w & 3u);
                if (!b.y) {
                    V3 o, d;
                    src(o, d);
                    float m[12];
#pragma unroll
                    for (int j = 0; j < 12; ++j) m[j] = __ldg(&bi->to_local[j]);
                    trav_ray(T, xf_point(m, o), xf_vector(m, d));
                    T.blas |= BLAS_MOVED;
                }
                T.cur = b.x;
                return false;
            }
        } else {
            const float range = T.best_t;  // what the reference holds the leaf's box against
            bool kept = false;
            uint32_t flags;
            do {
                const float4* tr = reinterpret_cast<const float4*>(S.tris + k);
                const float4 a = __ldg(tr), b = __ldg(tr + 1), c = __ldg(tr + 2);
                ++k;
                flags = __float_as_uint(c.w);
                const uint32_t see = flags | T.blas;
                if (T.camera && (see & 2u)) continue;
                // The scalar watertight test (triangle.rs:123), the reference's operations in its
                // order. The reference swaps the minor axes for a ray down the major one; that only
                // negates u, v and w, exactly (a t of zero, which takes a t_min of zero or less, may have
                // the other sign).
                const int kz = T.kz;
                auto px = [&](float x, float y, float z) { return kz == 0 ? y : (kz == 1 ? z : x); };
                auto py = [&](float x, float y, float z) { return kz == 0 ? z : (kz == 1 ? x : y); };
                auto pz = [&](float x, float y, float z) { return kz == 0 ? x : (kz == 1 ? y : z); };
                const float ex = a.x - T.org[0], ey = a.y - T.org[1], ez = a.z - T.org[2];
                const float gx = b.x - T.org[0], gy = b.y - T.org[1], gz = b.z - T.org[2];
                const float wx = c.x - T.org[0], wy = c.y - T.org[1], wz = c.z - T.org[2];
                const float a_z = pz(ex, ey, ez), b_z = pz(gx, gy, gz), c_z = pz(wx, wy, wz);
                const float ax = px(ex, ey, ez) - T.sx * a_z, ay = py(ex, ey, ez) - T.sy * a_z;
                const float bx = px(gx, gy, gz) - T.sx * b_z, by = py(gx, gy, gz) - T.sy * b_z;
                const float cx = px(wx, wy, wz) - T.sx * c_z, cy = py(wx, wy, wz) - T.sy * c_z;
                float u = cx * by - cy * bx, v = ax * cy - ay * cx, w = bx * ay - by * ax;
                if (T.flip) { u = -u; v = -v; w = -w; }
                const bool negative = u < 0.0f || v < 0.0f || w < 0.0f;
                const bool positive = u > 0.0f || v > 0.0f || w > 0.0f;
                const bool rejected = (see & 1u) ? negative : (negative && positive);
                const float det = u + v + w;
                if (rejected || det == 0.0f) continue;
                const float az = T.sz * a_z, bz = T.sz * b_z, cz = T.sz * c_z;
                const float t = (u * az + v * bz + w * cz) / det;
                if (!(t >= tmin && t <= T.best_t)) continue;
                uint32_t inst = __float_as_uint(b.w);
                if (!any) {
                    if (inst == 0xffffffffu) inst = __ldg(&S.blas[T.blas >> 3].instance);
                    if (!(t < T.best_t || inst < T.best_i || (inst == T.best_i && __float_as_uint(a.w) < __ldg(&S.tris[T.best_k].tri)))) continue;
                }
                if (!kept && !box_kept(S, T, S.leaf_boxes + 8 * (size_t)(flags >> TRI_LEAF_SHIFT), tmin, range, src)) break;
                kept = true;
                if (any) { hit = true; return true; }
                T.best_t = t;
                T.best_i = inst;
                T.best_k = k - 1;
            } while (!(flags & TRI_LAST));
        }
    }
    return !trav_pop<MODE>(S, T, stack, hit, src);
}

// A query's world ray kept by the query itself.
struct HeldRay {
    V3 o, d;
    RTG_D void operator()(V3& ro, V3& rd) const { ro = o; rd = d; }
};
// A whole query: false on a miss. Nearest-hit queries fill `res`.
template <bool ANY, bool POS = false, class Stack>
RTG_D bool traverse(const SceneDev& S, V3 o, V3 d, float tmin, float tmax, bool camera, TraceResult& res, uint32_t* err,
                    Stack& stack) {
    Trav T;
    if (!trav_init(S, T, o, d, tmin, tmax, camera)) return false;
    bool hit = false;
    const HeldRay src{o, d};
    constexpr TraceMode MODE = ANY ? TRACE_ANY : TRACE_NEAREST;
    for (bool over = false; !over;) {
        if (!trav_at_leaf(T)) over = trav_node<MODE, POS>(S, T, tmin, stack, err, hit, src);
        if (!over && trav_at_leaf(T)) over = trav_leaf<MODE, POS>(S, T, tmin, stack, err, hit, src);
    }
    if (hit && !ANY) { res.inst = T.best_i; res.tri = T.best_k; res.t = T.best_t; }
    return hit;
}

// ---- the section view (geometry/section.rs:127-448) --------------------------------------------------
// A query of a scene with a section sees the model as if the side of the plane its normal points to
// were empty: the ray is clipped to the interval where it is on the kept side; where it crosses the
// plane inside a closed solid (the next surface along it is met from behind) it hits the solid's cap
// on the plane; and the studio instances (exempt from the section) are found on the removed side by
// stepping over the cut model's surfaces, at most 48 deep.
constexpr uint32_t CAP_TRIANGLE = 0xffffffffu;  // the `tri` of a hit on a cap
constexpr int SECTION_MAX_SKIPS = 48;
enum : int { SPAN_REMOVED = 0, SPAN_WHOLE = 1, SPAN_ENTERS = 2, SPAN_LEAVES = 3 };

RTG_D int section_span(const SceneDev& S, V3 o, V3 d, float tmin, float tmax, float& t) {
    const V3 n = v3(S.section_n[0], S.section_n[1], S.section_n[2]);
    const float from_plane = dot(n, o) - S.section_d;
    const float towards = dot(n, d);
    if (towards == 0.0f) return from_plane <= 0.0f ? SPAN_WHOLE : SPAN_REMOVED;
    t = -from_plane / towards;
    if (towards > 0.0f) return t < tmin ? SPAN_REMOVED : (t >= tmax ? SPAN_WHOLE : SPAN_LEAVES);
    return t <= tmin ? SPAN_WHOLE : (t > tmax ? SPAN_REMOVED : SPAN_ENTERS);
}

RTG_D bool section_may_cap(const SceneDev& S, V3 p) {
    return S.cap_any && p.x >= S.cap_lo[0] && p.x <= S.cap_hi[0] && p.y >= S.cap_lo[1] && p.y <= S.cap_hi[1] &&
           p.z >= S.cap_lo[2] && p.z <= S.cap_hi[2];
}

RTG_D bool section_hidden(const SceneDev& S, bool camera, uint32_t inst) {
    return camera && inst < S.n_instances && (S.instances[inst].flags & 4u) != 0;  // INSTANCE_NO_CAMERA
}

// True when leaf triangle `tri` of capped instance `inst` is met by direction d from inside its solid.
RTG_D bool section_met_from_inside(const SceneDev& S, V3 d, uint32_t inst, uint32_t tri) {
    if (inst >= S.n_instances) return false;
    const DevInstance* I = S.instances + inst;
    if (!I->active || I->solid == 0u) return false;
    const float4* rec = reinterpret_cast<const float4*>(S.tris + tri);
    const float4 q0 = __ldg(rec), q1 = __ldg(rec + 1), q2 = __ldg(rec + 2);
    const V3 p0 = v3(q0.x, q0.y, q0.z), p1 = v3(q1.x, q1.y, q1.z), p2 = v3(q2.x, q2.y, q2.z);
    V3 w = cross(p1 - p0, p2 - p0);
    if (!I->identity) w = xf_transpose(I->to_local, w);
    const bool front = dot(w, d) < 0.0f;
    return I->solid == 1u ? !front : front;
}

// The first exempt instance within [near, far], stepping over the others' surfaces.
template <class Stack>
RTG_D bool section_first_exempt(const SceneDev& S, V3 o, V3 d, float near, float far, bool camera, TraceResult& res,
                                uint32_t* err, Stack& stack) {
    float t = near;
    for (int k = 0; k < SECTION_MAX_SKIPS; ++k) {
        TraceResult h;
        if (!traverse<false>(S, o, d, t, far, camera, h, err, stack)) return false;
        if (h.inst < S.n_instances && S.instances[h.inst].exempt) { res = h; return true; }
        t = __uint_as_float(__float_as_uint(fmaxf(h.t, 0.0f)) + 1u);  // strictly past the surface
        if (t > far) return false;
    }
    return false;
}

// The nearest exempt hit within [from, to] (a removed part of the ray's range), looked for inside
// each exempt instance's box only (Aabb::intersect, math.rs:388).
template <class Stack>
RTG_D bool section_exempt_in(const SceneDev& S, V3 o, V3 d, float from, float to, bool camera, TraceResult& res, uint32_t* err,
                             Stack& stack) {
    if (S.n_exempt == 0u || from != from || to != to || from > to) return false;
    const float inv[3] = {1.0f / d.x, 1.0f / d.y, 1.0f / d.z}, org[3] = {o.x, o.y, o.z};
    bool found = false;
    for (uint32_t b = 0; b < S.n_exempt; ++b) {
        const float* box = S.exempt_boxes + 6 * b;
        const float end = found ? fminf(res.t, to) : to;
        float near = from, far = end;
        for (int a = 0; a < 3; ++a) {
            const float x = (__ldg(box + a) - org[a]) * inv[a], y = (__ldg(box + 3 + a) - org[a]) * inv[a];
            if (x != x || y != y) continue;  // parallel to the slab, on its boundary
            near = fmaxf(near, fminf(x, y));
            far = fminf(far, fmaxf(x, y));
        }
        if (!(near <= far && near < f_inf())) continue;
        TraceResult h;
        if (section_first_exempt(S, o, d, near, fminf(far, end), camera, h, err, stack) && (!found || h.t < res.t)) {
            res = h;
            found = true;
        }
    }
    return found;
}

// The cap at t where the ray leaves the kept side having hit nothing: there when the next surface of
// the whole model beyond the plane is met from inside its solid.
template <class Stack>
RTG_D bool section_cap_beyond(const SceneDev& S, V3 o, V3 d, float t, TraceResult& res, uint32_t* err, Stack& stack) {
    if (!S.section_cap || !section_may_cap(S, o + d * t)) return false;
    TraceResult h;
    if (!traverse<false>(S, o, d, t, f_inf(), false, h, err, stack)) return false;
    if (!section_met_from_inside(S, d, h.inst, h.tri)) return false;
    res.inst = h.inst;
    res.tri = CAP_TRIANGLE;
    res.t = t;
    return true;
}

// Geometry::trace_sectioned / occluded_sectioned (section.rs:224-324). Out of line: scenes without
// a section never call it, and the kernels that can keep their registers for the plain traversal.
template <bool ANY, class Stack>
RTG_D_NI bool section_query(const SceneDev& S, V3 o, V3 d, float tmin, float tmax, bool camera, TraceResult& res,
                            uint32_t* err, Stack& stack) {
    float t = 0.0f;
    const int span = section_span(S, o, d, tmin, tmax, t);
    TraceResult other;
    if (ANY) {
        switch (span) {
            case SPAN_REMOVED: return section_exempt_in(S, o, d, tmin, tmax, camera, other, err, stack);
            case SPAN_WHOLE: return traverse<true>(S, o, d, tmin, tmax, camera, res, err, stack);
            case SPAN_LEAVES:
                return traverse<true>(S, o, d, tmin, t, camera, res, err, stack) || section_cap_beyond(S, o, d, t, other, err, stack) ||
                       section_exempt_in(S, o, d, t, tmax, camera, other, err, stack);
            default:  // the cap of a ray that enters is at the start of what it can hit anyway
                return traverse<true>(S, o, d, t, tmax, camera, res, err, stack) ||
                       section_exempt_in(S, o, d, tmin, t, camera, other, err, stack);
        }
    }
    switch (span) {
        case SPAN_REMOVED: return section_exempt_in(S, o, d, tmin, tmax, camera, res, err, stack);
        case SPAN_WHOLE: return traverse<false>(S, o, d, tmin, tmax, camera, res, err, stack);
        case SPAN_LEAVES:
            // The kept part; else a cap looked for beyond the plane; else the studio beyond it.
            if (traverse<false>(S, o, d, tmin, t, camera, res, err, stack)) return true;
            if (section_cap_beyond(S, o, d, t, other, err, stack) && !section_hidden(S, camera, other.inst)) {
                res = other;
                return true;
            }
            return section_exempt_in(S, o, d, t, tmax, camera, res, err, stack);
        default: {
            // The studio on the removed side is nearer than anything on the kept one; then the
            // nearest surface beyond the plane, whose side tells whether the crossing is a cap.
            if (section_exempt_in(S, o, d, tmin, t, camera, res, err, stack)) return true;
            const bool got = traverse<false>(S, o, d, t, tmax, camera, other, err, stack);
            if (got && S.section_cap && section_may_cap(S, o + d * t) && section_met_from_inside(S, d, other.inst, other.tri) &&
                !section_hidden(S, camera, other.inst)) {
                res.inst = other.inst;
                res.tri = CAP_TRIANGLE;
                res.t = t;
                return true;
            }
            if (got) res = other;
            return got;
        }
    }
}

// A whole query through the scene's section when it has one.
template <bool ANY, class Stack>
RTG_D bool trace_q(const SceneDev& S, V3 o, V3 d, float tmin, float tmax, bool camera, TraceResult& res, uint32_t* err,
                   Stack& stack) {
    if (!S.section_on) return traverse<ANY>(S, o, d, tmin, tmax, camera, res, err, stack);
    return section_query<ANY>(S, o, d, tmin, tmax, camera, res, err, stack);
}

struct HitInfo {
    V3 point, normal, geometric;
    float bary[3];
    bool front, outside;
    bool cap;  // on a section's cap: no triangle, the plane's normal
    uint32_t tri;  // the leaf triangle
};

// geometry/mod.rs:731 hit_details for an instance hit. `P`: a plain scene (SceneDev::plain), no section.
template <bool P = false>
RTG_D_NI bool hit_details(const SceneDev& S, V3 o, V3 d, float tmin, float tmax, uint32_t inst, uint32_t tri, float t_hit,
                       HitInfo& h, const DevInstance*& I_out) {
    if (inst >= S.n_instances) return false;
    const DevInstance* I = S.instances + inst;
    I_out = I;
    if (!I->active) return false;
    h.cap = !P && tri == CAP_TRIANGLE;
    if (h.cap) {  // Section::cap_details (section.rs:424-448): on the plane, facing where the ray came from
        if (!S.section_on) return false;
        const V3 n = v3(S.section_n[0], S.section_n[1], S.section_n[2]);
        const V3 at = o + d * t_hit;
        h.point = at - n * (dot(n, at) - S.section_d);
        h.front = dot(n, d) < 0.0f;
        h.normal = h.front ? n : -n;
        h.geometric = h.normal;
        h.bary[0] = 1.0f;
        h.bary[1] = h.bary[2] = 0.0f;
        h.outside = h.front;
        return true;
    }
    h.tri = tri;
    const float4* rec = reinterpret_cast<const float4*>(S.tris + tri);
    const float4 q0 = __ldg(rec), q1 = __ldg(rec + 1), q2 = __ldg(rec + 2);
    V3 p0 = v3(q0.x, q0.y, q0.z), p1 = v3(q1.x, q1.y, q1.z), p2 = v3(q2.x, q2.y, q2.z);
    bool identity = I->identity != 0;
    PRay r = identity ? prepare_ray(o, d, tmin, tmax) : prepare_ray(xf_point(I->to_local, o), xf_vector(I->to_local, d), tmin, tmax);
    float v0[3] = {p0.x, p0.y, p0.z}, v1[3] = {p1.x, p1.y, p1.z}, v2[3] = {p2.x, p2.y, p2.z};
    float t, u, v, w, det;
    if (watertight(r, v0, v1, v2, F_MAX, false, t, u, v, w, det)) {
        h.bary[0] = u / det; h.bary[1] = v / det; h.bary[2] = w / det;
    } else {
        h.bary[0] = h.bary[1] = h.bary[2] = 1.0f / 3.0f;
    }
    V3 pl = p0 * h.bary[0] + p1 * h.bary[1] + p2 * h.bary[2];
    V3 cr = cross(p1 - p0, p2 - p0);
    V3 winding = normalize(identity ? cr : xf_transpose(I->to_local, cr));
    V3 incoming = normalize(d);
    V3 geometric = len2(winding) > 0.0f ? winding : -incoming;
    h.front = dot(winding, d) < 0.0f;
    V3 smooth = v3(0, 0, 0);
    if (I->has_normals) {
        const float4* nr = S.tri_normals + 3 * (size_t)tri;
        const float4 m0 = __ldg(nr), m1 = __ldg(nr + 1), m2 = __ldg(nr + 2);
        V3 s = v3(m0.x, m0.y, m0.z) * h.bary[0] + v3(m1.x, m1.y, m1.z) * h.bary[1] + v3(m2.x, m2.y, m2.z) * h.bary[2];
        smooth = identity ? s : xf_transpose(I->to_local, s);
    }
    V3 normal = len2(smooth) > 1.0e-12f ? normalize(smooth) : geometric;
    h.normal = dot(normal, d) > 0.0f ? -normal : normal;
    h.geometric = dot(geometric, d) > 0.0f ? -geometric : geometric;
    h.point = identity ? pl : xf_point(I->to_world, pl);
    h.outside = h.front != (I->inside_out != 0);
    return true;
}

// geometry/mod.rs:682 terminator_point (Hanika 2021).
RTG_D_NI V3 terminator_point(const SceneDev& S, const DevInstance* I, const HitInfo& h) {
    if (h.cap || !I->has_normals) return h.point;
    const float4 *rec = reinterpret_cast<const float4*>(S.tris + h.tri), *nr = S.tri_normals + 3 * (size_t)h.tri;
    const float4 q[3] = {__ldg(rec), __ldg(rec + 1), __ldg(rec + 2)}, m[3] = {__ldg(nr), __ldg(nr + 1), __ldg(nr + 2)};
    V3 c[3], n[3];
    for (int k = 0; k < 3; ++k) { c[k] = v3(q[k].x, q[k].y, q[k].z); n[k] = v3(m[k].x, m[k].y, m[k].z); }
    float b0 = h.bary[0], b1 = h.bary[1], b2 = h.bary[2];
    V3 p = c[0] * b0 + c[1] * b1 + c[2] * b2;
    V3 interp = n[0] * b0 + n[1] * b1 + n[2] * b2;
    bool identity = I->identity != 0;
    V3 wn = identity ? interp : xf_transpose(I->to_local, interp);
    float side = dot(wn, h.geometric) < 0.0f ? -1.0f : 1.0f;
    V3 lifted = p;
    for (int k = 0; k < 3; ++k) {
        V3 nn = normalize(n[k]) * side;
        float below = dot(p - c[k], nn);
        if (below < 0.0f) lifted = lifted - nn * (below * h.bary[k]);
    }
    if (!vfinite(lifted)) return h.point;
    return identity ? lifted : xf_point(I->to_world, lifted);
}

}  // namespace rtg
