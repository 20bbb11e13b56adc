// CCD swept-sphere clamp (step.rs:1068-1155, :1210-1214; convex_sweep.rs:37-214, :263-295;
// gjk.rs:864-1044). One warp per body that has CCD settings finds its candidates: the bodies of its
// world that pass the collision filters (no-contact-response targets, joint-suppressed pairs,
// group/mask) and whose broad-phase proxy touches the swept box. A second kernel casts a sphere
// against each candidate, several casts a warp; a body's smallest hit fraction is its clamp. A third
// kernel, after the position integration, pulls each clamped body back along its step motion.
// The reference scans every body for every CCD body as well; the cast itself (a ternary search
// for the closest approach, then bisection, each probe a GJK point distance) matches its
// arithmetic step for step.
#include <algorithm>
#include "bgpu_kernels.cuh"

namespace bgpu {

namespace {

// A GJK simplex of up to four points, in the order the closest-feature tests keep them.
struct Simplex {
    V3 p[4];
    int n;
};

__device__ __forceinline__ void keep1(Simplex& s, V3 a) { s.p[0] = a; s.n = 1; }
__device__ __forceinline__ void keep2(Simplex& s, V3 a, V3 b) { s.p[0] = a; s.p[1] = b; s.n = 2; }

// gjk.rs:889-906
__device__ __forceinline__ V3 closest_segment(V3 a, V3 b, Simplex& keep) {
    const V3 ab = b - a;
    if (len2(ab) == 0.0f) { keep1(keep, a); return a; }
    const float t = -dot(a, ab) / len2(ab);
    if (t <= 0.0f) { keep1(keep, a); return a; }
    if (t >= 1.0f) { keep1(keep, b); return b; }
    keep2(keep, b, a);
    return a + ab * t;
}

__device__ __forceinline__ V3 sel(bool c, V3 x, V3 y) { return V3{c ? x.x : y.x, c ? x.y : y.y, c ? x.z : y.z}; }

// gjk.rs:911-989, a degenerate triangle: the closest of its three edges (a call of its own, rarely
// taken).
__device__ __noinline__ V3 closest_triangle_edges(V3 a, V3 b, V3 c, Simplex& keep) {
    Simplex kab, kbc, kca;
    const V3 qab = closest_segment(a, b, kab), qbc = closest_segment(b, c, kbc), qca = closest_segment(c, a, kca);
    if (len2(qab) <= len2(qbc) && len2(qab) <= len2(qca)) { keep = kab; return qab; }
    if (len2(qbc) <= len2(qca)) { keep = kbc; return qbc; }
    keep = kca;
    return qca;
}

// The point of the triangle a, b, c (gjk.rs:911-989), or with seg of the segment a, b (:889-906),
// closest to the origin, and the vertices that span it. One path for every region, by selects and a
// single division: the lanes of a warp walk different simplices, and with a branch per region a
// step cost the sum of all of them (10,000 cycles).
__device__ __forceinline__ V3 closest_feature(bool seg, V3 a, V3 b, V3 c, Simplex& keep) {
    const V3 ab = b - a, ac = c - a, ap = -a, bp = -b, cp = -c;
    const float d1 = dot(ab, ap), d2 = dot(ac, ap), d3 = dot(ab, bp), d4 = dot(ac, bp), d5 = dot(ab, cp), d6 = dot(ac, cp);
    const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
    const float sum = va + vb + vc, l2 = len2(ab);
    const float e43 = d4 - d3, e56 = d5 - d6;
    enum { A, B, AB, C, AC, BC, EDGES, FACE };
    int r = FACE;
    if (sum <= 0.0f || isnan(sum)) r = EDGES;
    if (va <= 0.0f && e43 >= 0.0f && e56 >= 0.0f) r = BC;
    if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) r = AC;
    if (d6 >= 0.0f && d5 <= d6) r = C;
    if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) r = AB;
    if (d3 >= 0.0f && d4 <= d3) r = B;
    if (d1 <= 0.0f && d2 <= 0.0f) r = A;
    if (seg) r = AB;
    if (r == EDGES) {
        Simplex k;  // (its address is taken: keep itself stays in registers)
        const V3 e = closest_triangle_edges(a, b, c, k);
        keep = k;
        return e;
    }
    const float num = r == AB ? d1 : (r == AC ? d2 : (r == BC ? e43 : 1.0f));
    const float den = r == AB ? (seg ? l2 : d1 - d3) : (r == AC ? d2 - d6 : (r == BC ? e43 + e56 : (r == FACE ? sum : 1.0f)));
    // Vanishing edges (the triangle tests d1 == d3, d2 == d6 and the sum, and the segment its length)
    if (r == AB && (seg ? l2 == 0.0f : d1 == d3)) r = A;
    if (r == AC && d2 == d6) r = A;
    if (r == BC && den == 0.0f) r = B;
    const float q = num / den;
    if (seg && r == AB) r = q <= 0.0f ? A : (q >= 1.0f ? B : AB);
    const bool face = r == FACE, vertex = r == A || r == B || r == C;
    const V3 base = sel(r == BC || r == B, b, sel(r == C, c, a));
    const V3 dir = sel(r == AC, ac, sel(r == BC, c - b, ab));
    V3 v = base + dir * (face ? vb * q : q);
    v = sel(face, v + ac * (vc * q), sel(vertex, base, v));
    // Kept: the vertex; b a, c a, c b for an edge; c b a for the face.
    keep.p[0] = sel(vertex, base, sel(r == AB, b, c));
    keep.p[1] = sel(r == BC || face, b, a);
    keep.p[2] = a;
    keep.n = vertex ? 1 : (face ? 3 : 2);
    return v;
}

// The target inflated by the swept sphere (convex_sweep.rs:107-125): its support point along d.
struct Inflated {
    Shape s;
    V3 pos;
    Q ori;
    float radius;
    const float4* hull;
    __device__ __forceinline__ V3 support(V3 d) const {
        const V3 sphere = len2(d) > 1e-12f ? d / len(d) * radius : V3{0.0f, 0.0f, 0.0f};
        return support_world(s, pos, ori, d, hull) + sphere;
    }
};

// Equal walk states between two iterations (at most three points are kept there).
__device__ __forceinline__ bool same_state(const Simplex& a, V3 av, const Simplex& b, V3 bv) {
    return a.n == b.n && same_bits(av, bv) && same_bits(a.p[0], b.p[0]) && (a.n < 2 || same_bits(a.p[1], b.p[1])) &&
           (a.n < 3 || same_bits(a.p[2], b.p[2]));
}

// convex_sweep.rs:72-103: squared distance from a point to the inflated target (zero when inside or
// touching), as a walk that is taken step by step, so that the lanes of a warp, each with a walk
// of its own, share every step. A step finds the next support point and the closest feature of the
// simplex; the four faces of a flat tetrahedron (gjk.rs:994-1044) take a step each.
//
// On a rounded target the walk seldom meets its stop tests: it falls, after some 10 to 20 iterations,
// into a cycle of 1, 2 or a few more states that it repeats up to the 64th. An iteration depends on
// the state (simplex, v) alone, so once a state equals an earlier one bit for bit, the whole
// periods that are left change nothing and are skipped. Compared with a state kept at iterations
// 4, 8, 12, 16, 24, 32 and 48: on 300,000 sweeps against plates, boxes, spheres and capsules 95 to
// 98 % of the walks that ran to the 64th end early, a probe taking 12 to 17 iterations instead of
// 45 to 62.
struct Walk {
    V3 point, v;
    Simplex s;
    V3 kv;           // the kept state
    Simplex ks;
    V3 best;         // of the faces tried so far
    Simplex bk;
    int it, kept_at, face;  // it < 0: the first support point; face >= 0: the faces of a flat tetrahedron
    float d2;
    bool done;

    __device__ __forceinline__ void start(V3 p) {
        point = p;
        v = len2(p) < 1e-12f ? V3{1.0f, 0.0f, 0.0f} : p;
        s.n = 0;
        it = -1;
        kept_at = 0;
        face = -1;
        done = false;
    }
    __device__ __forceinline__ void finish(float x) {
        d2 = x;
        done = true;
    }
    __device__ __forceinline__ void step(const Inflated& t) {
        bool seg = false, inside = false;
        V3 x = s.p[0], y = s.p[1], z = s.p[2];
        if (face < 0) {
            if (it >= 0) {
                const float l = len2(v);
                if (l < 1e-10f) return finish(0.0f);
                if (kept_at > 0 && same_state(s, v, ks, kv)) {
                    const int period = it - kept_at;
                    it += (64 - it) / period * period;
                    kept_at = -1;  // what is left is less than a period
                } else if (kept_at >= 0 && it >= 4 && (it & 3) == 0 && (it <= 16 || (it & 7) == 0) && (it <= 32 || it == 48)) {
                    ks = s;
                    kv = v;
                    kept_at = it;
                }
                if (it >= 64) return finish(l);
            }
            const V3 u = it < 0 ? v : -v;  // mink(u)
            const V3 w = point - t.support(-u);
            if (it < 0) {
                s.p[0] = w;
                s.n = 1;
                v = w;
                it = 0;
                return;
            }
            bool repeat = false;  // the simplex already holds w (constant indices keep s in registers)
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (k < s.n && len2(s.p[k] - w) < 1e-12f) repeat = true;
            if (repeat) return finish(len2(v));
            seg = s.n == 1;
            if (s.n == 1) s.p[1] = w;
            else if (s.n == 2) s.p[2] = w;
            else s.p[3] = w;
            ++s.n;
            y = s.p[1];
            z = seg ? s.p[0] : s.p[2];
            if (s.n == 4) {  // gjk.rs:994-1044
                const V3 a = s.p[0], b = s.p[1], c = s.p[2], d = s.p[3];
                const V3 ao = -a, ab = b - a, ac = c - a, ad = d - a, abc = cross(ab, ac);
                if (fabsf(dot(abc, ad)) < 1e-12f) {
                    face = 0;
                } else {
                    const V3 acd = cross(ac, ad), adb = cross(ad, ab), bcd = cross(c - b, d - b);
                    const bool f0 = dot(abc, ao) * dot(abc, ad) < 0.0f, f1 = dot(acd, ao) * dot(acd, ab) < 0.0f;
                    const bool f2 = dot(adb, ao) * dot(adb, ac) < 0.0f, f3 = dot(bcd, -b) * dot(bcd, a - b) < 0.0f;
                    inside = !(f0 || f1 || f2 || f3);  // else the first of abc, acd, adb, bcd
                    const bool k1 = !f0 && f1, k2 = !f0 && !f1 && f2, k3 = !f0 && !f1 && !f2;
                    x = sel(k3, b, a);
                    y = sel(k1 || k3, c, sel(k2, d, b));
                    z = sel(k1 || k3, d, sel(k2, b, c));
                }
            }
        }
        if (face >= 0) {  // abc, abd, acd, bcd
            x = sel(face == 3, s.p[1], s.p[0]);
            y = sel(face < 2, s.p[1], s.p[2]);
            z = sel(face == 0, s.p[2], s.p[3]);
        }
        Simplex k;
        V3 q = closest_feature(seg, x, y, z, k);
        if (face >= 0) {  // the first of equal ones
            if (face == 0 || len2(q) < len2(best)) {
                best = q;
                bk = k;
            }
            if (++face < 4) return;
            face = -1;
            q = best;
            k = bk;
        }
        if (inside) {  // v = 0: the next step ends the walk
            v = V3{0.0f, 0.0f, 0.0f};
        } else {
            v = q;
            s.p[0] = k.p[0];
            s.p[1] = k.p[1];
            s.p[2] = k.p[2];
            s.n = k.n;
        }
        ++it;
    }
};

__device__ __forceinline__ float point_distance2(const Inflated& t, V3 p) {
    Walk w;
    w.start(p);
    while (!w.done) w.step(t);
    return w.d2;
}

// convex_sweep.rs:155-214 (sweep_with_dist), the fraction only
__device__ bool sweep_convex(V3 from, V3 dir, float length, const Inflated& t, float& fraction) {
    float lo = 0.0f, hi = 1.0f;
    for (int it = 0; it < 40; ++it) {
        const float m1 = lo + (hi - lo) / 3.0f;
        const float m2 = hi - (hi - lo) / 3.0f;
        if (point_distance2(t, from + dir * (m1 * length)) < point_distance2(t, from + dir * (m2 * length))) hi = m2;
        else lo = m1;
    }
    const float s_min = (lo + hi) * 0.5f;
    if (point_distance2(t, from + dir * (s_min * length)) > 1e-8f) return false;
    float low = 0.0f, high = s_min;
    for (int it = 0; it < 60; ++it) {
        const float mid = (low + high) * 0.5f;
        if (point_distance2(t, from + dir * (mid * length)) <= 1e-8f) high = mid;
        else low = mid;
    }
    fraction = (low + high) * 0.5f;
    return true;
}

// convex_sweep.rs:217-262 (point_triangle_distance): squared distance to the triangle and the
// vector from its closest point to `p`.
__device__ float point_triangle_distance(V3 p, V3 a, V3 b, V3 c, V3& dv) {
    const V3 ab = b - a, ac = c - a, ap = p - a;
    const float d1 = dot(ab, ap), d2 = dot(ac, ap);
    if (d1 <= 0.0f && d2 <= 0.0f) { dv = p - a; return len2(dv); }
    const V3 bp = p - b;
    const float d3 = dot(ab, bp), d4 = dot(ac, bp);
    if (d3 >= 0.0f && d4 <= d3) { dv = p - b; return len2(dv); }
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
        const float v = d1 / (d1 - d3);
        dv = p - (a + ab * v);
        return len2(dv);
    }
    const V3 cp = p - c;
    const float d5 = dot(ab, cp), d6 = dot(ac, cp);
    if (d6 >= 0.0f && d5 <= d6) { dv = p - c; return len2(dv); }
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
        const float w = d2 / (d2 - d6);
        dv = p - (a + ac * w);
        return len2(dv);
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        dv = p - (b + (c - b) * w);
        return len2(dv);
    }
    const float denom = 1.0f / (va + vb + vc);
    const float v = vb * denom, w = vc * denom;
    dv = p - (a + ab * v + ac * w);
    return len2(dv);
}

// convex_sweep.rs:131-151 (sweep_triangle) distance: zero inside the inflated triangle.
__device__ __forceinline__ float tri_inflated_distance2(V3 p, V3 a, V3 b, V3 c, float radius) {
    V3 dv;
    const float q = point_triangle_distance(p, a, b, c, dv);
    if (q <= radius * radius) return 0.0f;
    const float d = sqrtf(q);
    return (d - radius) * (d - radius);
}

// convex_sweep.rs:155-214 (sweep_with_dist) against one triangle, the fraction only.
__device__ bool sweep_triangle(V3 from, V3 dir, float length, float radius, V3 a, V3 b, V3 c, float& fraction) {
    float lo = 0.0f, hi = 1.0f;
    for (int it = 0; it < 40; ++it) {
        const float m1 = lo + (hi - lo) / 3.0f;
        const float m2 = hi - (hi - lo) / 3.0f;
        if (tri_inflated_distance2(from + dir * (m1 * length), a, b, c, radius) <
            tri_inflated_distance2(from + dir * (m2 * length), a, b, c, radius))
            hi = m2;
        else
            lo = m1;
    }
    const float s_min = (lo + hi) * 0.5f;
    if (tri_inflated_distance2(from + dir * (s_min * length), a, b, c, radius) > 1e-8f) return false;
    float low = 0.0f, high = s_min;
    for (int it = 0; it < 60; ++it) {
        const float mid = (low + high) * 0.5f;
        if (tri_inflated_distance2(from + dir * (mid * length), a, b, c, radius) <= 1e-8f) high = mid;
        else low = mid;
    }
    fraction = (low + high) * 0.5f;
    return true;
}

// convex_sweep.rs:305-345 (sweep_mesh): the segment in the mesh frame, the BVH candidates of its
// swept box (bgpu_shapes.cuh's mesh layout), the smallest per-triangle fraction.
__device__ bool sweep_mesh(V3 from, V3 to, float radius, const Shape& ms, V3 pos, Q ori,
                           const float4* __restrict__ hull, uint32_t* status, float& fraction) {
    const Q inv = qinv(ori);
    const V3 lf = rotate(inv, from - pos), lt = rotate(inv, to - pos);
    const V3 delta = lt - lf;
    const float length = len(delta);
    if (length <= 1.1920929e-7f) return false;
    const V3 dir = delta / length;
    const V3 r = V3{radius, radius, radius};
    const V3 bmin = vmin(lf, lt) - r, bmax = vmax(lf, lt) + r;
    const uint32_t tri_base = mesh_tri_base(ms);
    bool any = false;
    float best = 1.0f;
    uint32_t stack[64];
    int sp = 0;
    if (ms.hull_cnt) stack[sp++] = 0;
    while (sp > 0) {
        const uint32_t k = stack[--sp];
        const float4 n0 = hull[ms.hull_off + 2 * k], n1 = hull[ms.hull_off + 2 * k + 1];
        if (!(n0.x <= bmax.x && n0.y <= bmax.y && n0.z <= bmax.z && bmin.x <= n1.x && bmin.y <= n1.y && bmin.z <= n1.z))
            continue;
        const uint32_t na = __float_as_uint(n0.w), nb = __float_as_uint(n1.w);
        if (!(na & MESH_LEAF)) {
            if (sp + 2 > 64) {
                atomicOr(status, ST_TRAVERSAL_STACK);
                continue;
            }
            stack[sp++] = na;
            stack[sp++] = nb;
            continue;
        }
        const uint32_t start = na & ~MESH_LEAF;
        for (uint32_t slot = start; slot < start + nb; ++slot) {
            const uint32_t o = tri_base + 3 * slot;
            float f;
            if (sweep_triangle(lf, dir, length, radius, from4(hull[o]), from4(hull[o + 1]), from4(hull[o + 2]), f) &&
                (!any || f < best)) {
                best = f;
                any = true;
            }
        }
    }
    if (any) fraction = best;
    return any;
}

// convex_sweep.rs:263-295 (sweep_plane), the fraction only
__device__ bool sweep_plane(V3 from, V3 dir, float length, float radius, const Shape& s, Q ori, float& fraction) {
    const V3 n = rotate(ori, V3{s.p0, s.p1, s.p2});
    const float dn0 = dot(n, from) - s.p3;
    if (fabsf(dn0) <= radius) { fraction = 0.0f; return true; }
    const float dd = dot(n, dir * length);
    if (dd >= 0.0f) return false;
    const float sign = dn0 > 0.0f ? 1.0f : -1.0f;
    const float f = (sign * radius - dn0) / dd;
    if (!(f >= 0.0f && f <= 1.0f)) return false;
    fraction = f;
    return true;
}

__device__ bool key_suppressed(const uint64_t* keys, uint32_t n, uint64_t k) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (keys[mid] < k) lo = mid + 1;
        else hi = mid;
    }
    return lo < n && keys[lo] == k;
}

__device__ __forceinline__ bool body_active(uint32_t act) {
    return act == ACT_ACTIVE || act == ACT_WANTS_DEACTIVATION || act == ACT_DISABLE_DEACTIVATION;
}

// One warp per CCD body. Candidates that pass the filters and the proxy-box pretest are kept in
// shared memory with a lower bound on their hit fraction and, ordered by it, handed to the casting
// kernel; a candidate whose bound is not below the best hit found so far is not cast. Two facts keep
// the result equal to casting every candidate: the inflated target lies inside the ball of radius
// bound + swept radius about its position, so a segment that misses that ball (by more than the
// 1e-4 distance the cast accepts as touching, plus rounding) is a miss; and a hit's fraction is at
// least where the segment enters that ball. A body with more candidates than the casting kernel takes
// casts them here, one a lane; overflowing the candidate buffer falls back to casting every candidate.
constexpr int CCD_THREADS = 32;
constexpr int CCD_CAP = 256;
constexpr uint32_t CCD_TREE_CAP = 1024;          // tree hits per CCD body before the world scan
constexpr uint32_t TREE_LEAF_REF = 0x80000000u;  // leaf children in the broad-phase node records
constexpr uint32_t CCD_RANKS = 8;                // candidates of a body handed to the casting kernel

struct CcdCtx {
    V3 from, to, dir;
    float length, radius;
    uint32_t* status;
};

__device__ __noinline__ float cast_mesh(const BodyDev& b, const Shape& sj, const float4* __restrict__ hull, const CcdCtx& c,
                                        uint32_t j) {
    float f;
    return sweep_mesh(c.from, c.to, c.radius, sj, from4(b.pos[j]), q4(b.quat[j]), hull, c.status, f) ? f : 1.0f;
}

__device__ __forceinline__ float cast_one(const BodyDev& b, const Shape* __restrict__ shapes, const float4* __restrict__ hull,
                                          const CcdCtx& c, uint32_t j) {
    const Shape& sj = shapes[b.info[j].x];
    float f;
    bool hit;
    if (sj.type == SHAPE_PLANE) {
        hit = sweep_plane(c.from, c.dir, c.length, c.radius, sj, q4(b.quat[j]), f);
    } else if (sj.type == SHAPE_MESH) {
        return cast_mesh(b, sj, hull, c, j);
    } else {
        Inflated t{sj, from4(b.pos[j]), q4(b.quat[j]), c.radius, hull};
        hit = sweep_convex(c.from, c.dir, c.length, t, f);
    }
    return hit ? f : 1.0f;
}

// The cast of one candidate by a segment of lanes, with the same result as sweep_convex: the
// ternary search's decisions depend only on the probes, so each round evaluates every probe of
// the next levels of its decision tree at once (on 32 lanes 4 levels: 15 nodes x 2 probes) and then
// follows the taken path; the bisection likewise (on 32 lanes 5 levels: 31 probes). A node's
// (lo, hi) is replayed from the round's root with the same operations as the sequential loop,
// so every probe point, and the fraction, is bit-identical to sweep_convex's.
__device__ __forceinline__ void replay_ternary(float& l, float& h, uint32_t node) {
    uint32_t path = 0, depth = 0;  // bit t: the branch taken at depth t + 1 (collected leaf first)
    for (uint32_t x = node; x > 0; x = (x - 1) >> 1) {
        path = (path << 1) | ((x & 1u) ? 0u : 1u);  // odd child: d(m1) < d(m2) (hi = m2)
        ++depth;
    }
    for (uint32_t t = 0; t < depth; ++t) {
        const float m1 = l + (h - l) / 3.0f;
        const float m2 = h - (h - l) / 3.0f;
        if (((path >> t) & 1u) == 0u) h = m2;
        else l = m1;
    }
}

__device__ __forceinline__ void replay_bisect(float& l, float& h, uint32_t node) {
    uint32_t path = 0, depth = 0;
    for (uint32_t x = node; x > 0; x = (x - 1) >> 1) {
        path = (path << 1) | ((x & 1u) ? 0u : 1u);  // odd child: d(mid) <= 1e-8 (high = mid)
        ++depth;
    }
    for (uint32_t t = 0; t < depth; ++t) {
        const float mid = (l + h) * 0.5f;
        if (((path >> t) & 1u) == 0u) h = mid;
        else l = mid;
    }
}

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Casts handed to k_ccd_cast: rank r holds every body's candidate with the r-th smallest bound,
// item = CCD list entry, target body, bound (float bits). count[r] items at items[r m].
struct CcdItems {
    uint4* items;
    uint32_t* count;
    uint32_t m;
};

// step.rs:1068-1155: the candidates of CCD list entry blockIdx.x, and its clamp fraction from the
// planes and from what it casts itself (1 when not clamped).
__global__ void __launch_bounds__(CCD_THREADS) k_ccd_sweep(BodyDev b, const Shape* __restrict__ shapes,
                                                           const float4* __restrict__ hull, const uint32_t* __restrict__ ids,
                                                           const float2* __restrict__ par, uint32_t n,
                                                           const uint32_t* __restrict__ world_off,
                                                           const uint32_t* __restrict__ world_of,
                                                           const uint64_t* __restrict__ suppressed, uint32_t nsuppressed,
                                                           float dt, float* clamp, uint32_t* status,
                                                           const float4* __restrict__ tree_rec,
                                                           const uint32_t* __restrict__ tree_leaf, int tree_m,
                                                           const uint32_t* __restrict__ unb, uint32_t nunb,
                                                           CcdItems items) {
    __shared__ uint32_t cand[CCD_CAP], sorted[CCD_CAP];
    __shared__ uint32_t tlist[CCD_TREE_CAP];
    __shared__ uint32_t ntl;
    __shared__ float lb[CCD_CAP], slb[CCD_CAP];
    __shared__ uint32_t ncand;
    const uint32_t k = blockIdx.x, lane = threadIdx.x;
    const uint32_t i = ids[k];
    const float threshold = par[k].x, radius = par[k].y;
    const uint4 info = b.info[i];
    const Shape& si = shapes[info.x];
    const V3 from = from4(b.pos[i]);
    const V3 to = from + from4(b.linvel[i]) * dt;
    bool eligible = body_active(info.z) && !(info.y & (BF_STATIC | BF_KINEMATIC)) && threshold > 0.0f && radius > 0.0f &&
                    si.type != SHAPE_PLANE;
    eligible = eligible && !(len2(to - from) <= threshold * threshold);
    if (!eligible) {
        if (lane == 0) clamp[k] = 1.0f;
        return;
    }
    const V3 smin = vmin(from, to) - V3{radius, radius, radius}, smax = vmax(from, to) + V3{radius, radius, radius};
    const V3 delta = to - from;
    CcdCtx c;
    c.length = len(delta);
    c.dir = delta / c.length;
    c.from = from;
    c.to = to;
    c.radius = radius;
    c.status = status;
    // convex_sweep.rs:45-50: a vanishing motion casts nothing
    if (c.length <= 1.1920929e-7f) {
        if (lane == 0) clamp[k] = 1.0f;
        return;
    }
    const uint32_t gi = info.w & 0xFFFFu, mi = info.w >> 16;
    uint32_t lo = 0, hi = n;
    if (world_of) { lo = world_off[world_of[i]]; hi = world_off[world_of[i] + 1]; }
    // The targets: in a plain world, the step's broad-phase tree gives the proxies whose boxes
    // touch the swept box (the same closed test as the scan below, so the same set), plus the
    // proxies kept out of the tree (planes, meshes); in a batch, or when the list overflows,
    // every body of the world.
    const bool use_tree = tree_rec && !world_of && tree_m >= 1;
    if (lane == 0) {
        ncand = 0;
        ntl = 0;
        if (use_tree) {
            uint32_t cnt = 0;
            auto push = [&](uint32_t j) {
                if (cnt < CCD_TREE_CAP) tlist[cnt] = j;
                ++cnt;
            };
            const float4 qmin = make_float4(smin.x, smin.y, smin.z, 0.0f), qmax = make_float4(smax.x, smax.y, smax.z, 0.0f);
            auto touch = [&](float4 a, float4 b) {
                return a.x <= qmax.x && a.y <= qmax.y && a.z <= qmax.z && qmin.x <= b.x && qmin.y <= b.y && qmin.z <= b.z;
            };
            if (tree_m == 1) {
                push(tree_leaf[0]);
            } else {
                uint32_t stack[64];
                int sp = 0;
                stack[sp++] = 0u;
                while (sp > 0 && cnt <= CCD_TREE_CAP) {
                    const float4* r = tree_rec + size_t(stack[--sp]) * 4;
                    const float4 a = r[0], bb = r[1], cc = r[2], d = r[3];
                    const uint32_t ref[2] = {__float_as_uint(a.w), __float_as_uint(bb.w)};
                    const bool hit[2] = {touch(a, bb), touch(cc, d)};
                    for (int q = 0; q < 2; ++q) {
                        if (!hit[q]) continue;
                        if (ref[q] & TREE_LEAF_REF) push(ref[q] & ~TREE_LEAF_REF);
                        else if (sp < 64) stack[sp++] = ref[q];
                        else atomicOr(status, ST_TRAVERSAL_STACK);
                    }
                }
            }
            for (uint32_t u = 0; u < nunb; ++u) push(unb[u]);
            ntl = cnt;
        }
    }
    __syncthreads();
    const bool from_tree = use_tree && ntl <= CCD_TREE_CAP;
    const uint32_t nsrc = from_tree ? ntl : hi - lo;
    float best = 1.0f;
    for (uint32_t s = lane; s < nsrc; s += CCD_THREADS) {
        const uint32_t j = from_tree ? tlist[s] : lo + s;
        if (j == i) continue;
        const uint4 oj = b.info[j];
        if (oj.y & BF_NO_RESPONSE) continue;
        const uint32_t gj = oj.w & 0xFFFFu, mj = oj.w >> 16;
        if ((gi & mj) == 0 || (gj & mi) == 0) continue;
        const float4 amin = b.aabb_min[j], amax = b.aabb_max[j];
        // Aabb::overlaps (util.rs:28-38), closed on every axis
        if (!(amin.x <= smax.x && amin.y <= smax.y && amin.z <= smax.z && smin.x <= amax.x && smin.y <= amax.y &&
              smin.z <= amax.z))
            continue;
        if (nsuppressed) {
            const uint64_t key = (uint64_t(min(i, j)) << 32) | max(i, j);
            if (key_suppressed(suppressed, nsuppressed, key)) continue;
        }
        const Shape& sj = shapes[oj.x];
        if (sj.type == SHAPE_PLANE) {  // analytic and cheap: cast now
            best = fminf(best, cast_one(b, shapes, hull, c, j));
            continue;
        }
        // bounding ball of the inflated target, widened by the touch distance and rounding
        const V3 cj = from4(b.pos[j]);
        const float bound = len(vmax(vabs(V3{sj.lmin[0], sj.lmin[1], sj.lmin[2]}), vabs(V3{sj.lmax[0], sj.lmax[1], sj.lmax[2]})));
        const float slack = 1e-3f + 1e-5f * (len(cj) + len(from) + c.length);
        const float rr = bound + radius + slack;
        const V3 m = from - cj;
        const float bb = dot(m, c.dir);
        const float tca = fminf(fmaxf(-bb, 0.0f), c.length);
        if (len2(m + c.dir * tca) > rr * rr) continue;  // the segment misses the ball: no hit
        const float cc = len2(m) - rr * rr;
        float lower = 0.0f;
        if (cc > 0.0f) {
            const float disc = fmaxf(bb * bb - cc, 0.0f);
            lower = fmaxf((-bb - sqrtf(disc)) / c.length - 1e-6f - slack / c.length, 0.0f);
        }
        const uint32_t slot = atomicAdd(&ncand, 1u);
        if (slot < CCD_CAP) {
            cand[slot] = j;
            lb[slot] = lower;
        }
    }
    best = warp_min(best);
    __syncthreads();
    const uint32_t nc = ncand;
    if (nc > CCD_CAP) {
        // too many candidates for the buffer: cast every candidate that passes the same tests
        float mine = best;
        for (uint32_t s = lane; s < nsrc; s += CCD_THREADS) {
            const uint32_t j = from_tree ? tlist[s] : lo + s;
            if (j == i) continue;
            const uint4 oj = b.info[j];
            if ((oj.y & BF_NO_RESPONSE) || shapes[oj.x].type == SHAPE_PLANE) continue;
            const uint32_t gj = oj.w & 0xFFFFu, mj = oj.w >> 16;
            if ((gi & mj) == 0 || (gj & mi) == 0) continue;
            const float4 amin = b.aabb_min[j], amax = b.aabb_max[j];
            if (!(amin.x <= smax.x && amin.y <= smax.y && amin.z <= smax.z && smin.x <= amax.x && smin.y <= amax.y &&
                  smin.z <= amax.z))
                continue;
            if (nsuppressed && key_suppressed(suppressed, nsuppressed, (uint64_t(min(i, j)) << 32) | max(i, j))) continue;
            mine = fminf(mine, cast_one(b, shapes, hull, c, j));
        }
        best = warp_min(mine);
    } else {
        // order the candidates by their lower bound (rank by counting; ties by slot)
        for (uint32_t s = lane; s < nc; s += CCD_THREADS) {
            uint32_t r = 0;
            const float v = lb[s];
            for (uint32_t t = 0; t < nc; ++t) r += (lb[t] < v || (lb[t] == v && t < s)) ? 1u : 0u;
            sorted[r] = cand[s];
            slb[r] = v;
        }
        __syncthreads();
        if (nc <= CCD_RANKS) {
            if (lane < nc && slb[lane] < best) {
                const uint32_t at = atomicAdd(&items.count[lane], 1u);
                items.items[size_t(lane) * items.m + at] = make_uint4(k, sorted[lane], __float_as_uint(slb[lane]), 0u);
            }
        } else
        for (uint32_t w0 = 0; w0 < nc; w0 += CCD_THREADS) {
            if (!(slb[w0] < best)) break;
            const uint32_t s = w0 + lane;
            float f = 1.0f;
            if (s < nc && slb[s] < best) f = cast_one(b, shapes, hull, c, sorted[s]);
            best = fminf(best, warp_min(f));
        }
    }
    if (lane == 0) clamp[k] = best;
}

// The casts, all the bodies' first candidates before their second ones (whose bound a hit may
// already have overtaken). A cast is about 100 dependent GJK point distances of up to 64 iterations,
// so with few casts the chain is what counts and each takes a warp (16 rounds of probes), and with
// many the probes that the speculation wastes count and a warp runs two or four casts side by side
// (19 rounds of 14 or 15 probes, 29 of 6 or 7). Measured at 1,045 casts (2,048 bodies), a launch:
// 2.27 ms on 32 lanes, 2.24 on 16, 2.78 on 8; from two casts a scheduler on the wider ones run one
// after the other. The whole warp for one body after the other, walks in lockstep to the 64th
// iteration and a branch for every kind of simplex took 16.1 ms. What bounds it now: the walks on the
// taken path, about 60 steps a round of 2,400 cycles each (square root, divisions, one
// dependent chain).
constexpr uint32_t CCD_CAST_THREADS = 128;
constexpr uint32_t CCD_CAST_BLOCKS = 148 * 4;
constexpr uint32_t CCD_WARP_CASTS = 1184;  // casts up to which each takes a whole warp

__global__ void __launch_bounds__(CCD_CAST_THREADS) k_ccd_cast(BodyDev b, const Shape* __restrict__ shapes,
                                                               const float4* __restrict__ hull,
                                                               const uint32_t* __restrict__ ids,
                                                               const float2* __restrict__ par, float dt, float* clamp,
                                                               uint32_t* status, CcdItems items) {
    uint32_t off[CCD_RANKS + 1];
    off[0] = 0u;
#pragma unroll
    for (uint32_t r = 0; r < CCD_RANKS; ++r) off[r + 1] = off[r] + items.count[r];
    const uint32_t total = off[CCD_RANKS];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t g = total <= CCD_WARP_CASTS ? 32u : (total <= 2u * CCD_WARP_CASTS ? 16u : 8u);
    const uint32_t td = g == 32u ? 4u : (g == 16u ? 3u : 2u), bd = td + 1u;
    const uint32_t segs = 32u / g, sl = lane % g;
    const uint32_t mine = (g == 32u ? 0xffffffffu : (1u << g) - 1u) << (lane - sl);  // the segment's lanes
    // A walk takes at most 258 steps (the first support point, 64 iterations of at most four, the end), a
    // cast 41 rounds of them, and each vote is a step of every walk: the loop below ends before `left` does.
    // The segment's cast (the same values on all its lanes) and the lane's walk.
    enum { TERNARY, CLOSEST, BISECT, IDLE };
    int phase = IDLE;
    uint32_t x = warp * segs + lane / g, entry = 0, steps = 0;
    V3 from{}, dir{};
    float length = 0.0f, lo = 0.0f, hi = 0.0f;
    Inflated t{};
    Walk w;
    w.done = true;
    w.d2 = 0.0f;
    bool ready = true;   // the segment's round is over and its decisions are taken
    uint32_t seen = 0u;  // the last vote on the walks that are done
    // The loop ends by itself: a segment's lanes hold the same cast, each vote is a step of every walk that is
    // not done, a walk has 258 steps at most (the first support point, 64 iterations of up to four, the end), a
    // cast 41 rounds of walks, and every cast is taken once. (A count of the votes beside it is one register too
    // many: it spills, and a launch takes 1.5 % longer; in shared memory 5 %.)
    for (;;) {
        if (ready) {
            // The next round of probes: of this cast, or of the segment's next one.
            w.done = true;
            bool ended = false;
            float f = 0.0f;
            if (phase == BISECT) {
                // The steps end early where they can change nothing any more: the midpoint rounds to
                // hi, whose probe touched, or to a lo whose probe did not.
                f = (lo + hi) * 0.5f;
                ended = steps == 60u || f == hi || (f == lo && lo > 0.0f);
            }
            while (ended || (phase == IDLE && x < total)) {
                if (ended) {
                    // Fractions are not negative, so their bits order as they do.
                    if (sl == 0u) atomicMin(reinterpret_cast<unsigned int*>(&clamp[entry]), __float_as_uint(f));
                    __syncwarp(mine);
                    ended = false;
                    phase = IDLE;
                    continue;
                }
                uint32_t r = 0, at = 0;
#pragma unroll
                for (uint32_t q = 0; q < CCD_RANKS; ++q)
                    if (x >= off[q]) { r = q; at = x - off[q]; }
                x += nwarps * segs;
                const uint4 it = items.items[size_t(r) * items.m + at];
                // A hit may have overtaken the cast's bound. One lane reads for the segment, which has to go
                // one way: other warps lower the clamp meanwhile.
                float reach = 0.0f;
                if (sl == 0u) reach = *(volatile float*)&clamp[it.x];
                reach = __shfl_sync(mine, reach, 0, int(g));
                if (!(__uint_as_float(it.z) < reach)) continue;
                entry = it.x;
                const uint32_t i = ids[entry];
                from = from4(b.pos[i]);
                const V3 to = from + from4(b.linvel[i]) * dt;
                const V3 delta = to - from;
                length = len(delta);
                dir = delta / length;
                const Shape& sj = shapes[b.info[it.y].x];
                if (sj.type == SHAPE_MESH) {
                    const CcdCtx c{from, to, dir, length, par[entry].y, status};
                    f = 1.0f;
                    if (sl == 0u) f = cast_mesh(b, sj, hull, c, it.y);
                    ended = true;
                    continue;
                }
                t = Inflated{sj, from4(b.pos[it.y]), q4(b.quat[it.y]), par[entry].y, hull};
                phase = TERNARY;
                steps = 0;
                lo = 0.0f;
                hi = 1.0f;
            }
            if (phase != IDLE) {
                float l = lo, h = hi;
                f = (lo + hi) * 0.5f;  // the closest approach, or replaced below
                bool on = sl == 0u;
                if (phase == TERNARY) {
                    on = sl < 2u * ((1u << min(td, 40u - steps)) - 1u);
                    replay_ternary(l, h, sl >> 1);
                    f = (sl & 1u) ? h - (h - l) / 3.0f : l + (h - l) / 3.0f;
                } else if (phase == BISECT) {
                    on = sl < (1u << min(bd, 60u - steps)) - 1u;
                    replay_bisect(l, h, sl);
                    f = (l + h) * 0.5f;
                }
                if (on) w.start(from + dir * (f * length));
            }
        }
        if (!__any_sync(0xffffffffu, phase != IDLE)) break;
        if (!w.done) w.step(t);
        // Follow the decisions as far as their probes are done: a round ends with the probes on the
        // taken path, whatever the walks beside it are still at.
        const uint32_t done = __ballot_sync(0xffffffffu, w.done);  // every lane votes, the idle ones too
        ready = false;
        if (done == seen) continue;  // uniform across the warp
        seen = done;
        const uint32_t here = done >> (lane - sl);  // bit k: the segment's probe k
        const uint32_t depth = phase == TERNARY ? min(td, 40u - steps) : (phase == BISECT ? min(bd, 60u - steps) : 0u);
        const float closest = __shfl_sync(0xffffffffu, w.d2, 0, int(g));
        float l = lo, h = hi;
        uint32_t n = 0;
        ready = phase != IDLE && (phase != CLOSEST || (here & 1u));
        for (uint32_t d = 0; d < bd; ++d) {  // (td < bd)
            const uint32_t at = min(phase == TERNARY ? 2u * n : n, g - 2u);
            const float d1 = __shfl_sync(0xffffffffu, w.d2, int(at), int(g));
            const float d2 = __shfl_sync(0xffffffffu, w.d2, int(at + 1u), int(g));
            if (d >= depth || !ready) continue;
            const uint32_t need = (phase == TERNARY ? 3u : 1u) << at;
            if ((here & need) != need) {
                ready = false;
                continue;
            }
            bool lower;
            if (phase == TERNARY) {
                const float m1 = l + (h - l) / 3.0f, m2 = h - (h - l) / 3.0f;
                lower = d1 < d2;
                if (lower) h = m2;
                else l = m1;
            } else {
                const float mid = (l + h) * 0.5f;
                lower = d1 <= 1e-8f;
                if (lower) h = mid;
                else l = mid;
            }
            n = 2u * n + (lower ? 1u : 2u);
        }
        if (!ready) continue;
        lo = l;
        hi = h;
        steps += depth;
        if (phase == TERNARY) {
            if (steps == 40u) phase = CLOSEST;
        } else if (phase == CLOSEST) {
            if (closest > 1e-8f) {
                phase = IDLE;  // a miss
            } else {
                phase = BISECT;
                steps = 0;
                hi = (lo + hi) * 0.5f;
                lo = 0.0f;
            }
        }
    }
}

// step.rs:1210-1214, after the position integration (which leaves the velocities unchanged).
__global__ void k_ccd_apply(BodyDev b, const uint32_t* __restrict__ ids, const float* __restrict__ clamp, uint32_t m,
                            float dt) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    const float c = clamp[k];
    if (!(c < 1.0f)) return;
    const uint32_t i = ids[k];
    const V3 p = from4(b.pos[i]);
    const V3 from = p - from4(b.linvel[i]) * dt;
    b.pos[i] = to4(from + (p - from) * c, 0.0f);
}

}  // namespace

void launch_ccd_sweep(const BodyDev& b, const Shape* shapes, const float4* hull, const uint32_t* ids, const float2* par,
                      uint32_t m, uint32_t n, const uint32_t* world_off, const uint32_t* world_of,
                      const uint64_t* suppressed, uint32_t nsuppressed, float dt, float* clamp, uint32_t* status,
                      const float4* tree_rec, const uint32_t* tree_leaf, int tree_m, const uint32_t* unb,
                      uint32_t nunb, CcdScratch& scratch, cudaStream_t s) {
    if (m == 0) return;
    scratch.items.reserve(size_t(m) * CCD_RANKS);
    scratch.count.reserve(CCD_RANKS);
    check_cuda(cudaMemsetAsync(scratch.count.p, 0, CCD_RANKS * sizeof(uint32_t), s), "memset");
    const CcdItems items{scratch.items.p, scratch.count.p, m};
    k_ccd_sweep<<<m, CCD_THREADS, 0, s>>>(b, shapes, hull, ids, par, n, world_off, world_of, suppressed, nsuppressed,
                                          dt, clamp, status, tree_rec, tree_leaf, tree_m, unb, nunb, items);
    const uint64_t lanes = uint64_t(m) * CCD_RANKS * 32u;  // a warp for every cast there may be
    const uint32_t blocks = uint32_t(std::min<uint64_t>((lanes + CCD_CAST_THREADS - 1) / CCD_CAST_THREADS, CCD_CAST_BLOCKS));
    k_ccd_cast<<<blocks, CCD_CAST_THREADS, 0, s>>>(b, shapes, hull, ids, par, dt, clamp, status, items);
}

void launch_ccd_apply(const BodyDev& b, const uint32_t* ids, const float* clamp, uint32_t m, float dt, cudaStream_t s) {
    if (m == 0) return;
    k_ccd_apply<<<(m + 127) / 128, 128, 0, s>>>(b, ids, clamp, m, dt);
}

}  // namespace bgpu
