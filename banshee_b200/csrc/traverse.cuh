// Closest-hit / any-hit traversal of the 4-wide BVH and of the 8-wide
// compressed BVH.
//
// Replaces Bvh::Intersect(ray, Hit&) and Bvh::Intersect(ray)
// (accelerator/bvh.cpp:499-647) together with Mesh::IntersectShape /
// IntersectFace (primitive/mesh.cpp:7-45, 216-261):
//   * a triangle is accepted when its Moller-Trumbore t is in (tmin, best],
//     computed with the reference's exact operation order in the bundle's
//     object space (ray transformed by minv as transform_ray does,
//     math/mathutils.h:154-157; skipped for identity bundles, where it is exact);
//   * the box test is this project's own: a slab test with a relative slack on
//     the exit distance, so no box that holds an accepted triangle is culled.
// Children are visited nearest-first; stack entries keep their entry distance
// and are culled against the current closest hit, widened by the same slack,
// when popped.
//
// Two kinds of walk share the code:
//   plain  slabs as (plane - o) * (1/d), slack 4e-7 (more than the 2*gamma(3)
//          rounding bound).  Among triangles whose t are equal to the last bit the
//          one visited last wins, so its visiting order is part of the result.
//   packed one fused multiply-add per plane with a per-ray bound of the roundings,
//          on the 64-byte QNode4 nodes, on the 128-byte nodes (fused) or on the
//          8-wide nodes, slack 1e-5.  Its boxes contain the plain ones, its order
//          differs in detail.  The plain walk decides, by a second walk of the ray on
//          the plain nodes, when two triangles share the closest t to the last bit and
//          when it might not come to the triangle that was hit (plain_reaches).  So an
//          any-hit answer is that of the plain walk, and so are ids, t, u and v, ties
//          included, unless the rounding of a triangle's t takes it in front of the
//          triangle's own box by more than 1e-5 of t: whether such a triangle hides a
//          surface within that distance behind it depends on which the walk comes to
//          first.  (t rounds by at most 12 x 2^-24 (t + 2 edges) / c, c = sine of the corner
//          x cosine of incidence: for triangles small against t, c above 0.07 rules it out.)
// Rays the packed arithmetic does not cover (components out of its range, not
// finite) take the plain walk from the start, as does the
// instrumented replay (COUNT).
#pragma once

#include <type_traits>

#include "device_common.cuh"
#include "scene_types.h"
#include "../../include/banshee_gpu.h"

namespace bg {

constexpr int kStackSize = 64;     // entries per ray, 4-wide; the builder checks max_stack against it
constexpr int kStackSize8 = 96;    // entries per ray, 8-wide (up to 7 pushes per level)
// Walks (template parameter WALK): kWalkPlain the plain walk alone; kWalkPacked
// and kWalkFused the packed arithmetic on QNode4 / QNode8 nodes and on the
// 128-byte nodes, one ray per lane; kWalkGroup the packed walk by a group of lanes.
constexpr int kWalkPlain = 0, kWalkPacked = 1, kWalkGroup = 2, kWalkFused = 3;

// stack entries per ray kept in shared memory: 8 for the 4-wide walks, 12 for the
// packed one (1M-triangle soup, closest / any incoherent: 4 entries 1241 / 1646
// Mrays/s, 8 1360 / 1779, 12 1436 / 1835), none for the 8-wide ones
template <int WIDTH, int WALK>
__host__ __device__ constexpr int smem_stack_entries() { return WIDTH == 8 ? 0 : WALK == kWalkPacked ? 12 : 8; }
template <int WIDTH>
__host__ __device__ constexpr int stack_entries() { return WIDTH == 8 ? kStackSize8 : kStackSize; }
// Traversal steps between warp refill points.  Renders (fused and plain walk):
// closest hit 24 > 16 > 12 by about 1 % of the frame, any hit 16 > 8, 32; 12 / 8
// cost the C3 frame 3 %.  Casts on packed nodes: 12 / 8 (coherent closest 1953
// against 1878 Mrays/s at 24 / 16, incoherent any 1865 against 1798), 8-wide nodes
// the same (incoherent any 1615 against 1530).
// (Measured and rejected: each lane's next ray prefetched into shared memory by
// cp.async from a per-warp pool of 32 indices, refilling every 24 / 12 / 8 / 4
// steps: C3 567 -> 528 / 519 / 511 / 280 Msamples/s with 4-wide nodes; and
// registers capped at 48 or 40 for 40 or 48 resident warps per SM: spills,
// 559 -> 544 / 495 Msamples/s.)
template <bool ANY, int WALK>
__host__ __device__ constexpr int refill_steps() { return WALK == kWalkPacked ? (ANY ? 8 : 12) : (ANY ? 16 : 24); }
constexpr float kBoxSlack = 4e-7f;
// The slack is applied as one fused multiply-add, t1 + |t1| * kBoxSlack rounded
// once: the same half-ulp guarantee as a multiply and an add (whose product
// term is exact to far below an ulp of t1), one instruction fewer per child
// box (measured: C3 extension and shadow traversal 1 % shorter, C2 coherent
// casts 1.2-1.6 % faster, hits unchanged).
// (Measured and rejected: slab distances as one fmaf(P, 1/d, -o/d) each, with a
// per-ray absolute error bound added to the slack.  The bound, 2^-24 max|o/d|,
// is huge for rays nearly parallel to an axis, so such rays visited most of the
// tree: C3 ran at 8 instead of 500 Msamples/s.)

// Slack of the packed walk: its box tests and its culling of popped entries.
constexpr float kFastSlack = 1e-5f;
constexpr float kZeroInv = 2e15f;    // its 1 / d for a component of 0

// Ray::flags: bits 0-2 sign of 1/d per axis
constexpr uint32_t kOctMask = 7u;
constexpr uint32_t kPlainWalk = 8u;   // walk the plain nodes
constexpr uint32_t kTie = 16u;        // packed walk: two triangles at the closest t, or no room on the stack

// kWalkPacked and kWalkFused keep the ray's origin and direction, which they need
// only for a new bundle's object-space ray and for a plain visit, in shared memory:
// six registers less during the walk (from global memory, C3 was 3 % slower).
template <int WALK>
constexpr bool kKeeps = WALK == kWalkPacked || WALK == kWalkFused;
struct RayFast {
    v3 inv;          // 1 / d
    v3 cn, cf;       // -o / d less / plus a bound of the roundings: near / far planes
    float tmin;
    uint32_t flags;
    int32_t idx;     // index in the ray array
};
template <int WALK>
struct Ray : RayFast {};
template <>
struct Ray<kWalkGroup> : RayFast {
    v3 o, d;
};
template <>
struct Ray<kWalkPlain> {
    v3 o, d, inv;
    float tmin;
    uint32_t flags;
    int32_t idx;
};

// the scene and the ray array of one launch
struct TraceScene : DevScene {
    const float4* rays;
    // kWalkPacked, kWalkFused: this lane's in shared memory, its ray at own[0] and
    // own[ownstep], its closest hit's TriRec and (any hit) t at own[2 ownstep]
    float4* own;
    int ownstep;
};

// Whether the packed arithmetic covers the scene, on its packed or 8-wide nodes and on
// the 128-byte ones (which need no room for packed nodes).
template <int WIDTH>
__host__ __device__ __forceinline__ bool packed_walk(const DevScene& S) {
    return S.extent <= 1e15f && (WIDTH == 8 || S.qnodes != nullptr);
}
__host__ __device__ __forceinline__ bool fused_walk(const DevScene& S) { return S.extent <= 1e15f && S.ranged; }

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ uint32_t octant(v3 inv) {
    return (__float_as_uint(inv.x) >> 31) | ((__float_as_uint(inv.y) >> 30) & 2u) | ((__float_as_uint(inv.z) >> 29) & 4u);
}

// walk: kPlainWalk to walk the plain nodes whatever the ray, 0 otherwise
__device__ __forceinline__ void make_ray(RayFast& r, float extent, uint32_t walk, float4 a, float4 b, int32_t idx) {
    r.idx = idx;
    r.tmin = a.w;
    r.inv = mk(1.f / b.x, 1.f / b.y, 1.f / b.z);
    const float far = max3(fabsf(a.x), fabsf(a.y), fabsf(a.z));
    const v3 ad = mk(fabsf(b.x), fabsf(b.y), fabsf(b.z));
    // A component of 0 (a camera's middle column) counts as 5e-16 while another is 1e-8 or
    // more and tmin is not negative: distances to its planes are then negative or beyond the
    // scene, as with the infinite inverse, except within the bound of the roundings.
    const bool zeros = a.w >= 0.f && max3(ad.x, ad.y, ad.z) >= 1e-8f;
    // the packed arithmetic's range (comparisons false for NaN: plain walk)
    auto in = [&](float x) { return x == 0.f ? zeros : x >= 1e-15f && x <= 1e15f; };
    const bool ok = far <= 1e15f && in(ad.x) && in(ad.y) && in(ad.z);
    if (ok && walk == 0u) {
        if (b.x == 0.f) r.inv.x = copysignf(kZeroInv, b.x);
        if (b.y == 0.f) r.inv.y = copysignf(kZeroInv, b.y);
        if (b.z == 0.f) r.inv.z = copysignf(kZeroInv, b.z);
    }
    r.flags = octant(r.inv) | (ok ? walk : kPlainWalk);
    const v3 ai = mk(fabsf(r.inv.x), fabsf(r.inv.y), fabsf(r.inv.z));
    // the bound of the roundings: those of a plane's distance here (of the intercepts and
    // the final multiply-add) are together at most 3 x 2^-24 of (|plane| + |o|) / |d|, and the
    // plain test reaches, by its slack and its own three roundings, 7e-7 of the distance
    // further than the exact one, on either plane.  So with 1e-6 this one enters every box
    // that the plain one enters.  (With 4.8e-7 a hit just behind tmin could be lost.)
    const float e = (extent + far) * 1e-6f;
    const float ex = fmaf(e, ai.x, 1e-36f), ey = fmaf(e, ai.y, 1e-36f), ez = fmaf(e, ai.z, 1e-36f);
    const float ox = a.x * r.inv.x, oy = a.y * r.inv.y, oz = a.z * r.inv.z;
    r.cn = mk(-ox - ex, -oy - ey, -oz - ez);
    r.cf = mk(ex - ox, ey - oy, ez - oz);
}
__device__ __forceinline__ void make_ray(Ray<kWalkPlain>& r, float, uint32_t, float4 a, float4 b, int32_t idx) {
    r.idx = idx;
    r.tmin = a.w;
    r.inv = mk(1.f / b.x, 1.f / b.y, 1.f / b.z);
    r.flags = octant(r.inv) | kPlainWalk;
}
// keeping and giving back the ray's origin and direction
__device__ __forceinline__ void keep_ray(const TraceScene& S, RayFast&, float4 a, float4 b) {
    S.own[0] = a;
    S.own[S.ownstep] = b;
}
__device__ __forceinline__ void world_ray(const TraceScene& S, const RayFast&, v3& o, v3& d) {
    const float4 a = S.own[0], b = S.own[S.ownstep];
    o = mk(a.x, a.y, a.z);
    d = mk(b.x, b.y, b.z);
}
template <class RAY>
__device__ __forceinline__ void keep_regs(RAY& r, float4 a, float4 b) {
    r.o = mk(a.x, a.y, a.z);
    r.d = mk(b.x, b.y, b.z);
}
__device__ __forceinline__ void keep_ray(const TraceScene&, Ray<kWalkGroup>& r, float4 a, float4 b) { keep_regs(r, a, b); }
__device__ __forceinline__ void keep_ray(const TraceScene&, Ray<kWalkPlain>& r, float4 a, float4 b) { keep_regs(r, a, b); }
__device__ __forceinline__ void world_ray(const TraceScene&, const Ray<kWalkGroup>& r, v3& o, v3& d) { o = r.o; d = r.d; }
__device__ __forceinline__ void world_ray(const TraceScene&, const Ray<kWalkPlain>& r, v3& o, v3& d) { o = r.o; d = r.d; }

// Mesh::IntersectFace (primitive/mesh.cpp:7-45), bit-exact.
__device__ __forceinline__ bool mt_test(v3 o, v3 d, v3 p1, v3 e1, v3 e2, float tmin, float tmax,
                                        float& t, float& a, float& b) {
    v3 s1 = cross(d, e2);
    float invd = 1.f / dot(s1, e1);
    v3 dd = sub(o, p1);
    float b1 = dot(dd, s1) * invd;
    if (b1 < 0.f || b1 > 1.f) return false;
    v3 s2 = cross(dd, e1);
    float b2 = dot(d, s2) * invd;
    if (b2 < 0.f || b1 + b2 > 1.f) return false;
    float tmp = dot(e2, s2) * invd;
    if (tmp > tmin && tmp <= tmax) {
        t = tmp; a = b1; b = b2;
        return true;
    }
    return false;
}

// ray in the object space of bundle `bundle`; with WT also the watertight
// test's shear (Woop, Benthin and Wald, "Watertight Ray/Triangle
// Intersection", JCGT 2(1), 2013): kz = the axis of the largest |d|, kx, ky
// the next two (swapped when d[kz] < 0, keeping the winding), sx = d[kx] /
// d[kz], sy = d[ky] / d[kz], sz = 1 / d[kz]
struct ObjRay {
    int bundle;
    v3 o, d;
};
struct ObjRayWT : ObjRay {
    int kx, ky, kz;
    float sx, sy, sz;
};

__device__ __forceinline__ float comp(v3 v, int k) { return k == 0 ? v.x : k == 1 ? v.y : v.z; }

__device__ __forceinline__ void shear(ObjRay&) {}
__device__ __forceinline__ void shear(ObjRayWT& c) {
    const float ax = fabsf(c.d.x), ay = fabsf(c.d.y), az = fabsf(c.d.z);
    c.kz = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
    c.kx = c.kz == 2 ? 0 : c.kz + 1;
    c.ky = c.kx == 2 ? 0 : c.kx + 1;
    const float dz = comp(c.d, c.kz);
    if (dz < 0.f) { const int t = c.kx; c.kx = c.ky; c.ky = t; }
    c.sx = comp(c.d, c.kx) / dz;
    c.sy = comp(c.d, c.ky) / dz;
    c.sz = 1.f / dz;
}

template <class RAY, class OR>
__device__ __forceinline__ void obj_ray(const TraceScene& S, const RAY& r, int b, OR& c) {
    if (b == c.bundle) return;
    c.bundle = b;
    world_ray(S, r, c.o, c.d);
    if (b >= 0) {
        const float4* mi = reinterpret_cast<const float4*>(S.bundles[b].minv);   // three 16-byte rows
        const float4 m0 = __ldg(mi), m1 = __ldg(mi + 1), m2 = __ldg(mi + 2);
        const float m[12] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w, m2.x, m2.y, m2.z, m2.w};
        c.o = xf_point(m, c.o);
        c.d = xf_vector(m, c.d);
    }
    shear(c);
}

// Watertight ray / triangle test (Woop, Benthin and Wald 2013) on the exact
// vertices: the edge functions U, V, W of an edge are computed from the same
// sheared vertex coordinates in both triangles that share it (and are exact
// negatives of each other there), so no ray passes between them.  Edges are
// inclusive; an edge function that comes out exactly 0 is recomputed in double
// precision.  Returns t and the barycentrics of p2 (a) and p3 (b), as
// Moller-Trumbore's b1, b2.
__device__ __forceinline__ bool wt_test(const ObjRayWT& c, v3 p1, v3 p2, v3 p3, float tmin, float tmax, float& t,
                                        float& a, float& b) {
    const v3 A = sub(p1, c.o), B = sub(p2, c.o), C = sub(p3, c.o);
    const float az = comp(A, c.kz), bz = comp(B, c.kz), cz = comp(C, c.kz);
    const float ax = comp(A, c.kx) - c.sx * az, ay = comp(A, c.ky) - c.sy * az;
    const float bx = comp(B, c.kx) - c.sx * bz, by = comp(B, c.ky) - c.sy * bz;
    const float cx = comp(C, c.kx) - c.sx * cz, cy = comp(C, c.ky) - c.sy * cz;
    float U = cx * by - cy * bx;
    float V = ax * cy - ay * cx;
    float W = bx * ay - by * ax;
    if (U == 0.f || V == 0.f || W == 0.f) {
        U = float(double(cx) * double(by) - double(cy) * double(bx));
        V = float(double(ax) * double(cy) - double(ay) * double(cx));
        W = float(double(bx) * double(ay) - double(by) * double(ax));
    }
    if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
    const float det = U + V + W;
    if (det == 0.f) return false;
    const float T = U * (c.sz * az) + V * (c.sz * bz) + W * (c.sz * cz);
    const float rcp = 1.f / det;
    const float tt = T * rcp;
    if (!(tt > tmin && tt <= tmax)) return false;
    t = tt;
    a = V * rcp;
    b = W * rcp;
    return true;
}

// Whether the plain walk comes to the triangle of a hit at t that another walk, with wider
// boxes, has found: the plain box test, with t as the closest hit so far, of a box inside the
// triangle's own.  Every box that holds the triangle has its planes at least as far out, the
// plain walk's closest hit is never closer (what it tests, the other walk has tested), and
// subtraction, multiplication, minimum and maximum round monotonously: if the plain test lets
// this box pass, it lets all those pass.  (Without it a ray by an edge, or to a point on a
// surface, got other answers from other walks: the rounding of the triangle's test grows with
// distance over edge length and with incidence, and takes the true hit out of the box.)
// Moller-Trumbore's record holds p2 - p1, rounded, not p2.  A little less of it, added to p1,
// comes out between p1 and p2, as the rounding of a sum is monotone and p2 a float.
// Once per ray, at its end (1M-triangle soup, closest / any incoherent 1400 / 1797 Mrays/s
// without it, 1440 / 1820 with it, any coherent 3845 and 3700; a 6M-triangle frame 29.0 and
// 29.4 ms, 29.8 with the record read by words).  Also measured: bounds of the test's rounding
// instead, at every hit casts 4-12 % slower, at the ray's end (the plain walk for what they
// leave open) the frame 44.6 ms; a call out of line 31.6 ms.
template <bool WT>
__device__ __forceinline__ bool plain_reaches(const DevScene& S, int tri, int prim, float t, const float* o, v3 inv, float tmin) {
    const float4* f = reinterpret_cast<const float4*>(S.tris + tri);
    float4 a = __ldg(f), b = __ldg(f + 1), c = __ldg(f + 2);
    const int bundle = __float_as_int(a.w);
    if (bundle >= 0) {                       // the corners themselves
        f = reinterpret_cast<const float4*>(S.shade + (prim & kPrimMask));
        a = __ldg(f); b = __ldg(f + 1); c = __ldg(f + 2);
        const float4* m = reinterpret_cast<const float4*>(S.bundles[bundle].m);
        auto row = [&](float4 r, float4 v) { return r.x * v.x + r.y * v.y + r.z * v.z + r.w; };
        const float4 m0 = __ldg(m), m1 = __ldg(m + 1), m2 = __ldg(m + 2);
        a = make_float4(row(m0, a), row(m1, a), row(m2, a), 0.f);
        b = make_float4(row(m0, b), row(m1, b), row(m2, b), 0.f);
        c = make_float4(row(m0, c), row(m1, c), row(m2, c), 0.f);
    } else if (!WT) {
        const float k = 1.f - 0x1p-20f;
        b = make_float4(fmaf(b.x, k, a.x), fmaf(b.y, k, a.y), fmaf(b.z, k, a.z), 0.f);
        c = make_float4(fmaf(c.x, k, a.x), fmaf(c.y, k, a.y), fmaf(c.z, k, a.z), 0.f);
    }
    float t0 = tmin, t1 = t;
    auto axis = [&](float x, float y, float z, float from, float i) {
        if (fabsf(i) == kZeroInv) i = copysignf(__int_as_float(0x7f800000), i);   // the plain walk's 1 / 0
        const float s0 = (min3(x, y, z) - from) * i, s1 = (max3(x, y, z) - from) * i;
        t0 = fmaxf(t0, fminf(s0, s1));
        t1 = fminf(t1, fmaxf(s0, s1));
    };
    axis(a.x, b.x, c.x, o[0], inv.x);
    axis(a.y, b.y, c.y, o[1], inv.y);
    axis(a.z, b.z, c.z, o[2], inv.z);
    return t0 <= fmaf(fabsf(t1), kBoxSlack, t1);
}

// entry distance of a child that is not hit: +inf
#define kMiss __int_as_float(0x7f800000)

// Orders four children by entry distance with a sorting network on registers
// (a missed child's +inf sorts last).
// ALL = false: only the nearest comes first (an any-hit ray: the order of the
// others does not pay for its two comparators).
template <bool ALL = true>
__device__ __forceinline__ void sort4(float (&t)[4], int32_t (&c)[4]) {
    auto cex = [&](int a, int b) {
        const bool sw = t[a] > t[b];
        const float ta = t[a], tb = t[b];
        const int ca = c[a], cb = c[b];
        t[a] = sw ? tb : ta; t[b] = sw ? ta : tb;
        c[a] = sw ? cb : ca; c[b] = sw ? ca : cb;
    };
    cex(0, 1); cex(2, 3); cex(0, 2);
    if (ALL) { cex(1, 3); cex(1, 2); }
}

// Plain visit of 4-wide node p: its children in order of entry distance, +inf for
// one that is not hit.  A ray with infinite direction components can enter an empty
// slot (all its slabs are 0 or NaN); such a child is dropped when it is popped, or
// here (DROP) where the walk's pops do not test for it: that test in every pop cost
// the fused any-hit walk 5 % (the plain one: 100 triangles, any hits 17.2 against 17.9
// Grays/s, 4.7 against 4.8 with 4,000).  (The near / far planes of each axis are picked by load
// address: the node stores lo and hi of an axis in adjacent float4s.)
struct Children4 {
    float t[4];
    int32_t c[4];
    int nh;      // the first nh were hit
};
template <bool DROP>
__device__ __forceinline__ Children4 box4_plain(const float4* __restrict__ p, v3 o, v3 inv, uint32_t flags, float tmin,
                                                float best) {
    const int fx = int(flags & 1u), fy = int((flags >> 1) & 1u), fz = int((flags >> 2) & 1u);
    const float4 nx4 = __ldg(p + fx), fx4 = __ldg(p + (1 - fx));
    const float4 ny4 = __ldg(p + 2 + fy), fy4 = __ldg(p + 3 - fy);
    const float4 nz4 = __ldg(p + 4 + fz), fz4 = __ldg(p + 5 - fz);
    const int4 c = __ldg(reinterpret_cast<const int4*>(p + 6));
    const float nxa[4] = {nx4.x, nx4.y, nx4.z, nx4.w}, fxa[4] = {fx4.x, fx4.y, fx4.z, fx4.w};
    const float nya[4] = {ny4.x, ny4.y, ny4.z, ny4.w}, fya[4] = {fy4.x, fy4.y, fy4.z, fy4.w};
    const float nza[4] = {nz4.x, nz4.y, nz4.z, nz4.w}, fza[4] = {fz4.x, fz4.y, fz4.z, fz4.w};
    Children4 r;
    r.c[0] = c.x; r.c[1] = c.y; r.c[2] = c.z; r.c[3] = c.w;
    r.nh = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float ax = (nxa[i] - o.x) * inv.x;
        float bx = (fxa[i] - o.x) * inv.x;
        float ay = (nya[i] - o.y) * inv.y;
        float by = (fya[i] - o.y) * inv.y;
        float az = (nza[i] - o.z) * inv.z;
        float bz = (fza[i] - o.z) * inv.z;
        float t0 = fmaxf(fmaxf(ax, ay), fmaxf(az, tmin));
        float t1 = fminf(fminf(bx, by), fminf(bz, best));
        t1 = fmaf(fabsf(t1), kBoxSlack, t1);
        const bool hit = t0 <= t1 && !(DROP && r.c[i] == kEmptyChild);
        r.t[i] = hit ? t0 : kMiss;
        r.nh += hit ? 1 : 0;
    }
    sort4(r.t, r.c);
    return r;
}

// 32 bytes in one load (32-byte aligned)
struct Words8 {
    uint32_t w[8];
};
__device__ __forceinline__ Words8 ldg256(const void* p) {
    Words8 r;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
        : "l"(p));
    return r;
}

// Two multiply-adds in one instruction: {a0, a1} * {m, m} + {c0, c1}
__device__ __forceinline__ float2 fma2(float a0, float a1, float m, float c0, float c1) {
    float2 r;
    asm("{\n\t.reg .b64 a, m, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 m, {%4, %4};\n\tmov.b64 c, {%5, %6};\n\t"
        "fma.rn.f32x2 d, a, m, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a0), "f"(a1), "f"(m), "f"(c0), "f"(c1));
    return r;
}
// Near and far distance of the slab whose plane bytes are byte `i` of words n
// and f: the bytes as the floats 2^15 + q, slope m, intercepts cn, cf.
__device__ __forceinline__ float2 slab(uint32_t n, uint32_t f, int i, float m, float cn, float cf) {
    const uint32_t sel = 0x7604u | (uint32_t(i) << 4);
    return fma2(__uint_as_float(__byte_perm(n, 0x47000000u, sel)), __uint_as_float(__byte_perm(f, 0x47000000u, sel)), m, cn, cf);
}

// Test the 4 children of packed node `ni` (packed walk): entry distances, +inf
// for a child that is not hit.  `cull`: the distance beyond which nothing
// matters.  (An empty slot's byte box is inverted, but the slack can be longer
// than a very small box: an empty child may come back as hit, and is dropped
// where it is visited.)
// What bounds the walk on incoherent rays is the L1's data pipe: 91-95 % of its
// peak with the 128-byte nodes (seven 16-byte loads per visit, each lane on a
// line of its own), issue slots 50 %.  Two 32-byte loads per visit bring it to
// 54-62 %; the instructions of the byte decode (one PRMT per plane) are paid for
// by the slabs' multiply-adds, two planes at a time.
__device__ __forceinline__ void box4_packed(const QNode4* __restrict__ nodes, int ni, const RayFast& r, float cull,
                                            float (&tn)[4], int32_t (&ch)[4]) {
    const Words8 A = ldg256(nodes + ni), B = ldg256(reinterpret_cast<const char*>(nodes + ni) + 32);
    auto F = [](uint32_t v) { return __uint_as_float(v); };
    const float ix = F(A.w[3]) * r.inv.x, iy = F(A.w[4]) * r.inv.y, iz = F(A.w[5]) * r.inv.z;
    const float2 cx = fma2(F(A.w[0]), F(A.w[0]), r.inv.x, r.cn.x, r.cf.x);
    const float2 cy = fma2(F(A.w[1]), F(A.w[1]), r.inv.y, r.cn.y, r.cf.y);
    const float2 cz = fma2(F(A.w[2]), F(A.w[2]), r.inv.z, r.cn.z, r.cf.z);
    const bool gx = r.flags & 1u, gy = r.flags & 2u, gz = r.flags & 4u;
    const uint32_t nx = gx ? A.w[7] : A.w[6], fx = gx ? A.w[6] : A.w[7];
    const uint32_t ny = gy ? B.w[1] : B.w[0], fy = gy ? B.w[0] : B.w[1];
    const uint32_t nz = gz ? B.w[3] : B.w[2], fz = gz ? B.w[2] : B.w[3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 x = slab(nx, fx, i, ix, cx.x, cx.y), y = slab(ny, fy, i, iy, cy.x, cy.y), z = slab(nz, fz, i, iz, cz.x, cz.y);
        const float t0 = fmaxf(max3(x.x, y.x, z.x), r.tmin), t1 = fminf(min3(x.y, y.y, z.y), cull);
        tn[i] = t0 <= t1 ? t0 : kMiss;
        ch[i] = int32_t(B.w[4 + i]);
    }
}

// Fused visit of 4-wide node `ni`: the plain node's planes with the packed walk's
// arithmetic, two children's planes in one instruction (12 multiply-adds instead
// of 48 operations, and no slack per child).
__device__ __forceinline__ void box4_fused(const WideNode4* __restrict__ nodes, int ni, const RayFast& r, float cull,
                                           float (&tn)[4], int32_t (&ch)[4]) {
    const float4* p = reinterpret_cast<const float4*>(nodes + ni);
    const int fx = int(r.flags & 1u), fy = int((r.flags >> 1) & 1u), fz = int((r.flags >> 2) & 1u);
    const float4 nx = __ldg(p + fx), gx = __ldg(p + (1 - fx));
    const float4 ny = __ldg(p + 2 + fy), gy = __ldg(p + 3 - fy);
    const float4 nz = __ldg(p + 4 + fz), gz = __ldg(p + 5 - fz);
    const int4 c = __ldg(reinterpret_cast<const int4*>(p + 6));
    ch[0] = c.x; ch[1] = c.y; ch[2] = c.z; ch[3] = c.w;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float2 ax = h ? fma2(nx.z, nx.w, r.inv.x, r.cn.x, r.cn.x) : fma2(nx.x, nx.y, r.inv.x, r.cn.x, r.cn.x);
        const float2 ay = h ? fma2(ny.z, ny.w, r.inv.y, r.cn.y, r.cn.y) : fma2(ny.x, ny.y, r.inv.y, r.cn.y, r.cn.y);
        const float2 az = h ? fma2(nz.z, nz.w, r.inv.z, r.cn.z, r.cn.z) : fma2(nz.x, nz.y, r.inv.z, r.cn.z, r.cn.z);
        const float2 bx = h ? fma2(gx.z, gx.w, r.inv.x, r.cf.x, r.cf.x) : fma2(gx.x, gx.y, r.inv.x, r.cf.x, r.cf.x);
        const float2 by = h ? fma2(gy.z, gy.w, r.inv.y, r.cf.y, r.cf.y) : fma2(gy.x, gy.y, r.inv.y, r.cf.y, r.cf.y);
        const float2 bz = h ? fma2(gz.z, gz.w, r.inv.z, r.cf.z, r.cf.z) : fma2(gz.x, gz.y, r.inv.z, r.cf.z, r.cf.z);
        const float t0 = fmaxf(max3(ax.x, ay.x, az.x), r.tmin), t1 = fmaxf(max3(ax.y, ay.y, az.y), r.tmin);
        tn[2 * h] = t0 <= fminf(min3(bx.x, by.x, bz.x), cull) ? t0 : kMiss;
        tn[2 * h + 1] = t1 <= fminf(min3(bx.y, by.y, bz.y), cull) ? t1 : kMiss;
    }
}

// The operands of an 8-wide node: header, child codes, and the near / far plane
// bytes of slots 0-3 (.x) and 4-7 (.y) for the ray's octant.
struct Node8 {
    v3 o2, s;
    uint32_t valid;
    int32_t ch[8];
    uint2 nx, fx, ny, fy, nz, fz;
};
__device__ __forceinline__ Node8 load8(const QNode8* __restrict__ node, uint32_t flags) {
    const char* p = reinterpret_cast<const char*>(node);
    const Words8 A = ldg256(p), B = ldg256(p + 32), C = ldg256(p + 64);
    Node8 n;
    n.o2 = mk(__uint_as_float(A.w[0]), __uint_as_float(A.w[1]), __uint_as_float(A.w[2]));
    const uint32_t meta = A.w[3];
    n.s = mk(__uint_as_float((meta & 0xffu) << 23), __uint_as_float(((meta >> 8) & 0xffu) << 23),
             __uint_as_float(((meta >> 16) & 0xffu) << 23));
    n.valid = meta >> 24;
#pragma unroll
    for (int i = 0; i < 4; ++i) { n.ch[i] = int32_t(A.w[4 + i]); n.ch[4 + i] = int32_t(B.w[i]); }
    const bool gx = flags & 1u, gy = flags & 2u, gz = flags & 4u;
    const uint2 lx = make_uint2(B.w[4], B.w[5]), hx = make_uint2(B.w[6], B.w[7]);
    const uint2 ly = make_uint2(C.w[0], C.w[1]), hy = make_uint2(C.w[2], C.w[3]);
    const uint2 lz = make_uint2(C.w[4], C.w[5]), hz = make_uint2(C.w[6], C.w[7]);
    n.nx = gx ? hx : lx; n.fx = gx ? lx : hx;
    n.ny = gy ? hy : ly; n.fy = gy ? ly : hy;
    n.nz = gz ? hz : lz; n.fz = gz ? lz : hz;
    return n;
}

// Plain visit of an 8-wide node: each plane is dequantised exactly (P = fmaf(2^23
// + q, s, o2), see QNode8) and then tested exactly as in box4_plain, so the same
// slack argument holds.  Entry distances of all slots and the mask of the hit ones.
struct Children8 {
    float t[8];
    uint32_t mask;
};
__device__ __forceinline__ Children8 box8_plain(const Node8& n, v3 o, v3 inv, float tmin, float best) {
    Children8 r;
    r.mask = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        // byte (i & 3) of the word as the float 2^23 + q
        const uint32_t sel = 0x7540u | uint32_t(i & 3);
        const float nqx = __uint_as_float(__byte_perm(i < 4 ? n.nx.x : n.nx.y, 0x4B000000u, sel));
        const float fqx = __uint_as_float(__byte_perm(i < 4 ? n.fx.x : n.fx.y, 0x4B000000u, sel));
        const float nqy = __uint_as_float(__byte_perm(i < 4 ? n.ny.x : n.ny.y, 0x4B000000u, sel));
        const float fqy = __uint_as_float(__byte_perm(i < 4 ? n.fy.x : n.fy.y, 0x4B000000u, sel));
        const float nqz = __uint_as_float(__byte_perm(i < 4 ? n.nz.x : n.nz.y, 0x4B000000u, sel));
        const float fqz = __uint_as_float(__byte_perm(i < 4 ? n.fz.x : n.fz.y, 0x4B000000u, sel));
        const float ax = (fmaf(nqx, n.s.x, n.o2.x) - o.x) * inv.x, bx = (fmaf(fqx, n.s.x, n.o2.x) - o.x) * inv.x;
        const float ay = (fmaf(nqy, n.s.y, n.o2.y) - o.y) * inv.y, by = (fmaf(fqy, n.s.y, n.o2.y) - o.y) * inv.y;
        const float az = (fmaf(nqz, n.s.z, n.o2.z) - o.z) * inv.z, bz = (fmaf(fqz, n.s.z, n.o2.z) - o.z) * inv.z;
        const float t0 = fmaxf(fmaxf(ax, ay), fmaxf(az, tmin));
        float t1 = fminf(fminf(bx, by), fminf(bz, best));
        t1 = fmaf(fabsf(t1), kBoxSlack, t1);
        r.t[i] = t0;
        if (t0 <= t1) r.mask |= 1u << i;
    }
    r.mask &= n.valid;
    return r;
}

// Packed visit of an 8-wide node: as box4_packed, the byte read as 2^15 + q against
// the origin moved by (2^23 - 2^15) steps (exact), the intercepts widened by 1/128
// of a step for the roundings at 2^15 steps.
__device__ __forceinline__ float2 cut8(float o2, float step, float inv, float slope, float cn, float cf) {
    const float o = fmaf(8355840.f, step, o2);   // 2^23 - 2^15
    const float2 c = fma2(o, o, inv, cn, cf);
    return make_float2(fmaf(fabsf(slope), -0.0078125f, c.x), fmaf(fabsf(slope), 0.0078125f, c.y));
}
__device__ __forceinline__ uint32_t box8_packed(const Node8& n, const RayFast& r, float cull, float (&tn)[8]) {
    const float ix = n.s.x * r.inv.x, iy = n.s.y * r.inv.y, iz = n.s.z * r.inv.z;
    const float2 cx = cut8(n.o2.x, n.s.x, r.inv.x, ix, r.cn.x, r.cf.x), cy = cut8(n.o2.y, n.s.y, r.inv.y, iy, r.cn.y, r.cf.y);
    const float2 cz = cut8(n.o2.z, n.s.z, r.inv.z, iz, r.cn.z, r.cf.z);
    uint32_t mask = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 x = slab(i < 4 ? n.nx.x : n.nx.y, i < 4 ? n.fx.x : n.fx.y, i & 3, ix, cx.x, cx.y);
        const float2 y = slab(i < 4 ? n.ny.x : n.ny.y, i < 4 ? n.fy.x : n.fy.y, i & 3, iy, cy.x, cy.y);
        const float2 z = slab(i < 4 ? n.nz.x : n.nz.y, i < 4 ? n.fz.x : n.fz.y, i & 3, iz, cz.x, cz.y);
        tn[i] = fmaxf(max3(x.x, y.x, z.x), r.tmin);
        if (tn[i] <= fminf(min3(x.y, y.y, z.y), cull)) mask |= 1u << i;
    }
    return mask & n.valid;
}

// Slot permutation s -> s ^ oct applied to an 8-bit mask.
__device__ __forceinline__ uint32_t octant_order(uint32_t m, uint32_t oct) {
    if (oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (oct & 4u) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
    return m;
}

// Traversal stack: the first SM entries of each ray live in shared memory
// (entry-major, one column per thread), deeper entries in local memory.
template <int SM>
struct RayStack {
    int2* sm;        // &shared[0][threadIdx.x]; entry i at sm[i * stride]
    int2* lm;        // local array; entry i >= SM at lm[i - SM]
    int stride;
    __device__ __forceinline__ void put(int i, int2 v) const {
        if (SM > 0 && i < SM) sm[i * stride] = v;
        else lm[i - SM] = v;
    }
    __device__ __forceinline__ int2 get(int i) const {
        if (SM > 0 && i < SM) return sm[i * stride];
        return lm[i - SM];
    }
};

struct Counters {
    unsigned long long rays, nodes, tris;
};

// Per-lane traversal state kept across refill points.
template <bool WT, int WALK>
struct TravState {
    Ray<WALK> r;
    typename std::conditional<WT, ObjRayWT, ObjRay>::type cache;
    float best, u, v;
    float cull;     // best with the walk's slack: nothing beyond it matters
    int prim;       // closest hit so far, its material class (TriRec e2.w) in bits 28-29; -1 = none
    int item;       // current node / leaf code; kNone when the stack must be popped
    int sp;
};
constexpr int kNone = 0x7fffffff;   // == kEmptyChild

template <class TS>
__device__ __forceinline__ float trav_cull(const TS& s, float t) {
    return fmaf(fabsf(t), (s.r.flags & kPlainWalk) ? kBoxSlack : kFastSlack, t);   // (a constant in the plain walk)
}

// walk: kPlainWalk to start on the plain nodes, 0 otherwise
template <class TS>
__device__ __forceinline__ void trav_init(TS& s, const TraceScene& S, uint32_t walk, float4 a, float4 b, int32_t idx, int root) {
    make_ray(s.r, S.extent, walk, a, b, idx);
    keep_ray(S, s.r, a, b);
    s.cache.bundle = -1;   // world space: the object-space ray of an identity bundle
    s.cache.o = mk(a.x, a.y, a.z);
    s.cache.d = mk(b.x, b.y, b.z);
    shear(s.cache);
    s.best = b.w;
    s.cull = trav_cull(s, b.w);
    s.prim = -1;
    s.u = s.v = 0.f;
    s.item = root;
    s.sp = 0;
    // A NaN in the origin or direction makes every triangle's t NaN, a miss, and
    // with all slabs NaN nothing would be culled.
    if ((s.r.flags & kPlainWalk) && (isnan(a.x) || isnan(a.y) || isnan(a.z) || isnan(b.x) || isnan(b.y) || isnan(b.z))) s.item = kNone;
}

// Pops the next stack entry, skipping entries that start beyond the closest
// hit; false when the stack is empty.
template <bool ANY, class STACK, bool WT, int WALK>
__device__ __forceinline__ bool trav_pop(TravState<WT, WALK>& s, const STACK& stack, int& item) {
    while (s.sp > 0) {
        const int2 e = stack.get(--s.sp);
        // the entry distance carries the box test's rounding: cull with its slack
        if (!ANY && __int_as_float(e.y) > s.cull) continue;
        if (WALK != kWalkFused && WALK != kWalkPlain && e.x == kNone) continue;   // an empty slot (box4_packed)
        item = e.x;
        return true;
    }
    return false;
}

// Visits internal node `item`: continues with the nearest hit child (s.item),
// pushes the others.  False on stack overflow (error flag raised).
template <bool ANY, bool COUNT, int WIDTH, class STACK, bool WT, int WALK>
__device__ __forceinline__ bool trav_node(const TraceScene& S, TravState<WT, WALK>& s, const STACK& stack, int item,
                                          bool fused, Counters& cnt) {
    if (COUNT) ++cnt.nodes;
    const bool plain = WALK == kWalkPlain || (s.r.flags & kPlainWalk) != 0;
    v3 o, d;
    if (WIDTH == 8) {
        float tn[8];
        uint32_t mask;
        const Node8 n = load8(S.nodes8 + item, s.r.flags);
        if (plain) {
            world_ray(S, s.r, o, d);
            const Children8 c = box8_plain(n, o, s.r.inv, s.r.tmin, s.best);
            mask = c.mask;
#pragma unroll
            for (int i = 0; i < 8; ++i) tn[i] = c.t[i];
        } else if constexpr (WALK != kWalkPlain) {
            mask = box8_packed(n, s.r, s.cull, tn);
        }
        if (mask == 0) { s.item = kNone; return true; }
        // visit order i = slot ^ octant: continue with the first hit, push the
        // others so that they pop in visit order
        const uint32_t oct = s.r.flags & kOctMask;
        const uint32_t om = octant_order(mask, oct);
        const uint32_t rest = om & (om - 1u);
        const int first = __ffs(om) - 1;
        const int nrest = __popc(rest);
        if (s.sp + nrest > kStackSize8) {
            atomicOr(S.errflags, BG_FLAG_STACK_OVERFLOW);
            return false;
        }
        int next = kNone;
#pragma unroll
        for (int sl = 0; sl < 8; ++sl) {
            const int i = sl ^ int(oct);
            if ((rest >> i) & 1u) stack.put(s.sp + __popc(rest >> (i + 1)), make_int2(n.ch[sl], __float_as_int(tn[sl])));
            if (i == first) next = n.ch[sl];
        }
        s.sp += nrest;
        s.item = next;
        return true;
    }
    if (plain) {
        world_ray(S, s.r, o, d);
        const Children4 h = box4_plain<WALK == kWalkFused || WALK == kWalkPlain>(reinterpret_cast<const float4*>(S.nodes + item), o, s.r.inv, s.r.flags, s.r.tmin, s.best);
        if (h.nh == 0) { s.item = kNone; return true; }
        // push the farther ones (farthest first), continue with the nearest
        if (s.sp + h.nh - 1 > kStackSize) {
            atomicOr(S.errflags, BG_FLAG_STACK_OVERFLOW);
            return false;
        }
#pragma unroll
        for (int i = 3; i >= 1; --i)
            if (i < h.nh) stack.put(s.sp++, make_int2(h.c[i], __float_as_int(h.t[i])));
        s.item = h.c[0];
    } else if constexpr (WALK != kWalkPlain) {
        float tn[4];
        int32_t ch[4];
        if (WALK == kWalkFused || fused) box4_fused(S.nodes, item, s.r, s.cull, tn, ch);
        else box4_packed(S.qnodes, item, s.r, s.cull, tn, ch);
        sort4<!ANY>(tn, ch);
        // (the commit has checked that no walk needs more than kStackSize entries; the packed
        // boxes can only let in an empty slot besides)
        if (s.sp + 3 > kStackSize) {
            s.r.flags |= kTie;   // no room to spare: the plain walk decides
            return false;
        }
#pragma unroll
        for (int i = 3; i >= 1; --i)
            if (tn[i] < kMiss) stack.put(s.sp++, make_int2(ch[i], __float_as_int(tn[i])));
        s.item = tn[0] < kMiss ? ch[0] : kNone;
    }
    return true;
}

// Tests the first triangle of leaf code `item` (bit 31 set, count-1 in bits
// 27..30, first triangle in bits 0..26) and sets the lane's next item: the
// rest of the leaf, or a pop.  True when an any-hit query found its hit.  One
// triangle per traversal step keeps lanes that are in a leaf in step with
// lanes that are in a node (measured against the whole leaf in one step: C2
// incoherent closest hits +4 %, any hits +3.5 %, C3 frame +1-2 %).
// WT: the scene's records hold the vertices (p1, p2, p3) and the test is the
// watertight one; otherwise they hold (p1, e1, e2) for Moller-Trumbore.
template <bool ANY, bool COUNT, bool WT, int WALK>
__device__ __forceinline__ bool trav_leaf(const TraceScene& S, TravState<WT, WALK>& s, int item, Counters& cnt) {
    const uint32_t code = uint32_t(item);
    const int count = int((code >> kLeafStartBits) & 15u) + 1;
    const int start = int(code & uint32_t(kMaxLeafStart));
    // the rest of the leaf: one triangle fewer, starting one later
    s.item = count > 1 ? int(code - (1u << kLeafStartBits) + 1u) : kNone;
    const float4* tp = reinterpret_cast<const float4*>(S.tris + start);
    float4 v0 = __ldg(tp), e1 = __ldg(tp + 1), e2 = __ldg(tp + 2);
    if (COUNT) ++cnt.tris;
    obj_ray(S, s.r, __float_as_int(v0.w), s.cache);
    float t, a, b;
    bool hit;
    if constexpr (WT)
        hit = wt_test(s.cache, mk(v0.x, v0.y, v0.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), s.r.tmin, s.best, t, a, b);
    else
        hit = mt_test(s.cache.o, s.cache.d, mk(v0.x, v0.y, v0.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z),
                      s.r.tmin, s.best, t, a, b);
    if (hit) {
        if (kKeeps<WALK> && !ANY && !(s.r.flags & kPlainWalk))   // (at tmax: a tie too, asked once more)
            s.r.flags = t == s.best ? s.r.flags | kTie : s.r.flags & ~kTie;
        s.prim = __float_as_int(e1.w) | (__float_as_int(e2.w) << kClassShift);
        if (kKeeps<WALK>) {
            S.own[2 * S.ownstep].x = __int_as_float(start);
            if (ANY) S.own[2 * S.ownstep].y = t;
        }
        if (ANY) return true;
        s.best = t; s.u = a; s.v = b;
        s.cull = trav_cull(s, t);
    }
    return false;
}

// Runs at most `steps` node / leaf visits.  Returns true when the ray is done.
// fused (kWalkPacked on 4-wide nodes, the same in all lanes of the warp): visit the
// 128-byte nodes instead of the packed ones.
// (Measured and rejected: node and leaf visits in two warp-wide phases,
// with or without postponing a lane's leaf while others still descend: the
// votes and the longer loops cost 2.5-4x on C2 and C3.)
template <bool ANY, bool COUNT, int WIDTH, class STACK, bool WT, int WALK>
__device__ __forceinline__ bool trav_steps(const TraceScene& S, TravState<WT, WALK>& s, const STACK& stack, int steps,
                                           bool fused, Counters& cnt) {
    for (int it = 0; it < steps; ++it) {
        int item = s.item;
        if (item == kNone && !trav_pop<ANY>(s, stack, item)) return true;
        if (item >= 0) {
            if (!trav_node<ANY, COUNT, WIDTH>(S, s, stack, item, fused, cnt)) return true;
        } else {
            if (trav_leaf<ANY, COUNT>(S, s, item, cnt)) return true;
        }
    }
    return false;
}

// ------------------------------------------------- a group of lanes per ray
// With few rays the time of a launch is the longest ray's chain of dependent
// visits (about 0.5 us each; a ray of the 1M-triangle soup makes 40, the
// longest of 4,096 shadow rays 150), whatever the chip could do beside it.  So
// a group of G = 32 or 8 lanes walks one ray: every step pops up to G entries
// of the group's stack, each lane visits one of them (a packed node, or a leaf's
// first triangle), and the lanes push what they found, the nearest lane's
// children on top.  A step's visits run side by side, so a ray takes about as
// many steps as the tree has levels; it visits more nodes than the serial walk,
// as entries are popped before nearer hits have culled them.
// The answer is that of the packed walk: an any-hit answer and the closest t do
// not depend on the order, and a closest hit with another one at the same t, a ray
// outside the packed arithmetic and a group whose stack runs full (8 entries
// per lane) are walked again serially on the plain nodes by the group's first
// lane.
// (Measured and rejected: four lanes per entry, one per child or triangle: fewer
// instructions per step, but a quarter of the entries: 4,096 rays 63 us, not 33.)
// Rays per warp of the grid (2,960 warps on 148 SMs) up to which 32 lanes walk a ray, and
// the most up to which 8 do (groups_walk says where).  100k-triangle soup, incoherent closest,
// 32 / 8 lanes: 256 rays 14 / 21 us, 1,024 14 / 24, 2,960 19 / 25, 4,096 25 / 27, 16,384 72 / 46.
constexpr int kCoop32 = 1, kCoop8 = 32;

// Lanes per ray of a launch of n rays on a grid of `warps` warps.
__host__ __device__ __forceinline__ int coop_group(int64_t n, int warps) { return n <= int64_t(warps) * kCoop32 ? 32 : 8; }

struct CoopHit {
    float t, u, v;
    int prim;       // with the material class in bits 28-29; -1 = none (any hit: >= 0 = occluded)
    bool writer;    // this lane holds the group's result
    bool redo;      // (first lane) walk the ray serially
};

// Lane `g` of the group of G lanes starting at lane `base`; entry j of the group's
// stack is sm[(j / G) * stride + base + j % G] (sm: the warp's columns).
// All 32 lanes of the warp call it; `live` = the group has a ray.
template <bool ANY, bool WT>
__device__ __forceinline__ CoopHit coop_walk(const TraceScene& S, bool live, int32_t idx, int root, int G, int g, int base,
                                             int2* sm, int stride) {
    constexpr unsigned kFull = 0xffffffffu;
    const unsigned gmask = G == 32 ? kFull : ((1u << G) - 1u) << base;
    const unsigned above = gmask & ~((2u << (base + g)) - 1u);   // lanes of the group after this one
    const int lg = 31 - __clz(G), cap = 8 * G;
    auto entry = [&](int j) -> int2& { return sm[(j >> lg) * stride + base + (j & (G - 1))]; };
    TravState<WT, 2> s;
    if (live) trav_init(s, S, 0u, __ldg(S.rays + 2 * int64_t(idx)), __ldg(S.rays + 2 * int64_t(idx) + 1), idx, root);
    else trav_init(s, S, 0u, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(1.f, 1.f, 1.f, 0.f), 0, 0);
    CoopHit r;
    r.prim = -1;
    r.t = s.best; r.u = r.v = 0.f;
    r.redo = live && (s.r.flags & kPlainWalk) != 0;
    float best = s.best;      // the group's closest t, and the lane that holds it
    int owner = -1;
    bool tie = false;
    int found = 0;            // (owner) TriRec of its hit
    int count = live && !r.redo ? 1 : 0;
    if (count && g == 0) entry(0) = make_int2(root, __float_as_int(s.r.tmin));
    __syncwarp();
    while (__any_sync(kFull, count > 0)) {
        // at most (room / 3) entries, as each visit adds up to three
        const int k = min(min(G, count), (cap - count) / 3);
        if (count > 0 && k == 0) { r.redo = true; count = 0; }
        int item = kNone;
        float entry_t = 0.f;
        if (count > 0 && g < k) {
            const int2 e = entry(count - 1 - g);
            item = e.x;
            entry_t = __int_as_float(e.y);
        }
        if (count > 0) count -= k;
        const float cull = fmaf(fabsf(best), kFastSlack, best);
        if (!ANY && entry_t > cull) item = kNone;
        float ht[4];
        int hc[4], npush = 0;
        float t = 0.f, u = 0.f, v = 0.f;
        int prim = -1, tri = 0;
        if (item >= 0 && item != kNone) {   // (kNone: none, culled, or an empty slot)
            box4_packed(S.qnodes, item, s.r, cull, ht, hc);
            sort4(ht, hc);
#pragma unroll
            for (int i = 0; i < 4; ++i) npush += ht[i] < kMiss ? 1 : 0;
        } else if (item < 0) {
            const uint32_t code = uint32_t(item);
            const int start = int(code & uint32_t(kMaxLeafStart)), rest = int((code >> kLeafStartBits) & 15u);
            // the other triangles of the leaf in up to three entries
            const int per = (rest + 2) / 3;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int first = i * per, c = min(per, rest - first);
                hc[i] = c > 0 ? encode_leaf(start + 1 + first, c) : 0;
                ht[i] = entry_t;
                npush += c > 0 ? 1 : 0;
            }
            const float4* tp = reinterpret_cast<const float4*>(S.tris + start);
            const float4 v0 = __ldg(tp), e1 = __ldg(tp + 1), e2 = __ldg(tp + 2);
            obj_ray(S, s.r, __float_as_int(v0.w), s.cache);
            bool hit;
            if constexpr (WT)
                hit = wt_test(s.cache, mk(v0.x, v0.y, v0.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), s.r.tmin, best, t, u, v);
            else
                hit = mt_test(s.cache.o, s.cache.d, mk(v0.x, v0.y, v0.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), s.r.tmin,
                              best, t, u, v);
            if (hit) prim = __float_as_int(e1.w) | (__float_as_int(e2.w) << kClassShift);
            tri = start;
        }
        const unsigned hits = __ballot_sync(kFull, prim >= 0);
        if (hits) {
            if (ANY) {
                if (hits & gmask) {
                    owner = __ffs(hits & gmask) - 1;
                    if (base + g == owner) { r.t = t; r.u = u; r.v = v; r.prim = prim; found = tri; }
                    count = 0;
                    npush = 0;
                }
            } else {
                float m = prim >= 0 ? t : kMiss;
                for (int o = G >> 1; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(kFull, m, o));
                const unsigned at = __ballot_sync(kFull, prim >= 0 && t == m) & gmask;
                if (hits & gmask) {
                    if (owner < 0 || m < best) {
                        tie = __popc(at) > 1;
                        best = m;
                        owner = __ffs(at) - 1;
                        if (base + g == owner) { r.t = t; r.u = u; r.v = v; r.prim = prim; found = tri; }
                    } else {
                        tie = true;      // (m = best)
                    }
                }
            }
        }
        // pushes: lane 0's children on top, each lane's farthest first
        const unsigned b0 = __ballot_sync(kFull, npush & 1), b1 = __ballot_sync(kFull, npush & 2), b2 = __ballot_sync(kFull, npush & 4);
        const int below = count + __popc(b0 & above) + 2 * __popc(b1 & above) + 4 * __popc(b2 & above);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < npush) entry(below + npush - 1 - i) = make_int2(hc[i], __float_as_int(ht[i]));
        count += __popc(b0 & gmask) + 2 * __popc(b1 & gmask) + 4 * __popc(b2 & gmask);
        __syncwarp();
    }
    bool unsure = false;
    if (owner >= 0 && base + g == owner)
        unsure = !plain_reaches<WT>(S, found, r.prim, r.t, &s.r.o.x, s.r.inv, s.r.tmin);
    const unsigned doubts = __ballot_sync(kFull, unsure) & gmask;   // (all lanes, tie or not)
    if (tie || doubts) r.redo = true;
    r.writer = live && !r.redo && base + g == (owner >= 0 ? owner : base);
    r.redo = r.redo && g == 0;
    return r;
}

}  // namespace bg
