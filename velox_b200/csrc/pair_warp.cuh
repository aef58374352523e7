// Pairs by a whole warp: the narrow phase's contacts of the pairs whose cores
// overlap or that involve a mesh or compound, and the rewind's gap probe.
// All lanes call every function with the same arguments; contacts are built by
// lane 0. A mesh's triangles go to the lanes, one query each, and the
// overlapping ones then take the warp query in turn; results are merged in the
// order of the mesh walk.
#pragma once
#include "gjk_warp.cuh"

namespace vxb {

// Up to 32 triangles of mesh `m`, lane by lane against `c`: `tri` is this
// lane's triangle when lane < have. Afterwards r holds the lane's result.
VXD void triangleQueries(const Convex& c, const Soup& soup, const vx_mesh& m, uint32_t tri, uint32_t have,
                         GjkResult& r) {
    const bool mine = warpLane() < have;
    bool open = false;
    if (mine) {
        Simplex s;
        open = gjkDistanceFast(c, meshTriangle(soup, m, tri), r, s) != kGjkSeparated;
    }
    for (unsigned mask = __ballot_sync(kFullWarp, open); mask; mask &= mask - 1u) {
        const int src = __ffs(mask) - 1;
        const GjkResult w = gjkDistanceWarp(c, meshTriangle(soup, m, __shfl_sync(kFullWarp, tri, src)));
        if ((int)warpLane() == src) r = w;
    }
}

// ---- narrow phase -------------------------------------------------------------

// meshConvex; out and n are lane 0's, the new count is returned to all.
static __device__ __noinline__ int meshConvexWarp(const BodyView& conv, const BodyView& mesh, uint32_t ic, uint32_t im,
                                                  const Soup& soup, float dt, vx_contact* out, int cap, int n) {
    const vx_mesh& m = soup.meshes[mesh.hullFirst];
    const float reach = aabbReach(conv.flags, conv.half, conv.radius, conv.hh, conv.margin, conv.v, conv.w, dt);
    const V3 lo = conv.p - V3{reach, reach, reach}, hi = conv.p + V3{reach, reach, reach};
    const Convex cc = makeConvex(conv, soup);
    const float touch = contactReach(conv, mesh, dt);
    const uint32_t lane = warpLane();
    uint32_t mine = 0u, have = 0u;
    auto flush = [&]() {
        GjkResult r;
        r.distance = 0.0f;
        r.normal = r.pointA = r.pointB = V3{0.0f, 0.0f, 0.0f};
        triangleQueries(cc, soup, m, mine, have, r);
        for (unsigned k = __ballot_sync(kFullWarp, lane < have && !(r.distance > touch)); k; k &= k - 1u) {
            const int src = __ffs(k) - 1;
            const V3 normal = shfl3(r.normal, src), pa = shfl3(r.pointA, src), pb = shfl3(r.pointB, src);
            const float distance = __shfl_sync(kFullWarp, r.distance, src);
            const uint32_t tri = __shfl_sync(kFullWarp, mine, src);
            if (lane == 0u)
                emitContact(conv, mesh, ic, im, normal, (pa + pb) * 0.5f, distance, dt, out, cap, n,
                            contactFeatureKey(kImplicitFeature, kTriangleFeature | tri));
        }
        have = 0u;
    };
    meshVisit(soup, m, lo, hi, [&](uint32_t tri) {
        if (lane == have) mine = tri;
        if (++have == 32u) flush();
        return true;
    });
    if (have) flush();
    return __shfl_sync(kFullWarp, n, 0);
}

VXD int collideSimpleWarp(const BodyView& a, const BodyView& b, uint32_t ia, uint32_t ib, const Soup& soup, float dt,
                          vx_contact* out, int cap) {
    int n = 0;
    const uint32_t sa = shapeOf(a.flags), sb = shapeOf(b.flags);
    const bool va = isConvexVolume(sa), vb = isConvexVolume(sb);
    if (va && vb) {
        const Convex ca = makeConvex(a, soup), cb = makeConvex(b, soup);
        const GjkResult r = gjkDistanceWarp(ca, cb);
        if (warpLane() == 0u) convexContacts(a, b, ia, ib, ca, cb, r, dt, out, cap, n);
    } else if (warpLane() == 0u && va && sb == kPlane) {
        planeConvex(a, b, ia, ib, soup, dt, out, cap, n);
    } else if (warpLane() == 0u && sa == kPlane && vb) {
        planeConvex(b, a, ib, ia, soup, dt, out, cap, n);
    }
    if (va && sb == kMesh) n = meshConvexWarp(a, b, ia, ib, soup, dt, out, cap, n);
    else if (sa == kMesh && vb) n = meshConvexWarp(b, a, ib, ia, soup, dt, out, cap, n);
    return __shfl_sync(kFullWarp, n, 0);
}

// collidePair: the contacts in lane 0's `out`, their number to all lanes.
static __device__ __noinline__ int collidePairWarp(const BodyView& a, const BodyView& b, uint32_t ia, uint32_t ib,
                                                   const Soup& soup, float dt, vx_contact* out, int cap) {
    const bool ca = shapeOf(a.flags) == kCompound, cb = shapeOf(b.flags) == kCompound;
    if (!ca && !cb) return collideSimpleWarp(a, b, ia, ib, soup, dt, out, cap);
    const int countA = ca ? (int)a.hullCount : 1, countB = cb ? (int)b.hullCount : 1;
    int total = 0;
    for (int x = 0; x < countA && total < cap; ++x) {
        const BodyView ga = ca ? compoundChildView(a, soup.children[a.hullFirst + x]) : a;
        for (int y = 0; y < countB && total < cap; ++y) {
            const BodyView gb = cb ? compoundChildView(b, soup.children[b.hullFirst + y]) : b;
            const int added = collideSimpleWarp(ga, gb, ia, ib, soup, dt, out + total, cap - total);
            if (warpLane() == 0u) ownContacts(a, b, ia, ib, x, y, out + total, added);
            total += added;
        }
    }
    return total;
}

// ---- rewind: gapAt (world.cpp:2916-2958) ---------------------------------------

struct GapProbe { float gap; V3 normal; };

// meshSimpleGapProbe (narrowphase.h:719-749): the smallest gap (strictly
// smaller replaces) between `a` and the triangles of mesh `b` whose BVH
// leaves overlap a cube of half width `search` around a's position.
static __device__ __noinline__ void meshGapWarp(const BodyView& a, const BodyView& b, const Soup& soup, float search,
                                                GapProbe& best) {
    const vx_mesh& m = soup.meshes[b.hullFirst];
    const V3 lo = a.p - V3{search, search, search}, hi = a.p + V3{search, search, search};
    const Convex ca = makeConvex(a, soup);
    const uint32_t lane = warpLane();
    uint32_t mine = 0u, have = 0u;
    auto flush = [&]() {
        GjkResult r;
        r.distance = 1e30f;
        r.normal = r.pointA = r.pointB = V3{0.0f, 0.0f, 0.0f};
        triangleQueries(ca, soup, m, mine, have, r);
        const bool counts = lane < have && r.distance == r.distance;
        const uint32_t key = counts ? sortBits(r.distance) : 0xffffffffu;
        const uint32_t low = __reduce_min_sync(kFullWarp, key);
        const unsigned at = __ballot_sync(kFullWarp, counts && key == low);
        if (at) {
            const int src = __ffs(at) - 1;
            const float d = __shfl_sync(kFullWarp, r.distance, src);
            const V3 normal = shfl3(r.normal, src);
            if (d < best.gap) best = GapProbe{d, normal};
        }
        have = 0u;
    };
    meshVisit(soup, m, lo, hi, [&](uint32_t tri) {
        if (lane == have) mine = tri;
        if (++have == 32u) flush();
        return true;
    });
    if (have) flush();
}

// gapAt for two non-compound bodies, b not a mesh.
VXD GapProbe gapConvexWarp(const BodyView& a, const BodyView& b, const Soup& soup) {
    if (shapeOf(b.flags) == kPlane) {
        const Convex c = makeConvex(a, soup);
        const V3 deep = c.position + supportOffset(c, -b.planeN);
        return GapProbe{dot(b.planeN, deep) - b.planeOff - c.radius, b.planeN};
    }
    const GjkResult r = gjkDistanceWarp(makeConvex(a, soup), makeConvex(b, soup));
    return GapProbe{r.distance, r.normal};
}

// Signed gap and normal (from b towards a) of the rewind's distance oracle;
// `dt` sizes the mesh search cube as the rewind loop does (world.cpp:4272-4273).
// Compounds and meshes: the minimum over every child pair (A's children outer,
// B's inner) and every searched triangle, the first minimum kept, starting
// from (1e30, +y) as the reference's recursion does.
static __device__ __noinline__ GapProbe gapAtWarp(const BodyView& a, const BodyView& b, const Soup& soup, float dt) {
    if (!isComplexShape(shapeOf(a.flags)) && !isComplexShape(shapeOf(b.flags))) return gapConvexWarp(a, b, soup);
    const float search = maxPointSpeed(a) * dt + a.radius + length(a.half) + a.hh + 0.1f;
    GapProbe best{1e30f, V3{0.0f, 1.0f, 0.0f}};
    const bool ca = shapeOf(a.flags) == kCompound, cb = shapeOf(b.flags) == kCompound;
    const uint32_t countA = ca ? a.hullCount : 1u, countB = cb ? b.hullCount : 1u;
    for (uint32_t x = 0; x < countA; ++x) {
        const BodyView ga = ca ? compoundChildView(a, soup.children[a.hullFirst + x]) : a;
        for (uint32_t y = 0; y < countB; ++y) {
            const BodyView gb = cb ? compoundChildView(b, soup.children[b.hullFirst + y]) : b;
            if (shapeOf(gb.flags) == kMesh) {
                meshGapWarp(ga, gb, soup, search, best);
            } else {
                const GapProbe g = gapConvexWarp(ga, gb, soup);
                if (g.gap < best.gap) best = g;
            }
        }
    }
    return best;
}

}  // namespace vxb
