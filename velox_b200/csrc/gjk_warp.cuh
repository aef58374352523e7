// Distance queries by a whole warp: gjkDistanceQuick's result, bit for bit.
//
// One thread's query is a long serial chain: support scans over a hull's
// points, and for overlapping shapes the search for a tetrahedron around the
// origin (up to 3,060 candidates) and EPA's scans of up to 128 faces, in a
// 10 KB stack frame of local memory (1-2 ms for the slowest queries). Here all
// lanes run the GJK loop on the same values (one pair per warp: no
// divergence, the simplex in registers) and share the scans: hull points,
// candidate tetrahedra, faces, horizon edges and new faces go to lanes, the
// polytope lies in shared memory. Where the serial code keeps the first of
// equals (or the first that passes), the lanes reduce to the lowest index.
//
// A query's code runs once per pair, so its size counts: with every function
// inlined two thirds of the issue slots waited for instructions (ncu, narrow
// phase of 1,000 boxes: 9.2 of 14 cycles per instruction). The shapes lie in
// shared memory and one out-of-line support mapping serves all callers; the
// faces of GJK's tetrahedron go to four lanes through one copy of the code.
//
// Robust and Paranoid pairs take the general routine on one lane; the kernels
// that can meet one carry it (255 registers and its 11 KB of stack).
#pragma once
#include "geom.cuh"

namespace vxb {

constexpr unsigned kFullWarp = 0xffffffffu;
constexpr int kEpaVerts = 64, kEpaFaces = 128, kEpaEdges = 192;

// Shared memory of one warp's queries.
struct WarpQuery {
    float4 face[kEpaFaces];          // normal, distance
    uint32_t faceIds[kEpaFaces];     // vertices (8 bits each), bit 31: valid
    SupportVert verts[kEpaVerts];    // EPA's vertices; the candidates of the tetrahedron search
    uint32_t edges[kEpaEdges];       // horizon, from | to << 8
    Convex shape[2];                 // the pair: A, B
    uint32_t pad[4 - (2 * sizeof(Convex) / 4) % 4];
};
static_assert(sizeof(WarpQuery) % 16 == 0, "one per warp, 16-byte aligned");

// Kernels that query by warps have one WarpQuery per warp as their dynamic shared memory.
VXD WarpQuery& warpQuery() {
    extern __shared__ float4 querySmem[];
    return reinterpret_cast<WarpQuery*>(querySmem)[threadIdx.x >> 5];
}

VXD uint32_t warpLane() { return threadIdx.x & 31u; }

// Order-preserving bits of a float that is not a NaN; -0 and +0 map to one value.
VXD uint32_t sortBits(float f) {
    const uint32_t u = __float_as_uint(f + 0.0f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

VXD V3 shfl3(const V3& v, int src) {
    return V3{__shfl_sync(kFullWarp, v.x, src), __shfl_sync(kFullWarp, v.y, src), __shfl_sync(kFullWarp, v.z, src)};
}

// supportVertex of the pair in shared memory: shape A's support on lanes 0-15,
// B's on lanes 16-31, a hull's points spread over the half (uniform argument,
// all lanes call).
static __device__ __noinline__ SupportVert supportVertexWarp(V3 dir) {
    const WarpQuery& W = warpQuery();
    const uint32_t half = warpLane() >> 4, at = warpLane() & 15u;
    const Convex& c = W.shape[half];
    const V3 d = half ? -dir : dir;
    V3 o;
    if (c.kind == cHull) {
        const unsigned group = 0xffffu << (16u * half);
        const V3 l = rotateInv(c.orientation, d);
        uint32_t key = 0u, index = at;
        bool firstNan = false;
#pragma unroll 1
        for (uint32_t i = at; i < c.hullCount; i += 16u) {
            const float t = dot(l, hullPoint(c.hullPts, i));
            if (t != t) {  // never larger; as the first point, never replaced
                firstNan |= i == 0u;
                continue;
            }
            const uint32_t k = sortBits(t);
            if (k > key) { key = k; index = i; }
        }
        const uint32_t top = __reduce_max_sync(group, key);
        uint32_t best = __reduce_min_sync(group, key == top ? index : 0xffffffffu);
        if (__any_sync(group, firstNan) || top == 0u) best = 0u;
        o = rotate(c.orientation, hullPoint(c.hullPts, best));
    } else {
        o = supportOffsetBody(c, d);
    }
    const V3 oa = shfl3(o, 0), ob = shfl3(o, 16);
    const V3 pa = W.shape[0].position, pb = W.shape[1].position;
    SupportVert v;
    v.a = pa + oa;
    v.b = pb + ob;
    v.p = (pa - pb) + (oa - ob);
    return v;
}

VXD SupportVert shflVert(const SupportVert& v, int src) {
    return SupportVert{shfl3(v.p, src), shfl3(v.a, src), shfl3(v.b, src)};
}

// solveTetrahedronV, face f on lane f. (The crosses only enter products and
// lengths, where a zero's sign does not matter.)
static __device__ __noinline__ bool solveTetrahedronWarp(SupportVert& v0, SupportVert& v1, SupportVert& v2,
                                                         const SupportVert& v3, float& b0, float& b1, float& b2,
                                                         int& count, float scale) {
    const float volume = dot(v1.p - v0.p, crossRaw(v2.p - v0.p, v3.p - v0.p));
    const float floorVol = 1e-10f * scale * scale * scale;
    const bool flat = fabsf(volume) < floorVol;
    const uint32_t f = warpLane() & 3u;
    SupportVert u0 = f == 3u ? v1 : v0, u1 = f < 2u ? v1 : v2, u2 = f == 0u ? v2 : v3;
    bool takes = true;
    if (!flat) {
        const V3 a = u0.p, o = f == 0u ? v3.p : f == 1u ? v2.p : f == 2u ? v1.p : v0.p;
        const V3 n = crossRaw(u1.p - a, u2.p - a);
        const float nLen = length(n);
        const float originDist = dot(n, -a) / nLen;
        const float oppositeDist = dot(n, o - a) / nLen;
        takes = !(nLen < 1e-20f) && (originDist * oppositeDist < 0.0f || fabsf(originDist) <= 3e-6f * scale);
        if (!__any_sync(kFullWarp, takes)) return true;
    }
    float e0 = 0.0f, e1 = 0.0f, e2 = 0.0f;
    int n = 3;
    solveTriangleV(u0, u1, u2, e0, e1, e2, n);
    V3 c{0.0f, 0.0f, 0.0f};
    c += u0.p * e0;
    if (n > 1) c += u1.p * e1;
    if (n > 2) c += u2.p * e2;
    const float d = lengthSq(c);
    const bool counts = takes && d < 1e30f;
    const uint32_t key = counts ? sortBits(d) : 0xffffffffu;
    const uint32_t low = __reduce_min_sync(kFullWarp, key);
    const unsigned at = __ballot_sync(kFullWarp, counts && key == low);
    if (!at) {  // no face with a finite distance
        v1 = v2 = v0;
        b0 = b1 = b2 = 0.0f;
        count = 0;
        return false;
    }
    const int src = __ffs(at) - 1;
    count = __shfl_sync(kFullWarp, n, src);
    b0 = __shfl_sync(kFullWarp, e0, src);
    b1 = __shfl_sync(kFullWarp, e1, src);
    b2 = __shfl_sync(kFullWarp, e2, src);
    v0 = shflVert(u0, src);
    if (count > 1) v1 = shflVert(u1, src);
    if (count > 2) v2 = shflVert(u2, src);
    return false;
}

struct WarpSupport {  // the pair's shapes are in shared memory already
    VXD SupportVert operator()(const Convex&, const Convex&, const V3& dir) const { return supportVertexWarp(dir); }
    VXD bool tetrahedron(SupportVert& v0, SupportVert& v1, SupportVert& v2, const SupportVert& v3, float& b0, float& b1,
                         float& b2, int& count, float scale) const {
        return solveTetrahedronWarp(v0, v1, v2, v3, b0, b1, b2, count, scale);
    }
};

// The 4-subsets of 18 candidates in lexicographic order, 5 bits per index;
// those of fewer candidates are a subsequence in the same order.
struct TetTable {
    uint32_t v[3060];
};
constexpr TetTable makeTetTable() {
    TetTable t{};
    int n = 0;
    for (uint32_t i = 0; i < 15; ++i)
        for (uint32_t j = i + 1; j < 16; ++j)
            for (uint32_t k = j + 1; k < 17; ++k)
                for (uint32_t l = k + 1; l < 18; ++l) t.v[n++] = i | j << 5 | k << 10 | l << 15;
    return t;
}
static __device__ const TetTable kTets = makeTetTable();

// expandOverlapSimplex: s is uniform in and out.
static __device__ __noinline__ bool expandOverlapWarp(Simplex& s) {
    WarpQuery& W = warpQuery();
    const Convex &A = W.shape[0], &B = W.shape[1];
    const uint32_t lane = warpLane();
    SupportVert* cand = W.verts;
    SupportVert* dirs = W.verts + 32;  // the 14 fixed directions' supports
    if (lane < 14u)
        dirs[lane] = supportVertex(A, B, V3{kExpandDirs[lane][0], kExpandDirs[lane][1], kExpandDirs[lane][2]});
    int count = s.count;
    if (lane == 0u)
        for (int i = 0; i < count; ++i) cand[i] = s.v[i];
    __syncwarp();
    const float dupSq = duplicateDistanceSq(A, B);
    for (int d = 0; d < 14 && count < 18; ++d) {
        const SupportVert w = dirs[d];
        const bool near = (int)lane < count && lengthSq(w.p - cand[lane].p) < dupSq;
        if (!__any_sync(kFullWarp, near)) {
            if (lane == 0u) cand[count] = w;
            ++count;
            __syncwarp();
        }
    }
    const float scale = pairScale(A, B);
    for (uint32_t base = 0; base < 3060u; base += 32u) {
        const uint32_t at = base + lane;
        bool hit = false;
        uint32_t t = 0u;
        if (at < 3060u) {
            t = kTets.v[at];
            if ((int)(t >> 15) < count)
                hit = originInsideTetrahedron(cand[t & 31u].p, cand[(t >> 5) & 31u].p, cand[(t >> 10) & 31u].p,
                                              cand[t >> 15].p, scale);
        }
        const unsigned hits = __ballot_sync(kFullWarp, hit);
        if (hits) {
            t = __shfl_sync(kFullWarp, t, __ffs(hits) - 1);
            s.count = 4;
            s.v[0] = cand[t & 31u]; s.v[1] = cand[(t >> 5) & 31u]; s.v[2] = cand[(t >> 10) & 31u]; s.v[3] = cand[t >> 15];
            __syncwarp();
            return true;
        }
    }
    __syncwarp();
    return false;
}

static __device__ __noinline__ void epaResult(uint32_t ids, const float4& face, GjkResult& r) {
    const WarpQuery& W = warpQuery();
    const Convex &A = W.shape[0], &B = W.shape[1];
    EpaFace f;
    f.a = (int)(ids & 255u); f.b = (int)(ids >> 8 & 255u); f.c = (int)(ids >> 16 & 255u);
    f.normal = f3(face);
    V3 ca, cb;
    SupportVert u0 = W.verts[f.a], u1 = W.verts[f.b];
    const SupportVert u2 = W.verts[f.c];
    SupportVert v2 = u2;
    float b0 = 0.0f, b1 = 0.0f, b2 = 0.0f;
    int n = 3;
    solveTriangleV(u0, u1, v2, b0, b1, b2, n);
    ca = cb = V3{0.0f, 0.0f, 0.0f};
    ca += u0.a * b0; cb += u0.b * b0;
    if (n > 1) { ca += u1.a * b1; cb += u1.b * b1; }
    if (n > 2) { ca += v2.a * b2; cb += v2.b * b2; }
    r.normal = -f.normal;
    r.distance = -(face.w + A.radius + B.radius);
    r.pointA = ca - r.normal * A.radius;
    r.pointB = cb + r.normal * B.radius;
    r.overlapping = true;
}

VXD uint32_t nthSet(unsigned mask, uint32_t n) {
    for (; n; --n) mask &= mask - 1u;
    return (uint32_t)__ffs(mask) - 1u;
}

// Adds the edges of the visible faces (`mask`: lanes whose face ids go) to the
// horizon in order: an edge whose reverse is listed removes it (the last one
// takes its place), any other is appended.
static __device__ __noinline__ void horizon(WarpQuery& W, unsigned mask, uint32_t ids, int& edgeCount,
                                            uint32_t& myEdge, bool& spilled) {
    const uint32_t lane = warpLane();
#pragma unroll 1
    for (; mask; mask &= mask - 1u) {
        uint32_t face = __shfl_sync(kFullWarp, ids, __ffs(mask) - 1) & 0x00ffffffu;
        face |= face << 24;  // a, b, c, a
#pragma unroll 1
        for (int e = 0; e < 3; ++e, face >>= 8) {
            const uint32_t edge = face & 0xffffu, back = (edge >> 8) | (edge & 255u) << 8;
            if (!spilled) {
                const unsigned at = __ballot_sync(kFullWarp, (int)lane < edgeCount && myEdge == back);
                if (at) {
                    --edgeCount;
                    const uint32_t last = __shfl_sync(kFullWarp, myEdge, edgeCount);
                    if ((int)lane == __ffs(at) - 1) myEdge = last;
                    continue;
                }
                if (edgeCount < 32) {
                    if ((int)lane == edgeCount) myEdge = edge;
                    ++edgeCount;
                    continue;
                }
                W.edges[lane] = myEdge;
                spilled = true;
                __syncwarp();
            }
            uint32_t reverse = 0xffffffffu;
            for (uint32_t k = lane; k < (uint32_t)edgeCount; k += 32u)
                if (W.edges[k] == back) { reverse = k; break; }
            reverse = __reduce_min_sync(kFullWarp, reverse);
            if (reverse != 0xffffffffu) {
                --edgeCount;
                if (lane == 0u) W.edges[reverse] = W.edges[edgeCount];
            } else if (edgeCount < kEpaEdges) {
                if (lane == 0u) W.edges[edgeCount] = edge;
                ++edgeCount;
            }
            __syncwarp();
        }
    }
}

// epaPenetration at Normal quality (other qualities take the general routine).
static __device__ __noinline__ bool epaWarp(const Simplex& s, GjkResult& result) {
    WarpQuery& W = warpQuery();
    const Convex &A = W.shape[0], &B = W.shape[1];
    constexpr uint32_t kValid = 0x80000000u;
    const uint32_t lane = warpLane();
    if (lane == 0u)
        for (int i = 0; i < 4; ++i) W.verts[i] = s.v[i];
    __syncwarp();
    constexpr float areaFloorSq = 1e-16f;
    int vertexCount = 4, faceCount = 4;
    auto put = [&](uint32_t slot, const EpaFace& f) {
        W.face[slot] = pack(f.normal, f.distance);
        W.faceIds[slot] = (uint32_t)f.a | (uint32_t)f.b << 8 | (uint32_t)f.c << 16 | kValid;
    };
    bool ok0 = true;  // the four first faces, one lane each; all must exist
    if (lane < 4u) {
        EpaFace f;
        ok0 = makeEpaFace(W.verts, kEpaInitial[lane][0], kEpaInitial[lane][1], kEpaInitial[lane][2],
                          areaFloorSq, f);
        if (ok0) put(lane, f);
    }
    if (!__all_sync(kFullWarp, ok0)) return false;
    __syncwarp();
    const float dupSq = duplicateDistanceSq(A, B);
    int bestFace = 0;
#pragma unroll 1
    for (int it = 0; it < 48; ++it) {
        uint32_t key = 0xffffffffu, index = 0xffffffffu;  // nearest valid face, the first of equals
        for (uint32_t i = lane; i < (uint32_t)faceCount; i += 32u) {
            const float dist = W.face[i].w;
            if (!(W.faceIds[i] & kValid) || !(dist < 1e30f)) continue;
            const uint32_t k = sortBits(dist);
            if (k < key) { key = k; index = i; }
        }
        const uint32_t low = __reduce_min_sync(kFullWarp, key);
        if (low == 0xffffffffu) return false;
        bestFace = (int)__reduce_min_sync(kFullWarp, key == low ? index : 0xffffffffu);
        const float4 closest = W.face[bestFace];
        const V3 normal = f3(closest);
        const SupportVert w = supportVertexWarp(normal);
        const float supportDistance = dot(normal, w.p);
        const float tolerance = 1e-4f * vmax(1.0f, supportDistance);
        bool near = false;
        for (uint32_t i = lane; i < (uint32_t)vertexCount; i += 32u)
            near |= lengthSq(w.p - W.verts[i].p) < dupSq;
        if (supportDistance - closest.w <= tolerance || __any_sync(kFullWarp, near)) {
            epaResult(W.faceIds[bestFace], closest, result);
            return true;
        }
        if (vertexCount >= kEpaVerts) break;
        const int nv = vertexCount++;
        if (lane == 0u) W.verts[nv] = w;
        // faces that see the new vertex go; their edges without a reverse are the
        // horizon, edge k on lane k (a longer horizon moves to shared memory)
        int edgeCount = 0;
        uint32_t myEdge = 0u;
        bool spilled = false;
        unsigned open[kEpaFaces / 32];  // invalid slots below faceCount
#pragma unroll
        for (int chunk = 0; chunk < kEpaFaces / 32; ++chunk) {
            open[chunk] = 0u;
            if (chunk * 32 >= faceCount) continue;
            const uint32_t i = (uint32_t)chunk * 32u + lane;
            uint32_t ids = i < (uint32_t)faceCount ? W.faceIds[i] : 0u;
            bool sees = false;
            if (ids & kValid) {
                const float4 f = W.face[i];
                sees = !(dot(f3(f), w.p - W.verts[ids & 255u].p) <= tolerance);
            }
            if (sees) W.faceIds[i] = ids & ~kValid;
            open[chunk] = __ballot_sync(kFullWarp, i < (uint32_t)faceCount && (sees || !(ids & kValid)));
            horizon(W, __ballot_sync(kFullWarp, sees), ids, edgeCount, myEdge, spilled);
        }
        // The new vertex and the cleared faces are other lanes' writes (votes and
        // shuffles order no memory), and the new faces reuse slots just read.
        __syncwarp();
        // the horizon's new faces, in order, into the lowest open slots, then behind the last
        uint32_t made = 0u, opened = 0u;
        for (int chunk = 0; chunk < kEpaFaces / 32; ++chunk) opened += (uint32_t)__popc(open[chunk]);
#pragma unroll 1
        for (int base = 0; base < edgeCount; base += 32) {
            const int e = base + (int)lane;
            EpaFace f;
            bool ok = false;
            const uint32_t edge = spilled && e < edgeCount ? W.edges[e] : myEdge;
            if (e < edgeCount) ok = makeEpaFace(W.verts, (int)(edge & 255u), (int)(edge >> 8), nv, areaFloorSq, f);
            const unsigned oks = __ballot_sync(kFullWarp, ok);
            uint32_t rank = made + (uint32_t)__popc(oks & ((1u << lane) - 1u));
            uint32_t slot = (uint32_t)faceCount + rank - opened;
            if (rank < opened) {
                slot = 0u;
#pragma unroll
                for (int chunk = 0; chunk < kEpaFaces / 32; ++chunk) {
                    const uint32_t here = (uint32_t)__popc(open[chunk]);
                    if (rank < here) { slot = (uint32_t)chunk * 32u + nthSet(open[chunk], rank); break; }
                    rank -= here;
                }
            }
            if (__any_sync(kFullWarp, ok && slot >= (uint32_t)kEpaFaces)) return false;
            if (ok) put(slot, f);
            made += (uint32_t)__popc(oks);
        }
        if (made > opened) faceCount += (int)(made - opened);
        __syncwarp();
    }
    if (bestFace >= 0 && (W.faceIds[bestFace] & kValid)) {
        epaResult(W.faceIds[bestFace], W.face[bestFace], result);
        return true;
    }
    return false;
}

// gjkOverlapTail at Normal quality.
static __device__ __noinline__ GjkResult overlapTailWarp(Simplex& s, bool expand) {
    const Convex &A = warpQuery().shape[0], &B = warpQuery().shape[1];
    if (expand && s.count < 4) expandOverlapWarp(s);
    GjkResult r;
    r.distance = 0.0f;
    r.normal = r.pointA = r.pointB = V3{0.0f, 0.0f, 0.0f};
    r.overlapping = true;
    if (s.count == 4 && epaWarp(s, r)) return r;
    V3 n = A.position - B.position;
    n = lengthSq(n) > 1e-12f ? normalize(n) : V3{0.0f, 1.0f, 0.0f};
    const SupportVert v = supportVertexWarp(-n);  // A's support along -n, B's along n
    const V3 sa = v.a, sb = v.b;
    const float depth = dot(n, sb - sa);
    r.normal = n;
    r.distance = -depth - A.radius - B.radius;
    r.pointA = sa;
    r.pointB = sb;
    return r;
}

// gjkDistanceQuick; all lanes call with the same pair and get its result.
static __device__ __noinline__ GjkResult gjkDistanceWarp(const Convex& A, const Convex& B) {
    WarpQuery& W = warpQuery();
    __syncwarp();  // an earlier query's reads of W are over
    if (warpLane() == 0u) W.shape[0] = A;
    if (warpLane() == 1u) W.shape[1] = B;
    __syncwarp();
    GjkResult r;
    Simplex s;
    const int status = gjkDistanceFast(W.shape[0], W.shape[1], r, s, WarpSupport{});
    if (status == kGjkSeparated) return r;
    if (status != kGjkGeneral) return overlapTailWarp(s, status == kGjkOverlapExpand);
    // Robust and Paranoid geometry: the general routine, one lane
    if (warpLane() == 0u) r = gjkDistance(A, B);
    r.distance = __shfl_sync(kFullWarp, r.distance, 0);
    r.normal = shfl3(r.normal, 0);
    r.pointA = shfl3(r.pointA, 0);
    r.pointB = shfl3(r.pointB, 0);
    r.overlapping = __shfl_sync(kFullWarp, r.overlapping ? 1 : 0, 0) != 0;
    return r;
}

}  // namespace vxb
