// Island solve on one warp or one block: the substep loop (integration, warm
// start, the coloured sweeps, transform integration) or the position correction
// of every island that one block's shared memory can hold.
//
// What bounds it: rows that share a body run in colour order, so an island costs
// its longest chain of such rows times the sweeps, and a link costs the latency
// of one row: read two bodies, two impulses through a world-space inverse inertia
// each, write two bodies. Everything here shortens that link:
//   * two lanes per row, one per body: each lane forms its own point velocity
//     and applies the impulses to its own body, and the two velocities cross
//     by shuffle, so a lane issues about half of the row's instructions;
//   * a row's prepared terms lie in planes of 16-byte words indexed by solve
//     position (a colour's rows are consecutive there, so a warp's loads are
//     whole lines), and a lane loads its next row while it computes the current
//     one;
//   * a lane keeps its own copy of the row's impulses (the side planes), so no
//     lane reads what another wrote except body velocities, which live in shared
//     memory; one warp orders them colour by colour, several by a tag on each
//     body (the dataflow below), without a barrier;
//   * no branch, predicate chain or general division where the operands allow
//     it (laneSweep, quotient): a warp alone on its scheduler pays each in full.
// Solve stage of one step, one row per thread on 128- and 176-byte records with a
// barrier a colour -> two lanes on planes -> the dataflow: 64 islands of 2,400
// rows (31 colours, 8 substeps) 13.3 -> 5.4 -> 4.5 ms, one of 310 rows (20
// colours) 4.8 -> 1.9 -> 1.6 ms.
// Measured and not kept: cross's sign rule behind a branch (20 % slower), one
// lane per row with the same planes (about equal for narrow colours, slower
// for wide ones).
#pragma once
#include "geom.cuh"
#include "quotient.cuh"

namespace vxb {

VXD Mass loadMass(const BodyArrays& B, uint32_t i) {
    const float4 in = B.inertia[i];
    Mass m;
    m.invI = V3{in.x, in.y, in.z};
    m.invMass = in.w;
    m.iq = q4(B.iq[i]);
    m.flags = B.filt[i].x;
    return m;
}

VXD SolverBody loadSolverBody(const BodyArrays& B, uint32_t i) {
    SolverBody s;
    s.p = f3(B.pos[i]);
    s.q = q4(B.rot[i]);
    s.v = f3(B.vel[i]);
    s.w = f3(B.ang[i]);
    s.m = loadMass(B, i);
    s.sphere = shapeOf(s.m.flags) == kSphere;
    return s;
}

VXD void loadRow(const vx_contact& c, RowContact& r) {
    r.normal = V3{c.normal.x, c.normal.y, c.normal.z};
    r.point = V3{c.point.x, c.point.y, c.point.z};
    r.la = V3{c.localAnchorA.x, c.localAnchorA.y, c.localAnchorA.z};
    r.lb = V3{c.localAnchorB.x, c.localAnchorB.y, c.localAnchorB.z};
    r.bias0 = c.bias0; r.vn0 = c.vn0; r.restitution = c.restitution;
    r.friction1 = c.friction1; r.friction2 = c.friction2;
    r.rolling = c.rollingFriction; r.spinning = c.spinningFriction;
    r.nImp = c.normalImpulse; r.t1Imp = c.tangentImpulse1; r.t2Imp = c.tangentImpulse2;
    r.r1Imp = c.rollingImpulse1; r.r2Imp = c.rollingImpulse2; r.sImp = c.spinningImpulse;
}
VXD void storeRow(vx_contact& c, const RowContact& r) {
    c.point = vx_vec3{r.point.x, r.point.y, r.point.z};
    c.normalImpulse = r.nImp; c.tangentImpulse1 = r.t1Imp; c.tangentImpulse2 = r.t2Imp;
    c.rollingImpulse1 = r.r1Imp; c.rollingImpulse2 = r.r2Imp; c.spinningImpulse = r.sImp;
}

struct SolveArgs {
    BodyArrays B;
    vx_contact* contacts;        // key-sorted storage
    const uint32_t* order;       // solve order -> contact index
    const uint32_t* islandStart; // islands + 1 (solve-order ranges)
    const uint32_t* segStart;    // segments + 1
    const uint32_t* islandSeg;   // islands + 1 (first segment)
    const uint32_t* bodyOrder;   // bodies sorted by island
    const uint32_t* bodyStart;   // islands + 2
    uint32_t islands;
    uint32_t realIslands;  // islands >= realIslands (the null island) own no bodies
    V3 gravity;
    float h;
    int substeps;
    int sweeps;
    int warmStart;     // warm start on the first substep
    int integrate;     // integrate velocities (s > 0) and transforms each substep
    int coneBlock;
    uint32_t tinyLimit;
    int positionIterations;  // position-correction mode when > 0
    RowPrep* prep;           // per solve-order row, rebuilt every substep (giant islands without a cooperative grid)
    float4* frames;          // per body inertia frame, rebuilt every substep (the same)
    float4* planes;          // per row terms of the block solve and the grid's flow (RowPlanes)
    uint32_t rows;           // rows of the plan (the planes' stride)
    int stackStabilization;
    float stackStiffness, stackDamping;
    uint32_t* fault;         // set when the island plan is inconsistent (Counters::planFault)
    uint32_t* timeout;       // set when a row's wait gave up (Counters::timeout)
    uint32_t waitLimit;      // polls before it does (Context::waitLimit)
};

VXD bool solvedContact(uint32_t fa, uint32_t fb) { return !isSensor(fa) && !isSensor(fb); }

// Island classes by what a block of the class holds (islandClassOf). Small: one
// warp, many per SM, or four warps (kSmallWide) where the GPU holds all islands
// at once. Medium: several blocks per SM. Large: one block per SM (the
// colouring's; the solve takes them as giants). Giant: the whole grid.
constexpr int kSmallThreads = 32, kSmallBodies = 64, kSmallRows = 256;
constexpr int kSmallWideThreads = 128;  // few small islands: four warps each
constexpr int kMediumThreads = 256, kMediumBodies = 512, kMediumRows = 3072;
constexpr int kLargeThreads = 512, kLargeBodies = 3072, kLargeRows = 16384;
enum IslandClass : int { kTinyIsland = 0, kSmallIsland, kMediumIsland, kLargeIsland, kGiantIsland,
                         kSmallWide };  // kSmallIsland's islands on four warps

VXD int islandClassOf(uint32_t nb, uint32_t rows, uint32_t tinyLimit) {
    if (rows <= tinyLimit) return kTinyIsland;
    if (nb <= (uint32_t)kSmallBodies && rows <= (uint32_t)kSmallRows) return kSmallIsland;
    if (nb <= (uint32_t)kMediumBodies && rows <= (uint32_t)kMediumRows) return kMediumIsland;
    if (nb <= (uint32_t)kLargeBodies && rows <= (uint32_t)kLargeRows) return kLargeIsland;
    return kGiantIsland;
}

// The solve's classes: large islands (one block's shared memory would hold
// them) run as the grid's flow, too. Solve stage of one step, one 512-thread
// block against the flow: 10,500 rows in 49 colours 7.9 / 4.8 ms, 6,100 in 40
// 5.5 / 4.1 ms, 3,500 in 17 4.1 / 3.2 ms. Medium islands stay in their blocks:
// 64 of 2,400 rows 5.4 / 7.2 ms, one of 310 1.9 / 2.6 ms.
VXD int solveClassOf(uint32_t nb, uint32_t rows, uint32_t tinyLimit) {
    const int cls = islandClassOf(nb, rows, tinyLimit);
    return cls == kLargeIsland ? kGiantIsland : cls;
}

template <int Class>
struct ClassShape {
    static constexpr bool kSmall = Class == kSmallIsland || Class == kSmallWide;
    static constexpr int kThreads = Class == kSmallIsland    ? kSmallThreads
                                    : Class == kSmallWide    ? kSmallWideThreads
                                    : Class == kMediumIsland ? kMediumThreads
                                                             : kLargeThreads;
    static constexpr int kBodies = kSmall ? kSmallBodies : Class == kMediumIsland ? kMediumBodies : kLargeBodies;
    static constexpr int kRows = kSmall ? kSmallRows : Class == kMediumIsland ? kMediumRows : kLargeRows;
    static constexpr int kBlocksPerSm = Class == kSmallIsland    ? 16
                                        : Class == kSmallWide    ? 4
                                        : Class == kMediumIsland ? 2
                                                                 : 1;
    static constexpr int kSegments = kSmall ? 64 : 256;  // colour starts kept in shared memory
    // dataflow (several warps): rows of a batch, a table of batches
    static constexpr bool kFlow = kThreads > 32;
    static constexpr int kBatch = kSmall ? 8 : 16;
    static constexpr size_t kSmem = (size_t)kBodies * 4 * sizeof(float4) + (size_t)kSegments * sizeof(uint32_t) +
                                    (kFlow ? (size_t)kRows * sizeof(uint16_t) : 0);
};

// The planes of one block's island, indexed by solve position. Velocity mode:
//   n    normal, kNormal (<= 0: the row is not solved)
//   t1   first tangent, k1          t2   second tangent, k2
//   g    normal target while not separating (vn <= 0) / while separating,
//        friction coefficients of the two tangents
//   aux  1 / kNormal, 1 / k1, 1 / k2; for the cone block kN1, kN2, k12
//   side (two per row, one per body) contact arm, body word
//   imp  (two per row) the three impulses, row bits (kRowExt: the row has
//        rolling or spinning terms; kRowSolved: no sensor; kRowRecip: the
//        effective masses are in quotient's range)
//   ext  (four per row, kRowExt only) per body: kr1, kr2, ks, rolling |
//        spinning and its three impulses
// Position mode: n normal, bias0; g correction factor, sum of inverse masses;
// side anchor offset, body word. Body word: index in the shared body table, or
// for a body outside it (never moved here) kAtRest when its velocities are
// zero, else the complement of its id: a body that is not at rest is read from
// global memory in every sweep, 300 cycles on the step's critical path.
constexpr size_t kRowPlaneBytes = 13 * sizeof(float4);
constexpr uint32_t kRowExt = 1u, kRowSolved = 2u, kRowRecip = 4u;
// Dataflow rows: the lane's body may turn; above it the row's rank among its
// body's rows, in a block 14 bits of it and 14 of the body's row count (at most
// kMediumRows), in the grid's flow 28 bits (the count lies with the body).
constexpr uint32_t kRowTurns = 8u, kRowLinkMask = 0x3fffu;
constexpr int kRowLinkShift = 4, kRowDegreeShift = kRowLinkShift + 14;
constexpr int kAtRest = INT_MIN;
struct RowPlanes {
    float4 *n, *t1, *t2, *g, *aux, *side, *imp, *ext;
};
VXD RowPlanes rowPlanes(const SolveArgs& A) {
    RowPlanes R;
    const size_t m = A.rows;
    R.n = A.planes;
    R.t1 = R.n + m;
    R.t2 = R.t1 + m;
    R.g = R.t2 + m;
    R.aux = R.g + m;
    R.side = R.aux + m;
    R.imp = R.side + 2 * m;
    R.ext = R.imp + 2 * m;
    return R;
}

// Shared body table. Velocity mode: v = velocity | 1 when rotation is locked,
// w = angular velocity, f = inertia frame, i = inverse inertia | inverse mass.
// Position mode: v = position | 1 when asleep, i as above.
struct BodyTable {
    float4 *v, *w, *f, *i;
};

struct RowRegs {
    float4 s, n, t1, t2, g, i, y;
};

enum RowOp : int { kRowWarm = 0, kRowSweep = 1, kRowPosition = 2 };

template <int Op>
VXD void loadRowRegs(const RowPlanes& R, uint32_t k, uint32_t side, RowRegs& r) {
    r.s = R.side[2 * (size_t)k + side];
    r.n = R.n[k];
    r.g = R.g[k];
    if (Op != kRowPosition) {
        r.t1 = R.t1[k];
        r.t2 = R.t2[k];
        r.i = R.imp[2 * (size_t)k + side];
        r.y = R.aux[k];
    }
}

// The pair's two values of `own`: (body a's, body b's).
VXD void pairBoth(const V3& own, uint32_t side, V3& a, V3& b) {
    const V3 o{__shfl_xor_sync(0xffffffffu, own.x, 1), __shfl_xor_sync(0xffffffffu, own.y, 1),
               __shfl_xor_sync(0xffffffffu, own.z, 1)};
    a = side ? o : own;
    b = side ? own : o;
}

// One lane's body in a velocity row.
struct LaneBody {
    V3 v, w, invI;
    Q4 frame;
    float im;
    bool dyn, turns;
};

template <bool Exact>
VXD V3 laneInvI(const LaneBody& b, const V3& x) {  // invIF
    const Q4 inv{-b.frame.x, -b.frame.y, -b.frame.z, b.frame.w};
    const V3 l = Exact ? rotate(inv, x) : rotateRaw(inv, x);
    const V3 s{l.x * b.invI.x, l.y * b.invI.y, l.z * b.invI.z};
    const V3 r = Exact ? rotate(b.frame, s) : rotateRaw(b.frame, s);
    return V3{b.turns ? r.x : 0.0f, b.turns ? r.y : 0.0f, b.turns ? r.z : 0.0f};
}

// x + d on body a's lane, x - d on body b's, x on a body that does not move.
VXD float laneAdd(const LaneBody& b, uint32_t flip, float x, float d) {
    const float y = x + __uint_as_float(__float_as_uint(d) ^ flip);
    return b.dyn ? y : x;
}
VXD V3 laneAdd(const LaneBody& b, uint32_t side, const V3& x, const V3& d) {
    const uint32_t flip = side << 31;
    return V3{laneAdd(b, flip, x.x, d.x), laneAdd(b, flip, x.y, d.y), laneAdd(b, flip, x.z, d.z)};
}
template <bool Exact>
VXD void laneImpulse(LaneBody& b, uint32_t side, const V3& arm, const V3& imp) {
    b.v = laneAdd(b, side, b.v, imp * b.im);
    b.w = laneAdd(b, side, b.w, laneInvI<Exact>(b, rowCross<Exact>(arm, imp)));
}
VXD void laneTorque(LaneBody& b, uint32_t side, const V3& tq) { b.w = laneAdd(b, side, b.w, laneInvI<true>(b, tq)); }

VXD float axisShare(float n, float mx) {  // (a zero numerator would cost the slow division)
    return !(mx > 0.0f) || (n == 0.0f && mx > 1e-10f) ? 0.0f : n * n / (mx * mx);
}
// Both lanes hold the same impulses; each divides one axis (all 32 lanes call).
VXD void clampToEllipse(uint32_t side, float max1, float max2, float& n1, float& n2) {
    if (max1 <= 0.0f) n1 = 0.0f;
    if (max2 <= 0.0f) n2 = 0.0f;
    float share = 0.0f;
    if (!(insideAxis(n1, max1) & insideAxis(n2, max2))) share = axisShare(side ? n2 : n1, side ? max2 : max1);
    const float ellipse = share + __shfl_xor_sync(0xffffffffu, share, 1);
    if (ellipse > 1.0f) {
        const float sc = 1.0f / sqrtf(ellipse);
        n1 *= sc;
        n2 *= sc;
    }
}

// One sweep of one row on the pair's two lanes: sweepRow's arithmetic in the
// same order (all 32 lanes call; `act`: this lane holds a row to solve).
//
// Exact = false as in sweepRowAs: for a warp whose rows have no -0 where it
// matters and no rolling or spinning terms.
template <bool Exact, bool Cone>
VXD void laneSweep(const RowPlanes& R, bool act, uint32_t k, uint32_t side, RowRegs& r, LaneBody& b) {
    const V3 arm = f3(r.s), n = f3(r.n), t1 = f3(r.t1), t2 = f3(r.t2);
    const float k1 = r.t1.w, k2 = r.t2.w;
    float nImp = r.i.x, i1 = r.i.y, i2 = r.i.z;
    V3 ua, ub;
    pairBoth(b.v + rowCross<Exact>(b.w, arm), side, ua, ub);
    const V3 rv0 = ua - ub;
    const float vn = dot(rv0, n);
    const float target = vn > 0.0f ? r.g.y : r.g.x;
    const bool friction = act && k1 > 0.0f && k2 > 0.0f;
    if (!Cone) {
        const float lack = target - vn;
        float jn;
        if (Exact) {
            jn = act ? lack / r.n.w : 0.0f;
        } else {
            jn = quotient(lack, r.n.w, r.y.x);
            if (act && !quotientRange(lack)) jn = lack / r.n.w;
        }
        const float next = vmax(nImp + jn, 0.0f);
        jn = next - nImp;
        nImp = next;
        laneImpulse<Exact>(b, side, arm, n * jn);
        pairBoth(b.v + rowCross<Exact>(b.w, arm), side, ua, ub);
        const V3 rv = ua - ub;
        const float d1 = dot(rv, t1), d2 = dot(rv, t2);
        float c1, c2;
        if (Exact) {
            c1 = friction ? d1 / k1 : 0.0f;
            c2 = friction ? d2 / k2 : 0.0f;
        } else {
            c1 = quotient(d1, k1, r.y.y);
            c2 = quotient(d2, k2, r.y.z);
            if (friction && !(quotientRange(d1) & quotientRange(d2))) {
                c1 = d1 / k1;
                c2 = d2 / k2;
            }
        }
        float n1 = i1 - c1, n2 = i2 - c2;
        // without friction terms: both axes read as inside, nothing changes
        const float max1 = friction ? r.g.z * nImp : 0.0f, max2 = friction ? r.g.w * nImp : 0.0f;
        clampToEllipse(side, max1, max2, n1, n2);
        if (friction) {
            laneImpulse<Exact>(b, side, arm, t1 * (n1 - i1) + t2 * (n2 - i2));
            i1 = n1;
            i2 = n2;
        }
    } else {
        float nextN = nImp, n1 = i1, n2 = i2;
        if (friction) {
            const float4 cn = act ? R.aux[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float kN = r.n.w, kN1 = cn.x, kN2 = cn.y, k12 = cn.z;
            const float det = kN * (k1 * k2 - k12 * k12) - kN1 * (kN1 * k2 - kN2 * k12) +
                              kN2 * (kN1 * k12 - kN2 * k1);
            if (fabsf(det) > 1e-12f) {
                const float bN = target - dot(rv0, n);
                const float b1 = -dot(rv0, t1);
                const float b2 = -dot(rv0, t2);
                const float dN = (bN * (k1 * k2 - k12 * k12) + b1 * (kN2 * k12 - kN1 * k2) +
                                  b2 * (kN1 * k12 - kN2 * k1)) / det;
                const float d1 = (bN * (kN2 * k12 - kN1 * k2) + b1 * (kN * k2 - kN2 * kN2) +
                                  b2 * (kN1 * kN2 - kN * k12)) / det;
                const float d2 = (bN * (kN1 * k12 - kN2 * k1) + b1 * (kN1 * kN2 - kN * k12) +
                                  b2 * (kN * k1 - kN1 * kN1)) / det;
                nextN = vmax(nImp + dN, 0.0f);
                n1 = i1 + d1;
                n2 = i2 + d2;
            }
        }
        const float max1 = r.g.z * nextN, max2 = r.g.w * nextN;
        clampToEllipse(side, max1, max2, n1, n2);
        laneImpulse<Exact>(b, side, arm, n * (nextN - nImp) + t1 * (n1 - i1) + t2 * (n2 - i2));
        nImp = nextN;
        i1 = n1;
        i2 = n2;
    }
    const uint32_t bits = __float_as_uint(r.i.w);
    if (Exact && __any_sync(0xffffffffu, act && (bits & kRowExt))) {  // rolling and spinning resistance
        const bool on = act && (bits & kRowExt);
        float4* E = R.ext + 2 * (2 * (size_t)k + side);
        const float4 e0 = on ? E[0] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float4 e1 = on ? E[1] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        V3 wa, wb;
        pairBoth(b.w, side, wa, wb);
        if (e0.w > 0.0f && e0.x > 0.0f && e0.y > 0.0f) {
            const V3 wr = wa - wb;
            float n1 = e1.y - dot(wr, t1) / e0.x;
            float n2 = e1.z - dot(wr, t2) / e0.y;
            const float limit = e0.w * nImp;
            const float mag = sqrtf(n1 * n1 + n2 * n2);
            if (mag > limit && mag > 1e-9f) {
                const float sc = limit / mag;
                n1 *= sc;
                n2 *= sc;
            }
            laneTorque(b, side, t1 * (n1 - e1.y) + t2 * (n2 - e1.z));
            e1.y = n1;
            e1.z = n2;
        }
        pairBoth(b.w, side, wa, wb);
        if (e1.x > 0.0f && e0.z > 0.0f) {
            const V3 wr = wa - wb;
            float next = e1.w - dot(wr, n) / e0.z;
            const float limit = e1.x * nImp;
            next = vclamp(next, -limit, limit);
            laneTorque(b, side, n * (next - e1.w));
            e1.w = next;
        }
        if (on) E[1] = e1;
    }
    r.i = make_float4(nImp, i1, i2, r.i.w);
}

// The lane's body in a velocity row.
VXD LaneBody loadLane(const SolveArgs& A, const BodyTable& T, int li) {
    LaneBody b;
    b.dyn = li >= 0;
    b.turns = false;
    b.im = 0.0f;
    b.v = b.w = b.invI = V3{0.0f, 0.0f, 0.0f};
    b.frame = Q4{0.0f, 0.0f, 0.0f, 1.0f};
    if (li >= 0) {
        const float4 tv = T.v[li], tw = T.w[li], tf = T.f[li], ti = T.i[li];
        b.v = f3(tv);
        b.turns = tv.w == 0.0f;
        b.w = f3(tw);
        b.frame = q4(tf);
        b.invI = f3(ti);
        b.im = ti.w;
    } else if (li != kAtRest) {
        b.v = f3(A.B.vel[~li]);
        b.w = f3(A.B.ang[~li]);
    }
    return b;
}

// One lane of one row (all 32 lanes call; `act`: this lane holds a row).
// warmPrepRow / sweepRow / positionRow on the pair's two lanes, the same
// arithmetic in the same order.
template <int Op, bool Cone>
VXD void laneRow(const SolveArgs& A, const RowPlanes& R, const BodyTable& T, bool act, uint32_t k, uint32_t side,
                 RowRegs& r, LaneBody& b) {
    const int li = act ? __float_as_int(r.s.w) : kAtRest;
    const V3 arm = f3(r.s), n = f3(r.n);
    if (Op == kRowPosition) {
        V3 p{0.0f, 0.0f, 0.0f};
        float asleep = 0.0f, im = 0.0f;
        if (li >= 0) {
            const float4 t = T.v[li];
            p = f3(t);
            asleep = t.w;
            im = T.i[li].w;
        } else if (act) {
            p = f3(A.B.pos[~li]);
        }
        V3 wa, wb;
        pairBoth(p + arm, side, wa, wb);
        const float gap = r.n.w + dot(n, wa - wb);
        if (!act || r.g.y <= 0.0f || gap >= -1e-3f) return;
        const float push = -r.g.x * (gap + 1e-3f) / r.g.y;
        if (li >= 0 && asleep == 0.0f) {
            const V3 d = n * (push * im);
            T.v[li] = pack(side ? p - d : p + d, 0.0f);
        }
        return;
    }
    const float locked = b.turns ? 0.0f : 1.0f;
    const V3 t1 = f3(r.t1), t2 = f3(r.t2);
    const uint32_t bits = __float_as_uint(r.i.w);
    if (Op == kRowWarm) {
        if (!act || !(bits & kRowSolved)) return;
        const vx_contact& c = A.contacts[A.order[k]];
        const float r1 = c.rollingImpulse1, r2 = c.rollingImpulse2, sp = c.spinningImpulse;
        if (r.i.x <= 0.0f && r.i.y == 0.0f && r.i.z == 0.0f && r1 == 0.0f && r2 == 0.0f && sp == 0.0f) return;
        laneImpulse<true>(b, side, arm, n * r.i.x + t1 * r.i.y + t2 * r.i.z);
        laneTorque(b, side, t1 * r1 + t2 * r2 + n * sp);
        if (li >= 0) { T.v[li] = pack(b.v, locked); T.w[li] = pack(b.w, 0.0f); }
        return;
    }
    act = act && !(r.n.w <= 0.0f);
    const bool special = act && ((bits & (kRowExt | (Cone ? 0u : kRowRecip))) != (Cone ? 0u : kRowRecip) || negativeZeroKey(b.w.x, b.w.y, b.w.z, r.i.y, r.i.z) == INT_MIN);
    if (__any_sync(0xffffffffu, special)) laneSweep<true, Cone>(R, act, k, side, r, b);
    else laneSweep<false, Cone>(R, act, k, side, r, b);
    if (!act) return;
    if (li >= 0) { T.v[li] = pack(b.v, locked); T.w[li] = pack(b.w, 0.0f); }
    R.imp[2 * (size_t)k + side] = r.i;
}

template <int Threads>
VXD void islandBarrier() {
    if (Threads == 32) __syncwarp();
    else __syncthreads();
}

// `units` passes over the island's colours. A lane's next row (this colour's
// next batch, else the next colour's first) is loaded before the current one
// runs; rows are always taken by the same lane, so a row's impulses come back
// to the lane that wrote them.
template <int Threads, int Op, bool Cone>
VXD void runColours(const SolveArgs& A, const RowPlanes& R, const BodyTable& T, const uint32_t* seg,
                    uint32_t colours, int units) {
    constexpr uint32_t kPairs = Threads / 2;
    const uint32_t pair = threadIdx.x >> 1, side = threadIdx.x & 1u, warpPair = (threadIdx.x & ~31u) >> 1;
    uint32_t start = seg[0], end = seg[1];
    uint32_t k = start + pair;
    RowRegs even, odd;  // the current and the next row, in turn
    even.s = even.n = even.t1 = even.t2 = even.g = even.i = even.y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (k < end) loadRowRegs<Op>(R, k, side, even);
    odd = even;
    uint32_t kw = start + warpPair, c = 0;
    const uint32_t steps = (uint32_t)units * colours;
    uint32_t done = 0;
    while (done < steps) {
        // one batch of this colour on `now`, the next batch loading into `then`
        auto batch = [&](RowRegs& now, RowRegs& then) {
            const bool more = kw + kPairs < end;  // the warp has another batch in this colour
            uint32_t nextStart = start, nextEnd = end;
            if (!more) {
                const uint32_t nc = c + 1 == colours ? 0u : c + 1;
                nextStart = seg[nc];
                nextEnd = done + 1 == steps ? 0u : seg[nc + 1];
            }
            const uint32_t kn = more ? k + kPairs : nextStart + pair;
            // the bodies first: shared loads queue behind global ones
            LaneBody b = loadLane(A, T, Op != kRowPosition && k < end ? __float_as_int(now.s.w) : kAtRest);
            if (kn < nextEnd) loadRowRegs<Op>(R, kn, side, then);
            if (kw < end) laneRow<Op, Cone>(A, R, T, k < end, k, side, now, b);
            if (kn == k) then.i = now.i;  // a lone row per lane: its impulses were just updated
            k = kn;
            if (more) {
                kw += kPairs;
            } else {
                start = nextStart;
                end = nextEnd;
                kw = start + warpPair;
                c = c + 1 == colours ? 0u : c + 1;
                ++done;
                islandBarrier<Threads>();
            }
        };
        batch(even, odd);
        if (done == steps) break;
        batch(odd, even);
    }
}

// ---- several warps on one island: a dataflow over the body table ------------
//
// Colour order only constrains rows that share a dynamic body, so with several
// warps the colours need no barrier: the table's velocities end in a tag that
// counts the body's row updates since the substep's start, and a row, which
// knows its rank among its body's rows, waits for the two tags it must find.
// The rows are cut into batches of one colour, taken by the warps in turn; a
// batch's predecessors all lie in earlier batches, so the waits end (each is
// bounded all the same). Solve stage of one step against the colour barrier:
// 5.3 -> 4.5 ms with 64 islands of 2,400 rows, 1.9 -> 1.6 ms with one of 310;
// 24 steps of 128 islands of 34 rows on four warps instead of one 27 -> 22 ms.
// Batches of 8 or 4 rows were slower (7.2 and 12.6 ms for the 64: more batches
// poll), as was sleeping between polls.
// Whole 16-byte accesses: a vector access is four scalar ones in any order to
// the memory model, a .b128 one is a single access, so a body's velocity
// arrives with the tag that announces it.
VXD float4 ldTable(const float4* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.cta.shared.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
    return make_float4(__uint_as_float((uint32_t)lo), __uint_as_float((uint32_t)(lo >> 32)),
                       __uint_as_float((uint32_t)hi), __uint_as_float((uint32_t)(hi >> 32)));
}
VXD void stTable(float4* p, const V3& v, uint32_t tag) {
    const unsigned long long lo = (unsigned long long)__float_as_uint(v.y) << 32 | __float_as_uint(v.x);
    const unsigned long long hi = (unsigned long long)tag << 32 | __float_as_uint(v.z);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.cta.shared.b128 [%0], t;\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(p)),
                 "l"(lo), "l"(hi)
                 : "memory");
}

// One batch (all 32 lanes call). u: the sweep counted from the substep's
// start. Returns false when a wait gave up.
template <bool Cone>
VXD bool tableRow(const SolveArgs& A, const RowPlanes& R, const BodyTable& T, bool act, uint32_t k, uint32_t side,
                  uint32_t u, bool warm, RowRegs& r, volatile int* dead) {
    const uint32_t bits = __float_as_uint(r.i.w);
    act = act && (bits & kRowSolved);
    const int li = act ? __float_as_int(r.s.w) : kAtRest;
    const uint32_t rank = (bits >> kRowLinkShift) & kRowLinkMask, degree = bits >> kRowDegreeShift;
    const uint32_t tag = u * degree + rank;
    LaneBody b;
    b.dyn = li >= 0;
    b.turns = b.dyn && (bits & kRowTurns);
    b.im = 0.0f;
    b.v = b.w = b.invI = V3{0.0f, 0.0f, 0.0f};
    b.frame = Q4{0.0f, 0.0f, 0.0f, 1.0f};
    if (li >= 0) {
        const float4 ti = T.i[li];
        b.frame = q4(T.f[li]);
        b.invI = f3(ti);
        b.im = ti.w;
    } else if (li != kAtRest) {
        b.v = f3(A.B.vel[~li]);
        b.w = f3(A.B.ang[~li]);
    }
    bool ok = li < 0;
    for (uint32_t spins = 0;; ++spins) {
        if (!ok) {
            const float4 tv = ldTable(T.v + li), tw = ldTable(T.w + li);
            ok = __float_as_uint(tv.w) == tag && __float_as_uint(tw.w) == tag;
            b.v = f3(tv);
            b.w = f3(tw);
        }
        if (__all_sync(0xffffffffu, ok)) break;
        if (spins > A.waitLimit) {
            atomicOr(A.timeout, 1u);
            *dead = 1;
        }
        if ((spins & 63u) == 63u && __any_sync(0xffffffffu, *dead != 0)) return false;
    }
    const V3 arm = f3(r.s), n = f3(r.n);
    if (warm) {
        if (act) {
            const vx_contact& c = A.contacts[A.order[k]];
            const float r1 = c.rollingImpulse1, r2 = c.rollingImpulse2, sp = c.spinningImpulse;
            const V3 t1 = f3(r.t1), t2 = f3(r.t2);
            if (!(r.i.x <= 0.0f && r.i.y == 0.0f && r.i.z == 0.0f && r1 == 0.0f && r2 == 0.0f && sp == 0.0f)) {
                laneImpulse<true>(b, side, arm, n * r.i.x + t1 * r.i.y + t2 * r.i.z);
                laneTorque(b, side, t1 * r1 + t2 * r2 + n * sp);
            }
        }
    } else {
        const bool solve = act && !(r.n.w <= 0.0f);
        const uint32_t plain = Cone ? 0u : kRowRecip;
        const bool special = solve && ((bits & (kRowExt | plain)) != plain ||
                                       negativeZeroKey(b.w.x, b.w.y, b.w.z, r.i.y, r.i.z) == INT_MIN);
        const float4 imp = r.i;
        const V3 v0 = b.v, w0 = b.w;
        if (__any_sync(0xffffffffu, special)) laneSweep<true, Cone>(R, solve, k, side, r, b);
        else laneSweep<false, Cone>(R, solve, k, side, r, b);
        if (!solve) {  // a row without normal mass passes its bodies on
            r.i = imp;
            b.v = v0;
            b.w = w0;
        } else {
            R.imp[2 * (size_t)k + side] = r.i;
        }
    }
    if (li >= 0) {
        stTable(T.v + li, b.v, tag + 1u);
        stTable(T.w + li, b.w, tag + 1u);
    }
    return true;
}

// `units` passes over the island's batches, of which the first `warmUnits`
// warm-start. batches: first row (12 bits, from s0) | rows - 1 << 12.
template <int Threads, bool Cone>
VXD void runBatches(const SolveArgs& A, const RowPlanes& R, const BodyTable& T, const uint16_t* batches,
                    uint32_t count, uint32_t s0, uint32_t units, uint32_t warmUnits, volatile int* dead) {
    constexpr uint32_t kWarps = Threads / 32;
    const uint32_t warp = threadIdx.x >> 5, pair = (threadIdx.x & 31u) >> 1, side = threadIdx.x & 1u;
    if (warp >= count) return;
    RowRegs even, odd;  // the current and the next batch, in turn
    even.s = even.n = even.t1 = even.t2 = even.g = even.i = even.y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    odd = even;
    uint32_t at = warp, u = 0, word = batches[at];
    if (pair <= word >> 12) loadRowRegs<kRowSweep>(R, s0 + (word & 0xfffu) + pair, side, even);
    bool alive = true;
    auto batch = [&](RowRegs& now, RowRegs& then) {
        const bool wrap = at + kWarps >= count;
        const uint32_t nat = wrap ? warp : at + kWarps, nu = wrap ? u + 1u : u, nword = batches[nat];
        if (nu < units && pair <= nword >> 12)
            loadRowRegs<kRowSweep>(R, s0 + (nword & 0xfffu) + pair, side, then);
        alive = tableRow<Cone>(A, R, T, pair <= word >> 12, s0 + (word & 0xfffu) + pair, side, u, u < warmUnits, now,
                               dead);
        if (nat == at) then.i = now.i;  // the warp's only batch: its impulses were just updated
        at = nat;
        u = nu;
        word = nword;
    };
    while (u < units && alive) {
        batch(even, odd);
        if (u >= units || !alive) break;
        batch(odd, even);
    }
}

// The body of a row for prepRow: pose and mass from global memory, the frame
// from the table.
VXD SolverBody tableBody(const SolveArgs& A, const BodyTable& T, int li, uint32_t id) {
    SolverBody b;
    b.p = f3(A.B.pos[id]);
    b.q = q4(A.B.rot[id]);
    const float4 in = A.B.inertia[id];
    b.m.invI = f3(in);
    b.m.invMass = in.w;
    b.m.iq = q4(A.B.iq[id]);
    b.m.flags = A.B.filt[id].x;
    b.sphere = shapeOf(b.m.flags) == kSphere;
    if (li >= 0) b.frame = q4(T.f[li]);
    else cacheFrame(b);
    return b;
}

// Body words of a row: its dynamic bodies' table indices. The null island
// (nb = 0: sensor contacts and contacts without a dynamic body) moves none. A
// dynamic body outside a real island's list means an inconsistent plan:
// reported, and the row then leaves that body alone.
VXD int bodyWord(const SolveArgs& A, const uint32_t* localIdx, uint32_t b0, uint32_t nb, uint32_t id, bool poses) {
    if (nb == 0u || !isDynamic(A.B.filt[id].x)) {
        if (poses) return ~(int)id;
        const float4 v = A.B.vel[id], w = A.B.ang[id];
        const int bits = __float_as_int(v.x) | __float_as_int(v.y) | __float_as_int(v.z) | __float_as_int(w.x) |
                         __float_as_int(w.y) | __float_as_int(w.z);
        return bits == 0 ? kAtRest : ~(int)id;
    }
    const uint32_t li = localIdx[id];
    if (li < nb && A.bodyOrder[b0 + li] == id) return (int)li;
    atomicOr(A.fault, 1u);
    return ~(int)id;
}

// A row's pose terms into the planes (all but its arms and impulses) for
// substep s; returns its bits.
template <bool Cone>
VXD uint32_t storeRowPlanes(const RowPlanes& R, uint32_t k, const RowContact& rc, const RowPrep& P, bool solved, int s) {
    R.n[k] = pack(rc.normal, solved ? P.kNormal : 0.0f);
    R.t1[k] = pack(P.t1, P.k1);
    R.t2[k] = pack(P.t2, P.k2);
    float closing = P.targetBase, parting = P.targetBase;
    if (rc.vn0 < -1.0f) {
        parting = vmax(P.targetBase, -rc.restitution * rc.vn0);
        if (P.liveGap <= 0.0f) closing = parting;
    }
    R.g[k] = make_float4(closing, parting, rc.friction1, rc.friction2);
    R.aux[k] = Cone ? make_float4(P.kN1, P.kN2, P.k12, 0.0f)
                    : make_float4(1.0f / P.kNormal, 1.0f / P.k1, 1.0f / P.k2, 0.0f);
    const bool ext = rc.rolling > 0.0f || rc.spinning > 0.0f;
    const bool recip = quotientBase(P.kNormal) &&
                       (!(P.k1 > 0.0f && P.k2 > 0.0f) || (quotientBase(P.k1) && quotientBase(P.k2)));
    if (ext)
        for (int side = 0; side < 2; ++side) {
            float4* E = R.ext + 2 * (2 * (size_t)k + side);
            E[0] = make_float4(P.kr1, P.kr2, P.ks, rc.rolling);
            if (s == 0) E[1] = make_float4(rc.spinning, rc.r1Imp, rc.r2Imp, rc.sImp);
        }
    return (ext ? kRowExt : 0u) | (solved ? kRowSolved : 0u) | (recip ? kRowRecip : 0u);
}

// The sweeps set a contact's point to these poses' anchors; a warm start
// without sweeps only for rows that carry impulses.
VXD bool setsPoint(const SolveArgs& A, int s, bool solved, const RowContact& rc) {
    return solved && (A.sweeps > 0 ||
                      (A.warmStart && s == 0 && !(rc.nImp <= 0.0f && rc.t1Imp == 0.0f && rc.t2Imp == 0.0f &&
                                                  rc.r1Imp == 0.0f && rc.r2Imp == 0.0f && rc.sImp == 0.0f)));
}

VXD void storeRowImpulses(const RowPlanes& R, uint32_t k, vx_contact& c) {
    const float4 imp = R.imp[2 * (size_t)k];
    c.normalImpulse = imp.x;
    c.tangentImpulse1 = imp.y;
    c.tangentImpulse2 = imp.z;
    if (__float_as_uint(imp.w) & kRowExt) {
        const float4 e1 = R.ext[4 * (size_t)k + 1];
        c.rollingImpulse1 = e1.y;
        c.rollingImpulse2 = e1.z;
        c.spinningImpulse = e1.w;
    }
}

template <int Class, bool Cone>
__global__ void __launch_bounds__(ClassShape<Class>::kThreads, ClassShape<Class>::kBlocksPerSm)
    solveIslandKernel(SolveArgs A, uint32_t* localIdx) {
    constexpr int Threads = ClassShape<Class>::kThreads, kBodies = ClassShape<Class>::kBodies;
    extern __shared__ float4 islandSmem[];
    BodyTable T;
    T.v = islandSmem;
    T.w = T.v + kBodies;
    T.f = T.w + kBodies;
    T.i = T.f + kBodies;
    uint32_t* segShared = reinterpret_cast<uint32_t*>(T.i + kBodies);
    uint16_t* batches = reinterpret_cast<uint16_t*>(segShared + ClassShape<Class>::kSegments);  // kFlow only
    constexpr bool kFlow = ClassShape<Class>::kFlow;
    __shared__ uint32_t batchCount;
    __shared__ int dead;
    const RowPlanes R = rowPlanes(A);
    for (uint32_t isl = blockIdx.x; isl < A.islands; isl += gridDim.x) {
        const uint32_t s0 = A.islandStart[isl], s1 = A.islandStart[isl + 1];
        const uint32_t b0 = isl < A.realIslands ? A.bodyStart[isl] : 0u;
        const uint32_t b1 = isl < A.realIslands ? A.bodyStart[isl + 1] : 0u;
        const uint32_t nb = b1 - b0;
        if (solveClassOf(nb, s1 - s0, A.tinyLimit) != (Class == kSmallWide ? (int)kSmallIsland : Class)) continue;
        const uint32_t g0 = A.islandSeg[isl], colours = A.islandSeg[isl + 1] - g0;
        const uint32_t* seg = A.segStart + g0;
        if (colours < (uint32_t)ClassShape<Class>::kSegments) {
            for (uint32_t c = threadIdx.x; c <= colours; c += Threads) segShared[c] = seg[c];
            seg = segShared;
        }
        const bool position = A.positionIterations > 0;
        for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
            const uint32_t id = A.bodyOrder[b0 + t];
            const Mass m{f3(A.B.inertia[id]), A.B.inertia[id].w, q4(A.B.iq[id]), A.B.filt[id].x};
            localIdx[id] = t;
            T.i[t] = pack(m.invI, solverInvMass(m));
            if (position) {
                T.v[t] = pack(f3(A.B.pos[id]), isAsleep(m.flags) ? 1.0f : 0.0f);
            } else {
                T.v[t] = pack(f3(A.B.vel[id]), !kFlow && isRotationLocked(m.flags) ? 1.0f : 0.0f);
                T.w[t] = A.B.ang[id];
            }
        }
        islandBarrier<Threads>();
        if (kFlow && !position) {
            // ranks of the rows on their bodies, colour by colour (a colour has one row a body)
            uint32_t* seen = reinterpret_cast<uint32_t*>(T.f);  // the frames come later
            for (uint32_t t = threadIdx.x; t < nb; t += Threads) seen[t] = 0u;
            // (a wait that gave up on another island ends this one's at once)
            if (threadIdx.x == 0u) dead = *static_cast<volatile uint32_t*>(A.timeout) != 0u;
            for (uint32_t k = s0 + threadIdx.x; k < s1; k += Threads) {
                const vx_contact& c = A.contacts[A.order[k]];
                const bool solved = solvedContact(A.B.filt[c.a].x, A.B.filt[c.b].x);
                const int la = bodyWord(A, localIdx, b0, nb, c.a, false), lb = bodyWord(A, localIdx, b0, nb, c.b, false);
                R.side[2 * (size_t)k].w = __int_as_float(solved ? la : kAtRest);
                R.side[2 * (size_t)k + 1].w = __int_as_float(solved ? lb : kAtRest);
            }
            islandBarrier<Threads>();
            for (uint32_t c = 0; c < colours; ++c) {
                for (uint32_t x = 2u * seg[c] + threadIdx.x; x < 2u * seg[c + 1]; x += Threads) {
                    const int li = __float_as_int(R.side[x].w);
                    if (li >= 0) R.imp[x].w = __uint_as_float(seen[li]++ << kRowLinkShift);
                }
                islandBarrier<Threads>();
            }
            for (uint32_t x = 2u * s0 + threadIdx.x; x < 2u * s1; x += Threads) {
                const int li = __float_as_int(R.side[x].w);
                R.imp[x].w = __uint_as_float(li >= 0 ? __float_as_uint(R.imp[x].w) | seen[li] << kRowDegreeShift : 0u);
            }
            if (threadIdx.x < 32u) {  // the batches of each colour, one lane a colour
                constexpr uint32_t kBatch = ClassShape<Class>::kBatch;
                uint32_t base = 0u;
                for (uint32_t c0 = 0; c0 < colours; c0 += 32u) {
                    const uint32_t c = c0 + threadIdx.x;
                    const uint32_t from = c < colours ? seg[c] : 0u, to = c < colours ? seg[c + 1] : 0u;
                    const uint32_t need = (to - from + kBatch - 1u) / kBatch;
                    uint32_t incl = need;
                    for (int off = 1; off < 32; off <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
                        if ((int)threadIdx.x >= off) incl += y;
                    }
                    uint32_t at = base + incl - need;
                    for (uint32_t k = from; k < to; k += kBatch)
                        batches[at++] = (uint16_t)((k - s0) | (min(kBatch, to - k) - 1u) << 12);
                    base += __shfl_sync(0xffffffffu, incl, 31);
                }
                if (threadIdx.x == 0u) batchCount = base;
            }
            islandBarrier<Threads>();
        }
        if (position) {
            for (uint32_t k = s0 + threadIdx.x; k < s1; k += Threads) {
                const vx_contact& c = A.contacts[A.order[k]];
                const int la = bodyWord(A, localIdx, b0, nb, c.a, true), lb = bodyWord(A, localIdx, b0, nb, c.b, true);
                const uint32_t fa = A.B.filt[c.a].x, fb = A.B.filt[c.b].x;
                const Mass ma = loadMass(A.B, c.a), mb = loadMass(A.B, c.b);
                const V3 na{c.localAnchorA.x, c.localAnchorA.y, c.localAnchorA.z};
                const V3 nbv{c.localAnchorB.x, c.localAnchorB.y, c.localAnchorB.z};
                R.side[2 * (size_t)k] =
                    pack(shapeOf(fa) == kSphere ? na : rotate(q4(A.B.rot[c.a]), na), __int_as_float(la));
                R.side[2 * (size_t)k + 1] =
                    pack(shapeOf(fb) == kSphere ? nbv : rotate(q4(A.B.rot[c.b]), nbv), __int_as_float(lb));
                R.n[k] = make_float4(c.normal.x, c.normal.y, c.normal.z, c.bias0);
                float resolve = 0.6f;
                if (A.stackStabilization && lengthSq(f3(A.B.vel[c.a]) - f3(A.B.vel[c.b])) < 1e-4f)
                    resolve += 0.2f * (A.stackStiffness / 1000.0f) / (1.0f + A.stackDamping * A.h);
                R.g[k] = make_float4(resolve, solvedContact(fa, fb) ? solverInvMass(ma) + solverInvMass(mb) : 0.0f,
                                     0.0f, 0.0f);
            }
            islandBarrier<Threads>();
            runColours<Threads, kRowPosition, Cone>(A, R, T, seg, colours, A.positionIterations);
            for (uint32_t t = threadIdx.x; t < nb; t += Threads)
                A.B.pos[A.bodyOrder[b0 + t]] = pack(f3(T.v[t]), 0.0f);
            islandBarrier<Threads>();
            continue;
        }
        for (int s = 0; s < A.substeps; ++s) {
            for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
                const uint32_t id = A.bodyOrder[b0 + t];
                const Mass m = loadMass(A.B, id);
                const Q4 q = q4(A.B.rot[id]);
                if (A.integrate && s > 0 && !isLocked(m.flags) && !isAsleep(m.flags)) {  // integrateVelocity
                    const float4 tv = T.v[t], ex = A.B.extra[id];
                    V3 v = f3(tv), w = f3(T.w[t]);
                    v += (A.gravity * ex.y + f3(A.B.force[id]) * solverInvMass(m)) * A.h;
                    w += invInertiaMulAt(m, f3(A.B.torque[id]), q) * A.h;
                    v *= 1.0f / (1.0f + ex.z * A.h);
                    w *= 1.0f / (1.0f + ex.w * A.h);
                    T.v[t] = pack(v, tv.w);
                    T.w[t] = pack(w, 0.0f);
                }
                if (kFlow) T.v[t].w = T.w[t].w = 0.0f;  // fresh tags
                T.f[t] = pack(inertiaFrameAt(m, q));
            }
            islandBarrier<Threads>();
            for (uint32_t k = s0 + threadIdx.x; k < s1; k += Threads) {
                vx_contact& c = A.contacts[A.order[k]];
                int la, lb;
                if (s == 0 && !kFlow) {
                    la = bodyWord(A, localIdx, b0, nb, c.a, false);
                    lb = bodyWord(A, localIdx, b0, nb, c.b, false);
                } else {
                    la = __float_as_int(R.side[2 * (size_t)k].w);
                    lb = __float_as_int(R.side[2 * (size_t)k + 1].w);
                }
                const SolverBody a = tableBody(A, T, la, c.a), b = tableBody(A, T, lb, c.b);
                RowContact rc;
                loadRow(c, rc);
                RowPrep P;
                prepRow(a, b, rc, A.h, Cone, P);
                const bool solved = solvedContact(a.m.flags, b.m.flags);
                const uint32_t bits = storeRowPlanes<Cone>(R, k, rc, P, solved, s);
                R.side[2 * (size_t)k] = pack(P.ra, __int_as_float(la));
                R.side[2 * (size_t)k + 1] = pack(P.rb, __int_as_float(lb));
                float4 imp = make_float4(rc.nImp, rc.t1Imp, rc.t2Imp, 0.0f);
                if (s > 0) imp = R.imp[2 * (size_t)k];
                uint32_t wordA = bits, wordB = bits;
                if (kFlow) {
                    const uint32_t link = ~((1u << kRowLinkShift) - 1u);
                    wordA |= (__float_as_uint(R.imp[2 * (size_t)k].w) & link) |
                             (isRotationLocked(a.m.flags) ? 0u : kRowTurns);
                    wordB |= (__float_as_uint(R.imp[2 * (size_t)k + 1].w) & link) |
                             (isRotationLocked(b.m.flags) ? 0u : kRowTurns);
                }
                imp.w = __uint_as_float(wordA);
                R.imp[2 * (size_t)k] = imp;
                imp.w = __uint_as_float(wordB);
                R.imp[2 * (size_t)k + 1] = imp;
                if (setsPoint(A, s, solved, rc)) c.point = vx_vec3{P.point.x, P.point.y, P.point.z};
            }
            islandBarrier<Threads>();
            const bool warm = A.warmStart && s == 0;
            if constexpr (kFlow) {
                runBatches<Threads, Cone>(A, R, T, batches, batchCount, s0, (warm ? 1u : 0u) + (uint32_t)A.sweeps,
                                          warm ? 1u : 0u, &dead);
                islandBarrier<Threads>();
            } else {
                if (warm) runColours<Threads, kRowWarm, Cone>(A, R, T, seg, colours, 1);
                runColours<Threads, kRowSweep, Cone>(A, R, T, seg, colours, A.sweeps);
            }
            if (A.integrate) {
                for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
                    const uint32_t id = A.bodyOrder[b0 + t];
                    const Mass m = loadMass(A.B, id);
                    if (isLocked(m.flags) || isAsleep(m.flags)) continue;
                    V3 p = f3(A.B.pos[id]), w = f3(T.w[t]);
                    Q4 q = q4(A.B.rot[id]);
                    advanceTransform(m, p, q, f3(T.v[t]), w, A.h);
                    A.B.pos[id] = pack(p, 0.0f);
                    A.B.rot[id] = pack(q);
                    T.w[t] = pack(w, 0.0f);
                }
                islandBarrier<Threads>();
            }
        }
        for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
            const uint32_t id = A.bodyOrder[b0 + t];
            A.B.vel[id] = pack(f3(T.v[t]), 0.0f);
            A.B.ang[id] = pack(f3(T.w[t]), 0.0f);
        }
        for (uint32_t k = s0 + threadIdx.x; k < s1; k += Threads) {
            storeRowImpulses(R, k, A.contacts[A.order[k]]);
        }
        islandBarrier<Threads>();
    }
}

}  // namespace vxb
