// Giant islands (beyond 512 bodies or 3,072 rows) by the whole grid, as a
// dataflow over their bodies.
//
// Colour order only constrains rows that share a dynamic body, so a row may
// run as soon as its two bodies carry the state that order gives it. Each body
// has a 64-byte record whose velocity and angular velocity end in a tag: the
// number of row updates the body has had since the substep's start. A row
// knows its rank among its body's rows and the body's row count, hence the tag
// to wait for in every sweep; it polls the records themselves, so the data
// arrives with the word that announces it (16-byte relaxed loads and stores
// are single accesses): no flag, no fence, no barrier between colours or
// sweeps. Rows are owned by warps (the bodies in Morton order are cut into as
// many clusters as the grid has warps; a row belongs to its first dynamic
// body's), a warp takes its rows in (sweep, colour) order, up to 16 of one
// colour at once, two lanes a row, and loads the next ones while it waits. All
// warps are resident (cooperative launch), and the earliest unfinished step of
// all is always runnable, so the waits end; each is bounded all the same.
//
// What bounds it: the longest chain of rows through shared bodies (about the
// largest body's rows times the sweeps), a link costing one row update and one
// trip through L2. The previous kernel walked colour by colour behind a block
// barrier and handed rows over with release / acquire flags: 6-8 us a colour
// step. Solve stage of one step of a heap of 40,000 bodies (48,000 rows, 24
// colours, 64 sweeps): 9.2 -> 4.3 ms.
#pragma once
#include "coop.cuh"
#include "solve_rows.cuh"

namespace vxb {

constexpr int kFlowThreads = 128;
constexpr int kFlowBlocksPerSm = 3;
constexpr uint32_t kLastColour = 65535;  // colours past it share a segment (the colour key's 16 bits)

struct FlowArgs {
    const uint32_t* start;    // first slot of each warp (warps + 1)
    const uint32_t* rows;     // slot -> solve position
    const uint32_t* colour;   // slot -> colour within its island
    const uint32_t* rank;     // 2 per solve position: rank among the rows of its bodies a and b (0: no dynamic body)
    const uint32_t* degree;   // body -> its rows
    const uint32_t* bodyIds;  // the islands' bodies
    float4* body;             // 4 per body: velocity | tag, angular velocity | tag, frame, inverse inertia | mass
    uint32_t bodies;
};

// The whole 16 bytes in one access, coherent over the GPU.
VXD float4 ldRelaxed16(const float4* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return make_float4(__uint_as_float((uint32_t)lo), __uint_as_float((uint32_t)(lo >> 32)),
                       __uint_as_float((uint32_t)hi), __uint_as_float((uint32_t)(hi >> 32)));
}
VXD void stRelaxed16(float4* p, const V3& v, uint32_t tag) {
    const unsigned long long lo = (unsigned long long)__float_as_uint(v.y) << 32 | __float_as_uint(v.x);
    const unsigned long long hi = (unsigned long long)tag << 32 | __float_as_uint(v.z);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(lo), "l"(hi)
                 : "memory");
}

struct FlowRegs {
    RowRegs r;
    float4 frame, inertia;
    uint32_t degree;
};

template <int Op>
VXD void loadFlowRegs(const RowPlanes& R, const FlowArgs& F, uint32_t slot, uint32_t side, FlowRegs& x) {
    x.r.s = R.side[2 * (size_t)slot + side];
    x.r.n = R.n[slot];
    x.r.g = R.g[slot];
    x.r.y = R.aux[slot];
    x.r.i = R.imp[2 * (size_t)slot + side];
    const int li = __float_as_int(x.r.s.w);
    if (Op != kRowPosition) {
        x.r.t1 = R.t1[slot];
        x.r.t2 = R.t2[slot];
        if (li >= 0) x.frame = __ldcg(F.body + 4 * (size_t)li + 2);
    }
    if (li >= 0) {
        x.inertia = __ldcg(F.body + 4 * (size_t)li + 3);
        x.degree = F.degree[li];
    }
}

// Waits until every lane's body record carries the lane's tag; false when a
// wait gave up (here or elsewhere).
template <bool Both>
VXD bool awaitTags(const float4* rec, bool need, uint32_t tag, float4& v, float4& w, CoopState* st) {
    bool ok = !need;
    for (uint32_t spins = 0;; ++spins) {
        if (!ok) {
            v = ldRelaxed16(rec);
            if (Both) w = ldRelaxed16(rec + 1);
            ok = __float_as_uint(v.w) == tag && (!Both || __float_as_uint(w.w) == tag);
        }
        if (__all_sync(0xffffffffu, ok)) return true;
        if (spins > st->spinLimit) atomicOr(&st->timeout, 1u);
        if ((spins & 63u) == 63u && __any_sync(0xffffffffu, loadVolatile(&st->timeout) != 0u)) return false;
        if (spins > 16u) __nanosleep(32);
    }
}

// One batch of rows of one colour (all 32 lanes call). u: the sweep counted
// from the substep's start. Returns false when a wait gave up.
template <int Op, bool Cone>
VXD bool flowRow(const SolveArgs& A, const FlowArgs& F, const RowPlanes& R, bool act, uint32_t slot, uint32_t side,
                 uint32_t u, bool warm, FlowRegs& x, CoopState* st) {
    RowRegs& r = x.r;
    const uint32_t bits = __float_as_uint(r.i.w);
    act = act && (bits & kRowSolved);
    const int li = act ? __float_as_int(r.s.w) : kAtRest;
    const uint32_t tag = u * x.degree + (bits >> kRowLinkShift);
    float4* rec = F.body + 4 * (size_t)(li >= 0 ? li : 0);
    float4 tv = make_float4(0.0f, 0.0f, 0.0f, 0.0f), tw = tv;
    if (!awaitTags<Op != kRowPosition>(rec, li >= 0, tag, tv, tw, st)) return false;
    const V3 arm = f3(r.s), n = f3(r.n);
    if (Op == kRowPosition) {
        V3 p = f3(tv);
        if (act && li < 0) p = f3(A.B.pos[~li]);
        V3 wa, wb;
        pairBoth(p + arm, side, wa, wb);
        const float gap = r.n.w + dot(n, wa - wb);
        if (act && li >= 0) {
            // (as laneRow's step, a gap that is not a number included; kRowTurns: asleep, in this mode)
            if (!(r.g.y <= 0.0f) && !(gap >= -1e-3f) && !(bits & kRowTurns)) {
                const float push = -r.g.x * (gap + 1e-3f) / r.g.y;
                const V3 d = n * (push * x.inertia.w);
                p = side ? p - d : p + d;
            }
            stRelaxed16(rec, p, tag + 1u);
        }
        return true;
    }
    LaneBody b;
    b.dyn = li >= 0;
    b.turns = b.dyn && (bits & kRowTurns);
    b.im = 0.0f;
    b.v = f3(tv);
    b.w = f3(tw);
    b.invI = V3{0.0f, 0.0f, 0.0f};
    b.frame = Q4{0.0f, 0.0f, 0.0f, 1.0f};
    if (li >= 0) {
        b.frame = q4(x.frame);
        b.invI = f3(x.inertia);
        b.im = x.inertia.w;
    } else if (li != kAtRest) {
        b.v = f3(A.B.vel[~li]);
        b.w = f3(A.B.ang[~li]);
    }
    if (warm) {
        if (act) {
            const vx_contact& c = A.contacts[A.order[F.rows[slot]]];
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
        const RowRegs before = r;
        const V3 v0 = b.v, w0 = b.w;
        if (__any_sync(0xffffffffu, special)) laneSweep<true, Cone>(R, solve, slot, side, r, b);
        else laneSweep<false, Cone>(R, solve, slot, side, r, b);
        if (!solve) {  // a row without normal mass passes its bodies on
            r.i = before.i;
            b.v = v0;
            b.w = w0;
        } else {
            R.imp[2 * (size_t)slot + side] = r.i;
        }
    }
    if (li >= 0) {
        stRelaxed16(rec, b.v, tag + 1u);
        stRelaxed16(rec + 1, b.w, tag + 1u);
    }
    return true;
}

// `units` passes over the warp's rows [s0, s1), of which the first `warmUnits`
// warm-start.
template <int Op, bool Cone>
VXD void runFlow(const SolveArgs& A, const FlowArgs& F, const RowPlanes& R, uint32_t s0, uint32_t s1, uint32_t units,
                 uint32_t warmUnits, CoopState* st) {
    if (s0 >= s1) return;
    const uint32_t pair = (threadIdx.x & 31u) >> 1, side = threadIdx.x & 1u;
    FlowRegs even, odd;  // the current and the next batch, in turn
    even.r.s = even.r.n = even.r.t1 = even.r.t2 = even.r.g = even.r.i = even.r.y = even.frame = even.inertia =
        make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    even.degree = 0u;
    odd = even;
    uint32_t i = s0, u = 0;
    if (i + pair < s1) loadFlowRegs<Op>(R, F, i + pair, side, even);
    bool alive = true;
    auto batch = [&](FlowRegs& now, FlowRegs& then) {
        // the leading rows of the first row's colour (rows lie in colour order)
        const bool valid = i + pair < s1;
        const uint32_t colour = __float_as_uint(now.r.y.w);
        const uint32_t first = __shfl_sync(0xffffffffu, colour, 0);
        uint32_t count = (uint32_t)__popc(__ballot_sync(0xffffffffu, valid && colour == first)) >> 1;
        if (first == kLastColour) count = 1u;  // rows of this one may share a body: in order, one by one
        const bool wrap = i + count >= s1;
        const uint32_t ni = wrap ? s0 : i + count, nu = wrap ? u + 1u : u;
        if (nu < units && ni + pair < s1) loadFlowRegs<Op>(R, F, ni + pair, side, then);
        alive = flowRow<Op, Cone>(A, F, R, pair < count, i + pair, side, u, u < warmUnits, now, st);
        if (ni == i) then.r.i = now.r.i;  // the warp's only batch: its impulses were just updated
        i = ni;
        u = nu;
    };
    while (u < units && alive) {
        batch(even, odd);
        if (u >= units || !alive) break;
        batch(odd, even);
    }
}

// A body's state at the row's poses, read through L2 (other SMs integrate it).
VXD SolverBody flowBody(const SolveArgs& A, const FlowArgs& F, uint32_t id) {
    SolverBody b;
    b.p = f3(__ldcg(A.B.pos + id));
    b.q = q4(__ldcg(A.B.rot + id));
    b.m = loadMass(A.B, id);
    b.sphere = shapeOf(b.m.flags) == kSphere;
    if (isDynamic(b.m.flags)) b.frame = q4(__ldcg(F.body + 4 * (size_t)id + 2));
    else cacheFrame(b);
    return b;
}

VXD int flowWord(const SolveArgs& A, uint32_t id, uint32_t flags, bool poses) {
    if (isDynamic(flags)) return (int)id;
    if (poses) return ~(int)id;
    const float4 v = A.B.vel[id], w = A.B.ang[id];
    const int bits = __float_as_int(v.x) | __float_as_int(v.y) | __float_as_int(v.z) | __float_as_int(w.x) |
                     __float_as_int(w.y) | __float_as_int(w.z);
    return bits == 0 ? kAtRest : ~(int)id;
}

template <bool Cone>
__global__ void __launch_bounds__(kFlowThreads, kFlowBlocksPerSm) solveFlowKernel(SolveArgs A, FlowArgs F,
                                                                                  CoopState* st) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const uint32_t warp = tid >> 5, lane = threadIdx.x & 31u;
    const uint32_t s0 = F.start[warp], s1 = F.start[warp + 1u];
    const RowPlanes R = rowPlanes(A);
    auto linkBits = [&](uint32_t k, uint32_t side) { return F.rank[2 * (size_t)k + side] << kRowLinkShift; };
    if (A.positionIterations > 0) {
        for (uint32_t t = tid; t < F.bodies; t += stride) {
            const uint32_t id = F.bodyIds[t];
            const Mass m = loadMass(A.B, id);
            stRelaxed16(F.body + 4 * (size_t)id, f3(A.B.pos[id]), 0u);
            __stcg(F.body + 4 * (size_t)id + 3, pack(m.invI, solverInvMass(m)));
        }
        for (uint32_t slot = s0 + lane; slot < s1; slot += 32u) {
            const uint32_t k = F.rows[slot];
            const vx_contact& c = A.contacts[A.order[k]];
            const Mass ma = loadMass(A.B, c.a), mb = loadMass(A.B, c.b);
            const V3 na{c.localAnchorA.x, c.localAnchorA.y, c.localAnchorA.z};
            const V3 nb{c.localAnchorB.x, c.localAnchorB.y, c.localAnchorB.z};
            R.side[2 * (size_t)slot] = pack(shapeOf(ma.flags) == kSphere ? na : rotate(q4(A.B.rot[c.a]), na),
                                            __int_as_float(flowWord(A, c.a, ma.flags, true)));
            R.side[2 * (size_t)slot + 1] = pack(shapeOf(mb.flags) == kSphere ? nb : rotate(q4(A.B.rot[c.b]), nb),
                                                __int_as_float(flowWord(A, c.b, mb.flags, true)));
            R.n[slot] = make_float4(c.normal.x, c.normal.y, c.normal.z, c.bias0);
            float resolve = 0.6f;
            if (A.stackStabilization && lengthSq(f3(A.B.vel[c.a]) - f3(A.B.vel[c.b])) < 1e-4f)
                resolve += 0.2f * (A.stackStiffness / 1000.0f) / (1.0f + A.stackDamping * A.h);
            R.g[slot] = make_float4(resolve, solverInvMass(ma) + solverInvMass(mb), 0.0f, 0.0f);
            R.aux[slot] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(F.colour[slot]));
            const uint32_t solved = solvedContact(ma.flags, mb.flags) ? kRowSolved : 0u;
            R.imp[2 * (size_t)slot] =
                make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(solved | (isAsleep(ma.flags) ? kRowTurns : 0u) | linkBits(k, 0)));
            R.imp[2 * (size_t)slot + 1] =
                make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(solved | (isAsleep(mb.flags) ? kRowTurns : 0u) | linkBits(k, 1)));
        }
        if (!gridSync(&st->bar, &st->timeout, st->spinLimit)) return;
        runFlow<kRowPosition, Cone>(A, F, R, s0, s1, (uint32_t)A.positionIterations, 0u, st);
        if (!gridSync(&st->bar, &st->timeout, st->spinLimit)) return;
        for (uint32_t t = tid; t < F.bodies; t += stride) {
            const uint32_t id = F.bodyIds[t];
            A.B.pos[id] = pack(f3(ldRelaxed16(F.body + 4 * (size_t)id)), 0.0f);
        }
        return;
    }
    // bodies of substep s: the previous substep's sweeps into the pose, then
    // this one's velocities, frame and fresh tags
    auto bodies = [&](int s) {
        for (uint32_t t = tid; t < F.bodies; t += stride) {
            const uint32_t id = F.bodyIds[t];
            float4* rec = F.body + 4 * (size_t)id;
            const Mass m = loadMass(A.B, id);
            const bool moves = !isLocked(m.flags) && !isAsleep(m.flags);
            V3 v, w;
            Q4 q = q4(__ldcg(A.B.rot + id));
            if (s == 0) {
                v = f3(__ldcg(A.B.vel + id));
                w = f3(__ldcg(A.B.ang + id));
            } else {
                v = f3(ldRelaxed16(rec));
                w = f3(ldRelaxed16(rec + 1));
                if (A.integrate && moves) {
                    V3 p = f3(__ldcg(A.B.pos + id));
                    advanceTransform(m, p, q, v, w, A.h);
                    __stcg(A.B.pos + id, pack(p, 0.0f));
                    __stcg(A.B.rot + id, pack(q));
                }
            }
            if (s == A.substeps) {
                __stcg(A.B.vel + id, pack(v, 0.0f));
                __stcg(A.B.ang + id, pack(w, 0.0f));
                continue;
            }
            if (A.integrate && s > 0 && moves) {  // integrateVelocity
                const float4 ex = A.B.extra[id];
                v += (A.gravity * ex.y + f3(A.B.force[id]) * solverInvMass(m)) * A.h;
                w += invInertiaMulAt(m, f3(A.B.torque[id]), q) * A.h;
                v *= 1.0f / (1.0f + ex.z * A.h);
                w *= 1.0f / (1.0f + ex.w * A.h);
            }
            stRelaxed16(rec, v, 0u);
            stRelaxed16(rec + 1, w, 0u);
            __stcg(rec + 2, pack(inertiaFrameAt(m, q)));
            if (s == 0) __stcg(rec + 3, pack(m.invI, solverInvMass(m)));
        }
    };
    for (int s = 0; s < A.substeps; ++s) {
        bodies(s);
        if (!gridSync(&st->bar, &st->timeout, st->spinLimit)) return;
        for (uint32_t slot = s0 + lane; slot < s1; slot += 32u) {
            const uint32_t k = F.rows[slot];
            vx_contact& c = A.contacts[A.order[k]];
            const SolverBody a = flowBody(A, F, c.a), b = flowBody(A, F, c.b);
            RowContact rc;
            loadRow(c, rc);
            RowPrep P;
            prepRow(a, b, rc, A.h, Cone, P);
            const bool solved = solvedContact(a.m.flags, b.m.flags);
            const uint32_t bits = storeRowPlanes<Cone>(R, slot, rc, P, solved, s);
            R.aux[slot].w = __uint_as_float(F.colour[slot]);
            R.side[2 * (size_t)slot] = pack(P.ra, __int_as_float(flowWord(A, c.a, a.m.flags, false)));
            R.side[2 * (size_t)slot + 1] = pack(P.rb, __int_as_float(flowWord(A, c.b, b.m.flags, false)));
            float4 imp = make_float4(rc.nImp, rc.t1Imp, rc.t2Imp, 0.0f);
            if (s > 0) imp = R.imp[2 * (size_t)slot];
            imp.w = __uint_as_float(bits | (isRotationLocked(a.m.flags) ? 0u : kRowTurns) | linkBits(k, 0));
            R.imp[2 * (size_t)slot] = imp;
            imp.w = __uint_as_float(bits | (isRotationLocked(b.m.flags) ? 0u : kRowTurns) | linkBits(k, 1));
            R.imp[2 * (size_t)slot + 1] = imp;
            if (setsPoint(A, s, solved, rc)) c.point = vx_vec3{P.point.x, P.point.y, P.point.z};
        }
        __syncwarp();
        const uint32_t warmUnits = A.warmStart && s == 0 ? 1u : 0u;
        runFlow<kRowSweep, Cone>(A, F, R, s0, s1, warmUnits + (uint32_t)A.sweeps, warmUnits, st);
        if (!gridSync(&st->bar, &st->timeout, st->spinLimit)) return;
    }
    bodies(A.substeps);
    for (uint32_t slot = s0 + lane; slot < s1; slot += 32u)
        storeRowImpulses(R, slot, A.contacts[A.order[F.rows[slot]]]);
}

}  // namespace vxb
