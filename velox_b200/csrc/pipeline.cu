// The per-step contact pipeline on the device.
//
// Step structure (src/world.cpp:3830-4521 with the CUDA backend's
// advanceSubsteps, src/backend_cuda.cu:691-761):
//   prepare      orientation normalisation, first-substep gravity, pre-solve poses
//   broad phase  swept AABBs, cell keys (world id in the high bits), radix sort,
//                cell hash table, 27-cell pair emission + per-world plane pairs
//   narrow phase collidePair per candidate pair, contacts sorted by (a, b, point)
//   warm start   impulse matching against the previous step's contacts
//   islands      union-find over dynamic-dynamic contacts; contacts grouped by
//                island keep their global order, so island-local greedy
//                colouring equals the reference's global greedy colouring and
//                island-local colour order equals its global colour order
//   solve        one launch runs every island's whole substep loop
//                (integration, warm start, 2*velocityIterations coloured
//                sweeps, transform integration); tiny islands share warps,
//                larger ones run one block each (solve_rows.cuh), the largest
//                the whole grid
//   rewind       conservative advancement for deep end-of-step overlaps
//   correction   split-impulse position correction, coloured per island
#include <algorithm>
#include <cstddef>
#include <cstring>

#include "context.cuh"
#include "pair_warp.cuh"
#include "solve_flow.cuh"
#include "solve_rows.cuh"

namespace vxb {

static_assert(sizeof(vx_contact) == 128 && offsetof(vx_contact, spinningImpulse) == 116,
              "contact record: 120 bytes of fields, 8 of padding");

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------

int fail(Context& c, int status, const std::string& message) {
    c.lastError = message;
    return status;
}

int cudaStatus(Context& c, cudaError_t e, const char* what) {
    if (e == cudaSuccess) return VXB_OK;
    std::string msg = std::string("velox_b200 CUDA failure: ") + cudaGetErrorString(e) + " (" + what + ")";
    if (e == cudaErrorMemoryAllocation) return fail(c, VXB_ERR_OOM, msg);
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return fail(c, VXB_ERR_NO_DEVICE, msg);
    if (e == cudaErrorLaunchFailure || e == cudaErrorLaunchTimeout || e == cudaErrorUnknown ||
        e == cudaErrorIllegalAddress || e == cudaErrorDevicesUnavailable)
        return fail(c, VXB_ERR_DEVICE_LOST, msg);
    return fail(c, VXB_ERR_INVALID, msg);
}

// cudaMalloc for `b`. When memory is short, what the tape holds without using
// it goes back first: everything of an ended tape, the scratch of a live one.
int allocate(Context& c, const DevBuf& b, void** out, size_t bytes) {
    cudaError_t e = cudaMalloc(out, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        if (!c.tape.active) {
            tapeEnd(c);
        } else if (&b != &c.tape.scratch && c.tape.scratch.ptr) {
            cudaFree(c.tape.scratch.ptr);
            c.tape.scratch = DevBuf{};
        }
        e = cudaMalloc(out, bytes);
    }
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess ? VXB_OK : cudaStatus(c, e, "cudaMalloc");
}

int ensure(Context& c, DevBuf& b, size_t bytes) {
    if (bytes <= b.bytes && b.ptr) return VXB_OK;
    if (b.ptr) cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
    size_t want = bytes + bytes / 2 + 256;
    if (const int rc = allocate(c, b, &b.ptr, want)) {
        b.ptr = nullptr;
        return rc;
    }
    b.bytes = want;
    return VXB_OK;
}

template <class T> T* P(DevBuf& b) { return reinterpret_cast<T*>(b.ptr); }

static cudaEvent_t takeEvent(Context& c) {
    if (c.timer.pool.empty()) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        return e;
    }
    cudaEvent_t e = c.timer.pool.back();
    c.timer.pool.pop_back();
    return e;
}

void stageBegin(Context& c, int stage) {
    if (!c.timing) return;
    cudaEvent_t e = takeEvent(c);
    cudaEventRecord(e, c.stream);
    c.timer.open[stage].push_back(e);
}

void stageEnd(Context& c, int stage) {
    if (!c.timing || c.timer.open[stage].empty()) return;
    cudaEvent_t e = takeEvent(c);
    cudaEventRecord(e, c.stream);
    c.timer.done[stage].push_back({c.timer.open[stage].back(), e});
    c.timer.open[stage].pop_back();
}

// Folds completed event pairs into the per-stage totals.
int stageResolve(Context& c) {
    cudaError_t e = cudaStreamSynchronize(c.stream);
    if (e != cudaSuccess) return cudaStatus(c, e, "stage timing");
    for (int s = 0; s < kStageCount; ++s) {
        for (auto& pr : c.timer.done[s]) {
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, pr.first, pr.second);
            c.timer.ms[s] += ms;
            c.timer.calls[s] += 1;
            c.timer.pool.push_back(pr.first);
            c.timer.pool.push_back(pr.second);
        }
        c.timer.done[s].clear();
    }
    return VXB_OK;
}

#define VXB_TRY(expr)                  \
    do {                               \
        int s_ = (expr);               \
        if (s_ != VXB_OK) return s_;   \
    } while (0)

#define VXB_CUDA(c, expr)                                             \
    do {                                                              \
        cudaError_t e_ = (expr);                                      \
        if (e_ != cudaSuccess) return cudaStatus((c), e_, #expr);     \
    } while (0)

static inline uint32_t blocksFor(uint64_t items, int threads, uint32_t cap = 65535u * 16u) {
    uint64_t b = (items + threads - 1) / threads;
    if (b == 0) b = 1;
    return (uint32_t)std::min<uint64_t>(b, cap);
}

static inline int bitsFor(uint64_t maxValue) { return keyBits(maxValue); }

#define LAUNCH(c, kernel, grid, block, ...)                                  \
    do {                                                                     \
        kernel<<<(grid), (block), 0, (c).stream>>>(__VA_ARGS__);            \
        ++(c).launches;                                                      \
    } while (0)


// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------

VXD uint32_t orderedBits(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
VXD float fromOrdered(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
VXD uint64_t mix64(uint64_t k) {
    k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull; k ^= k >> 33;
    return k;
}
VXD unsigned laneMaskLt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
// Warp-aggregated slot reservation for the currently active lanes.
VXD uint32_t aggregatedSlot(uint32_t* counter) {
    const unsigned active = __activemask();
    const int leader = __ffs(active) - 1;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(active));
    base = __shfl_sync(active, base, leader);
    return base + __popc(active & laneMaskLt());
}

// integrateKernel semantics (src/backend_cuda.cu:80-89) for body i.
VXD void integrateVelocity(const BodyArrays& B, uint32_t i, const V3& g, float dt) {
    const Mass m = loadMass(B, i);
    if (!isDynamic(m.flags) || isLocked(m.flags) || isAsleep(m.flags)) return;
    const Q4 q = q4(B.rot[i]);
    V3 v = f3(B.vel[i]);
    V3 w = f3(B.ang[i]);
    const V3 F = f3(B.force[i]);
    const V3 T = f3(B.torque[i]);
    const float4 ex = B.extra[i];
    v += (g * ex.y + F * solverInvMass(m)) * dt;
    w += invInertiaMulAt(m, T, q) * dt;
    v *= 1.0f / (1.0f + ex.z * dt);
    w *= 1.0f / (1.0f + ex.w * dt);
    B.vel[i] = pack(v, 0.0f);
    B.ang[i] = pack(w, 0.0f);
}

// integrateTransformsKernel semantics (src/backend_cuda.cu:91-97).
VXD void integrateTransform(const BodyArrays& B, uint32_t i, float dt) {
    const Mass m = loadMass(B, i);
    if (isStaticBody(m.flags) || isLocked(m.flags) || isAsleep(m.flags)) return;
    V3 p = f3(B.pos[i]);
    Q4 q = q4(B.rot[i]);
    const V3 v = f3(B.vel[i]);
    V3 w = f3(B.ang[i]);
    advanceTransform(m, p, q, v, w, dt);
    B.pos[i] = pack(p, 0.0f);
    B.rot[i] = pack(q);
    B.ang[i] = pack(w, 0.0f);
}

// ---------------------------------------------------------------------------
// body packing
// ---------------------------------------------------------------------------

__global__ void packBodiesKernel(const vx_body* __restrict__ in, uint32_t n, BodyArrays B) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const vx_body& b = in[i];
        B.pos[i] = make_float4(b.position.x, b.position.y, b.position.z, 0.0f);
        B.rot[i] = make_float4(b.orientation.x, b.orientation.y, b.orientation.z, b.orientation.w);
        B.vel[i] = make_float4(b.velocity.x, b.velocity.y, b.velocity.z, 0.0f);
        B.ang[i] = make_float4(b.angularVelocity.x, b.angularVelocity.y, b.angularVelocity.z, 0.0f);
        B.inertia[i] = make_float4(b.invInertia.x, b.invInertia.y, b.invInertia.z, b.invMass);
        B.iq[i] = make_float4(b.inertiaOrientation.x, b.inertiaOrientation.y, b.inertiaOrientation.z,
                              b.inertiaOrientation.w);
        B.dims[i] = make_float4(b.halfExtents.x, b.halfExtents.y, b.halfExtents.z, b.radius);
        B.extra[i] = make_float4(b.capsuleHalfHeight, b.gravityScale, b.linearDamping, b.angularDamping);
        B.mat[i] = make_float4(b.friction, b.restitution, b.rollingFriction, b.spinningFriction);
        B.fscale[i] = make_float4(b.frictionScale.x, b.frictionScale.y, b.frictionScale.z,
                                  b.ccdTuning.speculativeDistance);
        B.ccd[i] = make_float4(b.ccdTuning.collisionMargin, b.ccdTuning.minVelocityForCCD, 0.0f, 0.0f);
        B.plane[i] = make_float4(b.planeNormal.x, b.planeNormal.y, b.planeNormal.z, b.planeOffset);
        // the hull word: a mesh keeps its mesh index there, a compound its child range
        B.hull[i] = b.shape == VX_SHAPE_MESH       ? make_uint4(b.meshIndex, 0u, 0u, 0u)
                    : b.shape == VX_SHAPE_COMPOUND ? make_uint4(b.compoundFirst, b.compoundCount, 0u, 0u)
                                                   : make_uint4(b.hullFirst, b.hullCount, b.hullFaceFirst, b.hullFaceCount);
        const uint32_t flags = (uint32_t)(b.shape & 15u) | ((uint32_t)(b.motionType & 3u) << kMotionShift) |
                               ((uint32_t)(b.ccdTuning.quality & 3u) << kQualityShift) |
                               (b.ccdTuning.enableContinuous ? kContinuousBit : 0u) |
                               (b.sensor ? kSensorBit : 0u) | (b.fixedRotation ? kFixedRotationBit : 0u) |
                               (b.asleep == 1 ? kAsleepBit : 0u) |
                               ((uint32_t)(b.frictionCombine & 7u) << kFrictionCombineShift) |
                               ((uint32_t)(b.restitutionCombine & 7u) << kRestitutionCombineShift) |
                               ((uint32_t)(b.geometryQuality & 3u) << kGeomQualityShift);
        B.filt[i] = make_uint4(flags, b.categoryBits, b.maskBits, (uint32_t)b.groupIndex);
        B.force[i] = make_float4(b.force.x, b.force.y, b.force.z, 0.0f);
        B.torque[i] = make_float4(b.torque.x, b.torque.y, b.torque.z, 0.0f);
    }
}

__global__ void unpackBodiesKernel(vx_body* __restrict__ out, uint32_t n, BodyArrays B) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        vx_body& b = out[i];
        float4 t = B.pos[i]; b.position = vx_vec3{t.x, t.y, t.z};
        t = B.rot[i]; b.orientation = vx_quat{t.x, t.y, t.z, t.w};
        t = B.vel[i]; b.velocity = vx_vec3{t.x, t.y, t.z};
        t = B.ang[i]; b.angularVelocity = vx_vec3{t.x, t.y, t.z};
        t = B.force[i]; b.force = vx_vec3{t.x, t.y, t.z};
        t = B.torque[i]; b.torque = vx_vec3{t.x, t.y, t.z};
    }
}

__global__ void posesKernel(float* __restrict__ out, uint32_t n, BodyArrays B) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = B.pos[i], q = B.rot[i];
        float* o = out + 7 * (size_t)i;
        o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = q.x; o[4] = q.y; o[5] = q.z; o[6] = q.w;
    }
}

__global__ void forcesKernel(const float* __restrict__ in, uint32_t n, BodyArrays B) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* f = in + 6 * (size_t)i;
        B.force[i] = make_float4(f[0], f[1], f[2], 0.0f);
        B.torque[i] = make_float4(f[3], f[4], f[5], 0.0f);
    }
}

// ---------------------------------------------------------------------------
// prepare: World::stepImpl orientation normalisation (world.cpp:3930),
// first-substep gravity (world.cpp:4014) and the pre-solve poses (:4186-4188)
// ---------------------------------------------------------------------------

__global__ void prepareKernel(BodyArrays B, uint32_t n, V3 g, float h, float4* prevPos, float4* prevRot,
                              int normalizeOrientation) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (normalizeOrientation) B.rot[i] = pack(qnormalize(q4(B.rot[i])));
        integrateVelocity(B, i, g, h);
        if (prevPos) {
            prevPos[i] = B.pos[i];
            prevRot[i] = B.rot[i];
        }
    }
}

__global__ void integrateKernel(BodyArrays B, uint32_t n, V3 g, float h) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        integrateVelocity(B, i, g, h);
}

__global__ void transformsKernel(BodyArrays B, uint32_t n, float h) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        integrateTransform(B, i, h);
}

// ---------------------------------------------------------------------------
// broad phase
// ---------------------------------------------------------------------------

constexpr int kCellBits = 10;  // per axis; coordinates wrap modulo 1024 (exactness kept by the AABB test)
constexpr uint32_t kCellMask = (1u << kCellBits) - 1u;
constexpr uint64_t kEmptySlot = ~0ull;

// Swept AABBs (bodyAabb, narrowphase.h:369-398); planes unbounded, meshes
// their root bounds (src/backend_cuda.cu:100-129). Neither enters the cell
// size or the cell grid's extent.
__global__ void aabbKernel(BodyArrays B, uint32_t n, float dt, const vx_mesh* meshes, float4* lo, float4* hi,
                           Counters* C) {
    float ext = 0.0f;
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t flags = B.filt[i].x;
        if (shapeOf(flags) == kPlane) {
            lo[i] = make_float4(-1e30f, -1e30f, -1e30f, 0.0f);
            hi[i] = make_float4(1e30f, 1e30f, 1e30f, 0.0f);
            continue;
        }
        if (shapeOf(flags) == kMesh) {
            const vx_mesh& m = meshes[B.hull[i].x];
            lo[i] = make_float4(m.aabbMin.x, m.aabbMin.y, m.aabbMin.z, 0.0f);
            hi[i] = make_float4(m.aabbMax.x, m.aabbMax.y, m.aabbMax.z, 0.0f);
            continue;
        }
        const V3 p = f3(B.pos[i]);
        const float4 d = B.dims[i];
        const float reach = aabbReach(flags, V3{d.x, d.y, d.z}, d.w, B.extra[i].x, B.ccd[i].x,
                                      f3(B.vel[i]), f3(B.ang[i]), dt);
        const V3 L = p - V3{reach, reach, reach};
        const V3 H = p + V3{reach, reach, reach};
        lo[i] = pack(L, 0.0f);
        hi[i] = pack(H, 0.0f);
        const float e = fmaxf(H.x - L.x, fmaxf(H.y - L.y, H.z - L.z));
        if (e < 1e6f) ext = fmaxf(ext, e);
        const float c[3] = {(L.x + H.x) * 0.5f, (L.y + H.y) * 0.5f, (L.z + H.z) * 0.5f};
        for (int a = 0; a < 3; ++a) { mn[a] = fminf(mn[a], c[a]); mx[a] = fmaxf(mx[a], c[a]); }
    }
    for (int off = 16; off > 0; off >>= 1) {
        ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, off));
        for (int a = 0; a < 3; ++a) {
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], off));
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], off));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        if (ext > 0.0f) atomicMax(&C->extentBits, __float_as_uint(ext));
        for (int a = 0; a < 3; ++a)
            if (mn[a] <= mx[a]) {
                atomicMin(&C->cellMinBits[a], orderedBits(mn[a]));
                atomicMax(&C->cellMaxBits[a], orderedBits(mx[a]));
            }
    }
}

VXD float cellSizeOf(const Counters* C) {
    float s = __uint_as_float(C->extentBits);
    return s > 0.0f ? s : 1.0f;
}
VXD int cellCoord(float centre, float inv, float minCentre) {
    float f = floorf(centre * inv) - floorf(minCentre * inv);
    f = fminf(fmaxf(f, -1.0e9f), 1.0e9f);
    return (int)f;
}

__global__ void keyKernel(BodyArrays B, uint32_t n, const uint32_t* worldOf, const float4* lo, const float4* hi,
                          const Counters* C, uint64_t* keys, uint32_t* vals, uint64_t planeKey) {
    const float cs = cellSizeOf(C);
    const float inv = 1.0f / cs;
    const float m0 = fromOrdered(C->cellMinBits[0]), m1 = fromOrdered(C->cellMinBits[1]),
                m2 = fromOrdered(C->cellMinBits[2]);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        vals[i] = i;
        const uint32_t shape = shapeOf(B.filt[i].x);
        if (shape == kPlane || shape == kMesh) { keys[i] = planeKey; continue; }
        const float4 L = lo[i], H = hi[i];
        const int cx = cellCoord((L.x + H.x) * 0.5f, inv, m0);
        const int cy = cellCoord((L.y + H.y) * 0.5f, inv, m1);
        const int cz = cellCoord((L.z + H.z) * 0.5f, inv, m2);
        const uint64_t w = worldOf ? worldOf[i] : 0u;
        keys[i] = (w << (3 * kCellBits)) | ((uint64_t)((uint32_t)cz & kCellMask) << (2 * kCellBits)) |
                  ((uint64_t)((uint32_t)cy & kCellMask) << kCellBits) | (uint64_t)((uint32_t)cx & kCellMask);
    }
}

__global__ void cellTableKernel(const uint64_t* keys, uint32_t n, uint64_t planeKey, uint64_t* hk, uint32_t* hv,
                                uint32_t mask) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const uint64_t key = keys[s];
        if (key == planeKey) continue;
        if (s > 0 && keys[s - 1] == key) continue;
        uint32_t slot = (uint32_t)mix64(key) & mask;
        for (uint32_t probe = 0; probe <= mask; ++probe) {
            const unsigned long long prev = atomicCAS((unsigned long long*)&hk[slot], (unsigned long long)kEmptySlot,
                                                      (unsigned long long)key);
            if (prev == kEmptySlot) { hv[slot] = s; break; }
            slot = (slot + 1) & mask;
        }
    }
}

VXD uint32_t cellLookup(const uint64_t* hk, const uint32_t* hv, uint32_t mask, uint64_t key) {
    uint32_t slot = (uint32_t)mix64(key) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const uint64_t k = hk[slot];
        if (k == key) return hv[slot];
        if (k == kEmptySlot) return 0xffffffffu;
        slot = (slot + 1) & mask;
    }
    return 0xffffffffu;
}

VXD void emitPair(uint64_t pair, uint64_t* pairs, uint32_t cap, uint32_t* counter, Counters* C) {
    const uint32_t slot = aggregatedSlot(counter);
    if (slot < cap) pairs[slot] = pair;
    else atomicOr(&C->overflow, 1u);
}

// Candidate pairs (src/backend_cuda.cu:174-250): the 27 neighbouring cells of
// each body's cell (same world), pairs i<j discovered from i's side, plus the
// planes and meshes of the body's world (the list `planeList`; a mesh pair
// also needs overlapping AABBs). Plane pairs of simple convex bodies go to
// `planePairs`; mesh pairs and a compound's plane pairs join the general
// pairs, whose narrow phase handles every shape.
__global__ void pairKernel(BodyArrays B, uint32_t n, const uint64_t* keys, const uint32_t* vals, const float4* lo,
                           const float4* hi, const uint64_t* hk, const uint32_t* hv, uint32_t mask, uint64_t planeKey,
                           const uint32_t* worldOf, const uint32_t* planeStart, const uint32_t* planeList,
                           uint64_t* pairs, uint32_t cap, uint64_t* planePairs, uint32_t planeCap, Counters* C) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const uint64_t key = keys[s];
        if (key == planeKey) continue;
        const uint32_t i = vals[s];
        const uint4 fi = B.filt[i];
        const V3 Li = f3(lo[i]), Hi = f3(hi[i]);
        const int cx = (int)(key & kCellMask), cy = (int)((key >> kCellBits) & kCellMask),
                  cz = (int)((key >> (2 * kCellBits)) & kCellMask);
        const uint64_t wbits = key >> (3 * kCellBits);
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    const uint64_t nk = (wbits << (3 * kCellBits)) |
                                        ((uint64_t)((uint32_t)(cz + dz) & kCellMask) << (2 * kCellBits)) |
                                        ((uint64_t)((uint32_t)(cy + dy) & kCellMask) << kCellBits) |
                                        (uint64_t)((uint32_t)(cx + dx) & kCellMask);
                    const uint32_t start = cellLookup(hk, hv, mask, nk);
                    if (start == 0xffffffffu) continue;
                    for (uint32_t t = start; t < n && keys[t] == nk; ++t) {
                        const uint32_t j = vals[t];
                        if (j <= i) continue;
                        if (!aabbOverlap(Li, Hi, f3(lo[j]), f3(hi[j]))) continue;
                        const uint4 fj = B.filt[j];
                        if (inert(fi.x) && inert(fj.x)) continue;
                        if (!canCollide(fi.y, fi.z, (int32_t)fi.w, fj.y, fj.z, (int32_t)fj.w)) continue;
                        emitPair(((uint64_t)i << 32) | j, pairs, cap, &C->pairs, C);
                    }
                }
        const uint32_t w = worldOf ? worldOf[i] : 0u;
        const bool compound = shapeOf(fi.x) == kCompound;
        for (uint32_t k = planeStart[w]; k < planeStart[w + 1]; ++k) {
            const uint32_t p = planeList[k];
            const uint4 fp = B.filt[p];
            const bool mesh = shapeOf(fp.x) == kMesh;
            if (mesh && !aabbOverlap(Li, Hi, f3(lo[p]), f3(hi[p]))) continue;
            if (inert(fi.x) && inert(fp.x)) continue;
            const uint32_t a = i < p ? i : p, b = i < p ? p : i;
            const uint4 fa = a == i ? fi : fp, fb = a == i ? fp : fi;
            if (!canCollide(fa.y, fa.z, (int32_t)fa.w, fb.y, fb.z, (int32_t)fb.w)) continue;
            if (mesh || compound) emitPair(((uint64_t)a << 32) | b, pairs, cap, &C->pairs, C);
            else emitPair(((uint64_t)a << 32) | b, planePairs, planeCap, &C->planePairs, C);
        }
    }
}

// ---------------------------------------------------------------------------
// narrow phase
// ---------------------------------------------------------------------------

VXD bool pointLess(const vx_contact& x, const vx_contact& y) {
    if (x.point.x != y.point.x) return x.point.x < y.point.x;
    if (x.point.y != y.point.y) return x.point.y < y.point.y;
    return x.point.z < y.point.z;
}

// One thread per candidate pair: collidePair into a local buffer, order the
// pair's contacts by point (the host sort of src/backend_cuda.cu:587-595
// within one (a, b) key), append them and a record keyed for the global sort.
// mode 0: key = (a << bodyBits) | b; mode 1: key = pair index, emission order kept.
// Which pair classes one instantiation handles: plane pairs compile to a
// light kernel (high occupancy), convex pairs to the GJK kernel. Convex pairs
// whose cores overlap (or that are not Normal quality) and mesh and compound
// pairs are listed in `hard` for collideHardKernel: a thread's EPA runs up to
// 1 ms, and one such lane held its warp and the stage's tail for that long.
// Listed pairs: the contacts of those pairs from the query results that
// collideHardKernel left (face clipping fills a warp's lanes again). Thread
// pairs: the listed ones that a warp would waste (threadPair), one thread each
// from query to contacts (launched only when such bodies are loaded). Narrow phase
// of one step, a warp / a thread a pair: heap of 10,000 Robust bodies 11.5 / 7.7
// ms, Paranoid 22.6 / 10.9; heap of 30,000 compounds 14.4 / 4.0.
enum PairClass : int { kAnyPairs = 0, kPlanePairs = 1, kConvexPairs = 2, kListedPairs = 3, kThreadPairs = 4 };

// Listed pairs whose queries use a warp badly: Robust and Paranoid bodies (the
// general routine runs on one lane) and compounds (many child pairs, most of them
// apart, which all lanes follow alike); mesh pairs share the triangles among the
// lanes all the same. Where the list is longer than a few rounds of the GPU's
// resident warps they go to threads; of a shorter one a warp each is faster than
// 32 lanes that diverge (rewind stage with some 1,000 Paranoid pairs probed 14.2
// / 18.7 ms, narrow phase of 2,800 21 / 26 ms).
constexpr uint32_t kLoneLaneMax = 4096;
VXD bool threadPair(uint32_t listed, uint32_t flagsA, uint32_t flagsB) {
    const uint32_t sa = shapeOf(flagsA), sb = shapeOf(flagsB);
    return listed > kLoneLaneMax && sa != kMesh && sb != kMesh &&
           (((flagsA | flagsB) >> kGeomQualityShift & 3u) != 0u || sa == kCompound || sb == kCompound);
}

// Result of one listed pair's query.
struct HardResult {
    float distance;
    V3 normal, pointA, pointB;
};
// Mark on a listed pair whose query the thread kernel has answered: two boxes or
// hulls close to each other, whose face clipping waits for kListedPairs, where it
// runs beside that of the overlapping pairs instead of before it, in full warps
// (narrow phase of one step: heap of 3,000 bodies 0.57 -> 0.41 ms, of 40,000 1.40
// -> 0.98, 64 box pyramids 1.66 -> 1.14).
constexpr uint32_t kAnswered = 0x80000000u;
VXD bool clipsFaces(float distance, uint32_t flagsA, uint32_t flagsB) {
    const uint32_t sa = shapeOf(flagsA), sb = shapeOf(flagsB);
    return distance < 0.05f && (sa == kBox || sa == kHull) && (sb == kBox || sb == kHull);
}

// Contacts of one pair in the order of the reference's host sort within one
// (a, b) key (mode 0; mode 1 keeps the emission order).
VXD void orderContacts(vx_contact* buf, int count, int mode) {
    if (mode != 0) return;
    for (int x = 1; x < count; ++x) {
        vx_contact key = buf[x];
        int y = x - 1;
        while (y >= 0 && pointLess(key, buf[y])) { buf[y + 1] = buf[y]; --y; }
        buf[y + 1] = key;
    }
}

// A pair's contacts and record at reserved positions.
VXD void storeContacts(const vx_contact* buf, int count, uint32_t off, uint32_t rec, uint32_t p, int mode, int bodyBits,
                       vx_contact* tmp, uint32_t contactCap, uint64_t* recKeys, uint32_t* recVals, uint2* recInfo,
                       uint32_t recCap, Counters* C) {
    if (off + (uint32_t)count > contactCap || rec >= recCap) {
        atomicOr(&C->overflow, 2u);
        return;
    }
    for (int x = 0; x < count; ++x) {
        tmp[off + x] = buf[x];
        // the record's 8 tail bytes are padding: zero them so contact
        // images (snapshots, read-back) are deterministic bytes
        *reinterpret_cast<uint2*>(reinterpret_cast<char*>(tmp + off + x) + 120) = make_uint2(0u, 0u);
    }
    recKeys[rec] = mode == 0 ? (((uint64_t)buf[0].a << bodyBits) | buf[0].b) : (uint64_t)p;
    recVals[rec] = rec;
    recInfo[rec] = make_uint2(off, (uint32_t)count);
}

// `order` (optional): the pairs in the order to process them (convex pairs
// grouped by shape combination so that a warp runs one code path).
template <int Class>
__global__ void __launch_bounds__(128) collideKernel(BodyArrays B, Soup soup, const uint64_t* pairs,
                                                     const uint32_t* order, uint32_t npairs, float dt, int mode,
                                                     int bodyBits, vx_contact* tmp, uint32_t contactCap,
                                                     uint64_t* recKeys, uint32_t* recVals, uint2* recInfo,
                                                     uint32_t recCap, uint32_t* hard, HardResult* results,
                                                     Counters* C) {
    const uint32_t stride = gridDim.x * blockDim.x;
    if (Class == kListedPairs || Class == kThreadPairs) npairs = C->hardPairs;
    const uint32_t rounded = (npairs + 31u) & ~31u;
    for (uint32_t base = blockIdx.x * blockDim.x; base < rounded; base += stride) {
        const uint32_t slot = base + threadIdx.x;
        uint32_t p = slot < npairs && order ? order[slot] : slot;
        bool answered = false;
        if (Class == kListedPairs || Class == kThreadPairs) {
            answered = p & kAnswered;
            p &= ~kAnswered;
        }
        HardResult answer;
        vx_contact buf[kMaxContactsPerPair];
        int count = 0;
        bool later = false;
        if (slot < npairs) {
            const uint64_t pr = pairs[p];
            const uint32_t i = (uint32_t)(pr >> 32), j = (uint32_t)pr;
            const BodyView a = loadView(B, i);
            const BodyView b = loadView(B, j);
            if (Class == kAnyPairs) {
                count = collidePair(a, b, i, j, soup, dt, buf, kMaxContactsPerPair);
            } else if (Class == kPlanePairs) {
                if (shapeOf(b.flags) == kPlane) planeConvex(a, b, i, j, soup, dt, buf, kMaxContactsPerPair, count);
                else planeConvex(b, a, j, i, soup, dt, buf, kMaxContactsPerPair, count);
            } else if (Class == kThreadPairs) {
                if (!answered && threadPair(npairs, a.flags, b.flags)) count = collidePair(a, b, i, j, soup, dt, buf, kMaxContactsPerPair);
            } else if (isComplexShape(shapeOf(a.flags)) || isComplexShape(shapeOf(b.flags)) ||
                       (Class == kListedPairs && threadPair(npairs, a.flags, b.flags))) {
                later = Class == kConvexPairs;  // (as a listed pair: done by its warp or thread)
            } else if (Class == kListedPairs) {
                const HardResult h = results[slot];
                GjkResult r;
                r.distance = h.distance;
                r.normal = h.normal; r.pointA = h.pointA; r.pointB = h.pointB;
                r.overlapping = true;
                convexContacts(a, b, i, j, makeConvex(a, soup), makeConvex(b, soup), r, dt, buf, kMaxContactsPerPair,
                               count);
            } else {
                const Convex ca = makeConvex(a, soup), cb = makeConvex(b, soup);
                GjkResult r;
                Simplex s;
                later = gjkDistanceFast(ca, cb, r, s) != kGjkSeparated;
                if (!later && clipsFaces(r.distance, a.flags, b.flags)) {
                    later = answered = true;
                    answer = HardResult{r.distance, r.normal, r.pointA, r.pointB};
                }
                if (!later) convexContacts(a, b, i, j, ca, cb, r, dt, buf, kMaxContactsPerPair, count);
            }
            orderContacts(buf, count, mode);
        }
        if (Class == kConvexPairs) {
            const unsigned m = __ballot_sync(0xffffffffu, later);
            uint32_t at = 0;
            if (m && (threadIdx.x & 31) == 0) at = atomicAdd(&C->hardPairs, (uint32_t)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            at += __popc(m & laneMaskLt());
            if (later) hard[at] = answered ? p | kAnswered : p;
            if (answered) results[at] = answer;
        }
        // Warp-wide exclusive scan of the counts, one atomic per warp.
        const int lane = threadIdx.x & 31;
        uint32_t incl = (uint32_t)count;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        const unsigned hasMask = __ballot_sync(0xffffffffu, count > 0);
        uint32_t cbase = 0, rbase = 0;
        if (lane == 0 && total) {
            cbase = atomicAdd(&C->contactsTmp, total);
            rbase = atomicAdd(&C->records, (uint32_t)__popc(hasMask));
        }
        cbase = __shfl_sync(0xffffffffu, cbase, 0);
        rbase = __shfl_sync(0xffffffffu, rbase, 0);
        if (count > 0) {
            const uint32_t off = cbase + incl - (uint32_t)count;
            const uint32_t rec = rbase + __popc(hasMask & laneMaskLt());
            storeContacts(buf, count, off, rec, p, mode, bodyBits, tmp, contactCap, recKeys, recVals, recInfo, recCap,
                          C);
        }
    }
}

// The listed pairs' queries, a warp each; the contacts of convex pairs follow
// in collideKernel<kListedPairs>, mesh and compound pairs are finished here
// (pair_warp.cuh). The list's length stays on the device; the grid is what
// fits the GPU at once. Narrow phase of one step: 3.7 -> 0.5 ms with 2,500
// bodies on a mesh, 1.9 -> 0.5 ms in the falling scene of 100,000 bodies (a few
// deep pairs).
constexpr int kQueryThreads = 128;  // warps that share a block's shared memory for their queries
constexpr size_t kQuerySmem = kQueryThreads / 32 * sizeof(WarpQuery);

__global__ void __launch_bounds__(kQueryThreads) collideHardKernel(BodyArrays B, Soup soup, const uint64_t* pairs,
                                                                   const uint32_t* hard, float dt, int mode,
                                                                   int bodyBits, vx_contact* tmp, uint32_t contactCap,
                                                                   uint64_t* recKeys, uint32_t* recVals,
                                                                   uint2* recInfo, uint32_t recCap,
                                                                   HardResult* results, Counters* C) {
    const uint32_t count = C->hardPairs, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count; k += warps) {
        const uint32_t p = hard[k];
        if (p & kAnswered) continue;
        const uint64_t pr = pairs[p];
        const uint32_t i = (uint32_t)(pr >> 32), j = (uint32_t)pr;
        const BodyView a = loadView(B, i), b = loadView(B, j);
        if (threadPair(count, a.flags, b.flags)) continue;  // collideKernel<kThreadPairs>
        if (!isComplexShape(shapeOf(a.flags)) && !isComplexShape(shapeOf(b.flags))) {
            const GjkResult r = gjkDistanceWarp(makeConvex(a, soup), makeConvex(b, soup));
            if (warpLane() == 0u) results[k] = HardResult{r.distance, r.normal, r.pointA, r.pointB};
            __syncwarp();
            continue;
        }
        vx_contact buf[kMaxContactsPerPair];
        const int n = collidePairWarp(a, b, i, j, soup, dt, buf, kMaxContactsPerPair);
        if (n > 0 && warpLane() == 0u) {
            orderContacts(buf, n, mode);
            const uint32_t off = atomicAdd(&C->contactsTmp, (uint32_t)n), rec = atomicAdd(&C->records, 1u);
            storeContacts(buf, n, off, rec, p, mode, bodyBits, tmp, contactCap, recKeys, recVals, recInfo, recCap, C);
        }
        __syncwarp();
    }
}

__global__ void gatherCountsKernel(const uint32_t* recVals, const uint2* recInfo, uint32_t nrec, uint32_t* counts) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nrec; k += gridDim.x * blockDim.x)
        counts[k] = recInfo[recVals[k]].y;
}

// Shape combination of each convex pair (the processing-order sort key).
__global__ void pairClassKernel(const BodyArrays B, const uint64_t* pairs, uint32_t npairs, uint64_t* keys,
                                uint32_t* vals) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npairs; p += gridDim.x * blockDim.x) {
        const uint64_t pr = pairs[p];
        const uint32_t sa = shapeOf(B.filt[(uint32_t)(pr >> 32)].x), sb = shapeOf(B.filt[(uint32_t)pr].x);
        keys[p] = (uint64_t)(sa * 16u + sb);
        vals[p] = p;
    }
}

// Copies each record's contacts to their sorted position.
__global__ void placeKernel(const uint32_t* recVals, const uint2* recInfo, const uint32_t* offsets, uint32_t nrec,
                            const vx_contact* tmp, vx_contact* out, uint64_t* contactKeys, uint64_t* pairKeys,
                            uint32_t* recOffset) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nrec; k += gridDim.x * blockDim.x) {
        const uint2 info = recInfo[recVals[k]];
        const uint32_t dst = offsets[k];
        const float4* src = reinterpret_cast<const float4*>(tmp + info.x);
        float4* d = reinterpret_cast<float4*>(out + dst);
        for (uint32_t x = 0; x < info.y * 8u; ++x) d[x] = src[x];
        const uint64_t key = ((uint64_t)tmp[info.x].a << 32) | tmp[info.x].b;
        if (contactKeys)
            for (uint32_t x = 0; x < info.y; ++x) contactKeys[dst + x] = key;
        if (pairKeys) pairKeys[k] = key;
        if (recOffset) recOffset[k] = dst;
    }
}

// Multi-block exclusive scan: per-block sums, a single-block scan of the sums,
// then per-block scans with the carried offsets.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;

__device__ uint32_t blockExclusiveScan(uint32_t v, uint32_t* warpSums, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) warpSums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? warpSums[lane] : 0u;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        warpSums[lane] = w;
    }
    __syncthreads();
    const uint32_t r = x - v + (warp > 0 ? warpSums[warp - 1] : 0u);
    if (total) *total = warpSums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return r;
}

__global__ void scanReduceKernel(const uint32_t* in, uint32_t n, uint32_t* blockSums) {
    __shared__ uint32_t ws[32];
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t s = 0;
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < n) s += in[base + k];
    uint32_t total;
    blockExclusiveScan(s, ws, &total);
    if (threadIdx.x == 0) blockSums[blockIdx.x] = total;
}

__global__ void scanSumsKernel(uint32_t* sums, uint32_t len) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t start = 0; start < len; start += blockDim.x) {
        const uint32_t i = start + threadIdx.x;
        const uint32_t v = i < len ? sums[i] : 0u;
        uint32_t total;
        const uint32_t ex = blockExclusiveScan(v, ws, &total);
        if (i < len) sums[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

__global__ void scanApplyKernel(const uint32_t* in, uint32_t n, const uint32_t* blockSums, uint32_t* out,
                                uint32_t* grandTotal) {
    __shared__ uint32_t ws[32];
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0u;
        s += v[k];
    }
    uint32_t total;
    uint32_t ex = blockExclusiveScan(s, ws, &total) + blockSums[blockIdx.x];
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = ex;
        ex += v[k];
    }
    if (grandTotal && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *grandTotal = ex;
}

int exclusiveScan(Context& c, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* grandTotal) {
    if (n == 0) return VXB_OK;
    const uint32_t blocks = (n + kScanTile - 1) / kScanTile;
    VXB_TRY(ensure(c, c.scanTmp, (size_t)blocks * 4 + 16));
    uint32_t* sums = P<uint32_t>(c.scanTmp);
    LAUNCH(c, scanReduceKernel, blocks, kScanThreads, in, n, sums);
    LAUNCH(c, scanSumsKernel, 1, 1024, sums, blocks);
    LAUNCH(c, scanApplyKernel, blocks, kScanThreads, in, n, sums, out, grandTotal);
    return VXB_OK;
}

// ---------------------------------------------------------------------------
// warm-start matching (src/world.cpp:4133-4184)
// ---------------------------------------------------------------------------

__global__ void matchKernel(vx_contact* cur, uint32_t m, const vx_contact* prev, const uint64_t* prevKeys,
                            uint32_t mPrev, Counters* C) {
    uint32_t warm = 0;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        vx_contact c = cur[k];
        const uint64_t key = ((uint64_t)c.a << 32) | c.b;
        uint32_t lo = 0, hi = mPrev;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (prevKeys[mid] < key) lo = mid + 1;
            else hi = mid;
        }
        bool copied = false;
        bool matched = false;
        if (c.featureKey != 0) {
            for (uint32_t it = lo; it < mPrev && prevKeys[it] == key; ++it) {
                const vx_contact& p = prev[it];
                if (p.featureKey == c.featureKey) {
                    c.normalImpulse = p.normalImpulse; c.tangentImpulse1 = p.tangentImpulse1;
                    c.tangentImpulse2 = p.tangentImpulse2; c.rollingImpulse1 = p.rollingImpulse1;
                    c.rollingImpulse2 = p.rollingImpulse2; c.spinningImpulse = p.spinningImpulse;
                    if (c.vn0 < -1.0f && p.vn0 < c.vn0) c.vn0 = p.vn0;
                    matched = copied = true;
                    break;
                }
            }
        }
        if (!matched) {
            if (c.vn0 < -1.0f)
                for (uint32_t it = lo; it < mPrev && prevKeys[it] == key; ++it)
                    if (prev[it].vn0 < c.vn0) c.vn0 = prev[it].vn0;
            float best = 2.5e-3f;
            for (uint32_t it = lo; it < mPrev && prevKeys[it] == key; ++it) {
                const vx_contact& p = prev[it];
                const V3 d{p.point.x - c.point.x, p.point.y - c.point.y, p.point.z - c.point.z};
                const float ds = lengthSq(d);
                if (ds < best) {
                    best = ds;
                    c.normalImpulse = p.normalImpulse; c.tangentImpulse1 = p.tangentImpulse1;
                    c.tangentImpulse2 = p.tangentImpulse2; c.rollingImpulse1 = p.rollingImpulse1;
                    c.rollingImpulse2 = p.rollingImpulse2; c.spinningImpulse = p.spinningImpulse;
                    copied = true;
                }
            }
        }
        if (copied) ++warm;
        cur[k] = c;
    }
    for (int off = 16; off > 0; off >>= 1) warm += __shfl_xor_sync(0xffffffffu, warm, off);
    if ((threadIdx.x & 31) == 0 && warm) atomicAdd(&C->warmStarted, warm);
}

// ---------------------------------------------------------------------------
// islands and colouring
// ---------------------------------------------------------------------------

__global__ void iotaKernel(uint32_t* a, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = i;
}

// Union-find root with path halving. Parent links are read with ld.global.cg
// (L2, not the SM's L1): other SMs relink roots concurrently and a stale L1
// line would otherwise keep a thread spinning on an outdated root.
VXD uint32_t ufFind(uint32_t* parent, uint32_t x) {
    uint32_t p = __ldcg(parent + x);
    while (p != x) {
        const uint32_t gp = __ldcg(parent + p);
        if (gp != p) __stcg(parent + x, gp);  // path halving (benign race: any ancestor is valid)
        x = p;
        p = gp;
    }
    return x;
}

// Lock-free linking: a failed CAS means another thread linked that root, so
// the retry loop always makes global progress; the bound only turns a
// malfunction into a reported error instead of a hang.
constexpr uint32_t kUnionRetryLimit = 1u << 24;

__global__ void unionKernel(const vx_contact* cs, uint32_t m, const BodyArrays B, uint32_t* parent, Counters* C) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const uint32_t a = cs[k].a, b = cs[k].b;
        const uint32_t fa = B.filt[a].x, fb = B.filt[b].x;
        if (!solvedContact(fa, fb) || !isDynamic(fa) || !isDynamic(fb)) continue;
        uint32_t tries = 0;
        for (;; ++tries) {
            if (tries == kUnionRetryLimit) { atomicOr(&C->timeout, 1u); break; }
            uint32_t ra = ufFind(parent, a), rb = ufFind(parent, b);
            if (ra == rb) break;
            if (ra < rb) { const uint32_t t = ra; ra = rb; rb = t; }
            if (atomicCAS(&parent[ra], ra, rb) == ra) break;
        }
    }
}

// parent[i] = root of i. The walk writes nothing but the final root: a
// path-halving store racing with another thread's final store could leave a
// non-root ancestor behind, splitting one island into two keys.
__global__ void compressKernel(uint32_t* parent, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t x = i, p = __ldcg(parent + x);
        while (p != x) {
            x = p;
            p = __ldcg(parent + x);
        }
        __stcg(parent + i, x);
    }
}

// Island key of each contact: the root of its dynamic endpoint; contacts with
// no dynamic endpoint (or a sensor) go to the "null" island keyed n.
__global__ void islandKeyKernel(const vx_contact* cs, uint32_t m, const BodyArrays B, const uint32_t* root, uint32_t n,
                                uint64_t* keys, uint32_t* vals) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const uint32_t a = cs[k].a, b = cs[k].b;
        const uint32_t fa = B.filt[a].x, fb = B.filt[b].x;
        uint32_t key = n;
        if (solvedContact(fa, fb)) {
            if (isDynamic(fa)) key = root[a];
            else if (isDynamic(fb)) key = root[b];
        }
        keys[k] = key;
        vals[k] = k;
    }
}

__global__ void runFlagKernel(const uint64_t* keys, uint32_t m, uint32_t* flags) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        flags[k] = (k == 0 || keys[k] != keys[k - 1]) ? 1u : 0u;
}

// starts[index[k]] = k for run heads; also starts[runs] = m.
__global__ void runStartKernel(const uint32_t* flags, const uint32_t* index, uint32_t m, uint32_t* starts) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        if (flags[k]) starts[index[k]] = k;
        if (k == m - 1) starts[index[k] + flags[k]] = m;
    }
}

constexpr uint32_t kTinyLimit = 16;  // islands of at most this many contacts: packed tiny solve

// Class of an island of the plan (bodyStart: bodies sorted by island).
VXD int planClass(const uint32_t* islandStart, const uint32_t* bodyStart, uint32_t realIslands, uint32_t isl) {
    const uint32_t nb = isl < realIslands ? bodyStart[isl + 1] - bodyStart[isl] : 0u;
    return islandClassOf(nb, islandStart[isl + 1] - islandStart[isl], kTinyLimit);
}

// Greedy first-free-bit colouring (src/backend_cuda.cu:603-630), one thread
// per island (of at most sizeLimit contacts), contacts in their global (a, b, point) order. Static,
// kinematic and sensor endpoints do not constrain colours; past 64 colours
// each body continues from its own spill counter.
__global__ void colorKernel(const vx_contact* cs, const uint32_t* order, const uint32_t* islandStart,
                            uint32_t islands, const BodyArrays B, unsigned long long* mask, uint32_t* nextColor,
                            uint32_t* colorOf, uint64_t* colorKeys, Counters* C, uint32_t sizeLimit) {
    for (uint32_t isl = blockIdx.x * blockDim.x + threadIdx.x; isl < islands; isl += gridDim.x * blockDim.x) {
        const uint32_t s0 = islandStart[isl], s1 = islandStart[isl + 1];
        if (s1 - s0 > sizeLimit) continue;  // coloured in parallel
        for (uint32_t k = s0; k < s1; ++k) {
            const vx_contact& c = cs[order[k]];
            mask[c.a] = 0ull; mask[c.b] = 0ull;
            nextColor[c.a] = 64u; nextColor[c.b] = 64u;
        }
        uint32_t colors = 0;
        for (uint32_t k = s0; k < s1; ++k) {
            const uint32_t ci = order[k];
            const vx_contact& c = cs[ci];
            const uint32_t fa = B.filt[c.a].x, fb = B.filt[c.b].x;
            const bool sensor = isSensor(fa) || isSensor(fb);
            const bool sa = sensor || !isDynamic(fa);
            const bool sb = sensor || !isDynamic(fb);
            const unsigned long long used = (sa ? 0ull : mask[c.a]) | (sb ? 0ull : mask[c.b]);
            uint32_t color;
            if (~used) {
                color = (uint32_t)(__ffsll((long long)~used) - 1);
            } else {
                const uint32_t na = sa ? 64u : nextColor[c.a];
                const uint32_t nb = sb ? 64u : nextColor[c.b];
                color = na > nb ? na : nb;
                if (!sa) nextColor[c.a] = color + 1;
                if (!sb) nextColor[c.b] = color + 1;
            }
            if (color < 64) {
                if (!sa) mask[c.a] |= 1ull << color;
                if (!sb) mask[c.b] |= 1ull << color;
            }
            colorOf[ci] = color;
            colorKeys[k] = ((uint64_t)isl << 16) | (color < 65535u ? color : 65535u);
            if (color + 1 > colors) colors = color + 1;
        }
        atomicMax(&C->maxColors, colors);
        atomicMax(&C->largestIsland, s1 - s0);
    }
}

// Run number of each position: inclusive scan of the head flags minus one.
__global__ void runOfKernel(const uint32_t* flags, const uint32_t* index, uint32_t m, uint32_t* runOf) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        runOf[k] = index[k] + flags[k] - 1u;
}

__global__ void lastKeyKernel(const uint64_t* keys, uint32_t m, Counters* C) {
    if (blockIdx.x == 0 && threadIdx.x == 0) C->lastIslandKey = (uint32_t)keys[m - 1];
}

__global__ void islandMaxKernel(const uint32_t* islandStart, Counters* C) {
    const uint32_t islands = C->islands;
    uint32_t mx = 0;
    for (uint32_t isl = blockIdx.x * blockDim.x + threadIdx.x; isl < islands; isl += gridDim.x * blockDim.x)
        mx = max(mx, islandStart[isl + 1] - islandStart[isl]);
    for (int off = 16; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(&C->maxIslandSize, mx);
}

// Parallel greedy colouring of giant islands (beyond one block's shared memory). The greedy colour of a contact
// is the first colour below 64 unused by the earlier contacts (island order)
// that share one of its dynamic bodies (past that, one more than their
// highest colour): the unique fixed point of
//   colour[k] = rule({ colour[j] : j < k, j shares a body with k })
// reached by iterating the rule from all-zero colours (a contact is final
// once every earlier neighbour is). Every round runs over all contacts of the
// giant islands in parallel; a round without changes is the fixed point.
// Entries (body, 2k + side) sorted by body list each contact's earlier
// neighbours as the entries before its own in the body's run.
__global__ void colorEntryKernel(const vx_contact* cs, const uint32_t* order, uint32_t m, const uint32_t* islandIdx,
                                 const uint32_t* islandStart, const uint32_t* bodyStart, uint32_t realIslands,
                                 const BodyArrays B, uint32_t n, uint64_t* keys, uint32_t* vals, uint32_t* slot) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const bool big = planClass(islandStart, bodyStart, realIslands, islandIdx[k]) == kGiantIsland;
        const vx_contact& c = cs[order[k]];
        const uint32_t fa = B.filt[c.a].x, fb = B.filt[c.b].x;
        const bool sensor = isSensor(fa) || isSensor(fb);
        keys[2 * k] = big && !sensor && isDynamic(fa) ? c.a : n;
        keys[2 * k + 1] = big && !sensor && isDynamic(fb) ? c.b : n;
        vals[2 * k] = 2 * k;
        vals[2 * k + 1] = 2 * k + 1;
        slot[2 * k] = slot[2 * k + 1] = 0xffffffffu;
    }
}

__global__ void colorSlotKernel(const uint64_t* keys, const uint32_t* vals, uint32_t entries, uint32_t n,
                                uint32_t* slot, uint32_t* runStart) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < entries; e += gridDim.x * blockDim.x) {
        const uint64_t key = keys[e];
        if (key >= n) continue;
        slot[vals[e]] = e;
        if (e == 0 || keys[e - 1] != key) runStart[key] = e;
    }
}

// Cooperative launch. changed[3] rotate per round: the counter of round r + 1
// is cleared during round r, after every block has read round r - 2's value.
// color[] is indexed by island-order position and zero on entry; contacts of
// other islands have no slots and so keep their zero (looking their class up
// in every round: islands stage 4.17 / 4.05 ms with one island of 25,000
// contacts).
__global__ void colorFixedPointKernel(const uint64_t* keys, const uint32_t* vals, const uint32_t* slot,
                                      const uint32_t* runStart, uint32_t m, uint32_t* color, CoopState* st,
                                      uint32_t maxRounds) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t r = 0; r < maxRounds; ++r) {
        if (tid == 0) st->changed[(r + 1) % 3] = 0u;
        uint32_t local = 0;
        for (uint32_t k = tid; k < m; k += stride) {
            // Past 64 colours the greedy rule continues from a per-body
            // counter: one past the highest colour (>= 64) of the body's
            // earlier contacts, 64 when there is none.
            unsigned long long used = 0ull;
            uint32_t high = 63u;
            for (int side = 0; side < 2; ++side) {
                const uint32_t e = slot[2 * k + side];
                if (e == 0xffffffffu) continue;
                const uint32_t body = (uint32_t)keys[e];
                for (uint32_t f = runStart[body]; f < e; ++f) {
                    const uint32_t cq = __ldcg(color + (vals[f] >> 1));
                    if (cq < 64u) used |= 1ull << cq;
                    else high = max(high, cq);
                }
            }
            const uint32_t next = ~used != 0ull ? (uint32_t)(__ffsll((long long)~used) - 1) : high + 1u;
            if (next != __ldcg(color + k)) {
                __stcg(color + k, next);
                ++local;
            }
        }
        if (local) atomicAdd(&st->changed[r % 3], local);
        if (!gridSync(&st->bar, &st->timeout, st->spinLimit)) return;
        if (__ldcg(&st->changed[r % 3]) == 0u || __ldcg(&st->spill) != 0u) {
            if (tid == 0) st->rounds = r + 1;
            return;
        }
    }
    if (tid == 0) { st->rounds = maxRounds; atomicOr(&st->spill, 2u); }  // no fixed point within the bound
}

__global__ void colorFinishKernel(const uint32_t* order, uint32_t m, const uint32_t* islandIdx,
                                  const uint32_t* islandStart, const uint32_t* bodyStart, uint32_t realIslands,
                                  const uint32_t* color, uint32_t* colorOf, uint64_t* colorKeys, Counters* C) {
    uint32_t mx = 0;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const uint32_t isl = islandIdx[k];
        if (planClass(islandStart, bodyStart, realIslands, isl) != kGiantIsland) continue;
        const uint32_t size = islandStart[isl + 1] - islandStart[isl];
        const uint32_t c = color[k];
        colorOf[order[k]] = c;
        colorKeys[k] = ((uint64_t)isl << 16) | (c < 65535u ? c : 65535u);
        mx = max(mx, c + 1);
        if (k == islandStart[isl]) atomicMax(&C->largestIsland, size);
    }
    for (int off = 16; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(&C->maxColors, mx);
}

// ---------------------------------------------------------------------------
// colouring of one block's islands
// ---------------------------------------------------------------------------
//
// The greedy colour of a contact depends on the earlier contacts of its two
// bodies only. A block lists every body's contacts in order (shared memory),
// and one warp then follows the order as a dataflow: a contact whose
// predecessors on both bodies are coloured is ready, up to 32 ready contacts
// (they share no body) are coloured at once, and each releases its successor
// on either body. What bounds it is the longest chain, about 300 cycles a
// link; a chain through sorted contacts is long (hundreds of links on a pile
// of 1,000 bodies) and only a few contacts wide, so one warp without block
// barriers is enough. Before, one thread coloured an island of up to 4,096
// contacts (about 1 us each) and larger ones took a grid barrier per round of
// a fixed point. Islands stage of one step: 5.2 -> 0.66 ms with 64 islands of
// 2,400 contacts, 3.2 -> 0.41 ms with one of 3,500, 2.7 -> 0.64 ms with one of
// 10,500. Measured and not kept: block-wide rounds in which every waiting
// contact bids on its bodies (2.2 ms for the 10,500, 1.1 ms for the 2,400).
// A body's list is filled in any order and sorted by its thread while it is
// short; sorting a hub's there took most of the call (call on an island of 4,000
// rows of one body 31 ms, of 16,384 109 ms), so a warp picks a list of more than
// 64 rows out of the island's rows in order (2.3 and 8.3 ms).
template <int Class>
struct ColorShape {
    static constexpr int kRows = ClassShape<Class>::kRows;
    static constexpr int kBodies = ClassShape<Class>::kBodies;
    static_assert(kBodies < 0xfff && 2 * kRows < 0xffff, "12-bit body words, 16-bit list positions");
    static constexpr size_t kSmem = (size_t)kBodies * 16 + (size_t)kRows * 10;
};

template <int Class>
__global__ void __launch_bounds__(ClassShape<Class>::kThreads)
    colorIslandKernel(const vx_contact* cs, const uint32_t* order, const uint32_t* islandStart,
                      const uint32_t* bodyOrder, const uint32_t* bodyStart, uint32_t islands, uint32_t realIslands,
                      const BodyArrays B, uint32_t* localIdx, uint32_t* colorOf, uint64_t* colorKeys, Counters* C) {
    constexpr int Threads = ClassShape<Class>::kThreads, kBodies = ColorShape<Class>::kBodies;
    constexpr int kRows = ColorShape<Class>::kRows;
    constexpr uint32_t kNone = 0xfffu, kPred = 1u << 24;
    constexpr int kLongList = 64;
    extern __shared__ unsigned long long colorSmem[];
    unsigned long long* mask = colorSmem;
    uint32_t* next = reinterpret_cast<uint32_t*>(mask + kBodies);  // spill counter past 64 colours; entry counts first
    uint32_t* rows = next + kBodies;  // body words of a row (12 bits each) and predecessors; its colour when done
    uint16_t* list = reinterpret_cast<uint16_t*>(rows + kRows);  // the bodies' rows, each body's in order
    uint16_t* ready = list + 2 * kRows;                          // rows in the order they became ready
    uint16_t* head = ready + kRows;                              // the body's first waiting row in `list`
    uint16_t* stop = head + kBodies;
    __shared__ uint32_t tail;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t isl = blockIdx.x; isl < islands; isl += gridDim.x) {
        const uint32_t s0 = islandStart[isl], count = islandStart[isl + 1] - s0;
        const uint32_t b0 = isl < realIslands ? bodyStart[isl] : 0u;
        const uint32_t nb = isl < realIslands ? bodyStart[isl + 1] - b0 : 0u;
        if (islandClassOf(nb, count, kTinyLimit) != Class) continue;
        for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
            localIdx[bodyOrder[b0 + t]] = t;
            mask[t] = 0ull;
            next[t] = 0u;
        }
        if (threadIdx.x == 0u) tail = 0u;
        islandBarrier<Threads>();
        for (uint32_t r = threadIdx.x; r < count; r += Threads) {
            const vx_contact& c = cs[order[s0 + r]];
            const uint32_t fa = B.filt[c.a].x, fb = B.filt[c.b].x;
            const bool solved = nb > 0u && solvedContact(fa, fb);
            uint32_t la = kNone, lb = kNone;
            if (solved && isDynamic(fa)) la = localIdx[c.a];
            if (solved && isDynamic(fb)) lb = localIdx[c.b];
            // outside the island's list (an inconsistent plan, which the solve reports): no constraint
            if (la >= nb) la = kNone;
            if (lb >= nb) lb = kNone;
            rows[r] = la | (lb << 12);
            if (la != kNone) atomicAdd(next + la, 1u);
            if (lb != kNone) atomicAdd(next + lb, 1u);
        }
        islandBarrier<Threads>();
        if (threadIdx.x < 32u) {  // each body's range of the list
            uint32_t base = 0u;
            for (uint32_t t0 = 0; t0 < nb; t0 += 32u) {
                const uint32_t t = t0 + lane, v = t < nb ? next[t] : 0u;
                uint32_t incl = v;
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
                    if ((int)lane >= off) incl += y;
                }
                if (t < nb) {
                    next[t] = base + incl - v;  // fill position
                    head[t] = (uint16_t)(base + incl - v);
                    stop[t] = (uint16_t)(base + incl);
                }
                base += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        islandBarrier<Threads>();
        for (uint32_t r = threadIdx.x; r < count; r += Threads) {
            const uint32_t la = rows[r] & 0xfffu, lb = (rows[r] >> 12) & 0xfffu;
            if (la != kNone) list[atomicAdd(next + la, 1u)] = (uint16_t)r;
            if (lb != kNone) list[atomicAdd(next + lb, 1u)] = (uint16_t)r;
        }
        islandBarrier<Threads>();
        for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
            // (nearly sorted: the threads took the rows in ascending batches)
            const int from = head[t], to = stop[t];
            if (to - from > kLongList) continue;
            for (int x = from + 1; x < to; ++x) {
                const uint16_t v = list[x];
                int y = x - 1;
                while (y >= from && list[y] > v) { list[y + 1] = list[y]; --y; }
                list[y + 1] = v;
            }
        }
        for (uint32_t t = threadIdx.x >> 5; t < nb; t += Threads / 32) {  // a longer list: picked in order by a warp
            uint32_t at = head[t];
            if ((int)(stop[t] - at) <= kLongList) continue;
            for (uint32_t r0 = 0; r0 < count; r0 += 32u) {
                const uint32_t word = r0 + lane < count ? rows[r0 + lane] : 0xffffffu;
                const bool mine = (word & 0xfffu) == t || ((word >> 12) & 0xfffu) == t;
                const unsigned m = __ballot_sync(0xffffffffu, mine);
                if (mine) list[at + __popc(m & laneMaskLt())] = (uint16_t)(r0 + lane);
                at += __popc(m);
            }
        }
        islandBarrier<Threads>();
        for (uint32_t t = threadIdx.x; t < nb; t += Threads) {
            const int from = head[t], to = stop[t];
            for (int x = from + 1; x < to; ++x) atomicAdd(rows + list[x], kPred);
            next[t] = 64u;
        }
        islandBarrier<Threads>();
        for (uint32_t r = threadIdx.x; r < count; r += Threads)
            if (rows[r] < kPred) ready[atomicAdd(&tail, 1u)] = (uint16_t)r;
        islandBarrier<Threads>();
        if (threadIdx.x < 32u) {
            uint32_t colors = 0u, done = 0u, end = tail;
            while (done < end) {  // every pass colours at least one row; every row is queued once
                const uint32_t take = min(end - done, 32u);
                uint32_t push0 = 0xffffffffu, push1 = 0xffffffffu;
                if (lane < take) {
                    const uint32_t r = ready[done + lane], word = rows[r];
                    const uint32_t la = word & 0xfffu, lb = (word >> 12) & 0xfffu;
                    const unsigned long long used =
                        (la != kNone ? mask[la] : 0ull) | (lb != kNone ? mask[lb] : 0ull);
                    uint32_t color;
                    if (~used) {
                        color = (uint32_t)(__ffsll((long long)~used) - 1);
                        if (la != kNone) mask[la] |= 1ull << color;
                        if (lb != kNone) mask[lb] |= 1ull << color;
                    } else {
                        color = max(la != kNone ? next[la] : 64u, lb != kNone ? next[lb] : 64u);
                        if (la != kNone) next[la] = color + 1u;
                        if (lb != kNone) next[lb] = color + 1u;
                    }
                    rows[r] = color;
                    colors = max(colors, color + 1u);
                    if (la != kNone) {
                        const uint32_t h = head[la] + 1u;
                        head[la] = (uint16_t)h;
                        if (h < stop[la]) {
                            const uint32_t s = list[h];
                            if (atomicSub(rows + s, kPred) < 2u * kPred) push0 = s;
                        }
                    }
                    if (lb != kNone) {
                        const uint32_t h = head[lb] + 1u;
                        head[lb] = (uint16_t)h;
                        if (h < stop[lb]) {
                            const uint32_t s = list[h];
                            if (atomicSub(rows + s, kPred) < 2u * kPred) push1 = s;
                        }
                    }
                }
                const unsigned m0 = __ballot_sync(0xffffffffu, push0 != 0xffffffffu);
                const unsigned m1 = __ballot_sync(0xffffffffu, push1 != 0xffffffffu);
                if (push0 != 0xffffffffu) ready[end + __popc(m0 & laneMaskLt())] = (uint16_t)push0;
                if (push1 != 0xffffffffu) ready[end + __popc(m0) + __popc(m1 & laneMaskLt())] = (uint16_t)push1;
                done += take;
                end += __popc(m0) + __popc(m1);
                __syncwarp();
            }
            for (int off = 16; off > 0; off >>= 1) colors = max(colors, __shfl_xor_sync(0xffffffffu, colors, off));
            if (lane == 0u) {
                atomicMax(&C->maxColors, colors);
                atomicMax(&C->largestIsland, count);
            }
        }
        islandBarrier<Threads>();
        for (uint32_t r = threadIdx.x; r < count; r += Threads) {
            const uint32_t color = rows[r];
            colorOf[order[s0 + r]] = color;
            colorKeys[s0 + r] = ((uint64_t)isl << 16) | (color < 65535u ? color : 65535u);
        }
        islandBarrier<Threads>();
    }
}

// islandOfBody for the dynamic bodies of every real island's contacts, one
// thread per island-order position (islandOf[k]: island of position k).
__global__ void islandBodyKernel(const vx_contact* cs, const uint32_t* order, const uint32_t* islandOf, uint32_t m,
                                 uint32_t realIslands, const BodyArrays B, uint32_t* islandOfBody) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const uint32_t isl = islandOf[k];
        if (isl >= realIslands) continue;
        const vx_contact& c = cs[order[k]];
        if (isDynamic(B.filt[c.a].x)) islandOfBody[c.a] = isl;
        if (isDynamic(B.filt[c.b].x)) islandOfBody[c.b] = isl;
    }
}

__global__ void bodyKeyKernel(const uint32_t* islandOfBody, uint32_t n, uint32_t freeKey, uint64_t* keys,
                              uint32_t* vals) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t isl = islandOfBody[i];
        keys[i] = isl == 0xffffffffu ? freeKey : isl;
        vals[i] = i;
    }
}

// bodyStart[key] for each run of sorted body keys; bodyStart has islands+2 entries.
__global__ void bodyStartKernel(const uint64_t* keys, uint32_t n, uint32_t* bodyStart, uint32_t entries) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint64_t key = keys[k];
        const uint64_t prevKey = k == 0 ? ~0ull : keys[k - 1];
        if (key != prevKey) {
            // every key in (prevKey, key] starts at k (empty islands get empty ranges)
            const uint64_t from = k == 0 ? 0 : prevKey + 1;
            for (uint64_t x = from; x <= key && x < entries; ++x) bodyStart[x] = k;
        }
        if (k == n - 1)
            for (uint64_t x = key + 1; x < entries; ++x) bodyStart[x] = n;
    }
}

// Islands the block kernels cannot hold (the grid's flow), counted
// for the host's single read of the plan.
__global__ void giantCountKernel(const uint32_t* islandStart, const uint32_t* bodyStart, uint32_t islands,
                                 uint32_t realIslands, Counters* C) {
    uint32_t count = 0;
    for (uint32_t isl = blockIdx.x * blockDim.x + threadIdx.x; isl < islands; isl += gridDim.x * blockDim.x) {
        const uint32_t rows = islandStart[isl + 1] - islandStart[isl];
        const uint32_t nb = isl < realIslands ? bodyStart[isl + 1] - bodyStart[isl] : 0u;
        if (solveClassOf(nb, rows, kTinyLimit) == kGiantIsland) ++count;
    }
    for (int off = 16; off > 0; off >>= 1) count += __shfl_xor_sync(0xffffffffu, count, off);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd(&C->giantCount, count);
}

// Contact-free bodies: the last two bodyStart entries, for the host's single read.
__global__ void freeRangeKernel(const uint32_t* bodyStart, uint32_t entries, Counters* C) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        C->freeFrom = bodyStart[entries - 2];
        C->freeTo = bodyStart[entries - 1];
    }
}

// ---------------------------------------------------------------------------
// island solve (src/backend_cuda.cu:569-761 semantics)
// ---------------------------------------------------------------------------

VXD void positionRow(const SolveArgs& A, uint32_t ci) {
    const vx_contact& cc = A.contacts[ci];
    const uint32_t fa = A.B.filt[cc.a].x, fb = A.B.filt[cc.b].x;
    if (!solvedContact(fa, fb)) return;
    const Mass ma = loadMass(A.B, cc.a), mb = loadMass(A.B, cc.b);
    const float ima = solverInvMass(ma), imb = solverInvMass(mb);
    const float invMassSum = ima + imb;
    if (invMassSum <= 0.0f) return;
    V3 pa = f3(A.B.pos[cc.a]), pb = f3(A.B.pos[cc.b]);
    const Q4 qa = q4(A.B.rot[cc.a]), qb = q4(A.B.rot[cc.b]);
    const V3 n{cc.normal.x, cc.normal.y, cc.normal.z};
    const V3 wa = anchorWorld(shapeOf(fa) == kSphere, pa, qa, V3{cc.localAnchorA.x, cc.localAnchorA.y, cc.localAnchorA.z});
    const V3 wb = anchorWorld(shapeOf(fb) == kSphere, pb, qb, V3{cc.localAnchorB.x, cc.localAnchorB.y, cc.localAnchorB.z});
    const float g = cc.bias0 + dot(n, wa - wb);
    const float slop = 1e-3f;
    if (g >= -slop) return;
    float resolve = 0.6f;
    if (A.stackStabilization) {
        const V3 rv = f3(A.B.vel[cc.a]) - f3(A.B.vel[cc.b]);
        if (lengthSq(rv) < 1e-4f) {
            const float stiffness = A.stackStiffness / 1000.0f;
            const float damping = 1.0f + A.stackDamping * A.h;
            resolve += 0.2f * stiffness / damping;
        }
    }
    const float push = -resolve * (g + slop) / invMassSum;
    if (isDynamic(fa) && !isAsleep(fa)) { pa += n * (push * ima); A.B.pos[cc.a] = pack(pa, 0.0f); }
    if (isDynamic(fb) && !isAsleep(fb)) { pb -= n * (push * imb); A.B.pos[cc.b] = pack(pb, 0.0f); }
}



// Bodies of a pack of tiny islands in shared memory.
constexpr int kGiantBlockThreads = 256;  // one block per giant island (no cooperative grid)
constexpr size_t blockSmem(int bodies) { return (size_t)bodies * (7 * sizeof(float4) + sizeof(uint32_t)); }

struct SharedBodies {
    float4 *p, *q, *v, *w, *inertia, *iq, *frame;
    uint32_t* flags;
};

template <int Bodies>
VXD SharedBodies carve(float4* base) {
    SharedBodies S;
    S.p = base;
    S.q = S.p + Bodies;
    S.v = S.q + Bodies;
    S.w = S.v + Bodies;
    S.inertia = S.w + Bodies;
    S.iq = S.inertia + Bodies;
    S.frame = S.iq + Bodies;
    S.flags = reinterpret_cast<uint32_t*>(S.frame + Bodies);
    return S;
}

VXD SolverBody sharedBody(const SharedBodies& S, int li) {
    SolverBody b;
    b.p = f3(S.p[li]);
    b.q = q4(S.q[li]);
    b.v = f3(S.v[li]);
    b.w = f3(S.w[li]);
    const float4 in = S.inertia[li];
    b.m.invI = V3{in.x, in.y, in.z};
    b.m.invMass = in.w;
    b.m.iq = q4(S.iq[li]);
    b.m.flags = S.flags[li];
    b.sphere = shapeOf(b.m.flags) == kSphere;
    b.frame = q4(S.frame[li]);
    return b;
}

// A body outside the island's shared copy (static endpoints): frame computed here.
VXD SolverBody globalBody(const BodyArrays& B, uint32_t id) {
    SolverBody b = loadSolverBody(B, id);
    cacheFrame(b);
    return b;
}

VXD void sharedIntegrateVelocity(const SolveArgs& A, const SharedBodies& S, int li, uint32_t id) {
    SolverBody b = sharedBody(S, li);
    const Mass& m = b.m;
    if (!isDynamic(m.flags) || isLocked(m.flags) || isAsleep(m.flags)) return;
    const float4 ex = A.B.extra[id];
    b.v += (A.gravity * ex.y + f3(A.B.force[id]) * solverInvMass(m)) * A.h;
    b.w += invInertiaMulAt(m, f3(A.B.torque[id]), b.q) * A.h;
    b.v *= 1.0f / (1.0f + ex.z * A.h);
    b.w *= 1.0f / (1.0f + ex.w * A.h);
    S.v[li] = pack(b.v, 0.0f);
    S.w[li] = pack(b.w, 0.0f);
}

VXD void sharedIntegrateTransform(const SolveArgs& A, const SharedBodies& S, int li) {
    SolverBody b = sharedBody(S, li);
    if (isStaticBody(b.m.flags) || isLocked(b.m.flags) || isAsleep(b.m.flags)) return;
    advanceTransform(b.m, b.p, b.q, b.v, b.w, A.h);
    S.p[li] = pack(b.p, 0.0f);
    S.q[li] = pack(b.q);
    S.w[li] = pack(b.w, 0.0f);
}

// Island bodies read from global memory with frames from A.frames.
VXD SolverBody framedBody(const SolveArgs& A, uint32_t id) {
    SolverBody b = loadSolverBody(A.B, id);
    if (isDynamic(b.m.flags)) b.frame = q4(A.frames[id]);
    else cacheFrame(b);
    return b;
}

// op: 0 warm start, 1 velocity sweep, 3 prepare
VXD void globalRow(const SolveArgs& A, uint32_t pos, int op) {
    vx_contact& cc = A.contacts[A.order[pos]];
    SolverBody a = framedBody(A, cc.a), b = framedBody(A, cc.b);
    if (!solvedContact(a.m.flags, b.m.flags)) return;
    RowContact r;
    loadRow(cc, r);
    RowPrep& P = A.prep[pos];
    if (op == 3) { prepRow(a, b, r, A.h, A.coneBlock != 0, P); return; }
    if (op == 0) warmPrepRow(a, b, r, P);
    else sweepRow(a, b, r, P, A.coneBlock != 0);
    if (isDynamic(a.m.flags)) { A.B.vel[cc.a] = pack(a.v, 0.0f); A.B.ang[cc.a] = pack(a.w, 0.0f); }
    if (isDynamic(b.m.flags)) { A.B.vel[cc.b] = pack(b.v, 0.0f); A.B.ang[cc.b] = pack(b.w, 0.0f); }
    storeRow(cc, r);
}

__device__ void solveIslandGlobal(const SolveArgs& A, uint32_t isl) {
    const uint32_t g0 = A.islandSeg[isl], g1 = A.islandSeg[isl + 1];
    if (A.positionIterations > 0) {
        for (int it = 0; it < A.positionIterations; ++it)
            for (uint32_t g = g0; g < g1; ++g) {
                for (uint32_t k = A.segStart[g] + threadIdx.x; k < A.segStart[g + 1]; k += blockDim.x)
                    positionRow(A, A.order[k]);
                __syncthreads();
            }
        return;
    }
    const uint32_t s0 = A.islandStart[isl], s1 = A.islandStart[isl + 1];
    const uint32_t b0 = isl < A.realIslands ? A.bodyStart[isl] : 0u;
    const uint32_t b1 = isl < A.realIslands ? A.bodyStart[isl + 1] : 0u;
    for (int s = 0; s < A.substeps; ++s) {
        for (uint32_t k = b0 + threadIdx.x; k < b1; k += blockDim.x) {
            const uint32_t id = A.bodyOrder[k];
            if (A.integrate && s > 0) integrateVelocity(A.B, id, A.gravity, A.h);
            A.frames[id] = pack(inertiaFrameAt(loadMass(A.B, id), q4(A.B.rot[id])));
        }
        __syncthreads();
        for (uint32_t k = s0 + threadIdx.x; k < s1; k += blockDim.x) globalRow(A, k, 3);
        __syncthreads();
        if (A.warmStart && s == 0)
            for (uint32_t g = g0; g < g1; ++g) {
                for (uint32_t k = A.segStart[g] + threadIdx.x; k < A.segStart[g + 1]; k += blockDim.x)
                    globalRow(A, k, 0);
                __syncthreads();
            }
        for (int it = 0; it < A.sweeps; ++it)
            for (uint32_t g = g0; g < g1; ++g) {
                for (uint32_t k = A.segStart[g] + threadIdx.x; k < A.segStart[g + 1]; k += blockDim.x)
                    globalRow(A, k, 1);
                __syncthreads();
            }
        if (A.integrate) {
            for (uint32_t k = b0 + threadIdx.x; k < b1; k += blockDim.x)
                integrateTransform(A.B, A.bodyOrder[k], A.h);
            __syncthreads();
        }
    }
}

// ---- tiny islands packed into warps -----------------------------------------
//
// Islands of at most tinyLimit (16) contacts are packed, in island order, into
// warps of at most 32 rows and 64 bodies. Each lane owns one row and keeps its
// contact terms and per-substep pose terms in registers; the pack's bodies live
// in shared memory. A step runs colour slot c of every island in the pack at
// once (rows of different islands share no body; rows of one colour share no
// dynamic body), so each body sees its rows in colour order, as in the serial
// per-island loop. A pack needs (largest colour count) x sweeps x substeps
// warp steps instead of (rows x sweeps x substeps) thread steps, with no
// per-thread arrays in local memory.
constexpr int kPackRows = 32;
constexpr int kPackBodies = 64;
constexpr int kPackChunk = 64;      // tiny islands per packing thread (a serial greedy scan each)
constexpr int kPackWarps = 4;       // warps (packs) per block

// Sort key of a tiny island: its colour count (a pack runs as many colour
// slots per sweep as its most coloured island, so similar islands share packs).
// Over `cap` slots (an upper bound); slots past the device-side count sort last.
__global__ void tinyKeyKernel(SolveArgs A, const uint32_t* list, const uint32_t* countPtr, uint32_t cap,
                              uint64_t* keys, uint32_t* vals) {
    const uint32_t count = *countPtr;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < cap; t += gridDim.x * blockDim.x) {
        if (t < count) {
            const uint32_t isl = list[t];
            keys[t] = A.islandSeg[isl + 1] - A.islandSeg[isl];
            vals[t] = isl;
        } else {
            keys[t] = 0xffu;
            vals[t] = 0xffffffffu;
        }
    }
}

__global__ void tinyFlagKernel(SolveArgs A, uint32_t* flags) {
    for (uint32_t isl = blockIdx.x * blockDim.x + threadIdx.x; isl < A.islands; isl += gridDim.x * blockDim.x) {
        const uint32_t rows = A.islandStart[isl + 1] - A.islandStart[isl];
        flags[isl] = rows > 0 && rows <= A.tinyLimit ? 1u : 0u;
    }
}

VXD uint32_t islandBodies(const SolveArgs& A, uint32_t isl) {
    return isl < A.realIslands ? A.bodyStart[isl + 1] - A.bodyStart[isl] : 0u;
}

// Greedy packing of each chunk of the tiny-island list: pass 0 counts the
// packs of a chunk, pass 1 writes each pack's first list index.
__global__ void tinyPackKernel(SolveArgs A, const uint32_t* list, const uint32_t* countPtr, uint32_t chunksCap,
                               int pass, uint32_t* packCount, const uint32_t* packBase, uint32_t* packFirst) {
    const uint32_t count = *countPtr;
    for (uint32_t ch = blockIdx.x * blockDim.x + threadIdx.x; ch < chunksCap; ch += gridDim.x * blockDim.x) {
        if (ch * kPackChunk >= count) {  // past the list: no packs
            if (pass == 0) packCount[ch] = 0;
            continue;
        }
        const uint32_t t0 = ch * kPackChunk, t1 = min(count, t0 + kPackChunk);
        uint32_t packs = 0, rows = 0, bodies = 0;
        for (uint32_t t = t0; t < t1; ++t) {
            const uint32_t isl = list[t];
            const uint32_t r = A.islandStart[isl + 1] - A.islandStart[isl], b = islandBodies(A, isl);
            if (t == t0 || rows + r > (uint32_t)kPackRows || bodies + b > (uint32_t)kPackBodies) {
                if (pass == 1) packFirst[packBase[ch] + packs] = t;
                ++packs;
                rows = 0;
                bodies = 0;
            }
            rows += r;
            bodies += b;
        }
        if (pass == 0) packCount[ch] = packs;
    }
}

// Per-warp shared memory of the pack kernel: the bodies and their ids.
constexpr size_t kPackBodySmem = blockSmem(kPackBodies);
constexpr size_t kPackWarpSmem = (kPackBodySmem + kPackBodies * sizeof(uint32_t) + 15) / 16 * 16;

VXD void solveTinyPack(const SolveArgs& A, const uint32_t* list, const uint32_t* packFirst, uint32_t packs,
                       uint32_t listCount, uint32_t* localIdx, const SharedBodies& S, uint32_t* ids,
                       uint32_t packIdx, uint32_t lane);

// Packs come from device-side counts (no host read); warps stride over them.
__global__ void __launch_bounds__(32 * kPackWarps) solveTinyPackKernel(SolveArgs A, const uint32_t* list,
                                                                        const uint32_t* packFirst,
                                                                        const Counters* C, uint32_t* localIdx) {
    extern __shared__ float4 smemRaw[];
    const uint32_t warpInBlock = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    float4* base = smemRaw + warpInBlock * (kPackWarpSmem / sizeof(float4));
    const SharedBodies S = carve<kPackBodies>(base);
    uint32_t* ids = reinterpret_cast<uint32_t*>(base + kPackBodySmem / sizeof(float4));
    const uint32_t packs = C->tinyPacks, listCount = C->tinyIslands;
    for (uint32_t packIdx = blockIdx.x * kPackWarps + warpInBlock; packIdx < packs; packIdx += gridDim.x * kPackWarps) {
        solveTinyPack(A, list, packFirst, packs, listCount, localIdx, S, ids, packIdx, lane);
        __syncwarp();
    }
}

VXD void solveTinyPack(const SolveArgs& A, const uint32_t* list, const uint32_t* packFirst, uint32_t packs,
                       uint32_t listCount, uint32_t* localIdx, const SharedBodies& S, uint32_t* ids,
                       uint32_t packIdx, uint32_t lane) {
    const uint32_t first = packFirst[packIdx];
    const uint32_t last = packIdx + 1 < packs ? packFirst[packIdx + 1] : listCount;
    const uint32_t count = last - first;  // islands in this pack (1..32)
    uint32_t isl = 0, r = 0, nb = 0, colours = 0;
    if (lane < count) {
        isl = list[first + lane];
        r = A.islandStart[isl + 1] - A.islandStart[isl];
        nb = islandBodies(A, isl);
        colours = A.islandSeg[isl + 1] - A.islandSeg[isl];
    }
    // inclusive prefix sums of rows and bodies over the pack's islands, largest colour count
    uint32_t rp = r, bp = nb, maxC = colours;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, rp, off), y = __shfl_up_sync(0xffffffffu, bp, off);
        if ((int)lane >= off) { rp += x; bp += y; }
    }
    for (int off = 16; off > 0; off >>= 1) maxC = max(maxC, __shfl_xor_sync(0xffffffffu, maxC, off));
    rp -= r;  // exclusive
    bp -= nb;
    const uint32_t totalBodies = __shfl_sync(0xffffffffu, bp + nb, 31);
    // bodies into shared memory: island j's bodies at slots [bp_j, bp_j + nb_j)
    for (uint32_t j = 0; j < count; ++j) {
        const uint32_t jIsl = __shfl_sync(0xffffffffu, isl, j), jB = __shfl_sync(0xffffffffu, nb, j);
        const uint32_t jBase = __shfl_sync(0xffffffffu, bp, j);
        for (uint32_t k = lane; k < jB; k += 32) {
            const uint32_t id = A.bodyOrder[A.bodyStart[jIsl] + k], t = jBase + k;
            S.p[t] = A.B.pos[id]; S.q[t] = A.B.rot[id]; S.v[t] = A.B.vel[id]; S.w[t] = A.B.ang[id];
            S.inertia[t] = A.B.inertia[id]; S.iq[t] = A.B.iq[id]; S.flags[t] = A.B.filt[id].x;
            ids[t] = id;
            localIdx[id] = t;
        }
    }
    __syncwarp();
    // this lane's row: the island j with rp_j <= lane < rp_j + r_j
    bool has = false;
    uint32_t row = 0, myIsl = 0, myBase = 0, myNb = 0;
    for (uint32_t j = 0; j < count; ++j) {
        const uint32_t jr = __shfl_sync(0xffffffffu, r, j), jrp = __shfl_sync(0xffffffffu, rp, j);
        const uint32_t jIsl = __shfl_sync(0xffffffffu, isl, j), jBase = __shfl_sync(0xffffffffu, bp, j);
        const uint32_t jNb = __shfl_sync(0xffffffffu, nb, j);
        if (lane >= jrp && lane < jrp + jr) {
            has = true;
            myIsl = jIsl;
            row = A.islandStart[jIsl] + (lane - jrp);
            myBase = jBase;
            myNb = jNb;
        }
    }
    vx_contact* cp = nullptr;
    RowContact rc;
    RowPrep P;
    int la = -1, lb = -1;
    uint32_t ida = 0, idb = 0, myC = 0;
    bool live = false;
    if (has) {
        cp = A.contacts + A.order[row];
        loadRow(*cp, rc);
        ida = cp->a;
        idb = cp->b;
        const uint32_t fa = A.B.filt[ida].x, fb = A.B.filt[idb].x;
        live = solvedContact(fa, fb);
        // (a sensor's row lies in the null island, which owns no bodies)
        if (live && isDynamic(fa)) la = (int)localIdx[ida];
        if (live && isDynamic(fb)) lb = (int)localIdx[idb];
        // a dynamic body outside its island's slots means an inconsistent plan: report it, never index smem
        if (la >= 0 && ((uint32_t)la < myBase || (uint32_t)la >= myBase + myNb || ids[la] != ida)) {
            atomicOr(A.fault, 1u);
            la = -1;
        }
        if (lb >= 0 && ((uint32_t)lb < myBase || (uint32_t)lb >= myBase + myNb || ids[lb] != idb)) {
            atomicOr(A.fault, 1u);
            lb = -1;
        }
        const uint32_t g0 = A.islandSeg[myIsl], g1 = A.islandSeg[myIsl + 1];
        uint32_t g = g0;
        while (g + 1 < g1 && A.segStart[g + 1] <= row) ++g;
        myC = g - g0;
    }
    if (A.positionIterations > 0) {
        for (int it = 0; it < A.positionIterations; ++it)
            for (uint32_t c = 0; c < maxC; ++c) {
                if (live && myC == c) {
                    const SolverBody a = la >= 0 ? sharedBody(S, la) : globalBody(A.B, ida);
                    const SolverBody b = lb >= 0 ? sharedBody(S, lb) : globalBody(A.B, idb);
                    const float ima = solverInvMass(a.m), imb = solverInvMass(b.m);
                    const float invMassSum = ima + imb;
                    if (invMassSum > 0.0f) {
                        const V3 wa = anchorWorld(a.sphere, a.p, a.q, rc.la);
                        const V3 wb = anchorWorld(b.sphere, b.p, b.q, rc.lb);
                        const float gap = rc.bias0 + dot(rc.normal, wa - wb);
                        if (gap < -1e-3f) {
                            float resolve = 0.6f;
                            if (A.stackStabilization && lengthSq(a.v - b.v) < 1e-4f)
                                resolve += 0.2f * (A.stackStiffness / 1000.0f) / (1.0f + A.stackDamping * A.h);
                            const float push = -resolve * (gap + 1e-3f) / invMassSum;
                            if (isDynamic(a.m.flags) && !isAsleep(a.m.flags) && la >= 0)
                                S.p[la] = pack(a.p + rc.normal * (push * ima), 0.0f);
                            if (isDynamic(b.m.flags) && !isAsleep(b.m.flags) && lb >= 0)
                                S.p[lb] = pack(b.p - rc.normal * (push * imb), 0.0f);
                        }
                    }
                }
                __syncwarp();
            }
        for (uint32_t t = lane; t < totalBodies; t += 32)
            if (isDynamic(S.flags[t])) A.B.pos[ids[t]] = S.p[t];
        return;
    }
    for (int s = 0; s < A.substeps; ++s) {
        for (uint32_t t = lane; t < totalBodies; t += 32) {
            if (A.integrate && s > 0) sharedIntegrateVelocity(A, S, (int)t, ids[t]);
            Mass m;
            const float4 in = S.inertia[t];
            m.invI = V3{in.x, in.y, in.z};
            m.invMass = in.w;
            m.iq = q4(S.iq[t]);
            m.flags = S.flags[t];
            S.frame[t] = pack(inertiaFrameAt(m, q4(S.q[t])));
        }
        __syncwarp();
        if (live) {
            const SolverBody a = la >= 0 ? sharedBody(S, la) : globalBody(A.B, ida);
            const SolverBody b = lb >= 0 ? sharedBody(S, lb) : globalBody(A.B, idb);
            prepRow(a, b, rc, A.h, A.coneBlock != 0, P);
        }
        __syncwarp();
        const int units = (A.warmStart && s == 0 ? 1 : 0) + A.sweeps;
        for (int u = 0; u < units; ++u) {
            const bool warm = A.warmStart && s == 0 && u == 0;
            for (uint32_t c = 0; c < maxC; ++c) {
                if (live && myC == c) {
                    SolverBody a = la >= 0 ? sharedBody(S, la) : globalBody(A.B, ida);
                    SolverBody b = lb >= 0 ? sharedBody(S, lb) : globalBody(A.B, idb);
                    if (warm) warmPrepRow(a, b, rc, P);
                    else sweepRow(a, b, rc, P, A.coneBlock != 0);
                    if (la >= 0 && isDynamic(a.m.flags)) { S.v[la] = pack(a.v, 0.0f); S.w[la] = pack(a.w, 0.0f); }
                    if (lb >= 0 && isDynamic(b.m.flags)) { S.v[lb] = pack(b.v, 0.0f); S.w[lb] = pack(b.w, 0.0f); }
                }
                __syncwarp();
            }
        }
        if (A.integrate) {
            for (uint32_t t = lane; t < totalBodies; t += 32) sharedIntegrateTransform(A, S, (int)t);
            __syncwarp();
        }
    }
    for (uint32_t t = lane; t < totalBodies; t += 32) {
        if (!isDynamic(S.flags[t])) continue;
        const uint32_t id = ids[t];
        A.B.pos[id] = S.p[t]; A.B.rot[id] = S.q[t]; A.B.vel[id] = S.v[t]; A.B.ang[id] = S.w[t];
    }
    if (has) storeRow(*cp, rc);
}

// ---- giant islands: the plan of the grid's flow (solve_flow.cuh) ---------------

constexpr uint32_t kNoPred = 0xffffffffu;  // empty queue slot / no successor

// Entries (dynamic body, 2k + side) of every row of a giant island, other
// endpoints keyed n (no link).
__global__ void giantEntryKernel(SolveArgs A, const uint32_t* islandOf, uint32_t m, uint32_t n, uint64_t* keys,
                                 uint32_t* vals);
// For each body run of the sorted entries, its first entry.
__global__ void flowRunKernel(const uint64_t* keys, uint32_t entries, uint32_t n, uint32_t* first) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < entries; p += gridDim.x * blockDim.x) {
        const uint64_t key = keys[p];
        if (key != (uint64_t)n && (p == 0 || keys[p - 1] != key)) first[key] = p;
    }
}
// rank[2k + side]: the row's rank among its body's rows in colour order, 0
// without a dynamic body; degree: the body's rows.
__global__ void flowLinkKernel(const uint64_t* keys, const uint32_t* vals, uint32_t entries, uint32_t n,
                               const uint32_t* first, uint32_t* rank, uint32_t* degree) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < entries; p += gridDim.x * blockDim.x) {
        const uint64_t key = keys[p];
        const uint32_t v = key != (uint64_t)n ? p - first[key] : 0u;
        rank[vals[p]] = v;
        if (key != (uint64_t)n && (p + 1 == entries || keys[p + 1] != key)) degree[key] = v + 1u;
    }
}

// Spatial clusters: the islands' bodies in Morton order, cut into as many
// clusters as the grid has warps.
VXD uint32_t spreadBits10(uint32_t v) {  // 10 bits -> every third bit
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void clusterBodyKeyKernel(SolveArgs A, const uint32_t* bodyPos, uint32_t nb, const Counters* C,
                                     uint64_t* keys, uint32_t* vals) {
    const float lo[3] = {fromOrdered(C->cellMinBits[0]), fromOrdered(C->cellMinBits[1]), fromOrdered(C->cellMinBits[2])};
    const float hi[3] = {fromOrdered(C->cellMaxBits[0]), fromOrdered(C->cellMaxBits[1]), fromOrdered(C->cellMaxBits[2])};
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nb; k += gridDim.x * blockDim.x) {
        const uint32_t id = A.bodyOrder[bodyPos[k]];
        const float4 p = A.B.pos[id];
        const float x[3] = {p.x, p.y, p.z};
        uint32_t code = 0;
        for (int a = 0; a < 3; ++a) {
            const float span = fmaxf(hi[a] - lo[a], 1e-6f);
            float t = (x[a] - lo[a]) / span;
            t = t >= 0.0f ? fminf(t, 1.0f) : 0.0f;  // NaN (no bounds) -> 0
            code |= spreadBits10((uint32_t)(t * 1023.0f)) << a;
        }
        keys[k] = code;
        vals[k] = id;
    }
}

// Cluster of each giant-island body: its Morton rank chunked into `clusters`.
__global__ void clusterOfBodyKernel(const uint32_t* sortedIds, uint32_t nb, uint32_t clusters, uint32_t* clusterOf) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nb; r += gridDim.x * blockDim.x)
        clusterOf[sortedIds[r]] = (uint32_t)(((uint64_t)r * clusters) / nb);
}

VXD uint32_t segmentOf(const uint32_t* segStart, uint32_t g0, uint32_t g1, uint32_t k) {
    uint32_t lo = g0, hi = g1;  // last g with segStart[g] <= k
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (segStart[mid] <= k) lo = mid; else hi = mid;
    }
    return lo;
}

// Sort key of a giant row: its warp (the cluster of its first dynamic body),
// then its colour within its island. Rows of the null island (no dynamic body
// of their own island) have no links and go to any warp. Sorted rather than
// counted into a table of warps x colours: a body of 20,000 rows has as many
// colours, which made the table 0.6 GB.
__global__ void flowKeyKernel(SolveArgs A, const uint32_t* rowList, uint32_t R, const uint32_t* islandOf,
                              const uint32_t* clusterOf, uint32_t clusters, int colourBits, uint64_t* keys,
                              uint32_t* rows) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < R; t += gridDim.x * blockDim.x) {
        const uint32_t k = rowList[t], isl = islandOf[k];
        const uint32_t g0 = A.islandSeg[isl], g1 = A.islandSeg[isl + 1];
        uint32_t owner = k % clusters;
        if (isl < A.realIslands) {
            const vx_contact& c = A.contacts[A.order[k]];
            owner = clusterOf[isDynamic(A.B.filt[c.a].x) ? c.a : c.b];
        }
        keys[t] = (uint64_t)owner << colourBits | (segmentOf(A.segStart, g0, g1, k) - g0);
        rows[t] = k;
    }
}
// Colour and warp ranges of the sorted rows.
__global__ void flowStartKernel(const uint64_t* keys, uint32_t R, uint32_t clusters, int colourBits, uint32_t* colour,
                                uint32_t* start) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < R; t += gridDim.x * blockDim.x) {
        const uint64_t key = keys[t];
        colour[t] = (uint32_t)key & ((1u << colourBits) - 1u);
        const uint32_t w = (uint32_t)(key >> colourBits);
        for (uint32_t x = t ? (uint32_t)(keys[t - 1] >> colourBits) + 1u : 0u; x <= w; ++x) start[x] = t;
        if (t + 1 == R)
            for (uint32_t x = w + 1u; x <= clusters; ++x) start[x] = R;
    }
}

// The block kernel's complement among the islands above tinyLimit.
VXD bool isGiant(const SolveArgs& A, uint32_t isl) {
    const uint32_t rows = A.islandStart[isl + 1] - A.islandStart[isl];
    const uint32_t nb = isl < A.realIslands ? A.bodyStart[isl + 1] - A.bodyStart[isl] : 0u;
    return solveClassOf(nb, rows, A.tinyLimit) == kGiantIsland;
}

__global__ void giantEntryKernel(SolveArgs A, const uint32_t* islandOf, uint32_t m, uint32_t n, uint64_t* keys,
                                 uint32_t* vals) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const bool giant = isGiant(A, islandOf[k]);
        const vx_contact& c = A.contacts[A.order[k]];
        const uint32_t fa = A.B.filt[c.a].x, fb = A.B.filt[c.b].x;
        const bool solved = giant && solvedContact(fa, fb);
        keys[2 * k] = solved && isDynamic(fa) ? c.a : n;
        keys[2 * k + 1] = solved && isDynamic(fb) ? c.b : n;
        vals[2 * k] = 2 * k;
        vals[2 * k + 1] = 2 * k + 1;
    }
}

__global__ void coopTimeoutKernel(const CoopState* st, Counters* C) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && st->timeout) atomicOr(&C->timeout, 1u);
}

__global__ void giantListKernel(SolveArgs A, uint32_t* list, uint32_t* count) {
    for (uint32_t isl = blockIdx.x * blockDim.x + threadIdx.x; isl < A.islands; isl += gridDim.x * blockDim.x)
        if (isGiant(A, isl)) list[atomicAdd(count, 1u)] = isl;
}

// Giant-island membership of the sorted body positions and of the solve
// positions (flags for compaction), and the largest colour count of a giant.
__global__ void giantMemberKernel(SolveArgs A, const uint64_t* bodyKeys, uint32_t n, const uint32_t* islandOf,
                                  uint32_t m, uint32_t* bodyFlags, uint32_t* rowFlags, Counters* C) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const uint64_t isl = bodyKeys[k];
        bodyFlags[k] = isl < A.realIslands && isGiant(A, (uint32_t)isl) ? 1u : 0u;
    }
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += stride) {
        const uint32_t isl = islandOf[k];
        const bool g = isGiant(A, isl);
        rowFlags[k] = g ? 1u : 0u;
        if (g && k == A.islandStart[isl]) atomicMax(&C->clusterColours, A.islandSeg[isl + 1] - A.islandSeg[isl]);
    }
}

// Fallback when the device cannot run a cooperative grid: one block per giant island.
__global__ void __launch_bounds__(kGiantBlockThreads) solveGiantBlockKernel(SolveArgs A, const uint32_t* giants) {
    solveIslandGlobal(A, giants[blockIdx.x]);
}

// Bodies without contacts: the substep loop's integration only.
__global__ void freeBodiesKernel(BodyArrays B, const uint32_t* bodyOrder, uint32_t from, uint32_t to, V3 g, float h,
                                 int substeps) {
    for (uint32_t k = from + blockIdx.x * blockDim.x + threadIdx.x; k < to; k += gridDim.x * blockDim.x) {
        const uint32_t i = bodyOrder[k];
        for (int s = 0; s < substeps; ++s) {
            if (s > 0) integrateVelocity(B, i, g, h);
            integrateTransform(B, i, h);
        }
    }
}

// ---------------------------------------------------------------------------
// conservative-advancement rewind (src/world.cpp:4233-4357, gapAt :2916-2958)
// ---------------------------------------------------------------------------

VXD BodyView withPose(BodyView b, const V3& p, const Q4& q) {
    b.p = p;
    b.q = q;
    return b;
}

// Bounding spheres more than 1 mm apart give a positive end gap, so the
// rewind's `gap >= -8 mm` test skips the pair (planes, meshes and compounds
// have no bounding sphere here).
VXD bool spheresApart(const BodyView& a, const BodyView& b) {
    const float ea = coreExtent(shapeOf(a.flags), a.half, a.radius, a.hh);
    const float eb = coreExtent(shapeOf(b.flags), b.half, b.radius, b.hh);
    if (ea < 0.0f || eb < 0.0f) return false;
    const float reach = ea + eb + 1e-3f;
    return lengthSq(a.p - b.p) > reach * reach;
}

VXD Mass massOfView(const BodyArrays& B, uint32_t i) { return loadMass(B, i); }

// Conditions of the rewind loop for an oriented pair (a dynamic).
VXD bool caEligible(const BodyView& a, const BodyView& b, const BodyArrays& B, uint32_t ia) {
    if (isSensor(a.flags) || isSensor(b.flags)) return false;
    if (!isDynamic(a.flags)) return false;
    const float minVel = B.ccd[ia].y;
    if (!(a.flags & kContinuousBit) || qualityOf(a.flags) == kQualityLow || isLocked(a.flags) ||
        maxPointSpeed(a) < minVel)
        return false;
    return true;
}

VXD void orientPair(const BodyArrays& B, uint64_t key, uint32_t& i, uint32_t& j) {
    i = (uint32_t)(key >> 32);
    j = (uint32_t)key;
    if (!isDynamic(B.filt[i].x) && isDynamic(B.filt[j].x)) { const uint32_t t = i; i = j; j = t; }
}

// The probe: end-state gap of every pair, one thread each; pairs whose query
// overlaps (or that involve a mesh or compound) are listed in `hard` for
// caProbeHardKernel. `order` (optional): the pairs grouped by shape
// combination, so that a warp's lanes mostly take the same distance-query
// path; every outcome is written at the pair's own index.
VXD void caFlag(const BodyArrays& B, uint32_t r, uint32_t i, uint32_t j, uint32_t flagsB, const GapProbe& end,
                uint32_t* flags, uint32_t* bodyMark, float4* endGap) {
    uint32_t flag = 0;
    if (end.gap < -8e-3f) {
        flag = 1;
        endGap[r] = make_float4(end.gap, end.normal.x, end.normal.y, end.normal.z);
        bodyMark[i] = 1;  // only dynamic bodies move in a rewind
        if (isDynamic(flagsB)) bodyMark[j] = 1;
    }
    flags[r] = flag;
}

__global__ void caProbeKernel(BodyArrays B, Soup soup, const uint64_t* pairKeys, const uint32_t* order,
                              uint32_t npairs, uint32_t* flags, uint32_t* bodyMark, float4* endGap, uint32_t* hard,
                              Counters* C) {
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < npairs; slot += gridDim.x * blockDim.x) {
        const uint32_t r = order ? order[slot] : slot;
        uint32_t i, j;
        orientPair(B, pairKeys[r], i, j);
        const BodyView a = loadView(B, i), b = loadView(B, j);
        GapProbe end{0.0f, V3{0.0f, 0.0f, 0.0f}};
        bool later = false;
        if (!spheresApart(a, b) && caEligible(a, b, B, i)) {
            if (isComplexShape(shapeOf(a.flags)) || isComplexShape(shapeOf(b.flags))) {
                later = true;
            } else if (shapeOf(b.flags) == kPlane) {
                const Convex c = makeConvex(a, soup);
                const V3 deep = c.position + supportOffsetBody(c, -b.planeN);
                end = GapProbe{dot(b.planeN, deep) - b.planeOff - c.radius, b.planeN};
            } else {
                GjkResult g;
                Simplex s;
                later = gjkDistanceFast(makeConvex(a, soup), makeConvex(b, soup), g, s) != kGjkSeparated;
                if (!later) end = GapProbe{g.distance, g.normal};
            }
        }
        if (later) hard[aggregatedSlot(&C->caHard)] = r;
        else caFlag(B, r, i, j, b.flags, end, flags, bodyMark, endGap);
    }
}

// The listed convex pairs of Robust and Paranoid bodies, a thread each.
__global__ void caProbeGeneralKernel(BodyArrays B, Soup soup, const uint64_t* pairKeys, const uint32_t* hard,
                                     uint32_t* flags, uint32_t* bodyMark, float4* endGap, const Counters* C) {
    const uint32_t count = C->caHard;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const uint32_t r = hard[k];
        uint32_t i, j;
        orientPair(B, pairKeys[r], i, j);
        const BodyView a = loadView(B, i), b = loadView(B, j);
        if (!threadPair(count, a.flags, b.flags) || isComplexShape(shapeOf(a.flags)) || isComplexShape(shapeOf(b.flags)))
            continue;
        const GjkResult g = gjkDistance(makeConvex(a, soup), makeConvex(b, soup));
        caFlag(B, r, i, j, b.flags, GapProbe{g.distance, g.normal}, flags, bodyMark, endGap);
    }
}

__global__ void __launch_bounds__(kQueryThreads) caProbeHardKernel(BodyArrays B, Soup soup, const uint64_t* pairKeys,
                                                                   const uint32_t* hard, float dt, uint32_t* flags,
                                                                   uint32_t* bodyMark, float4* endGap,
                                                                   const Counters* C) {
    const uint32_t count = C->caHard, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count; k += warps) {
        const uint32_t r = hard[k];
        uint32_t i, j;
        orientPair(B, pairKeys[r], i, j);
        const BodyView a = loadView(B, i), b = loadView(B, j);
        if (threadPair(count, a.flags, b.flags) && !isComplexShape(shapeOf(a.flags)) && !isComplexShape(shapeOf(b.flags)))
            continue;  // caProbeGeneralKernel
        const GapProbe end = gapAtWarp(a, b, soup, dt);
        if (warpLane() == 0u) caFlag(B, r, i, j, b.flags, end, flags, bodyMark, endGap);
        __syncwarp();
    }
}

__global__ void caCandidateKernel(const BodyArrays B, const uint64_t* pairKeys, uint32_t npairs, uint32_t* flags,
                                  const uint32_t* bodyMark, uint32_t* candidates, Counters* C) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < npairs; r += gridDim.x * blockDim.x) {
        const uint32_t i = (uint32_t)(pairKeys[r] >> 32), j = (uint32_t)pairKeys[r];
        if (flags[r] || bodyMark[i] || bodyMark[j]) candidates[r] = 1;
        else candidates[r] = 0;
    }
}

VXD Q4 orientationAt(const Mass& m, const Q4& start, const V3& L, float elapsed) {
    Q4 q = start;
    V3 w = invInertiaMulAt(m, L, start);
    advanceOrientation(m, q, w, elapsed);
    return q;
}

// Full rewind logic for one oriented pair on the current state, by one warp.
// Returns true when the pair was rewound.
// `cached`: the probe's end-state gap for this pair when neither body has
// moved since the probe (else null: computed here). `spec` (optional): write
// the rewound states there (a: pos, rot, vel, ang; then b) instead of into B.
__device__ __noinline__ bool caRewind(BodyArrays& B, const Soup& soup, uint32_t i, uint32_t j, float dt,
                                      const float4* prevPos, const float4* prevRot, uint32_t* gapQueries,
                                      const float4* cached, float4* spec = nullptr) {
    BodyView a = loadViewCoherent(B, i), b = loadViewCoherent(B, j);
    if (!caEligible(a, b, B, i)) return false;
    if (spheresApart(a, b)) return false;  // positive end gap, no rewind (the probe's test)
    GapProbe end;
    if (cached) {
        const float4 g = *cached;
        end = GapProbe{g.x, V3{g.y, g.z, g.w}};
    } else {
        end = gapAtWarp(a, b, soup, dt);
    }
    if (end.gap >= -8e-3f) return false;
    const bool bStatic = isStaticBody(b.flags), bDyn = isDynamic(b.flags);
    const V3 pa0 = f3(prevPos[i]), da = a.p - pa0;
    const Q4 qa0 = q4(prevRot[i]);
    const V3 pb0 = bStatic ? b.p : f3(prevPos[j]);
    const V3 db = b.p - pb0;
    const Q4 qb0 = bStatic ? b.q : q4(prevRot[j]);
    const float bound = maxPointSpeed(a) * dt + (bStatic ? 0.0f : maxPointSpeed(b) * dt);
    if (bound < 1e-9f) return false;
    const Mass ma = loadMass(B, i), mb = loadMass(B, j);
    const V3 La = inertiaMulAt(ma, a.w, a.q);
    const V3 Lb = bDyn ? inertiaMulAt(mb, b.w, b.q) : V3{0.0f, 0.0f, 0.0f};
    float t = 0.0f;
    V3 n = end.normal;
    uint32_t queries = 1;
    for (int iter = 0; iter < 24 && t < 1.0f; ++iter) {
        ++queries;
        const Q4 qa = orientationAt(ma, qa0, La, dt * t);
        const Q4 qb = bStatic ? qb0 : orientationAt(mb, qb0, Lb, dt * t);
        const GapProbe g = gapAtWarp(withPose(a, pa0 + da * t, qa), withPose(b, pb0 + db * t, qb), soup, dt);
        n = g.normal;
        if (g.gap < 1e-3f) break;
        t = vmin(1.0f, t + g.gap / bound);
    }
    if (warpLane() == 0u) atomicAdd(gapQueries, queries);
    if (t >= 1.0f) return false;
    a.p = pa0 + da * t;
    a.q = qa0;
    a.w = invInertiaMulAt(ma, La, qa0);
    advanceOrientation(ma, a.q, a.w, dt * t);
    if (bDyn) {
        b.p = pb0 + db * t;
        b.q = qb0;
        b.w = invInertiaMulAt(mb, Lb, qb0);
        advanceOrientation(mb, b.q, b.w, dt * t);
    }
    const float ima = solverInvMass(ma), imb = solverInvMass(mb);
    const float vn = dot(a.v - b.v, n);
    const float invMassSum = ima + imb;
    if (vn < 0.0f && invMassSum > 0.0f) {
        const float restitution = vn < -1.0f
            ? combineMaterial(a.restitution, b.restitution, (a.flags >> kRestitutionCombineShift) & 7u,
                              (b.flags >> kRestitutionCombineShift) & 7u)
            : 0.0f;
        const float impulse = -(1.0f + restitution) * vn / invMassSum;
        a.v += n * (impulse * ima);
        if (bDyn) b.v -= n * (impulse * imb);
    }
    const float remaining = dt * (1.0f - t);
    advanceTransform(ma, a.p, a.q, a.v, a.w, remaining);
    if (bDyn) advanceTransform(mb, b.p, b.q, b.v, b.w, remaining);
    if (warpLane() != 0u) return true;
    if (spec) {
        spec[0] = pack(a.p, 0.0f); spec[1] = pack(a.q); spec[2] = pack(a.v, 0.0f); spec[3] = pack(a.w, 0.0f);
        spec[4] = pack(b.p, 0.0f); spec[5] = pack(b.q); spec[6] = pack(b.v, 0.0f); spec[7] = pack(b.w, 0.0f);
        return true;
    }
    B.pos[i] = pack(a.p, 0.0f); B.rot[i] = pack(a.q); B.vel[i] = pack(a.v, 0.0f); B.ang[i] = pack(a.w, 0.0f);
    if (bDyn) {
        B.pos[j] = pack(b.p, 0.0f); B.rot[j] = pack(b.q); B.vel[j] = pack(b.v, 0.0f); B.ang[j] = pack(b.w, 0.0f);
    }
    return true;
}

VXD uint64_t globalTimerNs() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every flagged pair evaluated in parallel on the probe's state (read-only):
// in the ordered pass, a flagged pair whose bodies no earlier rewind has moved
// sees exactly this state, so its outcome can be taken from here. A warp per
// pair: up to 25 dependent distance queries.
__global__ void __launch_bounds__(kQueryThreads) caSpeculateKernel(BodyArrays B, Soup soup, const uint64_t* pairKeys,
                                                                   const uint32_t* flaggedList, uint32_t flagged,
                                                                   const float4* endGap, float dt,
                                                                   const float4* prevPos, const float4* prevRot,
                                                                   float4* specState, uint32_t* specResult,
                                                                   Counters* C) {
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < flagged; k += warps) {
        const uint32_t r = flaggedList[k];
        uint32_t i, j;
        orientPair(B, pairKeys[r], i, j);
        const uint64_t t0 = globalTimerNs();
        const bool moved = caRewind(B, soup, i, j, dt, prevPos, prevRot, &C->caGapQueries, endGap + r,
                                    specState + 8 * (size_t)k);
        if (warpLane() == 0u) {
            specResult[k] = moved ? 1u : 0u;
            atomicMax(&C->caSpecMicros, (uint32_t)((globalTimerNs() - t0) / 1000u));
        }
        __syncwarp();
    }
}

// Rewind pass over the candidate pairs as a dataflow. A candidate's
// predecessors are the latest earlier candidates sharing one of its dynamic
// bodies; it becomes ready when both have finished and is then evaluated
// exactly as the reference's single ordered loop would evaluate it: it sees
// the same body states and rewound marks, as long as no rewind moves a body
// outside the marked set (that case is flagged; the caller widens the set and
// replays the pass from a snapshot). Workers (warps) take ready candidates
// from a queue, so independent chains never wait for one another; a worker
// goes on with a successor that it made ready, so a chain passes through the
// queue only where it forks. Cooperative launch (all workers resident); every
// wait is bounded.
//
// What bounds it: the longest chain of evaluations, each up to 25 dependent
// distance queries, and about 2.7 us a link where nothing is evaluated. Workers
// were one lane per SM, whose queries kept 10 KB stack frames in local memory
// (more lanes per SM evicted one another's); a warp keeps its polytope in
// shared memory and shares the scans. Rewind stage of one step: 7.2 -> 1.4 ms
// with 2,500 bodies on a mesh, 9.2 -> 6.6 ms in a heap of 40,000, 8.8 -> 6.5 ms
// among 1,000 tumbling boxes. One, two or four blocks of workers per SM: the
// same times (the chain binds).
constexpr int kCaWidenLimit = 8;  // replays with a widened marked set before the serial loop
constexpr uint32_t kProbeGroupMin = 8192;  // pairs from which the probe groups them by shape combination
constexpr int kCaWidenHops = 8;   // hops of widening per replay
constexpr int kCaInitialHops = 8; // hops of widening before the first pass
constexpr int kCaFlowBlocksPerSm = 2;

__global__ void __launch_bounds__(kQueryThreads) caFlowKernel(BodyArrays B, Soup soup, const uint32_t* flagRank,
                                                    const float4* specState, const uint32_t* specResult,
                                                    const uint4* info, uint32_t ncand, const uint32_t* succ,
                                                    uint32_t* pending, uint32_t* queue, uint32_t* depth,
                                                    uint32_t* crit, const uint32_t* bodyMark, uint32_t* rewound,
                                                    float dt, const float4* prevPos, const float4* prevRot,
                                                    Counters* C, CoopState* st) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    uint32_t* tail = &st->queued[0];
    uint32_t* head = &st->queued[1];
    uint32_t* finished = &st->queued[2];  // candidates done, added when a worker's chain ends
    for (uint32_t k = tid; k < ncand; k += stride)  // roots
        if (pending[k] == 0u) {
            const uint32_t t = atomicAdd(tail, 1u);
            if (t < ncand) __stcg(queue + t, k);
            else atomicOr(&st->spill, 4u);  // pushed twice: inconsistent links
        }
    // Every root is queued before any worker starts: a count that a finished
    // candidate has taken to zero must not read as a root.
    if (!gridSync(&st->bar, &st->timeout, st->spinLimit)) return;
    const bool lead = warpLane() == 0u;
    uint32_t rewinds = 0, maxDepth = 0, maxCrit = 0, mine = 0, k = kNoPred;
    for (;;) {
        if (k == kNoPred) {  // the chain ended: claim a queue slot and wait for it to be filled
            if (lead) {
                if (mine) atomicAdd(finished, mine);
                const uint32_t h = atomicAdd(head, 1u);
                // Idle workers back off (up to ~1 us) and read the shared words
                // only every 8th poll: polling them at full rate slows the
                // working warps' own loads.
                uint32_t spins = 0, nap = 32;
                while (h < ncand && (k = __ldcg(queue + h)) == kNoPred) {
                    if (++spins > st->spinLimit) atomicOr(&st->timeout, 1u);
                    if ((spins & 7u) == 0u && (__ldcg(finished) >= ncand || __ldcg(&st->timeout))) break;
                    __nanosleep(nap);
                    if (nap < 1024u) nap <<= 1;
                }
            }
            mine = 0;
            k = __shfl_sync(kFullWarp, k, 0);
            if (k == kNoPred) break;
        }
        if (lead) __threadfence();  // acquire the predecessors' writes
        __syncwarp();
        const uint64_t t0 = globalTimerNs();
        // record, successors and chain statistics in one round of loads (the
        // predecessors raised depth and crit before they released this one)
        const uint4 rec = info[k];
        const uint2 next = reinterpret_cast<const uint2*>(succ)[k];
        const uint32_t d = __ldcg(depth + k) + 1u;
        const uint32_t crit0 = __ldcg(crit + k);
        const uint32_t i = rec.y, j = rec.z;
        const bool jDyn = (rec.w & 2u) != 0u;
        const uint32_t seen = __ldcg(rewound + i) | __ldcg(rewound + j);
        const bool touched = __shfl_sync(kFullWarp, seen, 0) != 0u;
        if ((rec.w & 1u) || touched) {
            bool rewoundPair;
            if (!touched) {  // flagged, bodies as the probe saw them: the speculative outcome holds
                const uint32_t sk = flagRank[rec.x];
                rewoundPair = specResult[sk] != 0u;
                if (rewoundPair && warpLane() < (jDyn ? 8u : 4u)) {
                    const uint32_t lane = warpLane(), id = lane < 4u ? i : j;
                    float4* to = (lane & 3u) == 0u ? B.pos : (lane & 3u) == 1u ? B.rot : (lane & 3u) == 2u ? B.vel : B.ang;
                    __stcg(to + id, specState[8 * (size_t)sk + lane]);
                }
            } else {
                rewoundPair = caRewind(B, soup, i, j, dt, prevPos, prevRot, &C->caGapQueries, nullptr);
            }
            if (rewoundPair) {
                ++rewinds;
                if (lead) {
                    __stcg(rewound + i, 1u);
                    if (jDyn) __stcg(rewound + j, 1u);
                    if (!bodyMark[i] || (jDyn && !bodyMark[j])) atomicOr(&C->caOverflow, 1u);
                }
            }
        }
        const uint64_t elapsed = globalTimerNs() - t0;
        const uint32_t ck = crit0 + (uint32_t)(elapsed < 0x7fffffffull ? elapsed : 0x7fffffffull);
        maxDepth = max(maxDepth, d);
        maxCrit = max(maxCrit, ck);
        ++mine;
        k = kNoPred;
        __syncwarp();
        if (lead) {
            __threadfence();  // release this evaluation's writes before the successors can run
            // both successors' counts drop in one round; a count that reaches
            // zero makes its candidate ready (the same one twice only if it
            // follows this one on both bodies, and then only the second drop
            // reaches zero)
            uint32_t left0 = 0u, left1 = 0u;
            if (next.x != kNoPred) {
                atomicMax(depth + next.x, d);
                atomicMax(crit + next.x, ck);
                left0 = atomicSub(pending + next.x, 1u);
            }
            if (next.y != kNoPred) {
                atomicMax(depth + next.y, d);
                atomicMax(crit + next.y, ck);
                left1 = atomicSub(pending + next.y, 1u);
            }
            k = left0 == 1u ? next.x : left1 == 1u ? next.y : kNoPred;
            if (left0 == 1u && left1 == 1u) {
                const uint32_t t = atomicAdd(tail, 1u);
                if (t < ncand) __stcg(queue + t, next.y);
                else atomicOr(&st->spill, 4u);
            }
        }
        k = __shfl_sync(kFullWarp, k, 0);
    }
    if (!lead) return;
    if (rewinds) atomicAdd(&C->rewinds, rewinds);
    atomicMax(&st->rounds, maxDepth);
    atomicMax(&C->caCritMicros, maxCrit / 1000u);
}

// Entries (dynamic body, 2k + side) of the candidates; other endpoints sort last.
// Also the candidate's record for the pass: (pair, oriented bodies i and j,
// bit 0 flagged by the probe | bit 1 j dynamic), one load for the worker.
__global__ void caEntryKernel(const BodyArrays B, const uint64_t* pairKeys, const uint32_t* cand, uint32_t ncand,
                              uint32_t n, const uint32_t* flags, uint64_t* keys, uint32_t* vals, uint4* info) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < ncand; k += gridDim.x * blockDim.x) {
        const uint32_t r = cand[k];
        const uint64_t key = pairKeys[r];
        const uint32_t a = (uint32_t)(key >> 32), b = (uint32_t)key;
        keys[2 * k] = isDynamic(B.filt[a].x) ? a : n;
        keys[2 * k + 1] = isDynamic(B.filt[b].x) ? b : n;
        vals[2 * k] = 2 * k;
        vals[2 * k + 1] = 2 * k + 1;
        uint32_t i, j;
        orientPair(B, key, i, j);
        info[k] = make_uint4(r, i, j, (flags[r] ? 1u : 0u) | (isDynamic(B.filt[j].x) ? 2u : 0u));
    }
}

// Entries sorted stably by body: consecutive entries of one body link a
// candidate to its successor on that body (pending counts its predecessors).
__global__ void caLinkKernel(const uint64_t* keys, const uint32_t* vals, uint32_t entries, uint32_t n,
                             uint32_t* succ, uint32_t* pending) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < entries; p += gridDim.x * blockDim.x) {
        const uint64_t key = keys[p];
        const bool body = key != (uint64_t)n;
        const bool next = body && p + 1 < entries && keys[p + 1] == key;
        succ[vals[p]] = next ? (vals[p + 1] >> 1) : kNoPred;
        if (body && p > 0 && keys[p - 1] == key) atomicAdd(pending + (vals[p] >> 1), 1u);
    }
}

// Widen the marked set after a failed pass, one hop per launch: both dynamic
// endpoints of every pair touching a frontier body (the first frontier is
// the set of bodies the pass rewound); bodies marked here form the next one.
// Marking ahead of the cascade means fewer replays.
__global__ void caWidenKernel(const BodyArrays B, const uint64_t* pairKeys, uint32_t npairs, uint32_t* bodyMark,
                              const uint32_t* frontier, uint32_t* next) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < npairs; r += gridDim.x * blockDim.x) {
        const uint32_t i = (uint32_t)(pairKeys[r] >> 32), j = (uint32_t)pairKeys[r];
        if (!frontier[i] && !frontier[j]) continue;
        if (isDynamic(B.filt[i].x) && atomicExch(bodyMark + i, 1u) == 0u) next[i] = 1u;
        if (isDynamic(B.filt[j].x) && atomicExch(bodyMark + j, 1u) == 0u) next[j] = 1u;
    }
}

// The reference's loop verbatim in pair order (one warp): the fallback when
// a rewind cascades beyond the candidate neighbourhood.
__global__ void __launch_bounds__(32) caFullSerialKernel(BodyArrays B, Soup soup, const uint64_t* pairKeys, uint32_t npairs,
                                   const uint32_t* flags, uint32_t* rewound, float dt, const float4* prevPos,
                                   const float4* prevRot, Counters* C) {
    uint32_t rewinds = 0;
    for (uint32_t r = 0; r < npairs; ++r) {
        const uint64_t key = pairKeys[r];
        const uint32_t ri = (uint32_t)(key >> 32), rj = (uint32_t)key;
        if (!(flags[r] || __ldcg(rewound + ri) || __ldcg(rewound + rj))) continue;
        uint32_t i, j;
        orientPair(B, key, i, j);
        if (caRewind(B, soup, i, j, dt, prevPos, prevRot, &C->caGapQueries, nullptr)) {
            ++rewinds;
            if (threadIdx.x == 0) {
                __stcg(rewound + i, 1u);
                if (isDynamic(B.filt[j].x)) __stcg(rewound + j, 1u);
                __threadfence();
            }
        }
        __syncwarp();
    }
    if (threadIdx.x == 0) C->rewinds = rewinds;
}

__global__ void copyStateKernel(const BodyArrays B, uint32_t n, float4* snap, int restore) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4* s = snap + 4 * (size_t)i;
        if (restore) {
            B.pos[i] = s[0]; B.rot[i] = s[1]; B.vel[i] = s[2]; B.ang[i] = s[3];
        } else {
            s[0] = B.pos[i]; s[1] = B.rot[i]; s[2] = B.vel[i]; s[3] = B.ang[i];
        }
    }
}

// prefix ranks of candidate flags -> candidate index list
__global__ void compactKernel(const uint32_t* flags, const uint32_t* ranks, uint32_t n, uint32_t* out) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        if (flags[k]) out[ranks[k]] = k;
}

__global__ void clearForcesKernel(BodyArrays B, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        B.force[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        B.torque[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

__global__ void gatherContactsKernel(const vx_contact* in, const uint32_t* order, uint32_t m, vx_contact* out) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        out[k] = in[order[k]];
}

__global__ void contactKeysKernel(const vx_contact* cs, uint32_t m, uint64_t* keys) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        keys[k] = ((uint64_t)cs[k].a << 32) | cs[k].b;
}

// ===========================================================================
// host orchestration
// ===========================================================================

int sortPairs(Context& c, uint64_t* keys, uint32_t* vals, uint32_t n, int bits) {
    if (n <= 1 || bits <= 0) return VXB_OK;
    const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
    VXB_TRY(ensure(c, c.sortKeysAlt, (size_t)n * 8));
    VXB_TRY(ensure(c, c.sortValsAlt, (size_t)n * 4));
    VXB_TRY(ensure(c, c.sortHist, (size_t)tiles * 256 * 4));
    c.sortScratch.keysAlt = P<uint64_t>(c.sortKeysAlt);
    c.sortScratch.valsAlt = P<uint32_t>(c.sortValsAlt);
    c.sortScratch.hist = P<uint32_t>(c.sortHist);
    cudaError_t e = cudaSuccess;
    c.launches += radixSortPairs(keys, vals, n, 0, bits, c.sortScratch, c.stream, &e);
    if (e != cudaSuccess) return cudaStatus(c, e, "radix sort");
    return VXB_OK;
}

// Union-find roots (parent[i] = the root of i) over the dynamic-dynamic
// contacts of `cs` that involve no sensor (the islands of SleepManager::update,
// src/sleep.cpp:63-91, and of the solve).
int unionRoots(Context& c, const vx_contact* cs, uint32_t m, uint32_t* parent) {
    LAUNCH(c, iotaKernel, blocksFor(c.n, 256), 256, parent, c.n);
    if (m) {
        LAUNCH(c, unionKernel, blocksFor(m, 256), 256, cs, m, c.B, parent, c.dCounters);
        LAUNCH(c, compressKernel, blocksFor(c.n, 256), 256, parent, c.n);
    }
    return VXB_OK;
}

int resetCoop(Context& c, CoopState* st) {
    CoopState init;
    std::memset(&init, 0, sizeof(init));
    init.spinLimit = c.waitLimit;
    VXB_CUDA(c, cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, c.stream));
    return VXB_OK;
}

static int readCounters(Context& c) {
    VXB_CUDA(c, cudaMemcpyAsync(&c.hostCounters, c.dCounters, sizeof(Counters), cudaMemcpyDeviceToHost, c.stream));
    ++c.hostSyncs;
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

// Launch at a tuned site (tuner.h): `launch(shape)` issues the kernel with
// that block size and grid cap. While the size bucket of `items` has no shape,
// every candidate first runs on the same inputs, `restore()` putting back what
// a launch consumes before each trial and before the real launch.
template <class Launch, class Restore>
static int tunedLaunch(Context& c, int site, uint32_t items, Launch launch, Restore restore) {
    if (c.tuner.undecided(site, items)) {
        c.tuner.beginTrials();
        for (int round = 0; round < kTuneSamples; ++round)
            for (int k = 0; k < kTuneCandidates; ++k) {
                VXB_TRY(restore());
                c.tuner.trialStart(c.stream);
                launch(Tuner::candidate(site, k));
                ++c.hostSyncs;
                const cudaError_t e = c.tuner.trialStop(k, c.stream);
                if (e != cudaSuccess) return cudaStatus(c, e, "launch-shape trial");
            }
        c.tuner.decide(site, items);
        VXB_TRY(restore());
    }
    launch(c.tuner.shapeFor(site, items, nullptr));
    return VXB_OK;
}

// Restores the device counters a narrow-phase launch appends to (contacts,
// records, overflow flags): the first call keeps a device copy, later calls
// put it back.
struct CounterRestore {
    Context& c;
    bool saved = false;
    int operator()() {
        if (!saved) {
            VXB_TRY(ensure(c, c.tuneSaveBuf, sizeof(Counters)));
            VXB_CUDA(c, cudaMemcpyAsync(c.tuneSaveBuf.ptr, c.dCounters, sizeof(Counters), cudaMemcpyDeviceToDevice,
                                        c.stream));
            saved = true;
            return VXB_OK;
        }
        VXB_CUDA(c, cudaMemcpyAsync(c.dCounters, c.tuneSaveBuf.ptr, sizeof(Counters), cudaMemcpyDeviceToDevice,
                                    c.stream));
        return VXB_OK;
    }
};

static int resetCounters(Context& c) {
    Counters z;
    std::memset(&z, 0, sizeof(z));
    for (int a = 0; a < 3; ++a) { z.cellMinBits[a] = 0xffffffffu; z.cellMaxBits[a] = 0u; }
    VXB_CUDA(c, cudaMemcpyAsync(c.dCounters, &z, sizeof(Counters), cudaMemcpyHostToDevice, c.stream));
    return VXB_OK;
}

static uint64_t fnv1a(uint64_t h, const void* data, size_t bytes) {
    const unsigned char* p = static_cast<const unsigned char*>(data);
    for (size_t k = 0; k < bytes; ++k) h = (h ^ p[k]) * 0x100000001b3ull;
    return h;
}

int loadSoup(Context& c, const vx_soup* soup) {
    c.hullPointCount = soup ? soup->hullPointCount : 0;
    c.faceIndexCount = soup ? soup->hullFaceIndexCount : 0;
    VXB_TRY(ensure(c, c.hullPtsBuf, c.hullPointCount * 12 + 16));
    VXB_TRY(ensure(c, c.facesBuf, c.faceIndexCount * 4 + 16));
    if (c.hullPointCount)
        VXB_CUDA(c, cudaMemcpyAsync(c.hullPtsBuf.ptr, soup->hullPoints, c.hullPointCount * 12, cudaMemcpyHostToDevice,
                                    c.stream));
    if (c.faceIndexCount)
        VXB_CUDA(c, cudaMemcpyAsync(c.facesBuf.ptr, soup->hullFaceIndices, c.faceIndexCount * 4,
                                    cudaMemcpyHostToDevice, c.stream));
    // triangle meshes, their BVHs and compound children
    struct Part { DevBuf* buf; const void* src; size_t bytes; };
    const Part parts[] = {
        {&c.vertBuf, soup ? soup->vertices : nullptr, soup ? (size_t)soup->vertexCount * 12 : 0},
        {&c.indexBuf, soup ? soup->indices : nullptr, soup ? (size_t)soup->indexCount * 4 : 0},
        {&c.meshBuf, soup ? soup->meshes : nullptr, soup ? (size_t)soup->meshCount * sizeof(vx_mesh) : 0},
        {&c.nodeBuf, soup ? soup->bvhNodes : nullptr, soup ? (size_t)soup->bvhNodeCount * sizeof(vx_bvh_node) : 0},
        {&c.triRefBuf, soup ? soup->bvhTriRefs : nullptr, soup ? (size_t)soup->bvhTriRefCount * 4 : 0},
        {&c.childBuf, soup ? soup->compoundChildren : nullptr,
         soup ? (size_t)soup->compoundChildCount * sizeof(vx_compound_child) : 0}};
    for (const Part& part : parts) {
        VXB_TRY(ensure(c, *part.buf, part.bytes + 16));
        if (part.bytes)
            VXB_CUDA(c, cudaMemcpyAsync(part.buf->ptr, part.src, part.bytes, cudaMemcpyHostToDevice, c.stream));
    }
    if (soup && soup->meshCount) VXB_CUDA(c, cudaStreamSynchronize(c.stream));  // copies read the caller's arrays
    uint64_t key = 0xcbf29ce484222325ull;
    for (const Part& part : parts) key = fnv1a(key, &part.bytes, sizeof(part.bytes));
    const size_t hull[2] = {c.hullPointCount, c.faceIndexCount};
    c.soupGeometryKey = fnv1a(key, hull, sizeof(hull));
    return VXB_OK;
}

static Soup soupOf(Context& c) {
    return Soup{P<float>(c.hullPtsBuf), P<uint32_t>(c.facesBuf),  P<float>(c.vertBuf),
                P<uint32_t>(c.indexBuf), P<vx_mesh>(c.meshBuf),    P<vx_bvh_node>(c.nodeBuf),
                P<uint32_t>(c.triRefBuf), P<vx_compound_child>(c.childBuf)};
}

// What grows with the contacts of a world's first steps: the rows' planes and the
// listed pairs for two a body, the island plan and the rewind for fewer. Each was
// freed and allocated a dozen times on the way (4,096 worlds from rest, 60 steps:
// 170 allocations and 299 ms -> 27 and 279; a free now and then takes tens of ms
// more). Asked for, not required: a world that fits the device without it loads
// and steps. A small world's buffers grow from one small block to the next, and
// ten allocations would double its load (3,000 bodies 2 -> 4 ms).
constexpr uint32_t kReserveBodies = 16384;
static void reserve(Context& c, uint32_t n) {
    if (n < kReserveBodies) return;
    const size_t half = n / 2, few = n / 16;
    const struct {
        DevBuf* buf;
        size_t bytes;
    } later[] = {{&c.planeBuf, 4 * half * kRowPlaneBytes},
                 {&c.hardBuf, 4 * half * (4 + sizeof(HardResult))},
                 {&c.caFlagBuf, 2 * half * 28},
                 {&c.caCandBuf, 2 * half * 28},
                 {&c.islandBodyStartBuf, half * 4},
                 {&c.tinyBuf, half * 17},
                 {&c.tinyKeyBuf, half * 8},
                 {&c.caSpecBuf, few * 136},
                 {&c.islandInfoBuf, few * 24},
                 {&c.caInfoBuf, few * 16}};
    size_t free = 0, total = 0;
    for (const auto& r : later) {
        if (r.bytes <= r.buf->bytes) continue;
        if (!total && cudaMemGetInfo(&free, &total) != cudaSuccess) return;
        if (r.bytes > free / 8) continue;  // an eighth of what is free at most
        const std::string last = c.lastError;
        if (ensure(c, *r.buf, r.bytes) != VXB_OK) c.lastError = last;
    }
}

int loadBodies(Context& c, const vx_body* bodies, uint32_t n, const uint32_t* worldOf, bool deviceWorld) {
    if (n == 0) return fail(c, VXB_ERR_INVALID, "no bodies");
    // The Backend path reloads the same bodies between its calls of one step
    // (integrate between substeps' solves): the coloured contacts stay valid
    // unless the body set changed.
    if (n != c.n) {
        c.backendContacts = 0;
        c.backendColored = false;
    }
    bool threads = false;
    c.kinematic = false;
    uint64_t key = 0xcbf29ce484222325ull;
    for (uint32_t i = 0; i < n; ++i) {
        const vx_body& b = bodies[i];
        const uint32_t refs[6] = {b.shape, b.meshIndex, b.hullFirst, b.hullCount, b.compoundFirst, b.compoundCount};
        key = fnv1a(key, refs, sizeof(refs));
        key = fnv1a(key, &b.hullFaceFirst, 8);  // hullFaceFirst, hullFaceCount
    }
    c.bodyGeometryKey = key;
    for (uint32_t i = 0; i < n; ++i) {
        const uint8_t s = bodies[i].shape;
        if ((bodies[i].geometryQuality & 3u) || s == VX_SHAPE_COMPOUND) threads = true;
        if (s == VX_SHAPE_MESH && bodies[i].motionType != VX_MOTION_STATIC)
            return fail(c, VXB_ERR_INVALID, "mesh bodies are static");
        if (deviceWorld && bodies[i].motionType == VX_MOTION_KINEMATIC)
            return fail(c, VXB_ERR_UNSUPPORTED, "kinematic bodies are not supported by the device world");
        if (bodies[i].motionType == VX_MOTION_KINEMATIC) c.kinematic = true;
    }
    c.threadShapes = threads;
    c.n = n;
    // SoA arrays in one allocation (16 arrays of 16-byte elements).
    const size_t stride = ((size_t)n * 16 + 255) & ~(size_t)255;
    VXB_TRY(ensure(c, c.bodyBuf, stride * 16));
    char* base = P<char>(c.bodyBuf);
    float4** f4[] = {&c.B.pos, &c.B.rot, &c.B.vel, &c.B.ang, &c.B.inertia, &c.B.iq, &c.B.dims, &c.B.extra,
                     &c.B.mat, &c.B.fscale, &c.B.ccd, &c.B.plane, &c.B.force, &c.B.torque};
    int slot = 0;
    for (float4** p : f4) *p = reinterpret_cast<float4*>(base + stride * slot++);
    c.B.hull = reinterpret_cast<uint4*>(base + stride * slot++);
    c.B.filt = reinterpret_cast<uint4*>(base + stride * slot++);
    VXB_TRY(ensure(c, c.aosBuf, (size_t)n * sizeof(vx_body)));
    VXB_CUDA(c, cudaMemcpyAsync(c.aosBuf.ptr, bodies, (size_t)n * sizeof(vx_body), cudaMemcpyHostToDevice, c.stream));
    LAUNCH(c, packBodiesKernel, blocksFor(n, 256), 256, P<vx_body>(c.aosBuf), n, c.B);
    // worlds and per-world lists of planes and meshes (paired with every body of their world)
    c.hostWorldOf.assign(n, 0u);
    uint32_t worlds = 1;
    if (worldOf) {
        for (uint32_t i = 0; i < n; ++i) {
            c.hostWorldOf[i] = worldOf[i];
            if (i > 0 && worldOf[i] < worldOf[i - 1])
                return fail(c, VXB_ERR_INVALID, "bodies of one world must be contiguous and worlds ascending");
            worlds = std::max(worlds, worldOf[i] + 1);
        }
    }
    c.worlds = worlds;
    std::vector<uint32_t> planeStart(worlds + 1, 0), planeList;
    auto boundless = [&](uint32_t i) { return bodies[i].shape == VX_SHAPE_PLANE || bodies[i].shape == VX_SHAPE_MESH; };
    for (uint32_t i = 0; i < n; ++i)
        if (boundless(i)) ++planeStart[c.hostWorldOf[i] + 1];
    for (uint32_t w = 0; w < worlds; ++w) planeStart[w + 1] += planeStart[w];
    planeList.resize(planeStart[worlds]);
    {
        std::vector<uint32_t> fill(planeStart.begin(), planeStart.end() - 1);
        for (uint32_t i = 0; i < n; ++i)
            if (boundless(i)) planeList[fill[c.hostWorldOf[i]]++] = i;
    }
    VXB_TRY(ensure(c, c.worldOfBuf, (size_t)n * 4));
    VXB_TRY(ensure(c, c.planeStartBuf, planeStart.size() * 4));
    VXB_TRY(ensure(c, c.planeListBuf, planeList.size() * 4 + 4));
    c.hostPlaneStart = planeStart;
    VXB_CUDA(c, cudaMemcpyAsync(c.worldOfBuf.ptr, c.hostWorldOf.data(), (size_t)n * 4, cudaMemcpyHostToDevice, c.stream));
    VXB_CUDA(c, cudaMemcpyAsync(c.planeStartBuf.ptr, planeStart.data(), planeStart.size() * 4, cudaMemcpyHostToDevice,
                                c.stream));
    if (!planeList.empty())
        VXB_CUDA(c, cudaMemcpyAsync(c.planeListBuf.ptr, planeList.data(), planeList.size() * 4, cudaMemcpyHostToDevice,
                                    c.stream));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));  // host vectors above are freed on return
    // Reserve step buffers up front so steady stepping never reallocates
    // (cudaFree synchronises the device).
    if (c.pairCap < 16u * n) c.pairCap = 16u * n + 4096u;
    if (c.contactCap < 8u * n) c.contactCap = 8u * n + 4096u;
    if (c.recCap < 8u * n) c.recCap = 8u * n + 4096u;
    const size_t mcap = c.contactCap;
    VXB_TRY(ensure(c, c.pairBuf, (size_t)c.pairCap * 8));
    VXB_TRY(ensure(c, c.contactTmpBuf, mcap * sizeof(vx_contact)));
    VXB_TRY(ensure(c, c.contactBuf[0], mcap * sizeof(vx_contact) + 128));
    VXB_TRY(ensure(c, c.contactBuf[1], mcap * sizeof(vx_contact) + 128));
    VXB_TRY(ensure(c, c.coopBuf, sizeof(CoopState)));
    for (DevBuf* b : {&c.recValBuf, &c.recCountBuf, &c.recOffsetBuf, &c.islandValBuf, &c.colorBuf, &c.flagBuf,
                      &c.scanBuf, &c.islandStartBuf, &c.segStartBuf, &c.islandSegBuf, &c.fpIslandBuf})
        VXB_TRY(ensure(c, *b, mcap * 4 + 64));
    for (DevBuf* b : {&c.recKeyBuf, &c.recInfoBuf, &c.pairKeyBuf, &c.prevKeyBuf, &c.islandKeyBuf, &c.colorKeyBuf,
                      &c.sortKeysAlt})
        VXB_TRY(ensure(c, *b, mcap * 8 + 64));
    VXB_TRY(ensure(c, c.sortValsAlt, std::max<size_t>(mcap, (size_t)c.pairCap) * 4 + 64));
    reserve(c, n);
    c.prevCount = 0;
    c.stepContacts = 0;
    VXB_TRY(sleepLoad(c, bodies, n));
    return VXB_OK;
}

int readBodies(Context& c, vx_body* out, uint32_t n) {
    if (n != c.n) return fail(c, VXB_ERR_INVALID, "body count mismatch");
    LAUNCH(c, unpackBodiesKernel, blocksFor(n, 256), 256, P<vx_body>(c.aosBuf), n, c.B);
    VXB_TRY(sleepExport(c, P<vx_body>(c.aosBuf)));
    VXB_CUDA(c, cudaMemcpyAsync(out, c.aosBuf.ptr, (size_t)n * sizeof(vx_body), cudaMemcpyDeviceToHost, c.stream));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

int readPoses(Context& c, float* out, uint32_t n) {
    if (n != c.n) return fail(c, VXB_ERR_INVALID, "body count mismatch");
    VXB_TRY(ensure(c, c.scanBuf, (size_t)n * 28 + 16));
    LAUNCH(c, posesKernel, blocksFor(n, 256), 256, P<float>(c.scanBuf), n, c.B);
    VXB_CUDA(c, cudaMemcpyAsync(out, c.scanBuf.ptr, (size_t)n * 28, cudaMemcpyDeviceToHost, c.stream));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

int writeForces(Context& c, const float* in, uint32_t n) {
    if (n != c.n) return fail(c, VXB_ERR_INVALID, "body count mismatch");
    VXB_TRY(ensure(c, c.scanBuf, (size_t)n * 28 + 16));
    VXB_CUDA(c, cudaMemcpyAsync(c.scanBuf.ptr, in, (size_t)n * 24, cudaMemcpyHostToDevice, c.stream));
    LAUNCH(c, forcesKernel, blocksFor(n, 256), 256, P<float>(c.scanBuf), n, c.B);
    return VXB_OK;
}

// ---- broad phase ----------------------------------------------------------

static int broadPhase(Context& c, float dt, uint32_t* pairCount) {
    const uint32_t n = c.n;
    VXB_TRY(ensure(c, c.aabbBuf, (size_t)n * 32));
    float4* lo = P<float4>(c.aabbBuf);
    float4* hi = lo + n;
    stageBegin(c, kStageBroadphase);
    LAUNCH(c, aabbKernel, std::min<uint32_t>(blocksFor(n, 256), (uint32_t)c.smCount * 8), 256, c.B, n, dt,
           (const vx_mesh*)P<vx_mesh>(c.meshBuf), lo, hi, c.dCounters);
    const int worldBits = bitsFor(c.worlds > 1 ? c.worlds - 1 : 0);
    const int keyBitsTotal = 3 * kCellBits + worldBits + 1;
    const uint64_t planeKey = 1ull << (3 * kCellBits + worldBits);
    VXB_TRY(ensure(c, c.cellKeyBuf, (size_t)n * 8));
    VXB_TRY(ensure(c, c.cellValBuf, (size_t)n * 4));
    uint64_t* keys = P<uint64_t>(c.cellKeyBuf);
    uint32_t* vals = P<uint32_t>(c.cellValBuf);
    LAUNCH(c, keyKernel, blocksFor(n, 256), 256, c.B, n, c.worlds > 1 ? P<uint32_t>(c.worldOfBuf) : nullptr, lo, hi,
           c.dCounters, keys, vals, planeKey);
    stageEnd(c, kStageBroadphase);
    stageBegin(c, kStageCellSort);
    VXB_TRY(sortPairs(c, keys, vals, n, keyBitsTotal));
    stageEnd(c, kStageCellSort);
    stageBegin(c, kStageBroadphase);
    uint32_t hashCap = 1024;
    while (hashCap < 2 * n) hashCap <<= 1;
    c.hashCap = hashCap;
    VXB_TRY(ensure(c, c.hashKeyBuf, (size_t)hashCap * 8));
    VXB_TRY(ensure(c, c.hashValBuf, (size_t)hashCap * 4));
    VXB_CUDA(c, cudaMemsetAsync(c.hashKeyBuf.ptr, 0xff, (size_t)hashCap * 8, c.stream));
    LAUNCH(c, cellTableKernel, blocksFor(n, 256), 256, keys, n, planeKey, P<uint64_t>(c.hashKeyBuf),
           P<uint32_t>(c.hashValBuf), hashCap - 1);
    if (c.pairCap == 0) c.pairCap = std::max<uint32_t>(n * 8u, 4096u);
    // plane pairs: at most bodies x planes of a world
    uint32_t planeCap = 16;
    {
        uint32_t maxPlanes = 0;
        for (uint32_t w = 0; w < c.worlds; ++w) maxPlanes = std::max(maxPlanes, c.hostPlaneStart[w + 1] - c.hostPlaneStart[w]);
        planeCap = std::max<uint32_t>(16u, n * std::max<uint32_t>(maxPlanes, 1u));
    }
    for (int attempt = 0; attempt < 3; ++attempt) {
        VXB_TRY(ensure(c, c.pairBuf, ((size_t)c.pairCap + planeCap) * 8));
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->pairs, 0, 4, c.stream));
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->planePairs, 0, 4, c.stream));
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->overflow, 0, 4, c.stream));
        LAUNCH(c, pairKernel, blocksFor(n, 128), 128, c.B, n, keys, vals, lo, hi, P<uint64_t>(c.hashKeyBuf),
               P<uint32_t>(c.hashValBuf), hashCap - 1, planeKey,
               c.worlds > 1 ? P<uint32_t>(c.worldOfBuf) : nullptr, P<uint32_t>(c.planeStartBuf),
               P<uint32_t>(c.planeListBuf), P<uint64_t>(c.pairBuf), c.pairCap, P<uint64_t>(c.pairBuf) + c.pairCap,
               planeCap, c.dCounters);
        stageEnd(c, kStageBroadphase);
        VXB_TRY(readCounters(c));
        if (c.hostCounters.pairs <= c.pairCap && c.hostCounters.planePairs <= planeCap) break;
        c.pairCap = c.hostCounters.pairs + c.hostCounters.pairs / 4 + 1024;
    }
    // Convex pairs live at [0, pairs), plane pairs at [pairCap, pairCap + planePairs).
    c.convexPairs = c.hostCounters.pairs;
    c.planePairs = c.hostCounters.planePairs;
    *pairCount = c.convexPairs + c.planePairs;
    return VXB_OK;
}

// ---- narrow phase ---------------------------------------------------------

// Launch of a warp-per-item kernel over at most `items` items: no more blocks
// than run at once.
template <class Kernel, class... Args>
static int launchQueries(Context& c, uint32_t items, Kernel kernel, Args... args) {
    int perSm = 0;
    VXB_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, kQueryThreads, kQuerySmem));
    const uint32_t grid = std::min<uint32_t>(blocksFor(items, kQueryThreads / 32),
                                             (uint32_t)(std::max(perSm, 1) * c.smCount));
    kernel<<<grid, kQueryThreads, kQuerySmem, c.stream>>>(args...);
    ++c.launches;
    return VXB_OK;
}

// Runs the narrow phase on `npairs` device pairs and leaves the contacts
// sorted in contactBuf[c.cur] (mode 0) or grouped in pair order (mode 1).
// World path: `pairs` holds convexSplit convex-convex pairs and `planePairs`
// holds npairs - convexSplit plane pairs. Stage path (convexSplit = ~0u):
// `pairs` holds npairs unclassified pairs.
static int narrowPhase(Context& c, const uint64_t* pairs, uint32_t npairs, float dt, int mode, uint32_t* contactCount,
                       uint32_t* recordCount, uint32_t convexSplit = ~0u, const uint64_t* planePairs = nullptr) {
    const int bodyBits = std::max(1, bitsFor(c.n - 1));
    if (c.contactCap == 0) c.contactCap = std::max<uint32_t>(npairs * 2u, 4096u);
    if (c.recCap < npairs) c.recCap = npairs + 1024;
    for (int attempt = 0; attempt < 3; ++attempt) {
        VXB_TRY(ensure(c, c.contactTmpBuf, (size_t)c.contactCap * sizeof(vx_contact)));
        VXB_TRY(ensure(c, c.recKeyBuf, (size_t)c.recCap * 8));
        VXB_TRY(ensure(c, c.recValBuf, (size_t)c.recCap * 4));
        VXB_TRY(ensure(c, c.recInfoBuf, (size_t)c.recCap * 8));
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->contactsTmp, 0, 12, c.stream));  // contactsTmp, records, hardPairs
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->overflow, 0, 4, c.stream));
        stageBegin(c, kStageNarrowphase);
        vx_contact* tmp = P<vx_contact>(c.contactTmpBuf);
        uint64_t* recKeys = P<uint64_t>(c.recKeyBuf);
        uint32_t* recVals = P<uint32_t>(c.recValBuf);
        uint2* recInfo = P<uint2>(c.recInfoBuf);
        if (npairs && convexSplit <= npairs) {
            const uint32_t np = npairs - convexSplit;
            if (convexSplit) {
                // group the convex pairs by shape combination (records are keyed by body pair, so
                // the processing order does not change the result)
                VXB_TRY(ensure(c, c.classKeyBuf, (size_t)convexSplit * 8 + 64));
                VXB_TRY(ensure(c, c.classValBuf, (size_t)convexSplit * 4 + 64));
                if (attempt == 0) {
                    LAUNCH(c, pairClassKernel, blocksFor(convexSplit, 256), 256, c.B, pairs, convexSplit,
                           P<uint64_t>(c.classKeyBuf), P<uint32_t>(c.classValBuf));
                    VXB_TRY(sortPairs(c, P<uint64_t>(c.classKeyBuf), P<uint32_t>(c.classValBuf), convexSplit, 8));
                }
                const uint32_t* order = P<uint32_t>(c.classValBuf);
                VXB_TRY(ensure(c, c.hardBuf, (size_t)convexSplit * (4 + sizeof(HardResult)) + 64));
                HardResult* results = P<HardResult>(c.hardBuf);
                uint32_t* hard = reinterpret_cast<uint32_t*>(results + convexSplit);
                VXB_TRY(tunedLaunch(c, kTuneCollideConvex, convexSplit, [&](LaunchShape sh) {
                    LAUNCH(c, collideKernel<kConvexPairs>, sh.grid(convexSplit, c.smCount), sh.threads, c.B, soupOf(c),
                           pairs, order, convexSplit, dt, mode, bodyBits, tmp, c.contactCap, recKeys, recVals, recInfo,
                           c.recCap, hard, results, c.dCounters);
                }, CounterRestore{c}));
                const int rc = launchQueries(c, convexSplit, collideHardKernel, c.B, soupOf(c), pairs,
                                             (const uint32_t*)hard, dt, mode, bodyBits, tmp, c.contactCap, recKeys,
                                             recVals, recInfo, c.recCap, results, c.dCounters);
                if (rc != VXB_OK) return rc;
                LAUNCH(c, collideKernel<kListedPairs>, blocksFor(convexSplit, 64, (uint32_t)c.smCount * 16), 64, c.B,
                       soupOf(c), pairs, (const uint32_t*)hard, convexSplit, dt, mode, bodyBits, tmp, c.contactCap,
                       recKeys, recVals, recInfo, c.recCap, (uint32_t*)nullptr, results,
                       c.dCounters);
                if (c.threadShapes)
                    LAUNCH(c, collideKernel<kThreadPairs>, blocksFor(convexSplit, 64, (uint32_t)c.smCount * 16), 64,
                           c.B, soupOf(c), pairs, (const uint32_t*)hard, convexSplit, dt, mode, bodyBits, tmp,
                           c.contactCap, recKeys, recVals, recInfo, c.recCap, (uint32_t*)nullptr,
                           (HardResult*)nullptr, c.dCounters);
            }
            if (np)
                VXB_TRY(tunedLaunch(c, kTuneCollidePlane, np, [&](LaunchShape sh) {
                    LAUNCH(c, collideKernel<kPlanePairs>, sh.grid(np, c.smCount), sh.threads, c.B, soupOf(c), planePairs,
                           (const uint32_t*)nullptr, np, dt, mode, bodyBits, tmp, c.contactCap, recKeys, recVals,
                           recInfo, c.recCap, (uint32_t*)nullptr, (HardResult*)nullptr, c.dCounters);
                }, CounterRestore{c}));
        } else if (npairs) {
            VXB_TRY(tunedLaunch(c, kTuneCollideAny, npairs, [&](LaunchShape sh) {
                LAUNCH(c, collideKernel<kAnyPairs>, sh.grid(npairs, c.smCount), sh.threads, c.B, soupOf(c), pairs,
                       (const uint32_t*)nullptr, npairs, dt, mode, bodyBits, tmp, c.contactCap, recKeys, recVals,
                       recInfo, c.recCap, (uint32_t*)nullptr, (HardResult*)nullptr, c.dCounters);
            }, CounterRestore{c}));
        }
        stageEnd(c, kStageNarrowphase);
        VXB_TRY(readCounters(c));
        if (!(c.hostCounters.overflow & 2u)) break;
        c.contactCap = c.hostCounters.contactsTmp + c.hostCounters.contactsTmp / 4 + 1024;
        c.recCap = std::max(c.recCap, c.hostCounters.records + 1024);
    }
    const uint32_t m = c.hostCounters.contactsTmp, nrec = c.hostCounters.records;
    *contactCount = m;
    *recordCount = nrec;
    const int recBits = mode == 0 ? 2 * bodyBits : bitsFor(npairs);
    stageBegin(c, kStagePlacement);
    VXB_TRY(sortPairs(c, P<uint64_t>(c.recKeyBuf), P<uint32_t>(c.recValBuf), nrec, recBits));
    VXB_TRY(ensure(c, c.recCountBuf, (size_t)nrec * 4 + 16));
    VXB_TRY(ensure(c, c.recOffsetBuf, (size_t)nrec * 4 + 16));
    VXB_TRY(ensure(c, c.pairKeyBuf, (size_t)nrec * 8 + 16));
    VXB_TRY(ensure(c, c.contactBuf[c.cur], (size_t)m * sizeof(vx_contact) + 128));
    VXB_TRY(ensure(c, c.scanBuf, (size_t)nrec * 4 + 16));
    if (nrec) {
        LAUNCH(c, gatherCountsKernel, blocksFor(nrec, 256), 256, P<uint32_t>(c.recValBuf), P<uint2>(c.recInfoBuf), nrec,
               P<uint32_t>(c.recCountBuf));
        VXB_TRY(exclusiveScan(c, P<uint32_t>(c.recCountBuf), P<uint32_t>(c.scanBuf), nrec, nullptr));
        LAUNCH(c, placeKernel, blocksFor(nrec, 128), 128, P<uint32_t>(c.recValBuf), P<uint2>(c.recInfoBuf),
               P<uint32_t>(c.scanBuf), nrec, P<vx_contact>(c.contactTmpBuf), P<vx_contact>(c.contactBuf[c.cur]),
               (uint64_t*)nullptr, P<uint64_t>(c.pairKeyBuf), P<uint32_t>(c.recOffsetBuf));
    }
    stageEnd(c, kStagePlacement);
    return VXB_OK;
}

// ---- islands + colouring --------------------------------------------------

// Groups the m contacts of `cs` into islands, colours them and builds the
// solve order (island, colour, contact order) plus per-island body lists.
// Cooperative launch of `kernel` with as many blocks as fit on the device at
// once (at most maxPerSm per SM when maxPerSm > 0). VXB_ERR_UNSUPPORTED
// (nothing recorded) when the device cannot run it: callers then take their
// serial path.
template <class Kernel, class... Args>
static int launchCooperativeSmem(Context& c, int maxPerSm, size_t smem, Kernel kernel, int threads, Args... args) {
    int perSm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, threads, smem);
    if (e != cudaSuccess) return cudaStatus(c, e, "cooperative occupancy");
    if (perSm <= 0 || !c.cooperative) return VXB_ERR_UNSUPPORTED;
    if (maxPerSm > 0 && perSm > maxPerSm) perSm = maxPerSm;
    void* params[] = {&args...};
    e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(perSm * c.smCount), dim3(threads), params, smem,
                                    c.stream);
    ++c.launches;
    return cudaStatus(c, e, "cudaLaunchCooperativeKernel");
}

template <class Kernel, class... Args>
static int launchCooperative(Context& c, Kernel kernel, int threads, Args... args) {
    return launchCooperativeSmem(c, 0, 0, kernel, threads, args...);
}

// Colours of the giant islands (colorOf, colour keys, maxColors). VXB_ERR_UNSUPPORTED / VXB_ERR_TIMEOUT: the caller colours
// every island serially instead.
static int parallelColor(Context& c, const vx_contact* cs, const uint32_t* order, const uint32_t* islandIdx,
                         const uint32_t* islandStart, const uint32_t* bodyStart, uint32_t realIslands, uint32_t m,
                         uint64_t* colorKeys) {
    const uint32_t n = c.n;
    VXB_TRY(ensure(c, c.fpKeyBuf, (size_t)m * 16 + 64));
    VXB_TRY(ensure(c, c.fpValBuf, (size_t)m * 8 + 64));
    VXB_TRY(ensure(c, c.fpSlotBuf, (size_t)m * 8 + 64));
    VXB_TRY(ensure(c, c.fpColorBuf, (size_t)m * 4 + 64));
    VXB_TRY(ensure(c, c.fpRunStartBuf, (size_t)n * 4 + 64));
    VXB_TRY(ensure(c, c.coopBuf, sizeof(CoopState)));
    uint64_t* keys = P<uint64_t>(c.fpKeyBuf);
    uint32_t* vals = P<uint32_t>(c.fpValBuf);
    uint32_t* slot = P<uint32_t>(c.fpSlotBuf);
    uint32_t* color = P<uint32_t>(c.fpColorBuf);
    uint32_t* runStart = P<uint32_t>(c.fpRunStartBuf);
    CoopState* st = P<CoopState>(c.coopBuf);
    LAUNCH(c, colorEntryKernel, blocksFor(m, 256), 256, cs, order, m, islandIdx, islandStart, bodyStart,
           realIslands, c.B, n, keys, vals, slot);
    VXB_TRY(sortPairs(c, keys, vals, 2 * m, bitsFor(n)));
    LAUNCH(c, colorSlotKernel, blocksFor(2 * m, 256), 256, keys, vals, 2 * m, n, slot, runStart);
    VXB_CUDA(c, cudaMemsetAsync(color, 0, (size_t)m * 4, c.stream));
    VXB_TRY(resetCoop(c, st));
    const int rc = launchCooperative(c, colorFixedPointKernel, 256, (const uint64_t*)keys, (const uint32_t*)vals,
                                     (const uint32_t*)slot, (const uint32_t*)runStart, m, color, st, 4096u);
    if (rc != VXB_OK) return rc;
    CoopState host;
    VXB_CUDA(c, cudaMemcpyAsync(&host, st, sizeof(host), cudaMemcpyDeviceToHost, c.stream));
    ++c.hostSyncs;
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    c.stats.colorRounds = host.rounds;
    if (host.timeout || (host.spill & 2u)) return VXB_ERR_TIMEOUT;
    if (host.spill) return VXB_ERR_UNSUPPORTED;
    LAUNCH(c, colorFinishKernel, blocksFor(m, 256), 256, order, m, islandIdx, islandStart, bodyStart,
           realIslands, (const uint32_t*)color, P<uint32_t>(c.colorBuf), colorKeys, c.dCounters);
    return VXB_OK;
}

// Colours of the islands of one class, a block each.
template <int Class>
static int colorIslands(Context& c, const vx_contact* cs, const IslandPlan& plan) {
    using Shape = ColorShape<Class>;
    auto* kernel = colorIslandKernel<Class>;
    VXB_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape::kSmem));
    const uint32_t grid = std::min<uint32_t>(plan.islands, (uint32_t)(c.smCount * (Class == kSmallIsland ? 16 : Class == kMediumIsland ? 4 : 1)));
    kernel<<<grid, ClassShape<Class>::kThreads, Shape::kSmem, c.stream>>>(
        cs, P<uint32_t>(c.islandValBuf), P<uint32_t>(c.islandStartBuf), P<uint32_t>(c.bodyValBuf),
        P<uint32_t>(c.islandBodyStartBuf), plan.islands, plan.realIslands, c.B, P<uint32_t>(c.localIdxBuf),
        P<uint32_t>(c.colorBuf), P<uint64_t>(c.colorKeyBuf), c.dCounters);
    ++c.launches;
    return VXB_OK;
}

static int buildIslands(Context& c, const vx_contact* cs, uint32_t m, IslandPlan& plan, uint32_t* colorOut) {
    const uint32_t n = c.n;
    plan.contacts = m;
    c.planContacts = m;
    c.clusterBuilt = false;
    c.tinyPacked = false;
    VXB_TRY(ensure(c, c.parentBuf, (size_t)n * 4));
    VXB_TRY(ensure(c, c.islandOfBodyBuf, (size_t)n * 4));
    VXB_TRY(ensure(c, c.maskBuf, (size_t)n * 8));
    VXB_TRY(ensure(c, c.nextColorBuf, (size_t)n * 4));
    VXB_TRY(ensure(c, c.bodyKeyBuf, (size_t)n * 8));
    VXB_TRY(ensure(c, c.bodyValBuf, (size_t)n * 4));
    VXB_TRY(ensure(c, c.islandKeyBuf, (size_t)m * 8 + 16));
    VXB_TRY(ensure(c, c.islandValBuf, (size_t)m * 4 + 16));
    VXB_TRY(ensure(c, c.colorBuf, (size_t)m * 4 + 16));
    VXB_TRY(ensure(c, c.flagBuf, (size_t)m * 4 + 16));
    VXB_TRY(ensure(c, c.scanBuf, (size_t)m * 4 + 16));
    VXB_TRY(ensure(c, c.islandStartBuf, (size_t)m * 4 + 16));
    VXB_TRY(ensure(c, c.segStartBuf, (size_t)m * 4 + 16));
    VXB_TRY(ensure(c, c.islandSegBuf, (size_t)m * 4 + 16));
    uint32_t* parent = P<uint32_t>(c.parentBuf);
    LAUNCH(c, iotaKernel, blocksFor(n, 256), 256, parent, n);
    if (m == 0) {
        plan = IslandPlan{};
        plan.contacts = 0;
        VXB_CUDA(c, cudaMemsetAsync(c.islandOfBodyBuf.ptr, 0xff, (size_t)n * 4, c.stream));
    } else {
        LAUNCH(c, unionKernel, blocksFor(m, 256), 256, cs, m, c.B, parent, c.dCounters);
        LAUNCH(c, compressKernel, blocksFor(n, 256), 256, parent, n);
        uint64_t* ikeys = P<uint64_t>(c.islandKeyBuf);
        uint32_t* ivals = P<uint32_t>(c.islandValBuf);
        LAUNCH(c, islandKeyKernel, blocksFor(m, 256), 256, cs, m, c.B, parent, n, ikeys, ivals);
        VXB_TRY(sortPairs(c, ikeys, ivals, m, bitsFor(n)));
        uint32_t* flags = P<uint32_t>(c.flagBuf);
        uint32_t* index = P<uint32_t>(c.scanBuf);
        uint32_t* islandStart = P<uint32_t>(c.islandStartBuf);
        LAUNCH(c, runFlagKernel, blocksFor(m, 256), 256, ikeys, m, flags);
        VXB_TRY(exclusiveScan(c, flags, index, m, &c.dCounters->islands));
        LAUNCH(c, runStartKernel, blocksFor(m, 256), 256, flags, index, m, islandStart);
        VXB_TRY(ensure(c, c.fpIslandBuf, (size_t)m * 4 + 64));
        uint32_t* islandOf = P<uint32_t>(c.fpIslandBuf);
        LAUNCH(c, runOfKernel, blocksFor(m, 256), 256, flags, index, m, islandOf);
        LAUNCH(c, lastKeyKernel, 1, 32, ikeys, m, c.dCounters);
        LAUNCH(c, islandMaxKernel, std::min<uint32_t>(blocksFor(m, 256), (uint32_t)c.smCount * 4), 256, islandStart,
               c.dCounters);
        VXB_TRY(readCounters(c));
        plan.islands = c.hostCounters.islands;
        // is the last island the null island (key n)?
        plan.realIslands = c.hostCounters.lastIslandKey == n ? plan.islands - 1 : plan.islands;
        // island bodies (before the colouring, whose classes depend on them)
        VXB_CUDA(c, cudaMemsetAsync(c.islandOfBodyBuf.ptr, 0xff, (size_t)n * 4, c.stream));
        LAUNCH(c, islandBodyKernel, blocksFor(m, 256), 256, cs, ivals, (const uint32_t*)islandOf, m, plan.realIslands,
               c.B, P<uint32_t>(c.islandOfBodyBuf));
    }
    const uint32_t freeKey = plan.realIslands;
    LAUNCH(c, bodyKeyKernel, blocksFor(n, 256), 256, P<uint32_t>(c.islandOfBodyBuf), n, freeKey,
           P<uint64_t>(c.bodyKeyBuf), P<uint32_t>(c.bodyValBuf));
    VXB_TRY(sortPairs(c, P<uint64_t>(c.bodyKeyBuf), P<uint32_t>(c.bodyValBuf), n, bitsFor(freeKey)));
    VXB_TRY(ensure(c, c.islandBodyStartBuf, ((size_t)plan.realIslands + 2) * 4 + 16));
    uint32_t* bodyStart = P<uint32_t>(c.islandBodyStartBuf);
    LAUNCH(c, bodyStartKernel, blocksFor(n, 256), 256, P<uint64_t>(c.bodyKeyBuf), n, bodyStart, plan.realIslands + 2);
    LAUNCH(c, freeRangeKernel, 1, 32, bodyStart, plan.realIslands + 2, c.dCounters);
    VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->giantCount, 0, 4, c.stream));
    if (m) {
        uint32_t* ivals = P<uint32_t>(c.islandValBuf);
        uint32_t* flags = P<uint32_t>(c.flagBuf);
        uint32_t* index = P<uint32_t>(c.scanBuf);
        uint32_t* islandStart = P<uint32_t>(c.islandStartBuf);
        const uint32_t* islandOf = P<uint32_t>(c.fpIslandBuf);
        // colour each island; colour keys (island << 16 | colour) in island order
        VXB_TRY(ensure(c, c.colorKeyBuf, (size_t)m * 8 + 16));
        VXB_TRY(ensure(c, c.localIdxBuf, (size_t)n * 4 + 16));
        uint64_t* ckeys = P<uint64_t>(c.colorKeyBuf);
        bool serialAll = false;
        // which classes can exist: an island of k + 1 bodies has at least k contacts
        const uint32_t largest = c.planLargest = c.hostCounters.maxIslandSize;
        if (largest > (uint32_t)kLargeRows || (largest >= (uint32_t)kLargeBodies && n > (uint32_t)kLargeBodies)) {
            const int status = parallelColor(c, cs, ivals, islandOf, islandStart, bodyStart, plan.realIslands, m, ckeys);
            if (status == VXB_ERR_TIMEOUT || status == VXB_ERR_UNSUPPORTED) serialAll = true;  // exact serial path
            else if (status != VXB_OK) return status;
        }
        LAUNCH(c, colorKernel, blocksFor(plan.islands, 64), 64, cs, ivals, islandStart, plan.islands, c.B,
               P<unsigned long long>(c.maskBuf), P<uint32_t>(c.nextColorBuf), P<uint32_t>(c.colorBuf), ckeys,
               c.dCounters, serialAll ? 0xffffffffu : kTinyLimit);
        if (!serialAll && largest > kTinyLimit) {
            VXB_TRY(colorIslands<kSmallIsland>(c, cs, plan));
            if (largest >= (uint32_t)kSmallBodies) VXB_TRY(colorIslands<kMediumIsland>(c, cs, plan));
            if (largest >= (uint32_t)kMediumBodies) VXB_TRY(colorIslands<kLargeIsland>(c, cs, plan));
        }
        if (colorOut)
            VXB_CUDA(c, cudaMemcpyAsync(colorOut, c.colorBuf.ptr, (size_t)m * 4, cudaMemcpyDeviceToHost, c.stream));
        // solve order: stable sort by (island, colour)
        VXB_TRY(sortPairs(c, ckeys, ivals, m, 16 + bitsFor(plan.islands)));
        LAUNCH(c, runFlagKernel, blocksFor(m, 256), 256, ckeys, m, flags);
        VXB_TRY(exclusiveScan(c, flags, index, m, &c.dCounters->segments));
        LAUNCH(c, runStartKernel, blocksFor(m, 256), 256, flags, index, m, P<uint32_t>(c.segStartBuf));
        LAUNCH(c, giantCountKernel, std::min<uint32_t>(blocksFor(plan.islands, 256), (uint32_t)c.smCount * 4), 256,
               (const uint32_t*)islandStart, (const uint32_t*)bodyStart, plan.islands, plan.realIslands, c.dCounters);
    }
    VXB_TRY(readCounters(c));  // one read for the segment count, the free-body range and the giants
    plan.segments = m ? c.hostCounters.segments : 0;
    plan.freeFrom = c.hostCounters.freeFrom;
    plan.freeTo = c.hostCounters.freeTo;
    c.planGiants = m ? c.hostCounters.giantCount : 0u;
    return VXB_OK;
}

__global__ void islandSegKernel(const uint32_t* islandStart, const uint32_t* segIndex, uint32_t islands,
                                uint32_t segments, uint32_t* islandSeg) {
    for (uint32_t isl = blockIdx.x * blockDim.x + threadIdx.x; isl <= islands; isl += gridDim.x * blockDim.x)
        islandSeg[isl] = isl == islands ? segments : segIndex[islandStart[isl]];
}

static SolveArgs solveArgs(Context& c, vx_contact* cs, const IslandPlan& plan) {
    SolveArgs A;
    std::memset(&A, 0, sizeof(A));
    A.B = c.B;
    A.contacts = cs;
    A.order = P<uint32_t>(c.islandValBuf);
    A.islandStart = P<uint32_t>(c.islandStartBuf);
    A.segStart = P<uint32_t>(c.segStartBuf);
    A.islandSeg = P<uint32_t>(c.islandSegBuf);
    A.bodyOrder = P<uint32_t>(c.bodyValBuf);
    A.bodyStart = P<uint32_t>(c.islandBodyStartBuf);
    A.islands = plan.islands;
    A.realIslands = plan.realIslands;
    A.tinyLimit = kTinyLimit;
    A.fault = &c.dCounters->planFault;
    A.timeout = &c.dCounters->timeout;
    A.waitLimit = c.waitLimit;
    A.planes = P<float4>(c.planeBuf);
    A.rows = plan.contacts;
    return A;
}

static int prepareSegments(Context& c, const IslandPlan& plan) {
    if (plan.islands == 0) return VXB_OK;
    LAUNCH(c, islandSegKernel, blocksFor(plan.islands + 1, 256), 256, P<uint32_t>(c.islandStartBuf),
           P<uint32_t>(c.scanBuf), plan.islands, plan.segments, P<uint32_t>(c.islandSegBuf));
    return VXB_OK;
}

// The islands of one class, a block each, as many blocks as fit at once.
template <int Class>
static int launchIslands(Context& c, const SolveArgs& A) {
    using Shape = ClassShape<Class>;
    auto* kernel = A.coneBlock ? solveIslandKernel<Class, true> : solveIslandKernel<Class, false>;
    VXB_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape::kSmem));
    const uint32_t grid = std::min<uint32_t>(A.islands, (uint32_t)(c.smCount * Shape::kBlocksPerSm));
    kernel<<<grid, Shape::kThreads, Shape::kSmem, c.stream>>>(A, P<uint32_t>(c.localIdxBuf));
    ++c.launches;
    return VXB_OK;
}

// Plan of the giant islands' flow, once per island plan: every row's links on
// its bodies, the bodies' clusters and the warps' rows in colour order.
static int buildFlow(Context& c, const SolveArgs& A, uint32_t clusters) {
    const uint32_t m = c.planContacts, n = c.n;
    VXB_TRY(ensure(c, c.fpKeyBuf, (size_t)m * 16 + 64));
    VXB_TRY(ensure(c, c.fpValBuf, (size_t)m * 8 + 64));
    VXB_TRY(ensure(c, c.fpSlotBuf, (size_t)m * 8 + 64));
    VXB_TRY(ensure(c, c.fpRunStartBuf, (size_t)n * 4 + 64));
    VXB_TRY(ensure(c, c.flowDegreeBuf, (size_t)n * 4 + 64));
    VXB_TRY(ensure(c, c.flowBodyBuf, (size_t)n * 64 + 64));
    uint64_t* keys = P<uint64_t>(c.fpKeyBuf);
    uint32_t* vals = P<uint32_t>(c.fpValBuf);
    const uint32_t* islandOf = P<uint32_t>(c.fpIslandBuf);
    LAUNCH(c, giantEntryKernel, blocksFor(m, 256), 256, A, islandOf, m, n, keys, vals);
    VXB_TRY(sortPairs(c, keys, vals, 2 * m, bitsFor(n)));
    LAUNCH(c, flowRunKernel, blocksFor(2 * m, 256), 256, keys, 2 * m, n, P<uint32_t>(c.fpRunStartBuf));
    LAUNCH(c, flowLinkKernel, blocksFor(2 * m, 256), 256, keys, vals, 2 * m, n,
           (const uint32_t*)P<uint32_t>(c.fpRunStartBuf), P<uint32_t>(c.fpSlotBuf), P<uint32_t>(c.flowDegreeBuf));
    VXB_TRY(ensure(c, c.clusterInfoBuf, ((size_t)n * 3 + (size_t)m * 3 + 128) * 4));
    uint32_t* bodyFlags = P<uint32_t>(c.clusterInfoBuf);
    uint32_t* bodyRank = bodyFlags + n + 16;
    uint32_t* bodyPos = bodyRank + n + 16;
    uint32_t* rowFlags = bodyPos + n + 16;
    uint32_t* rowRank = rowFlags + m + 16;
    uint32_t* rowList = rowRank + m + 16;
    VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->clusterColours, 0, 4, c.stream));
    LAUNCH(c, giantMemberKernel, blocksFor(std::max(n, m), 256), 256, A, P<uint64_t>(c.bodyKeyBuf), n, islandOf, m,
           bodyFlags, rowFlags, c.dCounters);
    VXB_TRY(exclusiveScan(c, bodyFlags, bodyRank, n, &c.dCounters->clusterBodies));
    VXB_TRY(exclusiveScan(c, rowFlags, rowRank, m, &c.dCounters->clusterRows));
    LAUNCH(c, compactKernel, blocksFor(n, 256), 256, bodyFlags, bodyRank, n, bodyPos);
    LAUNCH(c, compactKernel, blocksFor(m, 256), 256, rowFlags, rowRank, m, rowList);
    VXB_TRY(readCounters(c));
    c.clusterNB = c.hostCounters.clusterBodies;
    c.clusterR = c.hostCounters.clusterRows;
    c.clusterG = c.hostCounters.clusterColours;
    c.clusterCount = clusters;
    c.clusterBuilt = true;
    const uint32_t nb = c.clusterNB, R = c.clusterR, G = c.clusterG;
    if (nb == 0 || R == 0 || G == 0) {
        c.clusterR = 0;
        return VXB_OK;
    }
    VXB_TRY(ensure(c, c.clusterKeyBuf, (size_t)nb * 8 + 64));
    VXB_TRY(ensure(c, c.clusterValBuf, (size_t)nb * 4 + 64));
    VXB_TRY(ensure(c, c.clusterOfBuf, (size_t)n * 4 + 64));
    VXB_TRY(ensure(c, c.flowColourBuf, (size_t)R * 4 + 64));
    VXB_TRY(ensure(c, c.clusterStartBuf, ((size_t)clusters + 1) * 4 + 64));
    VXB_TRY(ensure(c, c.clusterRowsBuf, (size_t)R * 4 + 64));
    const uint32_t* clusterOf = P<uint32_t>(c.clusterOfBuf);
    LAUNCH(c, clusterBodyKeyKernel, blocksFor(nb, 256), 256, A, (const uint32_t*)bodyPos, nb,
           (const Counters*)c.dCounters, P<uint64_t>(c.clusterKeyBuf), P<uint32_t>(c.clusterValBuf));
    VXB_TRY(sortPairs(c, P<uint64_t>(c.clusterKeyBuf), P<uint32_t>(c.clusterValBuf), nb, 30));
    LAUNCH(c, clusterOfBodyKernel, blocksFor(nb, 256), 256, (const uint32_t*)P<uint32_t>(c.clusterValBuf), nb, clusters,
           P<uint32_t>(c.clusterOfBuf));
    const int colourBits = bitsFor(G - 1);
    LAUNCH(c, flowKeyKernel, blocksFor(R, 256), 256, A, (const uint32_t*)rowList, R, islandOf, clusterOf, clusters,
           colourBits, keys, P<uint32_t>(c.clusterRowsBuf));
    VXB_TRY(sortPairs(c, keys, P<uint32_t>(c.clusterRowsBuf), R, colourBits + bitsFor(clusters - 1)));
    LAUNCH(c, flowStartKernel, blocksFor(R, 256), 256, (const uint64_t*)keys, R, clusters, colourBits,
           P<uint32_t>(c.flowColourBuf), P<uint32_t>(c.clusterStartBuf));
    return VXB_OK;
}

// Tiny islands: packed into warps once per island plan, then one launch.
static int launchTiny(Context& c, const SolveArgs& A) {
    const uint32_t islands = A.islands, chunksCap = (islands + kPackChunk - 1) / kPackChunk + 1;
    VXB_TRY(ensure(c, c.tinyBuf, ((size_t)islands * 4 + (size_t)chunksCap * 2 + 64) * 4));
    uint32_t* tFlags = P<uint32_t>(c.tinyBuf);
    uint32_t* tRanks = tFlags + islands + 16;
    uint32_t* tList = tRanks + islands + 16;
    uint32_t* tFirst = tList + islands + 16;
    uint32_t* tChunkCount = tFirst + islands + 16;
    uint32_t* tChunkBase = tChunkCount + chunksCap;
    // (counts stay on the device: sizes below are upper bounds, kernels read the counts)
    const uint32_t chunks = (islands + kPackChunk - 1) / kPackChunk;
    if (!c.tinyPacked) {
        LAUNCH(c, tinyFlagKernel, blocksFor(islands, 256), 256, A, tFlags);
        VXB_TRY(exclusiveScan(c, tFlags, tRanks, islands, &c.dCounters->tinyIslands));
        LAUNCH(c, compactKernel, blocksFor(islands, 256), 256, tFlags, tRanks, islands, tList);
        VXB_TRY(ensure(c, c.tinyKeyBuf, (size_t)islands * 8 + 64));
        LAUNCH(c, tinyKeyKernel, blocksFor(islands, 256), 256, A, (const uint32_t*)tList,
               (const uint32_t*)&c.dCounters->tinyIslands, islands, P<uint64_t>(c.tinyKeyBuf), tList);
        VXB_TRY(sortPairs(c, P<uint64_t>(c.tinyKeyBuf), tList, islands, 8));
        LAUNCH(c, tinyPackKernel, blocksFor(chunks, 128), 128, A, (const uint32_t*)tList,
               (const uint32_t*)&c.dCounters->tinyIslands, chunks, 0, tChunkCount, (const uint32_t*)tChunkBase, tFirst);
        VXB_TRY(exclusiveScan(c, tChunkCount, tChunkBase, chunks, &c.dCounters->tinyPacks));
        LAUNCH(c, tinyPackKernel, blocksFor(chunks, 128), 128, A, (const uint32_t*)tList,
               (const uint32_t*)&c.dCounters->tinyIslands, chunks, 1, tChunkCount, (const uint32_t*)tChunkBase, tFirst);
        c.tinyPacked = true;
    }
    VXB_TRY(ensure(c, c.localIdxBuf, (size_t)c.n * 4 + 16));
    {
        static bool packConfigured = false;
        if (!packConfigured) {
            cudaFuncSetAttribute(solveTinyPackKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(kPackWarpSmem * kPackWarps));
            packConfigured = true;
        }
        const uint32_t grid = std::min<uint32_t>((islands + kPackWarps - 1) / kPackWarps, (uint32_t)c.smCount * 8);
        solveTinyPackKernel<<<grid, 32 * kPackWarps, kPackWarpSmem * kPackWarps, c.stream>>>(
            A, (const uint32_t*)tList, (const uint32_t*)tFirst, (const Counters*)c.dCounters, P<uint32_t>(c.localIdxBuf));
        ++c.launches;
    }
    return VXB_OK;
}

// Runs `work` on the context's side stream `s`, forked from its stream at
// `forkEvent`; the caller joins with joinSide before anything depends on it.
template <class Work>
static int onSide(Context& c, int s, Work work) {
    VXB_CUDA(c, cudaStreamWaitEvent(c.side[s], c.forkEvent, 0));
    const cudaStream_t own = c.stream;
    c.stream = c.side[s];
    const int rc = work();
    c.stream = own;
    VXB_CUDA(c, cudaEventRecord(c.joinEvent[s], c.side[s]));
    return rc;
}
static int joinSide(Context& c, int s) {
    VXB_CUDA(c, cudaStreamWaitEvent(c.stream, c.joinEvent[s], 0));
    return VXB_OK;
}

// The classes' kernels touch different islands (their rows, bodies and
// planes), so tiny and small islands run beside the medium ones: one after
// the other, each class waited for the last's longest chain. Solve stage of one
// step, in turn -> side by side: a lattice of 65 bodies as it falls apart
// 1.65 -> 1.41 ms, 187,000 tiny islands beside some small ones 5.7 -> 5.1 ms,
// heaps of 3,000 and 40,000 bodies 3.0 -> 2.5 and 4.3 -> 3.8 ms; one class alone
// (the pyramids) stays at 4.5 ms. The flow starts after the join: it reuses the
// planes and fills the GPU.
static int launchSolve(Context& c, const SolveArgs& A) {
    if (A.islands == 0) return VXB_OK;
    VXB_TRY(ensure(c, c.localIdxBuf, (size_t)c.n * 4 + 16));
    VXB_TRY(ensure(c, c.coopBuf, sizeof(CoopState)));
    const uint32_t giants = c.planGiants;  // counted with the island plan
    int perSm = 0;
    uint32_t clusters = 0;
    auto* flow = A.coneBlock ? solveFlowKernel<true> : solveFlowKernel<false>;
    if (giants && c.cooperative) {  // (its sorts and scans share scratch with the tiny islands' packing)
        VXB_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, flow, kFlowThreads, 0));
        perSm = std::min(perSm, kFlowBlocksPerSm);
        clusters = (uint32_t)(perSm * c.smCount) * (kFlowThreads / 32);
        if (clusters > 0 && (!c.clusterBuilt || c.clusterCount != clusters)) VXB_TRY(buildFlow(c, A, clusters));
    }
    VXB_CUDA(c, cudaEventRecord(c.forkEvent, c.stream));
    const int tinyStatus = onSide(c, 0, [&] { return launchTiny(c, A); });
    int smallStatus = VXB_OK;
    if (c.planLargest > kTinyLimit)
        smallStatus = onSide(c, 1, [&] {
            // four warps an island while the GPU holds them all at once
            const bool few = A.islands <= (uint32_t)(c.smCount * ClassShape<kSmallWide>::kBlocksPerSm);
            return few ? launchIslands<kSmallWide>(c, A) : launchIslands<kSmallIsland>(c, A);
        });
    int mediumStatus = VXB_OK;
    if (c.planLargest >= (uint32_t)kSmallBodies) mediumStatus = launchIslands<kMediumIsland>(c, A);
    VXB_TRY(joinSide(c, 0));
    if (c.planLargest > kTinyLimit) VXB_TRY(joinSide(c, 1));
    VXB_TRY(tinyStatus);
    VXB_TRY(smallStatus);
    VXB_TRY(mediumStatus);
    if (!giants) return VXB_OK;
    // giant islands: list them, then one cooperative launch over all of them
    CoopState* st = P<CoopState>(c.coopBuf);
    VXB_TRY(ensure(c, c.giantBuf, ((size_t)A.islands + 1) * 4 + 64));
    uint32_t* list = P<uint32_t>(c.giantBuf);
    VXB_TRY(resetCoop(c, st));
    LAUNCH(c, giantListKernel, std::min<uint32_t>(blocksFor(A.islands, 256), (uint32_t)c.smCount * 4), 256, A, list,
           &st->rounds);
    c.stats.giantIslands = std::max(c.stats.giantIslands, giants);
    if (clusters > 0) {
        if (c.clusterR > 0) {
            FlowArgs F;
            F.start = P<uint32_t>(c.clusterStartBuf);
            F.rows = P<uint32_t>(c.clusterRowsBuf);
            F.colour = P<uint32_t>(c.flowColourBuf);
            F.rank = P<uint32_t>(c.fpSlotBuf);
            F.degree = P<uint32_t>(c.flowDegreeBuf);
            F.bodyIds = P<uint32_t>(c.clusterValBuf);
            F.body = P<float4>(c.flowBodyBuf);
            F.bodies = c.clusterNB;
            VXB_TRY(resetCoop(c, st));
            const int rcc = launchCooperativeSmem(c, perSm, 0, flow, kFlowThreads, A, F, st);
            if (rcc != VXB_ERR_UNSUPPORTED) {
                VXB_TRY(rcc);
                // a timed-out wait reaches the host with the step's final counter read
                LAUNCH(c, coopTimeoutKernel, 1, 32, (const CoopState*)st, c.dCounters);
                return VXB_OK;
            }
        }
    }
    // no cooperative grid (or no solvable giant rows): one block per giant island
    SolveArgs G = A;
    VXB_TRY(ensure(c, c.prepBuf, (size_t)A.rows * sizeof(RowPrep) + 256));
    VXB_TRY(ensure(c, c.frameBuf, (size_t)c.n * 16 + 256));
    G.prep = P<RowPrep>(c.prepBuf);
    G.frames = P<float4>(c.frameBuf);
    LAUNCH(c, solveGiantBlockKernel, giants, kGiantBlockThreads, G, (const uint32_t*)list);
    return VXB_OK;
}

// Substep loop over islands + contact-free bodies (advanceSubsteps).
static int runSubsteps(Context& c, vx_contact* cs, const IslandPlan& plan, const V3& g, float h, int substeps,
                       const vx_solver_options& o, bool warmStart, bool integrate) {
    VXB_TRY(ensure(c, c.planeBuf, ((size_t)plan.contacts + 1) * kRowPlaneBytes + 256));
    SolveArgs A = solveArgs(c, cs, plan);
    A.gravity = g;
    A.h = h;
    A.substeps = substeps;
    A.sweeps = 2 * o.velocityIterations;
    A.warmStart = warmStart ? 1 : 0;
    A.integrate = integrate ? 1 : 0;
    A.coneBlock = o.frictionModel == VX_FRICTION_CONE_BLOCK;
    VXB_TRY(launchSolve(c, A));
    if (integrate && plan.freeTo > plan.freeFrom)
        LAUNCH(c, freeBodiesKernel, blocksFor(plan.freeTo - plan.freeFrom, 128), 128, c.B, P<uint32_t>(c.bodyValBuf),
               plan.freeFrom, plan.freeTo, g, h, substeps);
    return VXB_OK;
}

static int positionCorrection(Context& c, vx_contact* cs, const IslandPlan& plan, const vx_solver_options& o, float h) {
    if (o.positionIterations <= 0 || plan.islands == 0) return VXB_OK;
    SolveArgs A = solveArgs(c, cs, plan);
    A.positionIterations = o.positionIterations;
    A.stackStabilization = o.enableStackStabilization;
    A.stackStiffness = o.stackStiffness;
    A.stackDamping = o.stackDamping;
    A.h = h;
    VXB_TRY(launchSolve(c, A));
    return VXB_OK;
}

static int conservativeAdvancement(Context& c, uint32_t npairs, float dt) {
    if (npairs == 0) return VXB_OK;
    const uint32_t n = c.n;
    VXB_TRY(ensure(c, c.caFlagBuf, (size_t)npairs * 28 + 64));
    VXB_TRY(ensure(c, c.caBodyMarkBuf, (size_t)n * 16 + 16));
    VXB_TRY(ensure(c, c.caCandBuf, (size_t)npairs * 28 + 64));
    float4* endGap = P<float4>(c.caFlagBuf);
    uint32_t* flags = reinterpret_cast<uint32_t*>(endGap + npairs);
    uint32_t* candFlags = flags + npairs;
    uint32_t* flagRank = candFlags + npairs;
    uint32_t* bodyMark = P<uint32_t>(c.caBodyMarkBuf);
    uint32_t* rewound = bodyMark + n;
    uint32_t* front[2] = {rewound + n, rewound + 2 * (size_t)n};  // widening frontiers
    uint32_t* queue = P<uint32_t>(c.caCandBuf);  // exclusive-scan ranks first, then the ready queue
    uint32_t* candIndex = queue + npairs;
    uint32_t* succ = candIndex + npairs;          // two per candidate
    uint32_t* pending = succ + 2 * (size_t)npairs;
    uint32_t* depth = pending + npairs;
    uint32_t* crit = depth + npairs;
    VXB_CUDA(c, cudaMemsetAsync(bodyMark, 0, (size_t)n * 8, c.stream));
    const uint64_t* pk = P<uint64_t>(c.pairKeyBuf);
    const float4* prevPos = P<float4>(c.prevPoseBuf);
    const float4* prevRot = prevPos + n;
    // group the pairs by shape combination for the probe (the narrow phase's
    // grouping buffers are free again at this point of the step)
    const uint32_t* probeOrder = nullptr;
    if (npairs >= kProbeGroupMin) {
        VXB_TRY(ensure(c, c.classKeyBuf, (size_t)npairs * 8 + 64));
        VXB_TRY(ensure(c, c.classValBuf, (size_t)npairs * 4 + 64));
        LAUNCH(c, pairClassKernel, blocksFor(npairs, 256), 256, c.B, pk, npairs, P<uint64_t>(c.classKeyBuf),
               P<uint32_t>(c.classValBuf));
        VXB_TRY(sortPairs(c, P<uint64_t>(c.classKeyBuf), P<uint32_t>(c.classValBuf), npairs, 8));
        probeOrder = P<uint32_t>(c.classValBuf);
    }
    // the probe writes each pair's outcome at its own index and only sets marks: trials restore its list's length
    uint32_t* hard = queue;
    auto emptyList = [&]() -> int {
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->caHard, 0, 4, c.stream));
        return VXB_OK;
    };
    VXB_TRY(emptyList());
    VXB_TRY(tunedLaunch(c, kTuneProbe, npairs, [&](LaunchShape sh) {
        LAUNCH(c, caProbeKernel, sh.grid(npairs, c.smCount), sh.threads, c.B, soupOf(c), pk, probeOrder, npairs,
               flags, bodyMark, endGap, hard, c.dCounters);
    }, emptyList));
    if (c.threadShapes)
        LAUNCH(c, caProbeGeneralKernel, blocksFor(npairs, 64, (uint32_t)c.smCount * 16), 64, c.B, soupOf(c), pk,
               (const uint32_t*)hard, flags, bodyMark, endGap, (const Counters*)c.dCounters);
    VXB_TRY(launchQueries(c, npairs, caProbeHardKernel, c.B, soupOf(c), pk, (const uint32_t*)hard, dt, flags, bodyMark,
                          endGap, (const Counters*)c.dCounters));
    // speculative outcomes of the flagged pairs on the probe's state
    VXB_TRY(exclusiveScan(c, flags, flagRank, npairs, &c.dCounters->caFlagged));
    VXB_TRY(readCounters(c));
    const uint32_t flagged = c.hostCounters.caFlagged;
    if (flagged == 0) return VXB_OK;  // nothing flagged: no pair is examined, nothing moves
    VXB_TRY(ensure(c, c.caSpecBuf, (size_t)flagged * (8 * sizeof(float4) + 8) + 64));
    float4* specState = P<float4>(c.caSpecBuf);
    uint32_t* specResult = reinterpret_cast<uint32_t*>(specState + 8 * (size_t)flagged);
    uint32_t* flaggedList = specResult + flagged;
    LAUNCH(c, compactKernel, blocksFor(npairs, 256), 256, flags, flagRank, npairs, flaggedList);
    VXB_TRY(launchQueries(c, flagged, caSpeculateKernel, c.B, soupOf(c), pk, (const uint32_t*)flaggedList, flagged,
                          (const float4*)endGap, dt, prevPos, prevRot, specState, specResult, c.dCounters));
    // mark ahead of the cascade before the first pass too (fewer replays)
    {
        const uint32_t* frontier = bodyMark;
        for (int hop = 0; hop < kCaInitialHops; ++hop) {
            uint32_t* next = front[hop & 1];
            VXB_CUDA(c, cudaMemsetAsync(next, 0, (size_t)n * 4, c.stream));
            LAUNCH(c, caWidenKernel, blocksFor(npairs, 256), 256, c.B, pk, npairs, bodyMark, frontier, next);
            frontier = next;
        }
    }
    VXB_TRY(ensure(c, c.snapBuf, (size_t)n * 64));
    VXB_TRY(ensure(c, c.coopBuf, sizeof(CoopState)));
    CoopState* st = P<CoopState>(c.coopBuf);
    bool snapped = false, serial = false;
    for (int pass = 0;; ++pass) {
        if (pass == kCaWidenLimit) { serial = true; break; }
        LAUNCH(c, caCandidateKernel, blocksFor(npairs, 256), 256, c.B, pk, npairs, flags, bodyMark, candFlags,
               c.dCounters);
        VXB_TRY(exclusiveScan(c, candFlags, queue, npairs, &c.dCounters->caCandidates));
        VXB_TRY(readCounters(c));
        const uint32_t ncand = c.hostCounters.caCandidates;
        if (ncand == 0) return VXB_OK;
        LAUNCH(c, compactKernel, blocksFor(npairs, 256), 256, candFlags, queue, npairs, candIndex);
        // successors and predecessor counts through shared dynamic bodies
        const size_t valsOffset = ((size_t)ncand * 16 + 255) & ~(size_t)255;  // both arrays 256-byte aligned
        VXB_TRY(ensure(c, c.islandInfoBuf, valsOffset + (size_t)ncand * 8 + 16));
        uint64_t* ekeys = P<uint64_t>(c.islandInfoBuf);
        uint32_t* evals = reinterpret_cast<uint32_t*>(P<char>(c.islandInfoBuf) + valsOffset);
        VXB_TRY(ensure(c, c.caInfoBuf, (size_t)ncand * 16 + 64));
        uint4* info = P<uint4>(c.caInfoBuf);
        LAUNCH(c, caEntryKernel, blocksFor(ncand, 256), 256, c.B, pk, (const uint32_t*)candIndex, ncand, n,
               (const uint32_t*)flags, ekeys, evals, info);
        VXB_TRY(sortPairs(c, ekeys, evals, 2 * ncand, bitsFor(n)));
        VXB_CUDA(c, cudaMemsetAsync(pending, 0, (size_t)ncand * 4, c.stream));
        VXB_CUDA(c, cudaMemsetAsync(depth, 0, (size_t)ncand * 4, c.stream));
        VXB_CUDA(c, cudaMemsetAsync(crit, 0, (size_t)ncand * 4, c.stream));
        LAUNCH(c, caLinkKernel, blocksFor(2 * ncand, 256), 256, ekeys, evals, 2 * ncand, n, succ, pending);
        if (!snapped) {
            LAUNCH(c, copyStateKernel, blocksFor(n, 256), 256, c.B, n, P<float4>(c.snapBuf), 0);
            snapped = true;
        }
        VXB_CUDA(c, cudaMemsetAsync(queue, 0xff, (size_t)ncand * 4, c.stream));
        VXB_TRY(resetCoop(c, st));
        const int rc = launchCooperativeSmem(c, kCaFlowBlocksPerSm, kQuerySmem, caFlowKernel, kQueryThreads, c.B, soupOf(c),
                                               (const uint32_t*)flagRank, (const float4*)specState,
                                               (const uint32_t*)specResult, (const uint4*)info, ncand,
                                               (const uint32_t*)succ, pending, queue, depth, crit,
                                               (const uint32_t*)bodyMark, rewound, dt, prevPos, prevRot, c.dCounters,
                                               st);
        if (rc == VXB_ERR_UNSUPPORTED) { serial = true; break; }
        VXB_TRY(rc);
        CoopState host;
        VXB_CUDA(c, cudaMemcpyAsync(&host, st, sizeof(host), cudaMemcpyDeviceToHost, c.stream));
        VXB_TRY(readCounters(c));
        if (host.timeout) return fail(c, VXB_ERR_TIMEOUT, "a wait timed out in the rewind pass");
        if (host.spill) return fail(c, VXB_ERR_INTERNAL, "inconsistent candidate links in the rewind pass");
        c.caRounds += host.rounds;
        if (!c.hostCounters.caOverflow) return VXB_OK;
        // a rewind reached an unmarked body: widen the marked set and replay from the snapshot
        LAUNCH(c, copyStateKernel, blocksFor(n, 256), 256, c.B, n, P<float4>(c.snapBuf), 1);
        {
            const uint32_t* frontier = rewound;
            for (int hop = 0; hop < kCaWidenHops; ++hop) {
                uint32_t* next = front[hop & 1];
                VXB_CUDA(c, cudaMemsetAsync(next, 0, (size_t)n * 4, c.stream));
                LAUNCH(c, caWidenKernel, blocksFor(npairs, 256), 256, c.B, pk, npairs, bodyMark, frontier, next);
                frontier = next;
            }
        }
        VXB_CUDA(c, cudaMemsetAsync(rewound, 0, (size_t)n * 4, c.stream));
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->rewinds, 0, 4, c.stream));
        VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->caOverflow, 0, 4, c.stream));
        ++c.caWidenings;
    }
    if (serial) {
        if (snapped) LAUNCH(c, copyStateKernel, blocksFor(n, 256), 256, c.B, n, P<float4>(c.snapBuf), 1);
        VXB_CUDA(c, cudaMemsetAsync(rewound, 0, (size_t)n * 4, c.stream));
        caFullSerialKernel<<<1, 32, sizeof(WarpQuery), c.stream>>>(c.B, soupOf(c), pk, npairs, flags, rewound, dt,
                                                                   prevPos, prevRot, c.dCounters);
        ++c.launches;
    }
    return VXB_OK;
}

// One World::step on the device world.
static int stepOnce(Context& c) {
    const vxb_step_config& cfg = c.config;
    const uint32_t n = c.n;
    const int substeps = cfg.substeps > 0 ? cfg.substeps : 1;
    const float dt = cfg.dt;
    const float h = dt / substeps;
    const V3 g{cfg.gravity.x, cfg.gravity.y, cfg.gravity.z};
    VXB_TRY(resetCounters(c));
    c.stats.colorRounds = 0;
    c.stats.giantIslands = 0;
    c.caRounds = 0;
    c.caWidenings = 0;
    VXB_TRY(ensure(c, c.prevPoseBuf, (size_t)n * 32));
    float4* prevPos = P<float4>(c.prevPoseBuf);
    if (c.tape.active) VXB_TRY(tapeStepBegin(c));
    stageBegin(c, kStagePrepare);
    LAUNCH(c, prepareKernel, blocksFor(n, 256), 256, c.B, n, g, h, prevPos, prevPos + n, 1);
    stageEnd(c, kStagePrepare);
    uint32_t npairs = 0, m = 0, nrec = 0;
    VXB_TRY(broadPhase(c, dt, &npairs));
    c.stats.candidatePairs = npairs;
    VXB_TRY(narrowPhase(c, P<uint64_t>(c.pairBuf), npairs, dt, 0, &m, &nrec, c.convexPairs,
                        P<uint64_t>(c.pairBuf) + c.pairCap));
    vx_contact* cs = P<vx_contact>(c.contactBuf[c.cur]);
    stageBegin(c, kStageWarmStart);
    VXB_TRY(wakePass(c, cs, m));  // src/world.cpp:4106-4128: after detection, before warm starting
    if (c.tape.active)
        VXB_TRY(tapeBeforeMatch(c, cs, m, P<vx_contact>(c.contactBuf[c.cur ^ 1]), P<uint64_t>(c.prevKeyBuf),
                                c.prevCount));
    if (c.prevCount && m)
        LAUNCH(c, matchKernel, blocksFor(m, 128), 128, cs, m, P<vx_contact>(c.contactBuf[c.cur ^ 1]),
               P<uint64_t>(c.prevKeyBuf), c.prevCount, c.dCounters);
    if (c.tape.active) VXB_TRY(tapeAfterMatch(c, cs, m));
    stageEnd(c, kStageWarmStart);
    IslandPlan plan;
    stageBegin(c, kStageIslands);
    VXB_TRY(buildIslands(c, cs, m, plan, nullptr));
    VXB_TRY(prepareSegments(c, plan));
    if (c.tape.active) VXB_TRY(tapeAfterIslands(c, P<uint32_t>(c.colorBuf), m));
    stageEnd(c, kStageIslands);
    stageBegin(c, kStageSolve);
    VXB_TRY(runSubsteps(c, cs, plan, g, h, substeps, cfg.solver, true, true));
    stageEnd(c, kStageSolve);
    stageBegin(c, kStageRewind);
    if (m) VXB_TRY(conservativeAdvancement(c, nrec, dt));
    if (c.tape.active && m && nrec) VXB_TRY(tapeAfterRewind(c, P<uint32_t>(c.caBodyMarkBuf) + n));
    stageEnd(c, kStageRewind);
    stageBegin(c, kStagePositions);
    VXB_TRY(positionCorrection(c, cs, plan, cfg.solver, h));
    stageEnd(c, kStagePositions);
    // events, sleeping and the resting pairs' cached contacts (before the
    // forces are cleared: the calm test reads them)
    uint32_t kept = 0;
    VXB_TRY(sleepAndEvents(c, cs, m, dt, &kept));
    LAUNCH(c, clearForcesKernel, blocksFor(n, 256), 256, c.B, n);
    // previous-contact cache: this step's contacts in (a, b, point) order, and
    // resting pairs' cached contacts merged in by pair
    if (kept) {
        VXB_TRY(mergeKeptContacts(c, m, kept));
        cs = P<vx_contact>(c.contactBuf[c.cur]);
    }
    const uint32_t cacheCount = m + kept;
    VXB_TRY(ensure(c, c.prevKeyBuf, (size_t)cacheCount * 8 + 16));
    if (cacheCount)
        LAUNCH(c, contactKeysKernel, blocksFor(cacheCount, 256), 256, cs, cacheCount, P<uint64_t>(c.prevKeyBuf));
    c.prevCount = cacheCount;
    c.stepContacts = m;
    c.cur ^= 1;
    if (c.tape.active) VXB_TRY(tapeStepEnd(c, m));
    VXB_TRY(readCounters(c));
    c.stats.contacts = m;
    c.stats.islands = plan.realIslands;
    c.stats.colors = c.hostCounters.maxColors;
    c.stats.largestIsland = c.hostCounters.largestIsland;
    c.stats.rewinds = c.hostCounters.rewinds;
    c.stats.rewindRounds = c.caRounds;
    c.stats.rewindReplays = c.caWidenings;
    c.stats.rewindGapQueries = c.hostCounters.caGapQueries;
    c.stats.rewindCriticalMicros = c.hostCounters.caCritMicros;
    c.stats.rewindSpeculateMicros = c.hostCounters.caSpecMicros;
    c.stats.warmStarted = c.hostCounters.warmStarted;
    c.stats.velocityIterations = (uint32_t)(2 * cfg.solver.velocityIterations * substeps);
    if (c.hostCounters.timeout) return fail(c, VXB_ERR_TIMEOUT, "a bounded device wait gave up");
    if (c.hostCounters.planFault) return fail(c, VXB_ERR_INTERNAL, "inconsistent island plan in the solve");
    return VXB_OK;
}

int worldStep(Context& c, int steps) {
    if (!c.configured) return fail(c, VXB_ERR_INVALID, "vxb_world_configure was not called");
    if (c.n == 0) return fail(c, VXB_ERR_INVALID, "no bodies loaded");
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    for (int s = 0; s < steps; ++s) VXB_TRY(stepOnce(c));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    VXB_CUDA(c, cudaGetLastError());
    return VXB_OK;
}

int readContacts(Context& c, vx_contact* out, uint32_t cap, uint32_t* count) {
    const uint32_t m = c.stepContacts;
    if (count) *count = m;
    if (out && m && c.prevCount != m) return readStepContacts(c, out, std::min(m, cap));
    if (out && m) {
        VXB_CUDA(c, cudaMemcpyAsync(out, c.contactBuf[c.cur ^ 1].ptr, (size_t)std::min(m, cap) * sizeof(vx_contact),
                                    cudaMemcpyDeviceToHost, c.stream));
        VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    }
    return VXB_OK;
}

int writeContacts(Context& c, const vx_contact* contacts, uint32_t m) {
    tapeEnd(c);
    VXB_TRY(ensure(c, c.contactBuf[c.cur ^ 1], (size_t)m * sizeof(vx_contact) + 128));
    VXB_TRY(ensure(c, c.prevKeyBuf, (size_t)m * 8 + 16));
    if (m) {
        VXB_CUDA(c, cudaMemcpyAsync(c.contactBuf[c.cur ^ 1].ptr, contacts, (size_t)m * sizeof(vx_contact),
                                    cudaMemcpyHostToDevice, c.stream));
        LAUNCH(c, contactKeysKernel, blocksFor(m, 256), 256, P<vx_contact>(c.contactBuf[c.cur ^ 1]), m,
               P<uint64_t>(c.prevKeyBuf));
    }
    c.prevCount = m;
    c.stepContacts = m;
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

// ---- stage entry points -----------------------------------------------------

int stagePairs(Context& c, float dt, uint64_t* out, uint32_t cap, uint32_t* count) {
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    VXB_TRY(resetCounters(c));
    uint32_t npairs = 0;
    VXB_TRY(broadPhase(c, dt, &npairs));
    *count = npairs;
    if (out) {
        std::vector<uint64_t> host(npairs);
        if (c.convexPairs)
            VXB_CUDA(c, cudaMemcpyAsync(host.data(), c.pairBuf.ptr, (size_t)c.convexPairs * 8, cudaMemcpyDeviceToHost,
                                        c.stream));
        if (c.planePairs)
            VXB_CUDA(c, cudaMemcpyAsync(host.data() + c.convexPairs, P<uint64_t>(c.pairBuf) + c.pairCap,
                                        (size_t)c.planePairs * 8, cudaMemcpyDeviceToHost, c.stream));
        VXB_CUDA(c, cudaStreamSynchronize(c.stream));
        std::sort(host.begin(), host.end());
        std::memcpy(out, host.data(), (size_t)std::min(npairs, cap) * 8);
    }
    return npairs > cap && out ? fail(c, VXB_ERR_CAPACITY, "pair buffer too small") : VXB_OK;
}

int stageCollide(Context& c, const uint64_t* pairs, uint32_t npairs, float dt, vx_contact* out, uint32_t cap,
                 uint32_t* counts, uint32_t* total) {
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    VXB_TRY(resetCounters(c));
    VXB_TRY(ensure(c, c.pairBuf, (size_t)npairs * 8 + 16));
    if (npairs)
        VXB_CUDA(c, cudaMemcpyAsync(c.pairBuf.ptr, pairs, (size_t)npairs * 8, cudaMemcpyHostToDevice, c.stream));
    uint32_t m = 0, nrec = 0;
    VXB_TRY(narrowPhase(c, P<uint64_t>(c.pairBuf), npairs, dt, 1, &m, &nrec));
    *total = m;
    if (m > cap) return fail(c, VXB_ERR_CAPACITY, "contact buffer too small");
    if (m) VXB_CUDA(c, cudaMemcpyAsync(out, c.contactBuf[c.cur].ptr, (size_t)m * sizeof(vx_contact),
                                       cudaMemcpyDeviceToHost, c.stream));
    if (counts) {
        std::vector<uint64_t> keys(nrec);
        std::vector<uint32_t> cnt(nrec);
        if (nrec) {
            VXB_CUDA(c, cudaMemcpyAsync(keys.data(), c.recKeyBuf.ptr, (size_t)nrec * 8, cudaMemcpyDeviceToHost, c.stream));
            VXB_CUDA(c, cudaMemcpyAsync(cnt.data(), c.recCountBuf.ptr, (size_t)nrec * 4, cudaMemcpyDeviceToHost, c.stream));
        }
        VXB_CUDA(c, cudaStreamSynchronize(c.stream));
        std::fill(counts, counts + npairs, 0u);
        for (uint32_t r = 0; r < nrec; ++r) counts[keys[r]] = cnt[r];
    }
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

int stageColor(Context& c, const vx_contact* contacts, uint32_t m, int32_t* colorOf, uint32_t* numColors) {
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    VXB_TRY(resetCounters(c));
    VXB_TRY(ensure(c, c.contactBuf[c.cur], (size_t)m * sizeof(vx_contact) + 128));
    if (m) VXB_CUDA(c, cudaMemcpyAsync(c.contactBuf[c.cur].ptr, contacts, (size_t)m * sizeof(vx_contact),
                                       cudaMemcpyHostToDevice, c.stream));
    IslandPlan plan;
    VXB_TRY(buildIslands(c, P<vx_contact>(c.contactBuf[c.cur]), m, plan, reinterpret_cast<uint32_t*>(colorOf)));
    VXB_TRY(readCounters(c));
    *numColors = c.hostCounters.maxColors;
    return VXB_OK;
}

VXD void storeDistance(const GjkResult& r, float* o) {
    o[0] = r.distance;
    o[1] = r.normal.x; o[2] = r.normal.y; o[3] = r.normal.z;
    o[4] = r.pointA.x; o[5] = r.pointA.y; o[6] = r.pointA.z;
    o[7] = r.pointB.x; o[8] = r.pointB.y; o[9] = r.pointB.z;
    o[10] = r.overlapping ? 1.0f : 0.0f;
}

__global__ void distanceKernel(BodyArrays B, Soup soup, const uint64_t* pairs, uint32_t npairs, int path, float* out,
                               uint32_t* hard, Counters* C) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npairs; p += gridDim.x * blockDim.x) {
        const Convex ca = makeConvex(loadView(B, (uint32_t)(pairs[p] >> 32)), soup);
        const Convex cb = makeConvex(loadView(B, (uint32_t)pairs[p]), soup);
        GjkResult r;
        Simplex s;
        if (path != 0) r = gjkDistance(ca, cb);
        else if (pairQuality(ca, cb) != 0) r = gjkDistance(ca, cb);
        else if (gjkDistanceFast(ca, cb, r, s) != kGjkSeparated) { hard[aggregatedSlot(&C->hardPairs)] = p; continue; }
        storeDistance(r, out + 11 * (size_t)p);
    }
}

__global__ void __launch_bounds__(kQueryThreads) distanceHardKernel(BodyArrays B, Soup soup, const uint64_t* pairs,
                                                                    const uint32_t* hard, float* out,
                                                                    const Counters* C) {
    const uint32_t count = C->hardPairs, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count; k += warps) {
        const uint32_t p = hard[k];
        const Convex ca = makeConvex(loadView(B, (uint32_t)(pairs[p] >> 32)), soup);
        const Convex cb = makeConvex(loadView(B, (uint32_t)pairs[p]), soup);
        const GjkResult r = gjkDistanceWarp(ca, cb);
        if (warpLane() == 0u) storeDistance(r, out + 11 * (size_t)p);
        __syncwarp();
    }
}

int stageDistance(Context& c, const uint64_t* pairs, uint32_t npairs, int path, float* out) {
    if (npairs == 0) return VXB_OK;
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    VXB_TRY(ensure(c, c.pairBuf, (size_t)npairs * 8 + 16));
    VXB_TRY(ensure(c, c.contactTmpBuf, (size_t)npairs * 44 + 16));
    VXB_TRY(ensure(c, c.hardBuf, (size_t)npairs * 4 + 64));
    VXB_CUDA(c, cudaMemcpyAsync(c.pairBuf.ptr, pairs, (size_t)npairs * 8, cudaMemcpyHostToDevice, c.stream));
    VXB_CUDA(c, cudaMemsetAsync(&c.dCounters->hardPairs, 0, 4, c.stream));
    LAUNCH(c, distanceKernel, blocksFor(npairs, 64), 64, c.B, soupOf(c), P<uint64_t>(c.pairBuf), npairs, path,
           P<float>(c.contactTmpBuf), P<uint32_t>(c.hardBuf), c.dCounters);
    if (path == 0)
        VXB_TRY(launchQueries(c, npairs, distanceHardKernel, c.B, soupOf(c), (const uint64_t*)P<uint64_t>(c.pairBuf),
                              (const uint32_t*)P<uint32_t>(c.hardBuf), P<float>(c.contactTmpBuf),
                              (const Counters*)c.dCounters));
    VXB_CUDA(c, cudaMemcpyAsync(out, c.contactTmpBuf.ptr, (size_t)npairs * 44, cudaMemcpyDeviceToHost, c.stream));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

// ---- Backend-interface mode ---------------------------------------------------

int backendIntegrate(Context& c, vx_vec3 gravity, float dt) {
    LAUNCH(c, integrateKernel, blocksFor(c.n, 256), 256, c.B, c.n, V3{gravity.x, gravity.y, gravity.z}, dt);
    return VXB_OK;
}

int backendIntegrateTransforms(Context& c, float dt) {
    LAUNCH(c, transformsKernel, blocksFor(c.n, 256), 256, c.B, c.n, dt);
    return VXB_OK;
}

int backendFindContacts(Context& c, float dt, uint32_t* count) {
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    VXB_TRY(resetCounters(c));
    uint32_t npairs = 0, m = 0, nrec = 0;
    VXB_TRY(broadPhase(c, dt, &npairs));
    VXB_TRY(narrowPhase(c, P<uint64_t>(c.pairBuf), npairs, dt, 0, &m, &nrec, c.convexPairs,
                        P<uint64_t>(c.pairBuf) + c.pairCap));
    c.backendContacts = m;
    c.backendColored = false;
    *count = m;
    return VXB_OK;
}

int backendCopyContacts(Context& c, vx_contact* out, uint32_t cap) {
    const uint32_t m = c.backendContacts;
    if (m > cap) return fail(c, VXB_ERR_CAPACITY, "contact buffer too small");
    if (m) VXB_CUDA(c, cudaMemcpyAsync(out, c.contactBuf[c.cur].ptr, (size_t)m * sizeof(vx_contact),
                                       cudaMemcpyDeviceToHost, c.stream));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

static bool hostContactLess(const vx_contact& x, const vx_contact& y) {
    const uint64_t kx = ((uint64_t)x.a << 32) | x.b, ky = ((uint64_t)y.a << 32) | y.b;
    if (kx != ky) return kx < ky;
    if (x.point.x != y.point.x) return x.point.x < y.point.x;
    if (x.point.y != y.point.y) return x.point.y < y.point.y;
    return x.point.z < y.point.z;
}

// solveVelocities / advanceSubsteps. On warm start the contacts are sorted,
// coloured, written back in colour order and kept resident; the solve then
// runs `substeps` substeps (fullSubsteps) or one velocity solve.
int backendSolve(Context& c, vx_contact* contacts, uint32_t m, float h, bool warmStart, const vx_solver_options& o,
                 vx_vec3 gravity, int substeps, bool fullSubsteps) {
    VXB_TRY(ensure(c, c.countersBuf, sizeof(Counters)));
    c.dCounters = P<Counters>(c.countersBuf);
    IslandPlan& plan = c.backendPlan;  // retained between the warm-start call and later calls
    if (warmStart) {
        VXB_TRY(resetCounters(c));
        c.hostSorted.assign(contacts, contacts + m);
        std::stable_sort(c.hostSorted.begin(), c.hostSorted.end(), hostContactLess);
        VXB_TRY(ensure(c, c.contactBuf[c.cur], (size_t)m * sizeof(vx_contact) + 128));
        if (m) VXB_CUDA(c, cudaMemcpyAsync(c.contactBuf[c.cur].ptr, c.hostSorted.data(), (size_t)m * sizeof(vx_contact),
                                           cudaMemcpyHostToDevice, c.stream));
        VXB_TRY(buildIslands(c, P<vx_contact>(c.contactBuf[c.cur]), m, plan, nullptr));
        VXB_TRY(prepareSegments(c, plan));
        // colour order back to the host (pre-solve values, like the reference's sorted_ copy)
        std::vector<uint32_t> order(m);
        if (m) VXB_CUDA(c, cudaMemcpyAsync(order.data(), c.islandValBuf.ptr, (size_t)m * 4, cudaMemcpyDeviceToHost,
                                           c.stream));
        VXB_CUDA(c, cudaStreamSynchronize(c.stream));
        for (uint32_t k = 0; k < m; ++k) contacts[k] = c.hostSorted[order[k]];
        c.backendContacts = m;
        c.backendColored = true;
    }
    if (m == 0 && !fullSubsteps) return VXB_OK;
    const V3 g{gravity.x, gravity.y, gravity.z};
    if (fullSubsteps) {
        VXB_TRY(runSubsteps(c, P<vx_contact>(c.contactBuf[c.cur]), plan, g, h, substeps, o, warmStart, true));
    } else {
        VXB_TRY(runSubsteps(c, P<vx_contact>(c.contactBuf[c.cur]), plan, g, h, 1, o, warmStart, false));
    }
    VXB_CUDA(c, cudaGetLastError());
    VXB_TRY(readCounters(c));
    if (c.hostCounters.timeout) return fail(c, VXB_ERR_TIMEOUT, "a bounded device wait gave up");
    if (c.hostCounters.planFault) return fail(c, VXB_ERR_INTERNAL, "inconsistent island plan in the solve");
    return VXB_OK;
}

int backendFetchImpulses(Context& c, vx_contact* contacts, uint32_t m) {
    if (!c.backendColored || m != c.backendContacts || m == 0) return VXB_OK;
    VXB_TRY(ensure(c, c.contactTmpBuf, (size_t)m * sizeof(vx_contact)));
    LAUNCH(c, gatherContactsKernel, blocksFor(m, 128), 128, P<vx_contact>(c.contactBuf[c.cur]),
           P<uint32_t>(c.islandValBuf), m, P<vx_contact>(c.contactTmpBuf));
    VXB_CUDA(c, cudaMemcpyAsync(contacts, c.contactTmpBuf.ptr, (size_t)m * sizeof(vx_contact), cudaMemcpyDeviceToHost,
                                c.stream));
    VXB_CUDA(c, cudaStreamSynchronize(c.stream));
    return VXB_OK;
}

}  // namespace vxb
