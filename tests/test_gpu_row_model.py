"""The rows of the contact solve (two-axis friction and the cone block, rolling
and spinning resistance, restitution) in packed islands and on lanes against a
plain float64 walk over the rows in colour order (src/narrowphase.h:80-366 of the
reference)."""
import numpy as np
import pytest

import velox_b200 as vb
from solve_model import tangents
from test_gpu_class_equality import H, island

pytestmark = pytest.mark.gpu

# As in test_gpu_island_classes: some 100 rounded operations a row, passed on
# without growth by the sweeps, against the repository's bar for a whole step.
TOL = 1e-4


def rotate(q, v):
    return v + 2.0 * np.cross(q[:3], np.cross(q[:3], v) + v * q[3])


def clamped(n1, n2, max1, max2):
    n1, n2 = (n1 if max1 > 0 else 0.0), (n2 if max2 > 0 else 0.0)
    e = (n1 / max1) ** 2 if max1 > 0 else 0.0
    e += (n2 / max2) ** 2 if max2 > 0 else 0.0
    return (n1 / np.sqrt(e), n2 / np.sqrt(e)) if e > 1.0 else (n1, n2)


def walk(body, c, colors, h, sweeps, cone):
    dyn = body["motionType"] == 2
    im = np.where(dyn, body["invMass"], 0.0).astype(np.float64)
    ii = np.where(dyn, body["invInertia"][:, 0], 0.0).astype(np.float64)  # isotropic bodies
    v, w = body["velocity"].astype(np.float64), body["angularVelocity"].astype(np.float64)
    p, q = body["position"].astype(np.float64), body["orientation"].astype(np.float64)
    order = np.argsort(colors, kind="stable")
    t1s, t2s = tangents(c["normal"].astype(np.float64))
    imp = {k: np.array([c[f][k] for f in ("normalImpulse", "tangentImpulse1", "tangentImpulse2", "rollingImpulse1",
                                          "rollingImpulse2", "spinningImpulse")], np.float64) for k in order}

    def push(a, b, ra, rb, f):
        v[a] += f * im[a]
        w[a] += np.cross(ra, f) * ii[a]
        v[b] -= f * im[b]
        w[b] -= np.cross(rb, f) * ii[b]

    def turn(a, b, t):
        w[a] += t * ii[a]
        w[b] -= t * ii[b]

    rows = {}
    for k in order:
        a, b, n = c["a"][k], c["b"][k], c["normal"][k].astype(np.float64)
        ra, rb = rotate(q[a], c["localAnchorA"][k].astype(np.float64)), rotate(q[b], c["localAnchorB"][k].astype(np.float64))
        gap = c["bias0"][k] + n @ (p[a] + ra - p[b] - rb)
        axes = [n, t1s[k], t2s[k]]
        xa, xb = [np.cross(ra, d) for d in axes], [np.cross(rb, d) for d in axes]
        K = np.array([[(im[a] + im[b] if i == j else 0.0) + ii[a] * xa[i] @ xa[j] + ii[b] * xb[i] @ xb[j]
                       for j in range(3)] for i in range(3)])
        rows[k] = (a, b, axes, ra, rb, gap, K)
        m = imp[k]
        push(a, b, ra, rb, axes[0] * m[0] + axes[1] * m[1] + axes[2] * m[2])
        turn(a, b, axes[1] * m[3] + axes[2] * m[4] + axes[0] * m[5])
    for k in np.tile(order, sweeps):
        a, b, axes, ra, rb, gap, K = rows[k]
        m = imp[k]

        def rel():
            return v[a] + np.cross(w[a], ra) - v[b] - np.cross(w[b], rb)

        vn = rel() @ axes[0]
        target = -gap / h if gap > 0.0 else 0.0
        if c["vn0"][k] < -1.0 and (gap <= 0.0 or vn > 0.0):
            target = max(target, -c["restitution"][k] * c["vn0"][k])
        f1, f2 = float(c["friction1"][k]), float(c["friction2"][k])
        if cone:
            r = rel()
            d = np.linalg.solve(K, [target - vn, -(r @ axes[1]), -(r @ axes[2])])
            new = max(m[0] + d[0], 0.0)
            n1, n2 = clamped(m[1] + d[1], m[2] + d[2], f1 * new, f2 * new)
            push(a, b, ra, rb, axes[0] * (new - m[0]) + axes[1] * (n1 - m[1]) + axes[2] * (n2 - m[2]))
        else:
            new = max(m[0] + (target - vn) / K[0, 0], 0.0)
            push(a, b, ra, rb, axes[0] * (new - m[0]))
            r = rel()
            n1, n2 = clamped(m[1] - (r @ axes[1]) / K[1, 1], m[2] - (r @ axes[2]) / K[2, 2], f1 * new, f2 * new)
            push(a, b, ra, rb, axes[1] * (n1 - m[1]) + axes[2] * (n2 - m[2]))
        m[:3] = new, n1, n2
        spread = ii[a] + ii[b]
        if c["rollingFriction"][k] > 0.0:
            wr = w[a] - w[b]
            r1, r2 = m[3] - wr @ axes[1] / spread, m[4] - wr @ axes[2] / spread
            limit, size = c["rollingFriction"][k] * new, np.hypot(r1, r2)
            if size > limit:
                r1, r2 = r1 * limit / size, r2 * limit / size
            turn(a, b, axes[1] * (r1 - m[3]) + axes[2] * (r2 - m[4]))
            m[3:5] = r1, r2
        if c["spinningFriction"][k] > 0.0:
            limit = c["spinningFriction"][k] * new
            s = np.clip(m[5] - (w[a] - w[b]) @ axes[0] / spread, -limit, limit)
            turn(a, b, axes[0] * (s - m[5]))
            m[5] = s
    return v, w, imp


@pytest.mark.parametrize("idle", [0, 40, 300, 3100])  # packed, one island on warps, a block, the grid
@pytest.mark.parametrize("mode", ["plain", "rolling"])
@pytest.mark.parametrize("friction", ["two axes", "cone"])
def test_rows(ctx, friction, mode, idle):
    body, c = island(mode, idle)
    body["invInertia"][1:] = [(2.0, 2.0, 2.0), (0.9, 0.9, 0.9)]
    options = vb.SolverOptions.default()
    options.velocityIterations = 4
    options.frictionModel = 1 if friction == "cone" else 0
    c = c[np.lexsort((c["point"][:, 0], c["b"], c["a"]))]
    c["featureKey"] = np.arange(len(c))  # (a solve moves the points)
    colors, _ = ctx.color(body, c)
    real = c["bias0"] < 999.0  # the others cannot act
    v, w, imp = walk(body, c[real], colors[real], H, 8, friction == "cone")
    want = np.array([imp[k] for k in range(real.sum())])
    got = body.copy()
    ctx.backend_advance_substeps(got, c, (0.0, 0.0, 0.0), H, 1, options)
    ctx.backend_fetch_impulses(c)
    c = c[np.argsort(c["featureKey"])][real]
    assert np.abs(got["velocity"] - v).max() < TOL * max(1.0, np.abs(v).max())
    assert np.abs(got["angularVelocity"] - w).max() < TOL * max(1.0, np.abs(w).max())
    for i, name in enumerate(("normalImpulse", "tangentImpulse1", "tangentImpulse2", "rollingImpulse1",
                              "rollingImpulse2", "spinningImpulse")):
        assert np.abs(c[name] - want[:, i]).max() < TOL * max(1.0, np.abs(want).max()), name
    if mode == "rolling":
        assert np.abs(want[:, 3:]).max() > 0.0
