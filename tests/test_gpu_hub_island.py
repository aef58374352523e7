"""A body with thousands of rows in the grid's flow: the rows follow one another
on the hub, so a plain float32 walk over them in colour order gives the same
bits, and the plan's memory grows with the rows."""
import numpy as np
import pytest
import torch

import velox_b200 as vb

pytestmark = pytest.mark.gpu

H = 1.0 / 240.0


def hub(spheres, rows):
    """A large sphere touched by small ones, several rows each."""
    rng = np.random.default_rng(rows)
    body = np.zeros(spheres + 1, vb.BODY)
    body["orientation"] = body["inertiaOrientation"] = (0, 0, 0, 1)
    body["motionType"] = 2
    body["radius"], body["invMass"], body["invInertia"] = 0.5, 1.0, 2.0
    body["radius"][0], body["invMass"][0] = 8.0, 1.0 / 1024.0
    body["velocity"] = rng.normal(0.0, 1.0, (spheres + 1, 3))
    c = np.zeros(rows, vb.CONTACT)
    other = np.sort(np.concatenate([np.arange(1, spheres + 1), rng.integers(1, spheres + 1, rows - spheres)]))
    c["a"], c["b"] = 0, other
    n = rng.normal(size=(spheres, 3))
    n = (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32)
    body["position"][1:] = -n * 8.4  # 0.1 m deep: the target velocity is zero
    tilt = n[other - 1] + rng.normal(0.0, 0.01, (rows, 3))
    normal = (tilt / np.linalg.norm(tilt, axis=1, keepdims=True)).astype(np.float32)
    c["normal"], c["localAnchorA"], c["localAnchorB"] = normal, normal * np.float32(-8.0), normal * np.float32(0.5)
    c["point"][:, 0] = np.arange(rows)  # the rows keep their order
    return body, c


def cross(a, b):
    return np.array([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]], np.float32)


def dot(a, b):
    p = a * b
    return (p[0] + p[1]) + p[2]


def walk(body, c, colors, sweeps):
    """Frictionless sweeps of isotropic spheres, row by row in colour order, in
    the solver's order of operations."""
    zero = np.float32(0.0)
    p, im, ii = body["position"], body["invMass"], body["invInertia"][:, 0]
    v, w = [x.copy() for x in body["velocity"]], [x.copy() for x in body["angularVelocity"]]
    rows = []
    for a, b, n, la, lb in zip(c["a"], c["b"], c["normal"], c["localAnchorA"], c["localAnchorB"]):
        ra, rb = (p[a] + la) - p[a], (p[b] + lb) - p[b]
        xa, xb = cross(ra, n), cross(rb, n)
        rows.append((a, b, n, ra, rb, im[a] + im[b] + dot(xa, xa * ii[a]) + dot(xb, xb * ii[b])))
    jn = np.zeros(len(c), np.float32)
    for k in np.tile(np.argsort(colors, kind="stable"), sweeps):
        a, b, n, ra, rb, mass = rows[k]
        vn = dot((v[a] + cross(w[a], ra)) - (v[b] + cross(w[b], rb)), n)
        new = max(jn[k] + (zero - vn) / mass, zero)
        imp = n * (new - jn[k])
        jn[k] = new
        v[a] = v[a] + imp * im[a]
        w[a] = w[a] + cross(ra, imp) * ii[a]
        v[b] = v[b] - imp * im[b]
        w[b] = w[b] - cross(rb, imp) * ii[b]
    return np.array(v), jn


# 16,383 and 16,384 rows on both sides of 14 bits; as many colours.
@pytest.mark.parametrize("spheres,rows", [(900, 4000), (3000, 16383), (3000, 16384)])
def test_hub_body(spheres, rows):
    body, contacts = hub(spheres, rows)
    ctx = vb.Context(0)
    colors, _ = ctx.color(body, contacts)
    assert colors.max() == rows - 1
    free = torch.cuda.mem_get_info()[0]
    options = vb.SolverOptions.default()
    options.velocityIterations = 1
    options.positionIterations = 0
    got, solved = body.copy(), contacts.copy()
    ctx.backend_advance_substeps(got, solved, (0.0, 0.0, 0.0), H, 1, options)
    held = free - torch.cuda.mem_get_info()[0]
    ctx.backend_fetch_impulses(solved)
    ctx.close()
    v, jn = walk(body, contacts, colors, 2)
    assert np.array_equal(got["velocity"], v)
    assert np.array_equal(np.sort(solved["normalImpulse"]), np.sort(jn))
    assert held < 100 << 20  # about 1 KB a row with the halves on top, and 2 MB steps
