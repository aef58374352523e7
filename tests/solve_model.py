"""One substep of the contact solve in plain numpy (float64), colour by colour:
prepared rows, warm start and two-axis friction sweeps of isotropic bodies
(src/narrowphase.h:80-366 of the reference), for checking the device's island
kernels."""
import numpy as np


def cross(a, b):
    return np.cross(a, b)


def dot(a, b):
    return (a * b).sum(axis=1)


def rotate(q, v):
    u, w = q[:, :3], q[:, 3:]
    return v + 2.0 * cross(u, cross(u, v) + v * w)


def tangents(n):
    a = np.abs(n)
    ref = np.where((a[:, 0] < a[:, 1])[:, None],
                   np.where((a[:, 0] < a[:, 2])[:, None], [[1.0, 0, 0]], [[0, 0, 1.0]]),
                   np.where((a[:, 1] < a[:, 2])[:, None], [[0, 1.0, 0]], [[0, 0, 1.0]]))
    t1 = cross(n, ref)
    t1 /= np.linalg.norm(t1, axis=1, keepdims=True)
    return t1, cross(n, t1)


def advance(bodies, contacts, colors, h, iterations):
    """(velocity, angular velocity, normal impulses) after one substep's warm
    start and sweeps; contacts carry the impulses to warm-start with."""
    f = lambda a: a.astype(np.float64)
    dyn = bodies["motionType"] == 2
    im = np.where(dyn, f(bodies["invMass"]), 0.0)
    ii = np.where(dyn, f(bodies["invInertia"][:, 0]), 0.0)  # isotropic bodies only
    p, q = f(bodies["position"]), f(bodies["orientation"])
    v, w = f(bodies["velocity"]), f(bodies["angularVelocity"])
    sphere = bodies["shape"] == 0
    a, b = contacts["a"].astype(int), contacts["b"].astype(int)
    n = f(contacts["normal"])

    def arm(body, local):
        local = f(local)
        return np.where(sphere[body][:, None], local, rotate(q[body], local))

    ra, rb = arm(a, contacts["localAnchorA"]), arm(b, contacts["localAnchorB"])
    gap = f(contacts["bias0"]) + dot(n, p[a] + ra - p[b] - rb)
    target = np.where(gap > 0.0, -gap / h, 0.0)
    rest = -f(contacts["restitution"]) * f(contacts["vn0"])
    bounce = contacts["vn0"] < -1.0
    t1, t2 = tangents(n)

    def mass(d):
        ca, cb = cross(ra, d), cross(rb, d)
        return im[a] + im[b] + ii[a] * dot(ca, ca) + ii[b] * dot(cb, cb)

    kn, k1, k2 = mass(n), mass(t1), mass(t2)
    jn, j1, j2 = f(contacts["normalImpulse"]), f(contacts["tangentImpulse1"]), f(contacts["tangentImpulse2"])
    f1, f2 = f(contacts["friction1"]), f(contacts["friction2"])
    order = [np.flatnonzero(colors == c) for c in range(int(colors.max()) + 1)]

    def push(k, imp):
        v[a[k]] += imp * im[a[k]][:, None]
        w[a[k]] += cross(ra[k], imp) * ii[a[k]][:, None]
        v[b[k]] -= imp * im[b[k]][:, None]
        w[b[k]] -= cross(rb[k], imp) * ii[b[k]][:, None]

    def relative(k):
        return v[a[k]] + cross(w[a[k]], ra[k]) - v[b[k]] - cross(w[b[k]], rb[k])

    for k in order:
        push(k, n[k] * jn[k][:, None] + t1[k] * j1[k][:, None] + t2[k] * j2[k][:, None])
    for _ in range(2 * iterations):
        for k in order:
            vn = dot(relative(k), n[k])
            tg = np.where(bounce[k] & ((gap[k] <= 0.0) | (vn > 0.0)), np.maximum(target[k], rest[k]), target[k])
            new = np.maximum(jn[k] + (tg - vn) / kn[k], 0.0)
            push(k, n[k] * (new - jn[k])[:, None])
            jn[k] = new
            rv = relative(k)
            m1, m2 = f1[k] * new, f2[k] * new
            n1 = np.where(m1 > 0.0, j1[k] - dot(rv, t1[k]) / k1[k], 0.0)
            n2 = np.where(m2 > 0.0, j2[k] - dot(rv, t2[k]) / k2[k], 0.0)
            e = np.where(m1 > 0.0, n1 / np.where(m1 > 0.0, m1, 1.0), 0.0) ** 2
            e += np.where(m2 > 0.0, n2 / np.where(m2 > 0.0, m2, 1.0), 0.0) ** 2
            s = np.where(e > 1.0, 1.0 / np.sqrt(np.maximum(e, 1.0)), 1.0)
            n1, n2 = n1 * s, n2 * s
            push(k, t1[k] * (n1 - j1[k])[:, None] + t2[k] * (n2 - j2[k])[:, None])
            j1[k], j2[k] = n1, n2
    return v, w, jn
