"""The same rows in every solve class, bit for bit. Rows that can never act (a
metre apart) are appended behind the real ones until the island is one of the
next class: packed, one warp, a block (in fewer and in more colours than its
table holds), the grid's flow. The packed solve runs the plain row routine, so
it is the reference for the lanes' split of a row."""
import numpy as np
import pytest

import velox_b200 as vb

pytestmark = pytest.mark.gpu

H = 1.0 / 240.0
REAL = 9
IDLE = [40, 240, 300, 3000, 3100]  # rows: 49, 249 (small), 309, 3009 (medium), 3109 (grid)


def island(mode, idle):
    """Two boxes of unequal inertia on the ground and against each other."""
    rng = np.random.default_rng(11)
    body = np.zeros(3, vb.BODY)
    body["orientation"] = body["inertiaOrientation"] = (0, 0, 0, 1)
    body["shape"], body["halfExtents"] = 2, (0.5, 0.4, 0.3)
    body["motionType"][1:], body["invMass"][1:] = 2, (1.0, 0.4)
    body["invInertia"][1:] = [(2.0, 3.0, 1.5), (0.7, 0.9, 1.3)]
    q = rng.normal(size=(2, 4))
    body["orientation"][1:] = q / np.linalg.norm(q, axis=1, keepdims=True)
    body["position"][1:] = [(0, 0.4, 0), (0.9, 0.45, 0.1)]
    body["velocity"][1:], body["angularVelocity"][1:] = rng.normal(0, 1, (2, 3)), rng.normal(0, 1, (2, 3))
    if mode == "locked":
        body["fixedRotation"][1] = 1
    if mode == "ground moves":
        body["motionType"][0] = 1  # kinematic
        body["velocity"][0], body["angularVelocity"][0] = (0.3, 0.0, -0.2), (0.0, 0.4, 0.0)
    if mode == "negative zeros":
        body["velocity"][1:], body["angularVelocity"][1:] = -0.0, -0.0
    c = np.zeros(REAL + idle, vb.CONTACT)
    c["a"], c["b"] = 1, 2
    c["a"][:6], c["b"][:6] = 0, [1, 1, 1, 2, 2, 2]
    n = rng.normal(0, 0.2, (REAL, 3)) + np.where(np.arange(REAL)[:, None] < 6, (0, -1, 0), (-1, 0, 0))
    c["normal"][:REAL] = n / np.linalg.norm(n, axis=1, keepdims=True)
    c["normal"][REAL:] = (-1, 0, 0)
    c["localAnchorA"][:REAL] = rng.normal(0, 0.4, (REAL, 3))
    c["localAnchorB"][:REAL] = rng.normal(0, 0.4, (REAL, 3))
    c["bias0"][:REAL] = rng.normal(0, 0.5, REAL)
    c["bias0"][REAL:] = 1000.0
    c["vn0"][:REAL], c["restitution"][:REAL] = rng.uniform(-2, 1, REAL), 0.3
    c["friction1"][:REAL], c["friction2"][:REAL] = 0.5, 0.3
    c["normalImpulse"][:REAL], c["tangentImpulse1"][:REAL] = 0.05, -0.02
    if mode == "nan":
        c["friction1"][[1, 7]], c["friction2"][4] = np.nan, np.nan
    if mode == "infinite":
        c["friction1"][[1, 7]], c["bias0"][3] = np.inf, np.inf
    if mode.startswith("rolling"):
        c["rollingFriction"][[0, 4, 7]], c["spinningFriction"][[0, 3, 8]] = 0.1, 0.2
        c["rollingImpulse1"][0], c["spinningImpulse"][8] = 0.01, -0.01
    c["point"][:, 0] = np.arange(len(c))  # order within a pair
    return body, c


@pytest.mark.parametrize("friction", ["two axes", "cone"])
@pytest.mark.parametrize("mode", ["plain", "nan", "infinite", "rolling", "locked", "ground moves", "negative zeros"])
def test_classes_agree(ctx, mode, friction):
    options = vb.SolverOptions.default()
    options.velocityIterations = 4
    options.frictionModel = 1 if friction == "cone" else 0

    def run(idle):
        body, c = island(mode, idle)
        ctx.backend_advance_substeps(body, c, (0.0, -9.81, 0.0), H, 3, options)
        ctx.backend_fetch_impulses(c)
        assert (c["bias0"] > 999).sum() == idle + (mode == "infinite")
        return body, c[np.lexsort((c["point"][:, 0], c["b"], c["a"]))]

    def bits(x):
        return np.where(np.isnan(x), np.float32(7.0), x).view(np.uint32)

    want, rows = run(0)
    assert np.abs(rows["normalImpulse"]).max() > 0.0
    for idle in IDLE:
        got, c = run(idle)
        for name in ("position", "orientation", "velocity", "angularVelocity"):
            assert np.array_equal(bits(got[name]), bits(want[name])), (idle, name)
        real = c[c["bias0"] != 1000.0] if mode != "infinite" else c[(c["bias0"] != 1000.0) | ~np.isfinite(c["bias0"])]
        for name in ("normalImpulse", "tangentImpulse1", "tangentImpulse2", "rollingImpulse1", "rollingImpulse2",
                     "spinningImpulse"):
            assert np.array_equal(bits(real[name]), bits(rows[name])), (idle, name)


# A body that the velocity solve drives to infinity: the position correction
# passes its gap on in every class alike.
def test_not_a_number_spreads_alike(ctx):
    masks = []
    for n in (40, 200, 700):
        s = np.zeros(n + 1, vb.binding.SPEC)
        s["orientation"] = (0, 0, 0, 1)
        s["shape"][n], s["planeNormal"][n] = 1, (0, 1, 0)  # last: contacts are written back with a < b
        s["mass"][:n], s["radius"][:n] = 1.0, 0.5
        s["position"][:n, 0], s["position"][:n, 1] = np.arange(n) * 0.995, 0.498
        bodies, hull, faces = vb.bodies_from_specs(s, np.zeros((0, 3), np.float32))
        ctx.load(bodies, vb.make_soup(hull, faces))
        ctx.configure(dt=4 * H, substeps=4)
        ctx.step(1)
        contacts = ctx.read_contacts()
        contacts["normalImpulse"][(contacts["a"] == 20) & (contacts["b"] == 21)] = np.inf
        ctx.write_contacts(contacts)
        ctx.step(1)
        assert (ctx.stats()["giantIslands"] == 1) == (n == 700)
        masks.append(np.isfinite(ctx.read_bodies()["position"]).all(axis=1)[:35])
    assert not masks[0].all() and masks[0].any()
    assert np.array_equal(masks[0], masks[1]) and np.array_equal(masks[0], masks[2])
