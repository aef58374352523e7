"""Sensor contacts take no part in the solve, however many there are: their rows
make up an island without bodies, in every solve class."""
import numpy as np
import pytest

import velox_b200 as vb
from velox_b200.binding import SPEC

pytestmark = pytest.mark.gpu


# Islands without bodies of 1 to 16 rows (packed), to 256 (one warp), to 3,072
# (a block), to 16,384 and beyond (the grid).
@pytest.mark.parametrize("touching", [1, 16, 17, 256, 257, 3072, 3073, 17000])
@pytest.mark.parametrize("moving", [False, True])
def test_sensor_rows(ctx, touching, moving):
    n = touching + 5
    s = np.zeros(n + 2, SPEC)
    s["orientation"] = (0, 0, 0, 1)
    s["shape"][0], s["planeNormal"][0] = 1, (0, 1, 0)
    side = int(np.ceil(np.sqrt(touching)))
    k = np.arange(touching)
    s["mass"], s["radius"], s["friction"] = 1.0, 0.5, 0.5
    s["mass"][0] = 0.0
    s["position"][1:touching + 1] = np.stack([k % side, np.full(touching, 0.2475), k // side], 1) * 2.0
    s["position"][touching + 1:n + 1, 0] = -20.0 - 3.0 * np.arange(5)  # beside the sensor
    s["position"][touching + 1:n + 1, 1] = 0.495
    s["velocity"][1:n + 1] = np.random.default_rng(touching).normal(0.0, 0.2, (n, 3))
    s["shape"][n + 1], s["halfExtents"][n + 1] = 2, (side + 1.0, 0.2, side + 1.0)
    s["position"][n + 1] = (side - 1.0, 1.1, side - 1.0)
    if not moving:
        s["mass"][n + 1] = 0.0
    bodies, hull, faces = vb.bodies_from_specs(s, np.zeros((0, 3), np.float32))
    soup = vb.make_soup(hull, faces)
    bodies["sensor"][n + 1] = 1
    out = []
    for world in (bodies, bodies[:n + 1].copy()):
        ctx.load(world, soup)
        ctx.configure(dt=1.0 / 60.0, substeps=4)
        ctx.step(1)
        out.append((ctx.read_bodies()[1:n + 1], ctx.read_contacts()))
    (got, contacts), (want, plain) = out
    assert len(contacts) >= len(plain) + touching
    for name in ("position", "orientation", "velocity", "angularVelocity"):
        assert np.array_equal(got[name], want[name]), name
    ctx.load(bodies, soup)
    ctx.step(3)  # warm-started
