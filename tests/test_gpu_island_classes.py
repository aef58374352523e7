"""The island solve at the edges of its classes (tiny packs, one warp, one
block, the grid's flow) against a plain numpy solve of
the same contacts, and against the same islands solved next to others."""
import numpy as np
import pytest

import velox_b200 as vb
from solve_model import advance
from velox_b200.binding import SPEC

pytestmark = pytest.mark.gpu

H = 1.0 / 240.0
# Single precision against float64 over 16 sweeps: each row rounds about 60
# operations (60 x 2^-24 = 4e-6 of the velocities), and a sweep passes them on
# without growth; 1e-4 of the largest velocity is the repository's bar for a
# whole step.
TOL = 1e-4


def chain(n, world=0, start=0.0):
    """n touching spheres in a row on a plane: one island of n bodies and about 2 n contacts."""
    s = np.zeros(n + 1, SPEC)
    s["orientation"] = (0, 0, 0, 1)
    s["world"] = world
    s["shape"][0] = 1
    s["planeNormal"][0] = (0, 1, 0)
    r = np.random.default_rng(n)
    s["mass"][1:] = r.uniform(0.5, 2.0, n)
    s["radius"][1:] = 0.5
    s["friction"][1:] = 0.5
    s["restitution"][1:] = 0.2
    s["position"][1:, 0] = start + np.arange(n) * 0.995
    s["position"][1:, 1] = 0.499
    s["velocity"][1:] = r.normal(0.0, 0.5, (n, 3))
    s["velocity"][1:, 1] -= 1.5
    s["angularVelocity"][1:] = r.normal(0.0, 1.0, (n, 3))
    return vb.bodies_from_specs(s, np.zeros((0, 3), np.float32))


def solved(ctx, bodies, soup):
    bodies = bodies.copy()
    contacts = ctx.backend_find_contacts(bodies, soup, 4 * H)
    contacts["normalImpulse"] = 0.01
    contacts["tangentImpulse1"] = -0.002
    colors, _ = ctx.color(bodies, contacts)
    want = advance(bodies, contacts, colors, H, 8)
    ctx.backend_advance_substeps(bodies, contacts, (0.0, 0.0, 0.0), H, 1)
    ctx.backend_fetch_impulses(contacts)
    return bodies, contacts, want


# bodies: 8 and 9 straddle the packed islands (16 contacts), 64 / 65 and
# 128 / 129 the one-warp class (64 bodies, 256 rows), 512 / 513 and 3072 / 3073
# the two block classes; 40 leaves a lone row in some colours.
@pytest.mark.parametrize("n", [1, 2, 8, 9, 40, 64, 65, 129, 512, 513, 3072, 3073])
def test_island_class_edges(ctx, n):
    bodies, hull, faces = chain(n)
    got, contacts, (v, w, jn) = solved(ctx, bodies, vb.make_soup(hull, faces))
    assert len(contacts) >= 2 * n - 1
    scale = max(1.0, np.abs(v).max())
    assert np.abs(got["velocity"] - v).max() < TOL * scale
    assert np.abs(got["angularVelocity"] - w).max() < TOL * max(1.0, np.abs(w).max())
    impulses = np.sort(contacts["normalImpulse"])
    assert np.abs(impulses - np.sort(jn)).max() < TOL * max(1.0, np.abs(jn).max())


def test_islands_of_every_class_side_by_side(ctx):
    """Chains of several sizes in one world, far apart: each solves as it does alone, bit for bit."""
    sizes = [3, 8, 9, 64, 65, 200, 513]
    parts, at, total = [], 0.0, 0
    for n in sizes:
        parts.append(chain(n, start=at)[0][1:])
        at += n * 0.995 + 30.0
    ground = chain(1)[0][:1]
    bodies = np.concatenate([ground] + parts).astype(vb.BODY)
    soup = vb.make_soup(np.zeros((0, 3)), np.zeros(0))
    both = vb.binding.records(bodies, vb.BODY).copy()
    contacts = ctx.backend_find_contacts(both, soup, 4 * H)
    ctx.backend_advance_substeps(both, contacts, (0.0, -9.81, 0.0), H, 4)
    at = 1
    for n, part in zip(sizes, parts):
        alone = vb.binding.records(np.concatenate([ground, part]), vb.BODY).copy()
        contacts = ctx.backend_find_contacts(alone, soup, 4 * H)
        ctx.backend_advance_substeps(alone, contacts, (0.0, -9.81, 0.0), H, 4)
        for name in ("position", "orientation", "velocity", "angularVelocity"):
            assert np.array_equal(both[name][at:at + n], alone[name][1:]), (n, name)
        at += n


def test_many_small_islands_on_one_warp_each(ctx):
    """More small islands than the GPU holds on four warps each: every one solves as it does alone, bit for bit."""
    n, islands = 12, 640
    part = chain(n)[0]
    ground, part = part[:1], part[1:]
    parts = [part.copy() for _ in range(islands)]
    for i, p in enumerate(parts):  # worlds keep the islands apart at equal coordinates
        p["velocity"][:, 0] += 0.001 * (i % 7)
    soup = vb.make_soup(np.zeros((0, 3)), np.zeros(0))
    many = np.concatenate([np.concatenate([ground, p]) for p in parts]).astype(vb.BODY)
    many = vb.binding.records(many, vb.BODY).copy()
    worlds = np.repeat(np.arange(islands, dtype=np.uint32), n + 1)
    c = vb.Context(0)
    c.load(many, soup, worlds)
    c.configure(dt=4 * H, substeps=4, gravity=(0.0, -9.81, 0.0))
    c.step(1)
    got = c.read_bodies()
    for i in (0, 3, 6, islands - 1):
        alone = vb.binding.records(np.concatenate([ground, parts[i]]).astype(vb.BODY), vb.BODY).copy()
        c.load(alone, soup)
        c.step(1)
        want = c.read_bodies()
        at = i * (n + 1)
        for name in ("position", "orientation", "velocity", "angularVelocity"):
            assert np.array_equal(got[name][at:at + n + 1], want[name]), (i, name)


# Rows of one body wait for one another through the tags in shared memory: equal
# worlds solved by many blocks at once, again and again, end in equal bits (a
# heap of 36 spheres is a small island, on four warps; one of 180 a medium one).
@pytest.mark.parametrize("layers", [1, 5])
def test_equal_crowded_islands_end_equal(ctx, layers):
    per, worlds = 36 * layers, 200
    k = np.arange(per)
    s = np.zeros(per + 1, SPEC)
    s["orientation"] = (0, 0, 0, 1)
    s["shape"][0] = 1
    s["planeNormal"][0] = (0, 1, 0)
    s["mass"][1:], s["radius"][1:], s["friction"][1:] = 1.0, 0.5, 0.5
    s["position"][1:] = np.stack([k % 6, k // 36, k // 6 % 6], 1) * 0.985 + (0.0, 0.49, 0.0)
    s["velocity"][1:] = np.random.default_rng(layers).normal(0.0, 0.3, (per, 3))
    bodies, hull, faces = vb.bodies_from_specs(s, np.zeros((0, 3), np.float32))
    many = vb.binding.records(np.concatenate([bodies] * worlds).astype(vb.BODY), vb.BODY).copy()
    world_of = np.repeat(np.arange(worlds, dtype=np.uint32), per + 1)
    first = None
    for _ in range(3):
        ctx.load(many, vb.make_soup(hull, faces), world_of)
        ctx.configure(dt=4 * H, substeps=4, gravity=(0.0, -9.81, 0.0))
        ctx.step(1)
        assert ctx.stats()["giantIslands"] == 0
        got = ctx.read_bodies()
        for name in ("position", "orientation", "velocity", "angularVelocity"):
            x = got[name].reshape(worlds, per + 1, -1)
            first = first or {}
            first.setdefault(name, x[0].copy())
            assert np.array_equal(x, np.broadcast_to(first[name], x.shape)), name
