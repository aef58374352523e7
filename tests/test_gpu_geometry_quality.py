"""Robust and Paranoid bodies among Normal ones: the step's narrow phase (lists
by kind of query) against the unclassified one-thread-per-pair entry point, and
the same through a snapshot that brings such bodies into another world."""
import numpy as np
import pytest

import velox_b200 as vb
from scenes import scene
from velox_b200.binding import COMPOUND_CHILD, CONTACT_FLOAT_FIELDS

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def world(size, qualities, compounds=True):
    specs, pool = scene("dense", size)
    bodies, hull, faces = vb.bodies_from_specs(specs, pool)
    rng = np.random.default_rng(size)
    bodies["geometryQuality"] = rng.choice(qualities, len(bodies))
    parts = {}
    if compounds:
        child = np.zeros(2, COMPOUND_CHILD)
        child["shape"], child["localOrientation"] = (0, 2), (0, 0, 0, 1)
        child["localPosition"] = [(0.3, 0, 0), (-0.3, 0, 0)]
        child["radius"], child["halfExtents"] = 0.4, (0.3, 0.2, 0.3)
        boxes = np.flatnonzero(bodies["shape"] == 2)[::3]
        bodies["shape"][boxes], bodies["compoundCount"][boxes], bodies["radius"][boxes] = vb.binding.SHAPE["compound"], 2, 0.8
        parts["children"] = child
    return bodies, vb.make_soup(hull, faces, **parts)


def ordered(contacts):
    return contacts[np.lexsort([contacts[f].reshape(len(contacts), -1)[:, 0] for f in ("featureKey", "gap", "point")] +
                               [contacts["b"], contacts["a"]])]


@pytest.mark.parametrize("qualities", [(0,), (1,), (2,), (0, 1, 2)])
def test_contacts_equal_the_unclassified_pairs(ctx, qualities):
    bodies, soup = world(700, qualities)
    got = ordered(ctx.backend_find_contacts(bodies, soup, DT))
    want = ordered(ctx.collide(bodies, soup, ctx.pairs(bodies, DT, soup), DT)[0])
    assert len(want) > 500
    for name in ["a", "b", "featureKey"] + CONTACT_FLOAT_FIELDS:
        assert np.array_equal(got[name], want[name]), name


def test_a_snapshot_brings_the_geometry_quality(ctx):
    bodies, soup = world(400, (1, 2), compounds=False)
    plain = bodies.copy()
    plain["geometryQuality"] = 0
    ctx.load(bodies, soup)
    ctx.configure(dt=DT, substeps=4)
    ctx.step(3)
    image = ctx.snapshot_bytes()
    other = vb.Context(0)
    other.load(plain, soup)
    for source in ("image", "slot"):
        if source == "image":
            other.snapshot_load(image)
            other.snapshot_save(1)
        else:
            other.load(plain, soup)
            other.snapshot_restore(1)
        if source == "image":
            ctx.step(3)
        other.step(3)
        assert other.stats()["contacts"] == ctx.stats()["contacts"] > 0
        for name in ("position", "orientation", "velocity", "angularVelocity"):
            assert np.array_equal(other.read_bodies()[name], ctx.read_bodies()[name]), name
    other.close()


# The serial routine runs a thread a pair: what the classified narrow phase adds
# to it is small, and one lane of a warp each took twice the time.
@pytest.mark.parametrize("quality", [1, 2])
def test_general_pairs_run_a_thread_each(quality):
    bodies, soup = world(12000, (quality,), compounds=False)
    c = vb.Context(0)
    pairs = c.pairs(bodies, DT)
    c.enable_timing(True)

    def stage(call):
        times = []
        for _ in range(4):
            before = c.stage_times()["narrowphase"][0]
            call()
            times.append(c.stage_times()["narrowphase"][0] - before)
        return min(times)

    classified = stage(lambda: c.backend_find_contacts(bodies, soup, DT))
    threads = stage(lambda: c.collide(bodies, soup, pairs, DT))
    c.close()
    print("narrow phase, quality", quality, len(pairs), "pairs:", classified, "against", threads, "ms")
    assert classified < 1.4 * threads


# Compounds: many child pairs, most of them apart. A warp a pair took three
# times the thread's time.
def test_compounds_run_a_thread_each():
    bodies, soup = world(12000, (0,))
    dyn = np.flatnonzero(bodies["motionType"] == 2)
    bodies["shape"][dyn], bodies["compoundFirst"][dyn], bodies["compoundCount"][dyn] = vb.binding.SHAPE["compound"], 0, 2
    bodies["radius"][dyn] = 0.8
    c = vb.Context(0)
    pairs = c.pairs(bodies, DT, soup)
    c.enable_timing(True)

    def stage(call):
        times = []
        for _ in range(4):
            before = c.stage_times()["narrowphase"][0]
            call()
            times.append(c.stage_times()["narrowphase"][0] - before)
        return min(times)

    classified = stage(lambda: c.backend_find_contacts(bodies, soup, DT))
    threads = stage(lambda: c.collide(bodies, soup, pairs, DT))
    c.close()
    print("narrow phase of compounds,", len(pairs), "pairs:", classified, "against", threads, "ms")
    assert classified < 1.4 * threads


# Box stacks: pairs in touch and just apart. Their face clipping runs in one pass;
# done in two, one behind the other, the classified phase lost to a thread a pair
# (0.48 against 0.41 ms; 0.27 in one).
def test_box_stacks_clip_their_faces_in_one_pass():
    specs, pool = vb.generate_scene(3, seed=3, size=2)
    bodies, hull, faces = vb.bodies_from_specs(specs, pool)
    soup = vb.make_soup(hull, faces)
    c = vb.Context(0)
    c.load(bodies, soup)
    c.configure(dt=DT, substeps=8)
    c.step(6)
    bodies = c.read_bodies()
    pairs = c.pairs(bodies, DT, soup)
    c.enable_timing(True)

    def stage(call):
        times = []
        for _ in range(6):
            before = c.stage_times()["narrowphase"][0]
            call()
            times.append(c.stage_times()["narrowphase"][0] - before)
        return min(times)

    classified = stage(lambda: c.backend_find_contacts(bodies, soup, DT))
    threads = stage(lambda: c.collide(bodies, soup, pairs, DT))
    c.close()
    print("narrow phase of box stacks:", classified, "against", threads, "ms")
    assert classified < threads
