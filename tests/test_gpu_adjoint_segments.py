"""The backward pass does not depend on how its segments are taped: every
checkpoint spacing (one slot, a remainder, one segment) and, beyond the scratch
limit, the step-by-step tape give the same gradients bit for bit, since each
recomputes the same states."""
import numpy as np
import pytest

import velox_b200 as vb
from velox_b200.binding import SPEC

pytestmark = pytest.mark.gpu


def taped(ctx, worlds, steps, every):
    specs, pool = vb.generate_scene(5, seed=3, size=worlds)
    bodies, hull, faces = vb.bodies_from_specs(specs, pool)
    ctx.load(bodies, vb.make_soup(hull, faces), world_of=np.ascontiguousarray(specs["world"], np.uint32))
    ctx.configure(substeps=4)
    ctx.tape_begin(steps, every)
    ctx.step(steps)
    seed = np.random.default_rng(1).normal(size=(len(bodies), 13)).astype(np.float32)
    return ctx.adjoint_backward(seed)


def gradients(worlds, steps, every):
    ctx = vb.Context(0)
    try:
        return taped(ctx, worlds, steps, every)
    finally:
        ctx.close()


# 900 worlds x 44 steps a segment exceed the 4 GiB of scratch (about 150 KB a
# world and step), 900 x 4 do not; 5 worlds share no block, 300 do. A world's
# rows lie in shared memory throughout (about 15 KB a world).
@pytest.mark.parametrize("worlds,steps,spacings", [(5, 7, (1, 2, 7)), (300, 6, (1, 4, 6)), (900, 44, (4, 44))])
def test_gradients_do_not_depend_on_the_tape(worlds, steps, spacings):
    first = gradients(worlds, steps, spacings[0])
    assert np.abs(first[0]).max() > 0.0 and (first[3] == 0).any()
    for every in spacings[1:]:
        for x, y in zip(first, gradients(worlds, steps, every)):
            assert np.array_equal(x, y), every


# A context's tapes share memory from one to the next: larger, smaller, after
# an untaped world (which gives it back) and after vxb_tape_end.
@pytest.mark.parametrize("between", ["nothing", "untaped", "end"])
def test_tapes_of_one_context_are_independent(ctx, between):
    for worlds, steps, every in [(20, 5, 2), (3, 9, 4), (40, 5, 5), (20, 5, 2)]:
        for x, y in zip(gradients(worlds, steps, every), taped(ctx, worlds, steps, every)):
            assert np.array_equal(x, y), (worlds, steps, every)
        if between == "untaped":
            specs, pool = vb.generate_scene(5, seed=4, size=7)
            bodies, hull, faces = vb.bodies_from_specs(specs, pool)
            for _ in range(2):
                ctx.load(bodies, vb.make_soup(hull, faces), world_of=np.ascontiguousarray(specs["world"], np.uint32))
                ctx.step(1)
        elif between == "end":
            ctx.tape_end()


def piles(heaps, per):
    """Worlds of `per` spheres dropped on a plane in a close grid."""
    s = np.zeros(heaps * (per + 1), SPEC)
    s["orientation"] = (0, 0, 0, 1)
    for h in range(heaps):
        at = h * (per + 1)
        s["world"][at:at + per + 1] = h
        s["shape"][at] = 1
        s["planeNormal"][at] = (0, 1, 0)
        r = np.random.default_rng(h)
        k = np.arange(per)
        body = slice(at + 1, at + 1 + per)
        s["mass"][body] = 1.0
        s["radius"][body] = 0.5
        s["friction"][body] = 0.5
        s["position"][body, 0] = (k % 8) * 0.98
        s["position"][body, 1] = 0.49 + (k // 64) * 0.98
        s["position"][body, 2] = (k // 8 % 8) * 0.98
        s["velocity"][body] = r.normal(0.0, 0.1, (per, 3))
    return s


# Worlds of 3 spheres hold their rows in shared memory, of 150 (about 500 rows
# of some 450 bytes, 225 KB) in global memory, and so does a small one that is
# taped beside a large one: its gradients are the same bit for bit. Two steps
# of frozen contacts without a rewind (the spheres start in touch).
def test_gradients_do_not_depend_on_where_the_rows_lie(ctx):
    small, large = piles(1, 3), piles(1, 150)
    large["world"] = 1
    both = np.concatenate([small, large]).astype(SPEC)  # (concatenate packs the records)

    def run(specs):
        bodies, hull, faces = vb.bodies_from_specs(specs, np.zeros((0, 3), np.float32))
        ctx.load(bodies, vb.make_soup(hull, faces), world_of=np.ascontiguousarray(specs["world"], np.uint32))
        ctx.configure(substeps=4)
        ctx.tape_begin(2, 2)
        ctx.step(2)
        seed = np.ones((len(bodies), 13), np.float32)
        return ctx.adjoint_backward(seed)

    alone, beside = run(small), run(both)
    assert alone[3][0] == beside[3][0] == 0
    assert np.abs(alone[0]).max() > 0.0
    for x, y in zip(alone[:3], beside[:3]):
        assert np.array_equal(x, y[:len(x)])
