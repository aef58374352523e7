"""The warp's distance query (overlapping pairs: tetrahedron search and EPA
shared by 32 lanes) against the one-thread GJK/EPA, bit for bit: every shape,
hulls of 4 to 70 points (one to three batches of lanes), grazing, deep and
concentric pairs, each geometry quality."""
import numpy as np
import pytest

import velox_b200 as vb

pytestmark = pytest.mark.gpu


def scene(seed, hull_points, spread):
    rng = np.random.default_rng(seed)
    kinds = [0, 2, 3, 5, 7, 8, 9, 10]
    n = 96
    body = np.zeros(n, vb.BODY)
    body["shape"] = rng.choice(kinds, n)
    body["motionType"], body["invMass"] = 2, 1.0
    body["inertiaOrientation"] = (0, 0, 0, 1)
    q = rng.normal(size=(n, 4))
    q[: n // 4] = (0, 0, 0, 1)  # aligned pairs meet face to face
    body["orientation"] = q / np.linalg.norm(q, axis=1, keepdims=True)
    body["radius"] = rng.uniform(0.1, 0.4, n)
    body["halfExtents"] = rng.uniform(0.1, 0.5, (n, 3))
    body["capsuleHalfHeight"] = rng.uniform(0.1, 0.5, n)
    body["position"] = rng.normal(0.0, spread, (n, 3))
    body["position"][: n // 4] = np.round(body["position"][: n // 4] * 2.0) / 2.0  # grid: exact touching
    body["position"][: n // 12] = 0.0  # concentric
    points = []
    for k in np.flatnonzero(body["shape"] == 5):
        count = int(rng.integers(4, hull_points + 1))
        d = rng.normal(size=(count, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        body["hullFirst"][k], body["hullCount"][k] = sum(len(p) for p in points), count
        body["radius"][k] = 0.5
        points.append(d * rng.uniform(0.2, 0.5, (count, 1)))
    soup = vb.make_soup(np.concatenate(points), np.zeros(0))
    a, b = np.triu_indices(n, 1)
    return body, soup, (a.astype(np.uint64) << np.uint64(32)) | b.astype(np.uint64)


@pytest.mark.parametrize("quality", [0, 1, 2])
@pytest.mark.parametrize("seed,hull_points,spread", [(1, 16, 0.15), (2, 16, 0.4), (3, 70, 0.2), (4, 4, 0.0)])
def test_warp_query_equals_the_thread_query(ctx, seed, hull_points, spread, quality):
    body, soup, pairs = scene(seed, hull_points, spread)
    body["geometryQuality"] = quality
    warp = ctx.distance(body, soup, pairs, path=0)
    thread = ctx.distance(body, soup, pairs, path=1)
    assert (thread[:, 10] == 1).sum() > 500
    assert np.array_equal(warp.view(np.uint32), thread.view(np.uint32))


# Hulls of many points on a sphere, deep in one another: EPA removes faces and
# reuses their slots in nearly every iteration, with horizons on both sides of
# 32 edges. Lanes pass vertices, faces and edges through shared memory, so the
# same bits must come back from every run.
@pytest.mark.parametrize("points", [24, 70])
def test_reused_face_slots(ctx, points):
    body, soup, pairs = scene(5, 4, 0.05)
    rng = np.random.default_rng(points)
    n = len(body)
    body["shape"], body["radius"] = 5, 0.5
    body["hullFirst"], body["hullCount"] = np.arange(n) * points, points
    d = rng.normal(size=(n * points, 3))
    soup = vb.make_soup(0.5 * d / np.linalg.norm(d, axis=1, keepdims=True), np.zeros(0))
    thread = ctx.distance(body, soup, pairs, path=1)
    assert (thread[:, 10] == 1).sum() > 4000
    for _ in range(3):
        assert np.array_equal(ctx.distance(body, soup, pairs, path=0).view(np.uint32), thread.view(np.uint32))
