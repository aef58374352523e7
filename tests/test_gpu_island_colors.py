"""Colouring of islands at the edges of their classes, bit for bit against the
serial greedy rule in plain Python (src/backend_cuda.cu:603-630 of the
reference): one thread, one warp, blocks of two sizes, the grid."""
import time

import numpy as np
import pytest

import velox_b200 as vb

pytestmark = pytest.mark.gpu


def greedy(contacts, dynamic, sensor):
    mask, spill, out = {}, {}, []
    for a, b in zip(contacts["a"].tolist(), contacts["b"].tolist()):
        solved = not (sensor[a] or sensor[b])
        ends = [x for x in (a, b) if solved and dynamic[x]]
        used = 0
        for x in ends:
            used |= mask.get(x, 0)
        color = next((k for k in range(64) if not used >> k & 1), None)
        if color is None:
            color = max([64] + [spill.get(x, 64) for x in ends])
            for x in ends:
                spill[x] = color + 1
        else:
            for x in ends:
                mask[x] = mask.get(x, 0) | 1 << color
        out.append(color)
    return np.array(out, np.int32)


# (bodies of the island, contacts): tiny 16 / 17 contacts, one warp 64 bodies
# or 256 contacts, blocks 512 bodies / 3,072 contacts and 3,072 bodies / 16,384
# contacts, and beyond; a hub body gives chains past 64 colours.
@pytest.mark.parametrize("bodies,rows,hub", [
    (5, 16, 0), (5, 17, 0), (64, 256, 0), (64, 257, 0), (65, 200, 0), (40, 250, 150), (512, 3072, 0),
    (512, 3073, 400), (513, 600, 0), (3072, 16384, 0), (3072, 16385, 200), (3073, 3500, 0)])
@pytest.mark.parametrize("seed", [1, 2])
def test_colors_equal_the_serial_rule(ctx, bodies, rows, hub, seed):
    rng = np.random.default_rng(seed)
    n = bodies + 3  # a static body, a sensor and a free body beside the island
    pairs = set()
    for k in range(1, bodies):  # connected
        pairs.add((int(rng.integers(max(0, k - 4), k)), k))
    listed = [p for p in pairs]
    while len(listed) < rows:
        if hub and len(listed) < bodies - 1 + hub:
            a, b = 0, int(rng.integers(1, bodies))
        else:
            a, b = sorted(int(x) for x in rng.integers(0, bodies + 2, 2))
        if a == b or a >= bodies:
            continue
        if b >= bodies and rng.random() < 0.5:
            continue
        listed.append((a, b))  # several contacts per pair are ordinary
    listed.sort()
    body = np.zeros(n, vb.BODY)
    body["orientation"] = (0, 0, 0, 1)
    body["inertiaOrientation"] = (0, 0, 0, 1)
    body["radius"], body["invMass"], body["motionType"] = 0.5, 1.0, 2
    body["motionType"][bodies], body["invMass"][bodies] = 0, 0.0
    body["sensor"][bodies + 1] = 1
    contacts = np.zeros(rows, vb.CONTACT)
    contacts["a"], contacts["b"] = np.array(listed, np.uint32).T
    colors, count = ctx.color(body, contacts)
    want = greedy(contacts, body["motionType"] == 2, body["sensor"] != 0)
    assert np.array_equal(colors, want)
    assert count == want.max() + 1


# Rows of one body: lists of up to 64 are sorted by a thread, longer ones picked
# in order by a warp. One warp, both block sizes.
@pytest.mark.parametrize("length", [64, 65, 250, 3000, 16384])
def test_long_lists_keep_their_order(ctx, length):
    rng = np.random.default_rng(length)
    bodies = min(length // 2 + 2, 3000)
    body = np.zeros(bodies, vb.BODY)
    body["orientation"] = body["inertiaOrientation"] = (0, 0, 0, 1)
    body["radius"], body["invMass"], body["motionType"] = 0.5, 1.0, 2
    hub = bodies // 2  # the first end of some rows, the second of others
    other = np.concatenate([np.delete(np.arange(bodies), hub), rng.integers(0, bodies, length)])
    other = other[other != hub][:length]
    contacts = np.zeros(len(other), vb.CONTACT)
    contacts["a"], contacts["b"] = np.sort(np.stack([other, np.full(len(other), hub)], 1), axis=1).T
    contacts = contacts[np.lexsort((contacts["b"], contacts["a"]))]
    times = []
    for _ in range(3):
        start = time.perf_counter()
        colors, count = ctx.color(body, contacts)
        times.append(time.perf_counter() - start)
    assert np.array_equal(colors, greedy(contacts, body["motionType"] == 2, body["sensor"] != 0))
    assert count == len(other)
    assert min(times) < 0.06  # 8 ms for the longest, 109 ms when its thread sorts it
