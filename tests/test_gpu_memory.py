"""What a solve allocates beyond what loading the bodies reserved."""
import numpy as np
import pytest
import torch

import velox_b200 as vb

pytestmark = pytest.mark.gpu


def test_rows_of_a_first_solve_fit_the_reserved_memory():
    n = 400_000
    body = np.zeros(n, vb.BODY)
    body["orientation"] = body["inertiaOrientation"] = (0, 0, 0, 1)
    body["motionType"], body["invMass"], body["invInertia"], body["radius"] = 2, 1.0, 2.0, 0.5
    body["position"][:, 0] = np.arange(n)
    contacts = np.zeros(2 * n, vb.CONTACT)  # pairs of bodies, four rows each
    contacts["a"] = np.arange(2 * n) // 4 * 2
    contacts["b"] = contacts["a"] + 1
    contacts["normal"] = (-1, 0, 0)
    contacts["localAnchorA"], contacts["localAnchorB"] = (0.5, 0, 0), (-0.5, 0, 0)
    ctx = vb.Context(0)
    ctx.backend_integrate(body, (0.0, 0.0, 0.0), 1.0 / 240.0)
    before = torch.cuda.mem_get_info()[0]
    ctx.backend_advance_substeps(body, contacts, (0.0, 0.0, 0.0), 1.0 / 240.0, 1)
    held = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    # the plan's per-body and per-row words: about 100 bytes a body and 60 a row,
    # half as much on top; the rows' prepared terms would be 384 bytes a row
    assert held < 250 << 20


def test_a_world_loads_without_the_reserve():
    """Memory for rows that a world may never have is asked for, not required."""
    n = 400_000
    body = np.zeros(n, vb.BODY)
    body["orientation"] = body["inertiaOrientation"] = (0, 0, 0, 1)
    body["motionType"], body["invMass"], body["invInertia"], body["radius"] = 2, 1.0, 2.0, 0.5
    body["position"][:, 0] = 3.0 * np.arange(n)

    def advance(ctx):
        moved = body.copy()
        ctx.backend_integrate(moved, (0.0, -9.81, 0.0), 1.0 / 60.0)
        return moved["velocity"]

    ctx = vb.Context(0)
    before = torch.cuda.mem_get_info()[0]
    want = advance(ctx)
    held = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    # the reserve is 2 x 252 bytes a body and half as much on top: 300 MB
    filler = torch.empty(torch.cuda.mem_get_info()[0] - held + (200 << 20), dtype=torch.uint8, device="cuda")
    ctx = vb.Context(0)
    try:
        assert np.array_equal(advance(ctx), want)
    finally:
        ctx.close()
        del filler
        torch.cuda.empty_cache()
