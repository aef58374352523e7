"""Device memory of tapes: a backward pass leaves as much free as it takes, what
an ended tape keeps is no more than is free beside it, and vxb_tape_end gives
everything back. Gradients do not depend on it."""
import numpy as np
import pytest
import torch

import velox_b200 as vb
from test_gpu_adjoint_segments import taped

pytestmark = pytest.mark.gpu


def free():
    return torch.cuda.mem_get_info()[0]


# 300 worlds x 44 steps of one segment: about 2 GB of tape. With 3 GiB free one
# step's tape is taken at a time, with 5 GiB the whole segment's, without room to
# grow on top.
@pytest.mark.parametrize("gib", [3, 5])
def test_a_tape_shares_the_device(gib):
    worlds, steps = 300, 44
    c = vb.Context(0)
    want = taped(c, worlds, steps, steps)
    c.tape_end()
    torch.cuda.empty_cache()
    full = free()
    filler = torch.empty(full - (gib << 30), dtype=torch.uint8, device="cuda")
    try:
        before = free()
        got = taped(c, worlds, steps, steps)
        after = free()
        assert after > 0.4 * before  # (the recorded steps themselves come on top)
        specs, pool = vb.generate_scene(5, seed=3, size=worlds)
        bodies, hull, faces = vb.bodies_from_specs(specs, pool)
        world_of = np.ascontiguousarray(specs["world"], np.uint32)
        c.load(bodies, vb.make_soup(hull, faces), world_of=world_of)  # ends the tape, memory kept
        assert before - free() <= free() + (64 << 20)
        c.tape_end()
        assert before - free() < 64 << 20
    finally:
        del filler
        torch.cuda.empty_cache()
        c.close()
    for x, y in zip(want, got):
        assert np.array_equal(x, y)
