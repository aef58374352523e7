"""The bounded waits of the island solve (rows that wait for their bodies): with
the context's limit cut to one poll they give up, the call reports a timeout,
and the context solves again under the default limit."""
import numpy as np
import pytest

import velox_b200 as vb
from test_gpu_island_classes import H, chain

pytestmark = pytest.mark.gpu


# A small island (four warps), a medium one (a block) and one for the grid.
@pytest.mark.parametrize("n", [40, 200, 700])
def test_a_wait_that_gives_up_is_a_timeout(ctx, n):
    bodies, hull, faces = chain(n)
    soup = vb.make_soup(hull, faces)
    c = vb.Context(0)

    def step():
        got = bodies.copy()
        contacts = c.backend_find_contacts(got, soup, 4 * H)
        c.backend_advance_substeps(got, contacts, (0.0, -9.81, 0.0), H, 4)
        return got

    want = step()
    c.set_wait_limit(1)
    with pytest.raises(vb.VeloxError) as info:
        step()
    assert info.value.status == 7  # VXB_ERR_TIMEOUT
    c.set_wait_limit(0)
    got = step()
    c.close()
    for name in ("position", "orientation", "velocity", "angularVelocity"):
        assert np.array_equal(got[name], want[name])
