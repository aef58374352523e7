"""Bodies and compounds against a triangle mesh, whose triangles the step's narrow
phase shares among a warp's lanes, against the unclassified one-thread-per-pair
entry point: one batch of triangles, several, and a remainder."""
import numpy as np
import pytest

import velox_b200 as vb
from test_gpu_geometry_quality import ordered
from velox_b200.binding import BVH_NODE, COMPOUND_CHILD, CONTACT_FLOAT_FIELDS, MESH, SHAPE

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def field(side, spacing):
    """A bumpy grid of triangles under a root with two leaves."""
    rng = np.random.default_rng(side)
    i, j = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    vertices = np.stack([i * spacing, 0.15 * rng.standard_normal(i.shape), j * spacing], -1).reshape(-1, 3)
    vertices = vertices.astype(np.float32)
    v = (i * side + j)[:-1, :-1].reshape(-1)
    tris = np.concatenate([np.stack([v, v + 1, v + side], 1), np.stack([v + 1, v + side + 1, v + side], 1)])
    corner = vertices[tris]
    order = np.argsort(corner[:, :, 0].mean(axis=1), kind="stable")
    half = len(order) // 2
    nodes = np.zeros(3, BVH_NODE)
    for k, part in enumerate((order, order[:half], order[half:])):
        nodes[k]["aabbMin"], nodes[k]["aabbMax"] = corner[part].min(axis=(0, 1)), corner[part].max(axis=(0, 1))
    nodes["leftFirst"], nodes["triCount"] = (1, 0, half), (0, half, len(order) - half)
    mesh = np.zeros(1, MESH)
    mesh["vertexCount"], mesh["indexCount"], mesh["nodeCount"] = len(vertices), 3 * len(tris), 3
    mesh["aabbMin"], mesh["aabbMax"] = vertices.min(axis=0), vertices.max(axis=0)
    return dict(vertices=vertices, indices=tris.astype(np.uint32), meshes=mesh, nodes=nodes,
                tri_refs=order.astype(np.uint32))


@pytest.mark.parametrize("side", [3, 6, 9])  # 8, 50 and 128 triangles
@pytest.mark.parametrize("qualities", [(0,), (0, 1, 2)])
def test_mesh_contacts_equal_the_unclassified_pairs(ctx, side, qualities):
    specs, pool = vb.generate_scene(2, seed=side, size=300)
    bodies, hull, faces = vb.bodies_from_specs(specs, pool)
    parts = field(side, 8.0 / side)
    rng = np.random.default_rng(side)
    ground = bodies["shape"] == SHAPE["plane"]
    bodies["shape"][ground], bodies["meshIndex"][ground] = SHAPE["mesh"], 0
    dyn = np.flatnonzero(~ground)
    bodies["position"][dyn] = rng.uniform((0, -0.2, 0), (8, 0.6, 8), (len(dyn), 3))
    bodies["geometryQuality"][dyn] = rng.choice(qualities, len(dyn))
    child = np.zeros(2, COMPOUND_CHILD)
    child["shape"], child["localOrientation"] = (SHAPE["capsule"], SHAPE["box"]), (0, 0, 0, 1)
    child["localPosition"] = [(0.3, 0, 0), (-0.3, 0, 0)]
    child["radius"], child["capsuleHalfHeight"], child["halfExtents"] = 0.3, 0.2, (0.3, 0.2, 0.3)
    boxes = np.flatnonzero(bodies["shape"] == SHAPE["box"])[::2]
    bodies["shape"][boxes], bodies["compoundCount"][boxes], bodies["radius"][boxes] = SHAPE["compound"], 2, 0.8
    soup = vb.make_soup(hull, faces, children=child, **parts)
    got = ordered(ctx.backend_find_contacts(bodies, soup, DT))
    want = ordered(ctx.collide(bodies, soup, ctx.pairs(bodies, DT, soup), DT)[0])
    mesh = np.flatnonzero(ground)
    assert (np.isin(want["a"], mesh) | np.isin(want["b"], mesh)).sum() > 200
    for name in ["a", "b", "featureKey"] + CONTACT_FLOAT_FIELDS:
        assert np.array_equal(got[name], want[name]), name
