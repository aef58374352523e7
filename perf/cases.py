"""Performance cases of the contact pipeline, through its public entry points.

A world case is a frame of a running simulation: the world is loaded and
stepped into the situation that the case is about when it is prepared, and a
pass rolls it back to that state (vxb_world_snapshot_restore, as a rollback or
a sampling controller does), steps it and reads the poses into pinned host
memory. The other two kinds are a training step through autograd and a frame
of a host engine that calls the Backend entry points with its own arrays.

Inputs come from the seed alone: the library's scene generators (the shapes,
sizes and densities of the benchmark workloads) and numpy.
"""
import math

import numpy as np
import torch

from velox_b200 import BODY, Context, SolverOptions, bodies_from_specs, generate_scene, make_soup
from velox_b200.autograd import Rollout
from velox_b200.binding import BVH_NODE, MESH, SHAPE

DT = 1.0 / 60.0
GRAVITY = (0.0, -9.81, 0.0)
CONTACT_SLOTS = 16  # contact or event records per body that a host program keeps room for

# Contacts per body in the state that a kind of case is measured in (rounded
# from vxb_world_stats), for the arithmetic that a step cannot do without.
CONTACTS = {"lattice": 4.0, "drop": 0.2, "heap": 5.0, "pyramids": 8.0, "batch": 0.7, "rollout": 4.0,
            "backend": 5.0, "sleep": 4.0, "terrain": 2.0}


def listed():
    return [
        # one agent's scene, four steps per control interval: launches and latency
        {"name": "lattice_64", "kind": "lattice", "size": 4, "settle": 40, "steps": 4, "substeps": 4, "forces": True},
        # a small game scene, a thousand boxes tumbling onto the ground, one frame with forces from the game
        {"name": "lattice_1000", "kind": "lattice", "size": 10, "settle": 45, "steps": 1, "substeps": 4,
         "forces": True},
        # the benchmark scene while most bodies still fall: broad phase and free bodies
        {"name": "drop_100000", "kind": "drop", "size": 100000, "settle": 4, "steps": 1, "substeps": 4,
         "forces": False},
        # heaps of mixed shapes: one island, many colours, rewinds; a mid-sized one of an odd size and a large one
        {"name": "heap_2999", "kind": "heap", "size": 2999, "settle": 60, "steps": 1, "substeps": 4, "forces": False},
        {"name": "heap_40000", "kind": "heap", "size": 40000, "settle": 60, "steps": 1, "substeps": 4,
         "forces": False},
        # stacking: box pyramids at eight substeps, islands of one block each
        {"name": "pyramids_64", "kind": "pyramids", "size": 64, "settle": 6, "steps": 1, "substeps": 8,
         "forces": False},
        # batches of independent worlds, as sampling and learning use them: a few and the benchmark's 4,096
        {"name": "batch_48", "kind": "batch", "size": 48, "settle": 50, "steps": 2, "substeps": 4, "forces": True},
        {"name": "batch_4096", "kind": "batch", "size": 4096, "settle": 60, "steps": 1, "substeps": 4,
         "forces": False},
        # gradients of a rollout: taped forward and adjoint backward through torch
        {"name": "rollout_128", "kind": "rollout", "size": 128, "settle": 24, "steps": 24, "substeps": 4,
         "forces": False},
        # a host engine on the Backend interface: its arrays in and out each frame
        {"name": "backend_4001", "kind": "backend", "size": 4001, "settle": 50, "steps": 1, "substeps": 4,
         "forces": False},
        # a scene coming to rest with sleeping and contact events on
        {"name": "sleep_729", "kind": "sleep", "size": 9, "settle": 75, "steps": 1, "substeps": 4, "forces": False},
        # mixed shapes landing on a heightfield mesh
        {"name": "terrain_2500", "kind": "terrain", "size": 2500, "settle": 35, "steps": 1, "substeps": 4,
         "forces": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; sizes log-uniform over the range that the listed cases of its kind stand for."""
    kind = rng.choice(["lattice", "drop", "heap", "heap", "pyramids", "batch", "rollout", "backend", "sleep",
                       "terrain"])
    c = {"kind": kind, "steps": 1, "substeps": 4, "forces": False}
    if kind == "lattice":
        c.update(size=rng.randint(3, 13), settle=rng.randint(20, 60), steps=rng.randint(1, 4),
                 forces=rng.random() < 0.5)
    elif kind == "drop":
        c.update(size=_log(rng, 500, 60000), settle=rng.randint(2, 12), substeps=rng.choice([1, 2, 4]))
    elif kind == "heap":
        c.update(size=_log(rng, 300, 30000), settle=rng.randint(40, 70), substeps=rng.choice([2, 4]))
    elif kind == "pyramids":
        c.update(size=_log(rng, 2, 90), settle=rng.randint(3, 9), substeps=rng.choice([4, 8]))
    elif kind == "batch":
        c.update(size=_log(rng, 8, 1500), settle=rng.randint(5, 50), steps=rng.randint(1, 2),
                 forces=rng.random() < 0.5)
    elif kind == "rollout":
        steps = rng.randint(10, 30)
        c.update(size=_log(rng, 8, 256), settle=steps, steps=steps)
    elif kind == "backend":
        c.update(size=_log(rng, 200, 12000), settle=rng.randint(30, 60))
    elif kind == "sleep":
        c.update(size=rng.randint(4, 11), settle=rng.randint(60, 90))
    else:
        c.update(size=_log(rng, 300, 8000), settle=rng.randint(25, 45))
    return c


# ---- scenes ----------------------------------------------------------------


def _heap_specs(n, seed):
    """The benchmark's mixed shapes on a jittered lattice 12 layers high, at rest: they drop into one heap."""
    specs, pool = generate_scene(2, seed=seed, size=n)
    rng = np.random.default_rng(seed)
    dyn = np.flatnonzero(specs["shape"] != SHAPE["plane"])
    side = int(math.ceil(math.sqrt(len(dyn) / 12.0)))
    cell = rng.permutation(len(dyn))
    at = np.stack([cell % side, cell // (side * side), (cell // side) % side], axis=1).astype(np.float64)
    at = at * 1.5 + rng.uniform(-0.1, 0.1, at.shape)
    at -= np.array([0.75 * side, -1.1, 0.75 * side])
    specs["position"][dyn] = at
    specs["velocity"][dyn] = rng.normal(0.0, 0.3, at.shape)
    return specs, pool


def _heightfield(side, spacing, seed):
    """A triangulated heightfield with a bounding volume hierarchy over its triangles (median splits, leaves of
    at most four, an inner node's children after it)."""
    rng = np.random.default_rng(seed)
    u = np.arange(side) - 0.5 * (side - 1)
    x, z = np.meshgrid(u * spacing, u * spacing, indexing="ij")
    a, b = rng.uniform(0.15, 0.3, 2)
    y = 0.8 * np.sin(a * x) * np.cos(b * z) + 0.1 * rng.standard_normal(x.shape)
    vertices = np.stack([x, y, z], axis=-1).reshape(-1, 3).astype(np.float32)
    i, j = np.meshgrid(np.arange(side - 1), np.arange(side - 1), indexing="ij")
    v = (i * side + j).reshape(-1)
    tris = np.concatenate([np.stack([v, v + 1, v + side], 1), np.stack([v + 1, v + side + 1, v + side], 1)])
    corner = vertices[tris]
    lo, hi = corner.min(axis=1), corner.max(axis=1)
    centre = (lo + hi) * 0.5
    nodes, refs, work = [None], [], [(0, np.arange(len(tris)))]
    while work:
        at, t = work.pop()
        box = (lo[t].min(axis=0), hi[t].max(axis=0))
        if len(t) <= 4:
            nodes[at] = (*box, len(refs), len(t))
            refs.extend(t.tolist())
            continue
        axis = int(np.argmax(centre[t].max(axis=0) - centre[t].min(axis=0)))
        t = t[np.argsort(centre[t, axis], kind="stable")]
        nodes[at] = (*box, len(nodes), 0)
        work += [(len(nodes), t[:len(t) // 2]), (len(nodes) + 1, t[len(t) // 2:])]
        nodes += [None, None]
    mesh = np.zeros(1, MESH)
    mesh["vertexCount"], mesh["indexCount"], mesh["nodeCount"] = len(vertices), 3 * len(tris), len(nodes)
    mesh["aabbMin"], mesh["aabbMax"] = vertices.min(axis=0), vertices.max(axis=0)
    return dict(vertices=vertices, indices=tris.astype(np.uint32), meshes=mesh, nodes=np.array(nodes, BVH_NODE),
                tri_refs=np.array(refs, np.uint32))


def _scene(case, seed):
    """(bodies, soup, world of each body or None)"""
    kind, size = case["kind"], case["size"]
    if kind in ("heap", "backend", "terrain"):
        specs, pool = _heap_specs(size, seed)
    else:
        number = {"lattice": 1, "sleep": 1, "drop": 2, "pyramids": 3, "batch": 4, "rollout": 5}[kind]
        # the worlds' sizes and shapes are the batch's own; the seed then moves its bodies
        specs, pool = generate_scene(number, seed=number if kind == "batch" else seed, size=size)
    if kind == "batch":
        rng = np.random.default_rng(seed + 4)
        dyn = specs["shape"] != SHAPE["plane"]
        specs["velocity"][dyn] = rng.normal(0.0, 0.5, (int(dyn.sum()), 3))
        specs["angularVelocity"][dyn] = rng.normal(0.0, 0.5, (int(dyn.sum()), 3))
    if kind == "sleep":
        specs["enableSleep"] = 1
    if kind == "terrain":
        # two layers over the field instead of the heap's twelve
        dyn = np.flatnonzero(specs["shape"] != SHAPE["plane"])
        rng = np.random.default_rng(seed + 1)
        side = int(math.ceil(math.sqrt(len(dyn) / 2.0)))
        cell = rng.permutation(len(dyn))
        at = np.stack([cell % side, cell // (side * side), (cell // side) % side], axis=1).astype(np.float64)
        specs["position"][dyn] = at * 1.7 + np.array([-0.85 * side, 2.2, -0.85 * side])
    bodies, hull, faces = bodies_from_specs(specs, pool)
    parts = {}
    if kind == "terrain":
        parts = _heightfield(int(1.7 * side / 1.25) + 6, 1.25, seed + 2)
        ground = bodies["shape"] == SHAPE["plane"]
        bodies["shape"][ground] = SHAPE["mesh"]
        bodies["meshIndex"][ground] = 0
    world_of = np.ascontiguousarray(specs["world"], np.uint32) if kind in ("batch", "rollout") else None
    return bodies, make_soup(hull, faces, **parts), world_of


# ---- the contract: prepare, run, work, exact ---------------------------------


def prepare(case, seed):
    seed = int(seed) % (1 << 31) + 1
    bodies, soup, world_of = _scene(case, seed)
    n = len(bodies)
    rng = np.random.default_rng(seed + 3)
    if case["kind"] == "rollout":
        rollout = Rollout(bodies, soup, world_of=world_of, steps=case["steps"], dt=DT, substeps=case["substeps"])
        mass = rollout.mass0 * rng.uniform(0.8, 1.25, n)

        def leaf(x):
            return torch.tensor(x, dtype=torch.float32, device="cuda", requires_grad=True)

        target = bodies["position"] + rng.uniform(-0.5, 0.5, (n, 3))
        return {"rollout": rollout, "v": leaf(bodies["velocity"]), "w": leaf(bodies["angularVelocity"]),
                "m": leaf(mass), "target": torch.tensor(target, dtype=torch.float32, device="cuda")}
    ctx = Context(0)
    ctx.load(bodies, soup, world_of=world_of)
    ctx.configure(dt=DT, substeps=case["substeps"], gravity=GRAVITY)
    if case["kind"] == "sleep":
        ctx.enable_events(True)
    ctx.step(case["settle"])
    if case["kind"] == "backend":
        # the engine keeps the bodies; its library context starts afresh
        settled = ctx.read_bodies()
        for name in ("position", "orientation", "velocity", "angularVelocity"):
            bodies[name] = settled[name]
        ctx.close()
        return {"ctx": Context(0), "bodies": bodies, "soup": soup, "substeps": case["substeps"]}
    ctx.snapshot_save(0)
    state = {"ctx": ctx, "soup": soup, "steps": case["steps"], "events": case["kind"] == "sleep",
             "poses": torch.empty((n, 7), dtype=torch.float32, pin_memory=True).numpy(), "forces": None}
    if case["forces"]:
        forces = torch.zeros((n, 6), dtype=torch.float32, pin_memory=True).numpy()
        forces[:] = rng.normal(0.0, 2.0, (n, 6))
        state["forces"] = forces
    return state


def _train(s):
    for x in (s["v"], s["w"], s["m"]):
        x.grad = None
    position = s["rollout"](s["v"], s["w"], s["m"])
    loss = ((position - s["target"]) ** 2).sum()
    loss.backward()
    return {"position": position.detach(), "v": s["v"].grad, "w": s["w"].grad, "m": s["m"].grad}


def _padded(records, names, slots):
    """Fields of the records as the caller's arrays of a fixed capacity, and how many there are."""
    count = min(len(records), slots)
    out = {"count": len(records)}
    for name in names:
        out[name] = np.zeros((slots,) + records.dtype[name].shape, records.dtype[name].base)
        out[name][:count] = records[name][:count]
    return out


def _engine_frame(s):
    ctx, h = s["ctx"], DT / s["substeps"]
    bodies = s["bodies"].copy()
    ctx.backend_integrate(bodies, GRAVITY, h)
    integrated = bodies["velocity"].copy()
    contacts = ctx.backend_find_contacts(bodies, s["soup"], DT)
    ctx.backend_advance_substeps(bodies, contacts, GRAVITY, h, s["substeps"], SolverOptions.default())
    ctx.backend_fetch_impulses(contacts)
    out = {"integrated": integrated, "position": bodies["position"], "orientation": bodies["orientation"],
           "velocity": bodies["velocity"], "angular": bodies["angularVelocity"]}
    out.update(_padded(contacts, ("a", "b", "point", "normal", "normalImpulse"), CONTACT_SLOTS * len(bodies)))
    return out


def run(state):
    if "rollout" in state:
        return _train(state)
    if "bodies" in state:
        return _engine_frame(state)
    ctx = state["ctx"]
    ctx.snapshot_restore(0)
    if state["forces"] is not None:
        ctx.write_forces(state["forces"])
    ctx.step(state["steps"])
    out = {"poses": ctx.read_poses(state["poses"])}
    if state["events"]:
        events = _padded(ctx.read_events(), ("a", "b", "type", "impulse"), CONTACT_SLOTS * len(state["poses"]))
        out.update({"event_" + k: v for k, v in events.items()})
    stats = ctx.stats()
    out.update({k: stats[k] for k in ("candidatePairs", "contacts", "colors", "islands", "rewinds")})
    return out


def _bodies(case):
    kind, size = case["kind"], case["size"]
    return {"lattice": size ** 3, "sleep": size ** 3, "pyramids": 210 * size, "batch": 122 * size,
            "rollout": 7 * size}.get(kind, size) + 1


def work(case):
    """Bytes: a body's 256-byte record read and its 64 bytes of state written once a step, a 128-byte record per
    contact written once, the poses (or the engine's 320-byte records, both ways) over the host boundary.
    Operations: 250 per contact row and sweep (relative velocity, three impulses, two bodies' updates), 16 sweeps a
    substep, 400 per body and substep for its integration; a gradient costs a second run and twice its operations
    backward."""
    n = _bodies(case)
    rows = n * CONTACTS[case["kind"]]
    passes = 4 if case["kind"] == "rollout" else 1
    step_bytes = n * (256 + 64) + rows * 128
    step_flops = case["substeps"] * (16 * 250 * rows + 400 * n)
    host = n * 640 if case["kind"] == "backend" else n * 28
    return {"bytes": passes * case["steps"] * step_bytes + host, "flops": passes * case["steps"] * step_flops}


def exact(case, seed):
    """A contact step has no value in 64 bits: which contacts exist, their order and the clamps of every sweep are
    decisions on single-precision state, and the sweeps are not run to convergence. The Backend frame's first part,
    the velocity integration, has one."""
    if case["kind"] != "backend":
        return None
    s = prepare(case, seed)
    b = s["bodies"]
    h = float(np.float32(DT / case["substeps"]))
    move = (b["motionType"] == 2) & (b["asleep"] == 0)
    v = b["velocity"].astype(np.float64)
    v[move] += h * b["gravityScale"][move, None].astype(np.float64) * np.array(np.float32(GRAVITY), np.float64)
    v[move] /= 1.0 + h * b["linearDamping"][move, None].astype(np.float64)
    s["ctx"].close()
    return {"integrated": v}
