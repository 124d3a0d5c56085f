"""The work the engine is timed on: whole public calls over the range of sizes,
contact geometries and options that simulations use.

A simulation builds an :class:`Engine` once and then alternates
``Engine.advance`` chunks with ``Engine.diagnostics`` reads; a packing is
prepared by repeated force passes; a shape library is packed once per run.
Each case here is one of those calls, from a handful of grains (where launches
and latency are the cost) to 50,000, with periodic cells, walls, batches of
specimens, the mesh and the signed-distance geometry, with and without normal
viscosity and the active-contact guard.  ``exact`` restates the same step in
64 bits by brute force (no neighbour lists, every triangle of the target) for
the cases small enough.
"""

import functools
import math
from pathlib import Path

import numpy as np
import torch

DATA = Path(__file__).resolve().parent.parent / "sand_atlas_dem_gb300" / "data"
RECORDS = {"loose": "packing-f4-1000-phi035.npz", "dense": "packing-f8-10000.npz",
           "uneven": "packing-uneven-6250.npz"}
RECORD_LIBRARY = {"loose": "f4", "dense": "f8", "uneven": "uneven"}
RECORD_GRAINS = {"loose": 1000, "dense": 10_000, "uneven": 6250}
# Contacts per grain of each start, and nodes and triangles per grain of each
# library: what work() and exact() size themselves by.
CONTACTS = {"loose": 0.4, "dense": 16, "uneven": 19, "lattice": 90, "walled": 72, "spheres": 6, "rough": 40}
NODES = {"f4": 162, "f8": 642, "uneven": 900}
TRIANGLES = {"f4": 320, "f8": 1280, "uneven": 1800}
EXACT_RATE = 2.5e9  # node-triangle tests exact() makes in a second


def listed():
    return [
        # The smallest call a servo or a test makes: one step of a handful of
        # grains and the diagnostics after it.
        dict(name="call-125", kind="lattice", side=5, library="f4", shapes=8, steps=1, solid=0.56, rate=-0.5,
             damping=0.0, drag=0.0, speed=0.02, policy="conservative"),
        # A loose gas of grains: few contacts, moving fast, the validation
        # configuration of the method.
        dict(name="loose-1000", kind="packing", record="loose", reps_x=1, reps_y=1, reps_z=1, steps=10, rate=0.0,
             damping=0.3, drag=0.0, speed=0.05, policy="conservative"),
        # The headline: a dense packing under isotropic compression.
        dict(name="dense-10000", kind="packing", record="dense", reps_x=1, reps_y=1, reps_z=1, steps=10, rate=-0.5,
             damping=0.3, drag=0.0, speed=0.005, policy="conservative"),
        # The largest production size: 50,000 uneven grains.
        dict(name="uneven-50000", kind="packing", record="uneven", reps_x=2, reps_y=2, reps_z=2, steps=10, rate=-0.5,
             damping=0.3, drag=0.0, speed=0.005, policy="conservative"),
        # A wall stage: grains boxed by six moving planes.
        dict(name="walled-4913", kind="walled", side=17, library="f8", shapes=64, steps=10, solid=0.58, damping=0.3,
             drag=0.0, speed=0.0, policy="conservative"),
        # A small wall stage under the active-contact timestep guard, odd sizes.
        dict(name="walled-343-guarded", kind="walled", side=7, library="f4", shapes=5, steps=7, solid=0.57,
             damping=0.3, drag=0.0, speed=0.01, policy="active-contact"),
        # The signed-distance geometry on spheres in a simple cubic lattice.
        dict(name="spheres-1000", kind="sdf", side=10, shape="spheres", nodes=512, steps=10, drag=0.0, speed=0.01),
        # The same geometry on rough grains.
        dict(name="rough-sdf-2197", kind="sdf", side=13, shape="rough", nodes=162, steps=5, drag=0.0, speed=0.01),
        # A batch of independent specimens, each with its own rate.
        dict(name="batch-16", kind="batch", specimens=16, low=216, high=1000, library="uneven", shapes=64, steps=5,
             damping=0.3, drag=0.0, speed=0.0),
        # An overlapped lattice relaxing: many contacts, frequent list builds.
        dict(name="relaxing-15625", kind="lattice", side=25, library="uneven", shapes=64, steps=5, solid=0.58,
             rate=-0.5, damping=0.3, drag=0.0, speed=0.0, policy="conservative"),
        # Packing preparation: new centres, a zero-timestep force pass with
        # all lists built again, forces read back.
        dict(name="descent-4096", kind="descent", side=16, library="f8", shapes=64, solid=0.56),
        # Packing a shape library: the source-node trees of eight shapes.
        dict(name="trees-8x262144", kind="trees", shapes=8, items=262_144, leaf=64),
    ]


def log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["lattice", "packing", "packing", "walled", "sdf", "batch", "descent", "trees"])
    steps = log_uniform(rng, 1, 20)
    drag = rng.choice([0.0, 0.0, round(rng.uniform(1e3, 1e5), 1)])
    damping = rng.choice([0.0, round(rng.uniform(0.05, 0.4), 3)])
    policy = rng.choice(["conservative", "conservative", "active-contact"])
    speed = round(rng.uniform(0.001, 0.05), 4)
    solid = round(rng.uniform(0.54, 0.59), 3)
    library = rng.choice(["f4", "f8", "uneven"])
    shapes = log_uniform(rng, 3, 64)
    if kind == "lattice":
        side = log_uniform(rng, 5, 22)
        return dict(kind=kind, side=side, library=library, shapes=shapes, steps=min(steps, max(1, 60_000 // side**3)),
                    solid=solid, rate=round(rng.uniform(-0.8, 0.3), 3), damping=damping, drag=drag, speed=speed,
                    policy=policy)
    if kind == "packing":
        record = rng.choice(["loose", "loose", "dense", "uneven"])
        reps = [rng.choice([1, 2]) if record != "dense" else 1 for _ in range(3)]
        return dict(kind=kind, record=record, reps_x=reps[0], reps_y=reps[1], reps_z=reps[2], steps=min(steps, 10),
                    rate=round(rng.uniform(-0.8, 0.3), 3), damping=damping, drag=drag,
                    speed=speed if record == "loose" else round(0.2 * speed, 5), policy=policy)
    if kind == "walled":
        return dict(kind=kind, side=log_uniform(rng, 5, 18), library=rng.choice(["f4", "f8"]), shapes=shapes,
                    steps=min(steps, 10), solid=solid, damping=damping, drag=drag, speed=speed, policy=policy)
    if kind == "sdf":
        shape = rng.choice(["spheres", "rough"])
        return dict(kind=kind, side=log_uniform(rng, 5, 14), shape=shape,
                    nodes=rng.choice([128, 300, 512]) if shape == "spheres" else 162, steps=min(steps, 10), drag=drag,
                    speed=speed)
    if kind == "batch":
        count = log_uniform(rng, 2, 24)
        return dict(kind=kind, specimens=count, low=216, high=log_uniform(rng, 300, 1200), library=library,
                    shapes=shapes, steps=min(steps, 8), damping=damping, drag=drag, speed=speed)
    if kind == "descent":
        return dict(kind=kind, side=log_uniform(rng, 5, 18), library=library, shapes=shapes, solid=solid)
    leaf = rng.choice([64, 4])
    return dict(kind=kind, shapes=log_uniform(rng, 1, 16), items=log_uniform(rng, 300, 130_000), leaf=leaf)


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def library_of(kind, count):
    from sand_atlas_dem_gb300.shapes import synthetic_library

    return synthetic_library(kind, count)


@functools.lru_cache(maxsize=None)
def sdf_library(shape, nodes):
    from sand_atlas_dem_gb300.shapes import ShapeLibrary, analytic_sphere, perturbed_grain, with_sdf

    if shape == "spheres":
        return ShapeLibrary([analytic_sphere(resolution=32, samples=nodes)])
    return ShapeLibrary([with_sdf(perturbed_grain(4, seed=1000 + k), resolution=16) for k in range(3)])


@functools.lru_cache(maxsize=None)
def record_of(name):
    from sand_atlas_dem_gb300.workloads import load_packing

    return load_packing(DATA / RECORDS[name])


def experiment(library, ids, scales, case, **more):
    from dataclasses import replace

    from sand_atlas_dem_gb300.workloads import material_spec

    spec = material_spec(library, ids, scales, damping_ratio=case["damping"], policy=case["policy"], **more)
    # The guard bounds both grains' stiffness: half the conservative step.
    return replace(spec, timestep=0.5 * spec.timestep) if case["policy"] == "active-contact" else spec


def inputs(case, seed):
    """Everything a program has before it builds its engine: library, spec,
    specimens (centres, cell, shape ids, scales), rotations, velocities, rates."""
    from sand_atlas_dem_gb300 import workloads
    from sand_atlas_dem_gb300.spec import Experiment

    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("lattice", "descent"):
        library = library_of(case["library"], case["shapes"])
        start = workloads.lattice_at(library, case["side"], case["solid"], seed=seed % (1 << 31))
        if kind == "descent":
            case = dict(case, damping=0.0, policy="active-contact", speed=0.0, rate=0.0)
        more = dict(friction=0.0, contacts_per_particle=512) if kind == "descent" else {}
        spec = experiment(library, start["ids"], start["scales"], case, max_overlap_fraction=0.5,
                          pairs_per_particle=16, **more)
        rates = np.full(3, case["rate"])
    elif kind == "packing":
        library = library_of(RECORD_LIBRARY[case["record"]], 64)
        start = workloads.tile_packing(record_of(case["record"]), (case["reps_x"], case["reps_y"], case["reps_z"]))
        # Another origin of the periodic cell.
        start["positions"] = np.mod(start["positions"] + rng.uniform(0, 1, 3) * start["cell"], start["cell"])
        spec = experiment(library, start["ids"], start["scales"], case, max_overlap_fraction=0.1)
        rates = case["rate"] * (1 + 0.2 * rng.uniform(-1, 1, 3))
    elif kind == "walled":
        library = library_of(case["library"], case["shapes"])
        start = workloads.walled_lattice(library, case["side"], case["solid"], seed=seed % (1 << 31))
        spec = experiment(library, start["ids"], start["scales"], case, max_overlap_fraction=0.5, periodic=False,
                          planes=start["planes"], boundary_box=list(range(6)), pairs_per_particle=16)
        rates = np.zeros(3)
    elif kind == "sdf":
        library = sdf_library(case["shape"], case["nodes"])
        side, n = case["side"], case["side"] ** 3
        if case["shape"] == "spheres":
            spacing = 1.99 * library.shapes[0].radius
            index = np.stack(np.meshgrid(*([np.arange(side)] * 3), indexing="ij"), -1).reshape(-1, 3)
            jitter = 0.002 * spacing * rng.uniform(-1, 1, (n, 3))
            start = dict(positions=(index + 0.5) * spacing + jitter, cell=np.full(3, side * spacing),
                         ids=np.zeros(n, np.uint32), scales=np.ones(n),
                         rotations=workloads.random_rotations(n, seed))
        else:
            start = workloads.lattice_at(library, side, 0.55, seed=seed % (1 << 31))
        spec = Experiment(particles=n, contact_geometry="sdf", timestep=2e-9, pairs_per_particle=16,
                          contacts_per_particle=256, max_overlap_fraction=0.5)
        rates = np.zeros(3)
    else:
        library = library_of(case["library"], case["shapes"])
        # Grain counts spread over the range in a fixed order; packings,
        # orientations and rates are the seed's.
        sides = [round((case["low"] + (case["high"] - case["low"]) * ((7 * k) % case["specimens"])
                        / case["specimens"]) ** (1 / 3)) for k in range(case["specimens"])]
        starts = [workloads.lattice_at(library, side, rng.uniform(0.55, 0.6), seed=(seed + 1000 + k) % (1 << 31))
                  for k, side in enumerate(sides)]
        specimens = [(s["positions"], s["cell"], s["ids"], s["scales"]) for s in starts]
        rotations, rates = np.concatenate([s["rotations"] for s in starts]), rng.uniform(0.1, 1.0, len(starts))
        ids, scales = (np.concatenate([s[k] for s in specimens]) for k in (2, 3))
        spec = experiment(library, ids, scales, dict(case, policy="conservative"), max_overlap_fraction=0.5,
                          pairs_per_particle=16)
        velocities = rng.normal(0, 1, (len(ids), 3)) * case["speed"]
        return dict(library=library, spec=spec, specimens=specimens, rotations=rotations, velocities=velocities,
                    rates=-np.repeat(rates[:, None], 3, axis=1))
    velocities = rng.normal(0, 1, (len(start["ids"]), 3)) * case.get("speed", 0.0)
    return dict(library=library, spec=spec, rotations=np.asarray(start["rotations"], np.float32),
                specimens=[(start["positions"], start["cell"], start["ids"], start["scales"])], velocities=velocities,
                rates=rates)


def tree_items(case, seed):
    """Per shape (keys, low, high): points on a rough ellipsoid, or the
    centres and boxes of small triangles on it (leaf 4)."""
    rng = np.random.default_rng(seed)
    items = []
    for _ in range(case["shapes"]):
        x = rng.normal(size=(case["items"], 3)).astype(np.float32)
        x /= np.linalg.norm(x, axis=1, keepdims=True)
        x *= (0.5 * rng.uniform(0.6, 1.0, 3) * (1 + 0.05 * np.sin(7 * x[:, :1]))).astype(np.float32)
        if case["leaf"] == 64:
            items.append((x, None, None))
        else:
            reach = (1.5 / math.sqrt(case["items"]) * rng.uniform(0.2, 1, x.shape)).astype(np.float32)
            items.append((x, x - reach, x + reach))
    return items


def scaled(velocities, engine):
    out = np.zeros((engine.n, 4), np.float32)
    out[:, :3] = velocities * engine.time_unit / engine.length_unit
    return out


def descent_centres(start, seed):
    """Two sets of centres a descent visits, 0.02 mean spacings apart."""
    positions, cell = np.asarray(start["specimens"][0][0]), start["specimens"][0][1]
    rng = np.random.default_rng(seed + 1)
    step = 0.02 * (np.prod(cell) / len(positions)) ** (1 / 3)
    return [positions, np.mod(positions + step * rng.uniform(-1, 1, positions.shape), cell)]


def prepare(case, seed):
    if case["kind"] == "trees":
        return dict(case=case, items=tree_items(case, seed))
    from sand_atlas_dem_gb300.engine import Engine

    start = inputs(case, seed)
    library, spec, specimens = start["library"], start["spec"], start["specimens"]
    if len(specimens) == 1:
        engine = Engine(library, spec, *specimens[0])
    else:
        engine = Engine.batch(library, spec, specimens)
    engine.buffers["rotation"].copy_from_numpy(start["rotations"])
    state = dict(case=case, engine=engine)
    if case["kind"] == "descent":
        rows = []
        for x in descent_centres(start, seed):
            x = x / engine.length_unit
            high = x.astype(np.float32)
            rows.append([np.pad(a, ((0, 0), (0, 1))) for a in (high, (x - high).astype(np.float32))])
        return dict(state, rows=rows, turn=0, config=engine.config(dt=0, history=False))
    engine.buffers["velocity"].copy_from_numpy(scaled(start["velocities"], engine))
    engine.initialize()
    state["arguments"] = dict(rate=tuple(start["rates"]) if start["rates"].ndim == 1 else start["rates"],
                              drag=case["drag"])
    if case["kind"] == "walled":
        state["arguments"]["wall_velocities"] = np.array([p["velocity"] for p in spec.planes])
    return state


# -------------------------------------------------------------------- pass
def rows_of(buffer, rows, width=4, dtype=torch.float32):
    return buffer.tensor.view(dtype)[: 4 * rows].view(rows, 4)[:, :width]


def run(state):
    case = state["case"]
    if case["kind"] == "trees":
        from sand_atlas_dem_gb300.trees import device_median_trees

        order, records, low, high = device_median_trees(state["items"], case["leaf"])
        return dict(order=order.astype(np.int64), records=records.astype(np.int64), low=low[:, :3], high=high[:, :3])
    if case["kind"] == "descent":
        return descend(state)
    engine = state["engine"]
    engine.advance(case["steps"], **state["arguments"])
    d = engine.diagnostics()
    committed = engine.sides[1 - engine.active]
    # The committed contacts fill the first rows of these buffers; as many
    # rows come back whatever the number of contacts.
    count = min(engine.contact_capacity, contact_rows(case, engine.n))
    out = {k: rows_of(engine.buffers[k], engine.n, 3) for k in ("position", "velocity", "momentum", "force", "torque")}
    out["rotation"] = rows_of(engine.buffers["rotation"], engine.n)
    out["meta"] = rows_of(committed["meta"], count, dtype=torch.int32)
    out["slip"] = rows_of(committed["slip"], count)
    out["normalArea"] = rows_of(committed["normalArea"], count)
    for key in ("stress", "kinetic_energy", "elastic_energy_proxy", "max_overlap_fraction", "candidate_pairs",
                "active_surface_contacts", "active_grain_pairs"):
        out[key] = d[key]
    out["walls"] = [w["reaction"] + [w["work"]] for w in d["walls"]]
    return out


def descend(state):
    """One force evaluation at new centres, as a packing's descent makes it."""
    engine, n = state["engine"], state["engine"].n
    high, low = state["rows"][state["turn"]]
    state["turn"] ^= 1
    control = np.zeros(16, np.uint32)
    control[4] = 1
    engine.buffers["position"].copy_from_numpy(high)
    engine.buffers["positionRemainder"].copy_from_numpy(low)
    engine.buffers["control"].copy_from_numpy(control)
    engine.forces(state["config"], capture_kinematics=False)
    force = engine.read("force", np.float32, (n, 4))
    torque = engine.read("torque", np.float32, (n, 4))
    control = engine.read("control", np.uint32, (16,))
    side, count = engine.sides[engine.active], min(engine.contact_capacity, contact_rows(state["case"], n))
    return dict(force=force[:, :3], torque=torque[:, :3], flags=int(control[0]), pairs=int(control[1]),
                contacts=int(control[2]), meta=rows_of(side["meta"], count, dtype=torch.int32),
                normalArea=rows_of(side["normalArea"], count))


# -------------------------------------------------------------------- work
def start_of(case):
    return {"packing": case.get("record"), "sdf": case.get("shape"), "walled": "walled"}.get(case["kind"], "lattice")


def contact_rows(case, n):
    """Rows that hold every contact of the case."""
    return 64 + 2 * n * math.ceil(CONTACTS[start_of(case)])


def grains_of(case):
    kind = case["kind"]
    if kind == "packing":
        return RECORD_GRAINS[case["record"]] * case["reps_x"] * case["reps_y"] * case["reps_z"]
    if kind == "batch":
        return case["specimens"] * (case["low"] + case["high"]) / 2
    return case["side"] ** 3


def work(case):
    """Per step: a grain's eight state rows in and out, its constant rows and
    its force, torque and stress (416 B); a contact's committed history in
    and out (96 B).  A contact takes about 600 operations (placement, nearest
    triangle, law, gather), a grain 600; a signed-distance node 150.  Trees:
    12 B in per item, 4 B out, 48 B per node; a comparison per item and level."""
    kind = case["kind"]
    if kind == "trees":
        items = case["shapes"] * case["items"]
        nodes = 2 * items / case["leaf"] * 1.5
        return dict(bytes=16 * items + 48 * nodes + (24 * items if case["leaf"] == 4 else 0),
                    flops=items * max(1, math.log2(case["items"] / case["leaf"])))
    n = grains_of(case)
    contacts = CONTACTS[start_of(case)] * n
    steps = case.get("steps", 1)
    tests = 6 * n * case["nodes"] if kind == "sdf" else 0
    return dict(bytes=steps * (416 * n + 96 * contacts), flops=steps * (600 * n + 600 * contacts + 150 * tests))


# ------------------------------------------------------------------- exact
def cross(a, b):
    return torch.cross(a, b, dim=-1)


def dot(a, b):
    return (a * b).sum(-1)


def turn(q, v):
    u = q[..., :3].expand_as(v)
    return v + 2 * cross(u, cross(u, v) + q[..., 3:] * v)


def unturn(q, v):
    return turn(torch.cat([-q[..., :3], q[..., 3:]], -1), v)


def nearest(p, a, b, c):
    """Closest points of the triangles (a, b, c) to p (all (..., 3))."""
    ab, ac, bc = b - a, c - a, c - b

    def on_segment(o, d):
        return o + (dot(p - o, d) / dot(d, d)).clamp(0, 1)[..., None] * d

    n = cross(ab, ac)
    n = n / n.norm(dim=-1, keepdim=True)
    inside = ((dot(cross(ab, p - a), n) >= 0) & (dot(cross(bc, p - b), n) >= 0) & (dot(cross(-ac, p - c), n) >= 0))
    best = p - dot(p - a, n)[..., None] * n
    far = torch.where(inside, dot(p - best, p - best), torch.full_like(dot(p, p), math.inf))
    for q in (on_segment(a, ab), on_segment(b, bc), on_segment(a, ac)):
        d = dot(p - q, p - q)
        closer = d < far
        best, far = torch.where(closer[..., None], q, best), torch.minimum(d, far)
    return best, far


class Shape64:
    """A shape in normalized 64-bit units: depth and outward normal at points."""

    def __init__(self, shape, unit, sdf, device):
        def t(a):
            return torch.as_tensor(np.asarray(a, np.float64), device=device)

        self.samples, self.areas = t(shape.samples) / unit, t(shape.areas) / unit**2
        self.radius = shape.radius / unit
        if sdf:
            self.grid = t(np.asarray((shape.sdf / unit), np.float32))
            self.origin, self.spacing = t(shape.origin) / unit, shape.spacing / unit
        else:
            self.grid, self.tri = None, t(shape.vertices / unit)[torch.as_tensor(np.asarray(shape.faces), device=device)]

    def query(self, p):
        """(inside mask, signed distance, gradient) at the points p."""
        if self.grid is not None:
            g = (p - self.origin) / self.spacing
            size = torch.as_tensor(self.grid.shape, device=p.device)
            k = g.floor().long()
            valid = ((k >= 0) & (k < size - 1)).all(-1)
            k = torch.where(valid[:, None], k, torch.zeros_like(k))
            f, value, grad = g - k, 0.0, torch.zeros_like(p)
            for corner in range(8):
                bit = [(corner >> a) & 1 for a in range(3)]
                w = [f[:, a] if bit[a] else 1 - f[:, a] for a in range(3)]
                s = [2 * b - 1 for b in bit]
                v = self.grid[k[:, 0] + bit[0], k[:, 1] + bit[1], k[:, 2] + bit[2]]
                value = value + v * w[0] * w[1] * w[2]
                grad = grad + v[:, None] * torch.stack([s[0] * w[1] * w[2], s[1] * w[0] * w[2], s[2] * w[0] * w[1]], -1)
            return valid & (value < 0), value, grad / self.spacing
        inside = torch.zeros(len(p), dtype=torch.bool, device=p.device)
        phi, grad = torch.zeros_like(p[:, 0]), torch.zeros_like(p)
        rows = max(1, 4_000_000 // len(self.tri))
        for k in range(0, len(p), rows):
            a, b, c = (self.tri[None, :, j] - p[k:k + rows, None] for j in range(3))
            la, lb, lc = a.norm(dim=-1), b.norm(dim=-1), c.norm(dim=-1)
            angle = torch.atan2(dot(a, cross(b, c)), la * lb * lc + dot(a, b) * lc + dot(b, c) * la + dot(c, a) * lb)
            inside[k:k + rows] = angle.sum(1) > math.pi
        where = inside.nonzero()[:, 0]
        for k in range(0, len(where), rows):
            i = where[k:k + rows]
            q, far = nearest(p[i, None].expand(-1, len(self.tri), 3), *(self.tri[None, :, j].expand(len(i), -1, 3) for j in range(3)))
            d, best = far.min(1)
            q = q[torch.arange(len(i), device=p.device), best]
            phi[i] = -d.sqrt()
            grad[i] = (q - p[i]) / d.sqrt()[:, None]
        return inside, phi, grad


class World64:
    """The specimens of a case in 64 bits: forces by testing every node of
    every grain against every grain it can reach, and the same kick, drift and
    contact law the engine documents."""

    def __init__(self, start, device):
        library, spec = start["library"], start["spec"]
        self.spec, self.device = spec, device
        diameters = [(6 * s.volume / math.pi) ** (1 / 3) for s in library.shapes]
        self.unit = float(np.median(diameters))
        self.time = math.sqrt(spec.density * self.unit / spec.normal_stiffness)
        sdf = spec.contact_geometry == "sdf"
        ids = np.concatenate([s[2] for s in start["specimens"]]).astype(np.int64)
        scales = np.concatenate([s[3] for s in start["specimens"]]).astype(float)
        self.ids, self.n = ids, len(ids)
        self.shapes = {int(k): Shape64(library.shapes[int(k)], self.unit, sdf, device) for k in np.unique(ids)}
        shape = [library.shapes[int(i)] for i in ids]

        def t(a):
            return torch.as_tensor(np.asarray(a, np.float64), device=device)

        counts = np.array([len(s.samples) for s in library.shapes])
        self.counts = torch.as_tensor(counts, device=device)
        self.first = torch.as_tensor(np.cumsum(counts) - counts, device=device)
        self.samples = t(np.concatenate([s.samples for s in library.shapes])) / self.unit
        self.areas = t(np.concatenate([s.areas for s in library.shapes])) / self.unit**2
        self.scale = t(scales)
        self.mass = t([s.volume for s in shape]) * self.scale**3 / self.unit**3
        inverse = np.array([np.linalg.inv(s.inertia / self.unit**5) for s in library.shapes])
        self.inverse = t(inverse[ids]) / (self.scale**5)[:, None, None]
        self.reach = t([s.radius for s in shape]) * self.scale / self.unit
        self.specimen = torch.as_tensor(np.repeat(np.arange(len(start["specimens"])), [len(s[2]) for s in start["specimens"]]), device=device)
        self.x = t(np.concatenate([s[0] for s in start["specimens"]])) / self.unit
        self.box0 = t(np.array([s[1] for s in start["specimens"]])) / self.unit
        self.box, self.strain = self.box0.clone(), torch.zeros_like(self.box0)
        self.rate = t(start["rates"]).reshape(-1, 3).expand_as(self.box0) * self.time
        self.q = t(start["rotations"])
        self.v = t(np.asarray(start["velocities"] * self.time / self.unit, np.float32))
        self.l = torch.zeros_like(self.v)
        self.kt = spec.tangential_stiffness / spec.normal_stiffness
        self.eta = spec.normal_viscosity / (spec.normal_stiffness * self.time)
        planes = spec.planes
        self.planes = [dict(n=t(p["normal"]), d=p["offset"] / self.unit, v=t(p["velocity"]) * self.time / self.unit,
                            kn=p["normal_stiffness"] / spec.normal_stiffness, mu=p["friction"],
                            kt=p["tangential_stiffness"] / spec.normal_stiffness,
                            eta=p.get("normal_viscosity", 0) / (spec.normal_stiffness * self.time)) for p in planes]
        self.history = None

    def spin(self, q, l):
        return turn(q, (self.inverse @ unturn(q, l)[..., None])[..., 0])

    def pairs(self):
        """Directed pairs (i, j, branch j - i) whose bounding spheres meet."""
        found = []
        for s in range(len(self.box)):
            at = (self.specimen == s).nonzero()[:, 0]
            for k in range(0, len(at), 512):
                d = self.x[at][None] - self.x[at[k:k + 512]][:, None]
                if self.spec.periodic:
                    d = d - torch.floor(d / self.box[s] + 0.5) * self.box[s]
                near = d.norm(dim=-1) <= self.reach[at[k:k + 512]][:, None] + self.reach[at][None]
                i, j = near.nonzero().T
                i, j, d = at[k + i], at[j], d[i, j]
                found.append((i[i != j], j[i != j], d[i != j]))
        return [torch.cat(a) for a in zip(*found)]

    def contacts(self):
        """Grain contacts: source, target, node, arm, branch, depth, normal, area."""
        i, j, branch = self.pairs()
        ids = torch.as_tensor(self.ids, device=self.device)
        nodes = self.counts[ids[i]]
        out = []
        for part in torch.arange(len(i), device=self.device).split(8192):
            # Every node of each pair's source: pair row and node index.
            row = part.repeat_interleave(nodes[part])
            first = nodes[part].cumsum(0) - nodes[part]
            node = torch.arange(len(row), device=self.device) - first.repeat_interleave(nodes[part])
            src, dst, at = i[row], j[row], self.first[ids[i[row]]] + node
            arm = turn(self.q[src], self.samples[at] * self.scale[src, None])
            local = unturn(self.q[dst], arm - branch[row]) / self.scale[dst, None]
            near = (local.norm(dim=-1) * self.scale[dst] <= self.reach[dst] * 1.0001).nonzero()[:, 0]
            for s, shape in self.shapes.items():
                k = near[ids[dst[near]] == s]
                if not len(k):
                    continue
                inside, phi, grad = shape.query(local[k])
                k, phi, grad = k[inside], phi[inside], grad[inside]
                normal = turn(self.q[dst[k]], grad)
                out.append((src[k], dst[k], node[k], arm[k], branch[row[k]], -phi * self.scale[dst[k]],
                            normal / normal.norm(dim=-1, keepdim=True), self.areas[at[k]] * self.scale[src[k]] ** 2))
        if not out:
            z, e = torch.zeros(0, dtype=torch.long, device=self.device), torch.zeros(0, 3, dtype=torch.float64, device=self.device)
            return z, z, z, e, e, e[:, 0], e, e[:, 0]
        return [torch.cat(x) for x in zip(*out)]

    def carried(self, key, normal, spin, dt):
        """The committed slip of each contact, carried to its new normal."""
        slip = torch.zeros_like(normal)
        if self.history is None or not len(self.history[0]) or not len(key):
            return slip
        keys, slips, normals = self.history
        at = torch.searchsorted(keys, key).clamp(max=len(keys) - 1)
        hit = keys[at] == key
        x, a, b = slips[at], normals[at], normal
        c = dot(a, b).clamp(-1, 1)
        v = cross(a, b)
        x = x + cross(v, x) + cross(v, cross(v, x)) / (1 + c)[:, None]
        angle = 0.5 * spin * dt
        x = x * angle.cos()[:, None] + cross(b, x) * angle.sin()[:, None] + b * (dot(b, x) * (1 - angle.cos()))[:, None]
        x = x - b * dot(x, b)[:, None]
        return torch.where((hit & (c >= -0.999999))[:, None], x, slip)

    def law(self, slip, rv, normal, depth, area, dt, kn, kt, eta, mu, weight):
        slip = slip + (rv - normal * dot(rv, normal)[:, None]) * dt
        fn = weight * kn * area * depth
        if eta > 0:
            fn = (fn - weight * eta * area * dot(rv, normal)).clamp(min=0)
        ft = -(weight * kt * area)[:, None] * slip
        size = ft.norm(dim=-1)
        slide = (size > mu * fn) & (size > 0)
        ft = torch.where(slide[:, None], ft * (mu * fn / size.clamp(min=1e-300))[:, None], ft)
        slip = torch.where(slide[:, None], -ft / (weight * kt * area)[:, None], slip)
        return fn[:, None] * normal + ft, slip

    def forces(self, dt):
        w = self.spin(self.q, self.l)
        i, j, node, arm, branch, depth, normal, area = self.contacts()
        wi, wj = w[i], w[j]
        rate = self.rate[self.specimen[i]]
        rv = self.v[i] - self.v[j] - rate * branch + cross(wi, arm) - cross(wj, arm - branch)
        key = (i * (self.n + 64) + j) * (1 << 20) + node
        slip = self.carried(key, normal, dot(wi + wj, normal), dt)
        force, slip = self.law(slip, rv, normal, depth, area, dt, 1.0, self.kt, self.eta, self.spec.friction, 0.5)
        self.f, self.t = torch.zeros_like(self.v), torch.zeros_like(self.v)
        self.f.index_add_(0, i, force).index_add_(0, j, -force)
        self.t.index_add_(0, i, cross(arm, force)).index_add_(0, j, -cross(arm - branch, force))
        kept = [(key, slip, normal)]
        for number, p in enumerate(self.planes):
            for s, shape in self.shapes.items():
                g = torch.as_tensor((self.ids == s).nonzero()[0], device=self.device)
                arm = turn(self.q[g][:, None], shape.samples[None] * self.scale[g][:, None, None])
                phi = dot(self.x[g][:, None] + arm, p["n"]) - p["d"]
                row, node = (phi < 0).nonzero().T
                b, arm, depth = g[row], arm[row, node], -phi[row, node]
                normal = p["n"].expand_as(arm)
                rv = self.v[b] + cross(w[b], arm) - p["v"]
                key = (b * (self.n + 64) + self.n + number) * (1 << 20) + node
                slip = self.carried(key, normal, dot(w[b], normal), dt)
                force, slip = self.law(slip, rv, normal, depth, shape.areas[node] * self.scale[b] ** 2, dt, p["kn"],
                                       p["kt"], p["eta"], p["mu"], 1.0)
                self.f.index_add_(0, b, force)
                self.t.index_add_(0, b, cross(arm, force))
                kept.append((key, slip, normal))
        key, slip, normal = (torch.cat(x) for x in zip(*kept))
        order = key.argsort()
        self.history = key[order], slip[order], normal[order]

    def kick(self, dt, drag):
        self.v = self.v + 0.5 * dt * self.f / self.mass[:, None]
        self.l = self.l + 0.5 * dt * self.t
        self.v, self.l = self.v * math.exp(-0.5 * drag * dt), self.l * math.exp(-0.5 * drag * dt)

    def step(self, dt, drag):
        self.kick(dt, drag)

        def turned(w, h):
            size = w.norm(dim=-1, keepdim=True)
            part = torch.where(size > 0, torch.sin(0.5 * size * h) / size.clamp(min=1e-300), torch.full_like(size, 0.5 * h))
            a = torch.cat([part * w, torch.cos(0.5 * size * h)], -1)
            v = a[:, 3:] * self.q[:, :3] + self.q[:, 3:] * a[:, :3] + cross(a[:, :3], self.q[:, :3])
            return torch.cat([v, a[:, 3:] * self.q[:, 3:] - dot(a[:, :3], self.q[:, :3])[:, None]], -1)

        middle = turned(self.spin(self.q, self.l), 0.5 * dt)
        self.q = turned(self.spin(middle / middle.norm(dim=-1, keepdim=True), self.l), dt)
        self.strain = self.strain + self.rate * dt
        self.box = self.box0 * self.strain.exp()
        rate = self.rate[self.specimen]
        self.x = self.x * torch.exp(rate * dt) + dt * self.v
        if self.spec.periodic:
            box = self.box[self.specimen]
            self.x = self.x - torch.floor(self.x / box) * box
        self.v = self.v * torch.exp(-rate * dt)
        for p in self.planes:
            p["d"] = p["d"] + float(dot(p["n"], p["v"])) * dt
        self.forces(dt)
        self.kick(dt, drag)


def exact_trees(case, seed):
    """Bounds of every node of the median-split trees, preorder."""
    low, high = [], []
    for keys, lo, hi in tree_items(case, seed):
        lo, hi = (keys if lo is None else lo), (keys if hi is None else hi)
        stack = [np.arange(len(keys))]
        while stack:
            at = stack.pop()
            low.append(lo[at].min(0))
            high.append(hi[at].max(0))
            if len(at) > case["leaf"]:
                axis = int(np.ptp(keys[at], axis=0).argmax())
                at = at[np.argsort(keys[at, axis], kind="stable")]
                stack += [at[len(at) // 2:], at[:len(at) // 2]]
    return dict(order=None, records=None, low=np.array(low, np.float64), high=np.array(high, np.float64))


def exact(case, seed):
    kind = case["kind"]
    if kind == "trees":
        return exact_trees(case, seed) if case["shapes"] * case["items"] / case["leaf"] < 200_000 else None
    # Node-triangle tests of one force pass, and the shapes looped over.
    if kind == "sdf":
        tests, kinds = 40 * grains_of(case) * case["nodes"], 3
    else:
        library = RECORD_LIBRARY[case["record"]] if kind == "packing" else case["library"]
        tests = 1.5 * grains_of(case) * NODES[library] * TRIANGLES[library]
        kinds = 64 if kind == "packing" else case["shapes"]
    evaluations = 1 if kind == "descent" else case["steps"] + 1
    if evaluations * (tests / EXACT_RATE + kinds / 400) > 14 or grains_of(case) > 12_000:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    start = inputs(case, seed)
    world = World64(start, device)
    world.forces(0.0)
    if kind == "descent":
        return dict(force=world.f, torque=world.t, flags=None, pairs=None, contacts=None, meta=None, normalArea=None)
    # A zero-timestep pass commits no slip beyond zero; then the steps.
    for _ in range(case["steps"]):
        world.step(start["spec"].timestep / world.time, case["drag"] * world.time)
    # The nodal torques of a sphere cancel: what is left of them is rounding.
    spheres = case.get("shape") == "spheres"
    return dict(position=world.x, velocity=world.v, momentum=None if spheres else world.l, force=world.f,
                torque=None if spheres else world.t, rotation=world.q)
