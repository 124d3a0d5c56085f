"""Exact queries from certificates and per-cell triangle lists against walks.

A stored exact-query slot is answered from its certificate's triangles, from
its grid cell's triangle list, by a scan of the shape's leaves or by a walk of
the BVH; without the lists every lapsed slot is scanned or walked, and with no
filter margin every node is walked every step.  The three engines must hold
bit-identical states through list builds, lapsing certificates and reuse: on
rough grains of one, few and many triangles per cell, and on boxes, whose
edges and corners tie several triangles exactly.
"""

import numpy as np
import pytest

from sand_atlas_dem_gb300 import engine as engine_module
from sand_atlas_dem_gb300.engine import Engine
from sand_atlas_dem_gb300.shapes import ShapeLibrary, box_shape, exact_cube, perturbed_grain
from sand_atlas_dem_gb300.spec import Experiment
from sand_atlas_dem_gb300.workloads import contact_lattice
from tests.specimens import build

pytestmark = pytest.mark.gpu
RATE = (-0.5, -0.3, 0.2)


def grains(kind):
    if kind == "boxes":
        return ShapeLibrary([exact_cube(1e-3), box_shape([1e-3, 9e-4, 8e-4], shape_id="brick")])
    if kind == "fine":  # 5,120 triangles: cells with more triangles than a list holds
        return ShapeLibrary([perturbed_grain(16, seed=77, nodes=300), perturbed_grain(3, seed=78)])
    return ShapeLibrary([perturbed_grain(4, seed=1000 + k) for k in range(3)])


@pytest.mark.parametrize("kind,spacing", [("rough", 0.985), ("rough", 0.8), ("boxes", 0.9), ("fine", 0.9)])
@pytest.mark.parametrize("speed", [0.05, 5.0])
def test_lists_walks_and_plain_filters_agree(gpu_library, monkeypatch, kind, spacing, speed):
    library = grains(kind)
    case = contact_lattice(library, 4, spacing=spacing, seed=3, speed=speed)
    spec = Experiment(particles=64, contact_geometry="mesh", timestep=2e-9, normal_viscosity=4e5,
                      max_overlap_fraction=0.9, contacts_per_particle=2048, pairs_per_particle=32)
    engines = [build(Engine, library, spec, case), build(Engine, library, spec, case, filter_margin=0.0)]
    monkeypatch.setattr(engine_module, "CELL_LIST_LIMIT", 0)
    engines.append(build(Engine, library, spec, case))
    lists = [e.buffers["cellLists"].size for e in engines]
    assert lists[0] > 16 and lists[1] == lists[2] == 16
    for e in engines:
        e.initialize()
    for chunk in (1, 7, 40):
        for e in engines:
            e.advance(chunk, rate=RATE)
        first = engines[0].state()
        assert first["contacts"] > 0
        for e in engines[1:]:
            other = e.state()
            assert other["contacts"] == first["contacts"]
            for key, value in first.items():
                if isinstance(value, np.ndarray):
                    assert value.tobytes() == other[key].tobytes(), (kind, speed, key)
        for name in ("particleStress", "contactForce"):
            rows = 3 * spec.particles if name == "particleStress" else first["contacts"]
            got = [e.read(name, np.float32)[:4 * rows].tobytes() for e in engines]
            assert got[0] == got[1] == got[2], name


def test_contact_counts_and_starts_follow_the_contacts(gpu_library):
    """The per-pair first contacts and counts of the compaction, also for
    pairs without a stored slot, against the committed contact keys."""
    library = grains("rough")
    case = contact_lattice(library, 5, spacing=1.12, seed=5, scale_sigma=0.2)  # many pairs, few contacts
    spec = Experiment(particles=125, contact_geometry="mesh", timestep=2e-9, max_overlap_fraction=0.9,
                      contacts_per_particle=512, pairs_per_particle=32, skin=0.3)
    e = build(Engine, library, spec, case)
    e.initialize()
    e.advance(3, rate=RATE)
    state = e.state()
    pairs = int(e.check_errors()[1])
    ij = e.read("pairs", np.uint32, (e.pair_capacity, 2))[:pairs].astype(np.int64)
    side = e.sides[1 - e.active]
    starts = e.m.read_prefix(side["sideContactStart"], pairs + 1, np.uint32).astype(np.int64)
    counts = e.read("contactCounts", np.uint32)[:pairs]
    meta = state["meta"].astype(np.int64)
    assert 0 < state["contacts"] == starts[-1]
    np.testing.assert_array_equal(np.diff(starts), counts)
    owner = np.repeat(np.arange(pairs), np.diff(starts))
    np.testing.assert_array_equal(np.sort(meta[:, :2], axis=1), ij[owner])
    assert (counts == 0).sum() > pairs // 4


def test_lists_without_the_distance_grid(gpu_library):
    """Without the grid's bound a stored node may lie in any cell: every cell
    has its list, and a new slot is certified from it instead of by a scan."""
    library = grains("rough")
    case = contact_lattice(library, 4, spacing=0.985, seed=3, speed=0.05)
    spec = Experiment(particles=64, contact_geometry="mesh", timestep=2e-9, max_overlap_fraction=0.9,
                      contacts_per_particle=256, pairs_per_particle=32)
    engines = [build(Engine, library, spec, case, distance_grid=flag) for flag in (True, False)]
    first = [e.read("cellLists", np.uint32).reshape(-1, 64)[:, 2] for e in engines]
    assert (first[0] == 0xFFFFFFFF).any() and not (first[1] == 0xFFFFFFFF).any()
    for e in engines:
        e.initialize()
        kept, slow, lapsed = (int(e.read("work", np.uint32, (64,))[k]) for k in (3, 14, 20))
        assert kept > 0 and lapsed == slow == 0
        e.advance(5)
    a, b = (e.state() for e in engines)
    assert a["contacts"] == b["contacts"] > 0
    for key, value in a.items():
        if isinstance(value, np.ndarray):
            assert value.tobytes() == b[key].tobytes(), key
