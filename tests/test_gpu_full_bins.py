"""Cell lists of few, full bins: one grain of many times the others' size sets
the bin width.  The persistent step orders such bins by itself; pairs equal the
oracle's and the launched step's, after builds in which the grains arrive at
their bins in any order.
"""

import numpy as np
import pytest

from oracle.engine import OracleEngine
from sand_atlas_dem_gb300.engine import Engine
from sand_atlas_dem_gb300.shapes import ShapeLibrary, exact_cube
from sand_atlas_dem_gb300.spec import Experiment
from tests.specimens import build, read, upload


def bitonic(v):
    """The warp's in-place sort (``sortWarp``), restated: compare places
    low < high, the mirrored ones first, leaving out those past the end."""
    v, n, size = list(v), len(v), 2
    while size < 2 * n:
        stride = size >> 1
        while stride:
            k = 0
            while (low := 2 * k - (k & (stride - 1))) < n:
                high = low ^ (size - 1) if stride == size >> 1 else low + stride
                if high < n and v[low] > v[high]:
                    v[low], v[high] = v[high], v[low]
                k += 1
            stride >>= 1
        size <<= 1
    return v


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 127, 129, 500, 512, 513])
def test_in_place_sort_of_any_length(n):
    rng = np.random.default_rng(n)
    for _ in range(5):
        v = rng.permutation(3 * n)[:n].tolist()
        assert bitonic(v) == sorted(v)


def specimen(side, spacing=7e-4):
    """Small cubes on a jittered lattice, too far apart to touch, around one of six times
    their size; ids in random order over the lattice."""
    rng = np.random.default_rng(side)
    box = side * spacing
    at = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * spacing + 0.5 * spacing
    at += rng.uniform(-0.02, 0.02, at.shape) * spacing
    at = at[np.linalg.norm(at - 0.5 * box, axis=1) > 3.2e-3]
    at = np.r_[[[0.5 * box] * 3], rng.permutation(at)]
    n = len(at)
    case = dict(positions=at, cell=[box] * 3, ids=[0] * n, scales=[3.0] + [0.5] * (n - 1),
                rotations=np.tile([0, 0, 0, 1], (n, 1)).astype(np.float32), velocities=np.zeros((n, 3)))
    spec = Experiment(particles=n, contact_geometry="mesh", timestep=1e-9, pairs_per_particle=64, bin_capacity=2048,
                      contacts_per_particle=16)
    return ShapeLibrary([exact_cube(1e-3)]), spec, case


@pytest.mark.gpu
@pytest.mark.parametrize("side", [16, 18])
def test_pairs_of_full_bins(gpu_library, side):
    library, spec, case = specimen(side)
    engines = [build(Engine, library, spec, case, use_graph=flag) for flag in (True, False)]
    engines.append(build(OracleEngine, library, spec, case))
    for e in engines:
        e.initialize()
        for _ in range(2):
            # Far from the reference positions: the next step builds.
            upload(e, "referencePosition", np.full((spec.particles, 4), 3.0, np.float32))
            e.advance(1)
    assert engines[0].lib.sdg_engine_persistent(engines[0]._native) == 1
    pairs = [read(e, "pairs", e.pair_capacity, np.uint32, 2) for e in engines]
    counts = [int(e.read("control", np.uint32, (16,))[1]) if isinstance(e, Engine) else int(e.buffers["control"][1])
              for e in engines]
    assert counts[0] == counts[1] == counts[2] > spec.particles
    occupancy = engines[0].read("binCounts", np.uint32)[:engines[0].bin_count]
    assert occupancy.max() > 256
    for other in pairs[1:]:
        np.testing.assert_array_equal(pairs[0][:counts[0]], other[:counts[0]])
    work = [e.read("work", np.uint32, (64,))[17] for e in engines[:2]]
    assert work[0] == work[1] == 3  # the initialization's build and both steps'
