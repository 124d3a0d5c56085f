"""Pairs at the edge of the search range, across the boundary of boxes of
hundreds of thousands of grain sizes: the pair list is the oracle's, whose
every separation is FP64."""

import numpy as np
import pytest

from oracle.engine import OracleEngine
from sand_atlas_dem_gb300.engine import Engine
from sand_atlas_dem_gb300.model import HostLayout
from sand_atlas_dem_gb300.shapes import ShapeLibrary, exact_cube
from sand_atlas_dem_gb300.spec import Experiment
from tests.specimens import build, read

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [8, 14, 18, 20])
def test_pairs_across_the_boundary(gpu_library, power):
    library = ShapeLibrary([exact_cube(1e-3)])
    n, box = 256, 1e-3 * 2.0**power
    spec = Experiment(particles=n, contact_geometry="mesh", timestep=1e-9)
    rng = np.random.default_rng(power)
    at = rng.uniform(0.1, 0.9, (n, 3)) * box
    h = HostLayout(library, spec, at, [box] * 3, [0] * n, [1.0] * n)
    reach = (2 * h.body[0, 2] + h.skin) * h.length_unit
    # Pairs of grains k, k + n/2 either side of the x = 0 face, near the range.
    half = n // 2
    k = np.arange(half)
    at[:half, 1:] = (np.c_[k % 16, k // 16] + 2 + rng.uniform(-0.2, 0.2, (half, 2))) / 20 * box
    direction = rng.normal(size=(half, 3)) * [1.0, 0.3, 0.3]
    direction *= (np.sign(direction[:, :1]) + (direction[:, :1] == 0)) / np.linalg.norm(direction, axis=1)[:, None]
    at[:half, 0] = box - rng.uniform(0.01, 0.3, half) * reach
    at[half:] = at[:half] + direction * reach * rng.uniform(0.985, 1.015, half)[:, None]
    at = np.mod(at, box)
    case = dict(positions=at, cell=[box] * 3, ids=[0] * n, scales=[1.0] * n,
                rotations=np.tile([0, 0, 0, 1], (n, 1)).astype(np.float32), velocities=np.zeros((n, 3)))
    engines = [build(cls, library, spec, case) for cls in (Engine, OracleEngine)]
    for e in engines:
        e.initialize()
    count = int(engines[0].read("control", np.uint32, (16,))[1])
    assert count == int(engines[1].buffers["control"][1]) and 0 < count < half
    got, want = (read(e, "pairs", e.pair_capacity, np.uint32, 2)[:count] for e in engines)
    np.testing.assert_array_equal(got, want)
