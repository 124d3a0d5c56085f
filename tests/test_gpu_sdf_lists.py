"""The SDF node lists at their edges: node counts below and between whole
rounds of 32 and 128, pairs deep enough to fill the list many times over and
to give one virtual lane several contacts, and pairs without any; contact
keys, order and geometry, forces and slip equal the oracle's bit for bit, in
the persistent, the launched and the dispatched forms.
"""

import numpy as np
import pytest

from oracle.engine import OracleEngine
from sand_atlas_dem_gb300.engine import Engine
from sand_atlas_dem_gb300.model import RejectedStep
from sand_atlas_dem_gb300.shapes import ShapeLibrary, analytic_sphere
from sand_atlas_dem_gb300.spec import Experiment
from sand_atlas_dem_gb300.workloads import contact_lattice
from tests.specimens import build

pytestmark = pytest.mark.gpu


def rejected(call, *args):
    try:
        call(*args)
    except RejectedStep as exc:
        return exc.flags
    return 0


@pytest.mark.parametrize("nodes", [1, 31, 130, 700])
@pytest.mark.parametrize("spacing,friction", [(0.99, 0.5), (0.55, 0.2)])
def test_against_the_oracle(gpu_library, nodes, spacing, friction):
    library = ShapeLibrary([analytic_sphere(resolution=24, samples=nodes)])
    case = contact_lattice(library, 6, spacing=spacing, seed=5, speed=0.5, scale_sigma=0.02)
    spec = Experiment(particles=216, contact_geometry="sdf", timestep=1e-10, friction=friction, normal_viscosity=4e5,
                      max_overlap_fraction=2.0, contacts_per_particle=8192, pairs_per_particle=64)
    o = build(OracleEngine, library, spec, case)
    engines = [build(Engine, library, spec, case, use_graph=flag) for flag in (True, False)]
    # Spheres this deep can put a node at another's centre: a rejection is the
    # oracle's too, with the same flags.
    flags = [rejected(e.initialize) for e in (o, *engines)]
    assert flags[0] == flags[1] == flags[2], flags
    if flags[0]:
        return
    so = o.state()
    assert nodes == 1 or so["contacts"] > 0
    count = int(so["contacts"])
    for g in engines:
        sg = g.state()
        assert sg["contacts"] == count
        for key in ("meta", "slip", "normalArea", "force", "torque"):
            assert sg[key].tobytes() == so[key].tobytes(), key
        assert g.read("pointDepth", np.float32)[:4 * count].tobytes() == o.buffers["pointDepth"][:count].tobytes()
    flags = [rejected(e.advance, 5) for e in (o, *engines)]
    assert flags[0] == flags[1] == flags[2], flags
    if flags[0]:
        return
    first, second = (g.state() for g in engines)
    for key, value in first.items():
        if isinstance(value, np.ndarray):
            assert value.tobytes() == second[key].tobytes(), key
    assert engines[0].lib.sdg_engine_persistent(engines[0]._native) == 1
    # The phases by name, on the committed contacts.
    g = engines[1]
    for phase in ("collect", "resolveContacts"):
        g.dispatch(phase, g.n, g.config(dt=0))
    np.testing.assert_array_equal(first["meta"], o.state()["meta"])
