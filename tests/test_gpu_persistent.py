"""The persistent step against the launched one.

With graphs on, an engine runs its steps in one cooperative launch where its
stored exact-query list is small, and replays a captured graph above that;
without, it launches kernel by kernel.  All three hold the same state, bit for
bit, with neighbour rebuilds and filter builds on the way, over chunks shorter
and longer than a launch's steps, periodic and between planes.
"""

from dataclasses import replace

import numpy as np
import pytest

from sand_atlas_dem_gb300.engine import Engine
from sand_atlas_dem_gb300.model import RejectedStep
from tests.specimens import build, lattice_case, walled_lattice

pytestmark = pytest.mark.gpu


def assert_same(a, b):
    sa, sb = a.state(), b.state()
    assert sa["contacts"] == sb["contacts"] > 0
    for key, value in sa.items():
        if isinstance(value, np.ndarray):
            assert value.tobytes() == sb[key].tobytes(), key
    assert a.read("work", np.uint32, (64,)).tobytes() == b.read("work", np.uint32, (64,)).tobytes()
    for name in ("particleStress", "particleDiagnostic", "timestepRows", "normalDamping", "control"):
        assert a.read(name, np.uint8).tobytes() == b.read(name, np.uint8).tobytes(), name


@pytest.mark.parametrize("side,frequency,persistent,chunks", [
    (3, 4, 1, (1, 2, 130)), (5, 4, 1, (63, 64, 65)), (14, 8, 0, (1, 6, 7))])
@pytest.mark.parametrize("policy", ["conservative", "active-contact"])
def test_periodic(gpu_library, side, frequency, persistent, chunks, policy):
    # 14^3 grains of 642 nodes hold more live slots than the persistent step takes.
    library, spec, case = lattice_case(side=side, frequency=frequency, viscosity=4e5, policy=policy,
                                       speed=50.0 if side < 14 else 0.05, spacing=0.9 if side == 14 else 0.985)
    engines = [build(Engine, library, spec, case, use_graph=flag) for flag in (True, False)]
    for e in engines:
        e.initialize()
    for steps in chunks:
        for e in engines:
            e.advance(steps, rate=(-0.5, -0.4, 0.3), drag=1e3)
    assert engines[0].lib.sdg_engine_persistent(engines[0]._native) == persistent
    assert_same(*engines)
    if side == 5:
        assert int(engines[0].read("work", np.uint32, (64,))[17]) > 1  # neighbour rebuilds on the way


@pytest.mark.parametrize("policy", ["conservative", "active-contact"])
@pytest.mark.parametrize("viscosity", [0.0, 4e5])
def test_between_planes(gpu_library, policy, viscosity):
    library, spec, case, velocities = walled_lattice(viscosity=viscosity, policy=policy)
    engines = [build(Engine, library, spec, case, use_graph=flag) for flag in (True, False)]
    for e in engines:
        e.initialize()
        for steps in (1, 70, 5):
            e.advance(steps, wall_velocities=velocities)
    assert engines[0].lib.sdg_engine_persistent(engines[0]._native) == 1
    assert_same(*engines)


@pytest.mark.parametrize("side,persistent", [(19, 1), (26, 0)])  # 768-thread CTAs; the captured step
def test_many_grains_between_planes(gpu_library, side, persistent):
    library, spec, case, velocities = walled_lattice(side=side, viscosity=4e5)
    spec = replace(spec, contacts_per_particle=64)
    engines = [build(Engine, library, spec, case, use_graph=flag) for flag in (True, False)]
    for e in engines:
        e.initialize()
        e.advance(4, wall_velocities=velocities)
    assert engines[0].lib.sdg_engine_persistent(engines[0]._native) == persistent
    assert_same(*engines)


def rejected(e, **kwargs):
    with pytest.raises(RejectedStep) as info:
        e.advance(100, **kwargs)
    return info.value.flags


@pytest.mark.parametrize("kind", ["periodic", "planes", "guarded"])
def test_a_chunk_rejected_on_the_way(gpu_library, kind):
    """Steps of a launch that follow a rejected one change nothing: the flags, the
    restored state and the next chunk are the launched step's.  Fast grains run too
    deep into each other (the periodic case) or into fast planes, with and without the
    timestep guard, some steps after a list build."""
    if kind == "periodic":
        library, spec, case = lattice_case(side=4, speed=1000.0)
        spec = replace(spec, max_overlap_fraction=0.25)
        chunk, calm = dict(rate=(-0.5, -0.4, 0.3)), {}
    else:
        library, spec, case, velocities = walled_lattice(policy="active-contact" if kind == "guarded" else "conservative")
        calm = dict(wall_velocities=0.1 * velocities)
        chunk = dict(wall_velocities=velocities * (1.5e5 if kind == "guarded" else 1e5))
    engines = [build(Engine, library, spec, case, use_graph=flag) for flag in (True, False)]
    for e in engines:
        e.initialize()
        e.advance(2, **calm)
    before = engines[0].state()
    flags = [rejected(e, **chunk) for e in engines]
    assert flags[0] == flags[1] != 0
    for e in engines:
        after = e.state()
        assert e.step == 2 and after["contacts"] == before["contacts"]
        for key, value in before.items():
            if isinstance(value, np.ndarray):
                assert value.tobytes() == after[key].tobytes(), key
    for e in engines:
        e.advance(3, **calm)
    sa, sb = (e.state() for e in engines)
    for key, value in sa.items():
        if isinstance(value, np.ndarray):
            assert value.tobytes() == sb[key].tobytes(), key
    assert engines[0].lib.sdg_engine_persistent(engines[0]._native) == 1
