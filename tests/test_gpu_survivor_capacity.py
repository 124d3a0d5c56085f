"""A filter build that finds more surviving nodes than the engine holds.

The build raises the contact-capacity flag and returns early, with the keep
flags of an earlier step left in place; the scans over them must write no place
at or past the capacity, and the engine's capacity retry must hold the state of an
engine that had room.  Slots had lapsed before the
build, and the grains move fast enough that each build doubles the margin.
"""

import numpy as np
import pytest

from sand_atlas_dem_gb300.engine import Engine
from tests.specimens import build, lattice_case

W_SURVIVORS, W_LAPSED = 2, 20


def places(values, room):
    """The places at which a compaction of the nonzero values is stored: the
    exclusive scan of the values (32-bit), where it lies below `room`."""
    offsets = np.cumsum(np.r_[np.uint32(0), values.astype(np.uint32)], dtype=np.uint32)[:-1]
    at = offsets[values != 0]
    return at[at < room]


@pytest.mark.parametrize("slots,lapsed", [(100_000, 40), (300_000, 1000), (2592, 89)])
def test_compaction_places_stay_below_the_capacity(slots, lapsed):
    rng = np.random.default_rng(slots)
    flags = (rng.random(slots) < 0.7).astype(np.uint32)
    np.testing.assert_array_equal(places(flags, slots), np.arange(flags.sum()))
    # Slot numbers where flags are expected: their sums pass the capacity.
    stale = flags.copy()
    stale[:lapsed] = rng.choice(slots, lapsed, replace=False)
    assert places(stale, 1 << 32).max() >= slots
    assert places(stale, slots).max(initial=0) < slots


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [True, False], ids=["persistent", "launched"])
@pytest.mark.parametrize("chunks", [(1,) * 9, (4, 20)], ids=["single", "long"])
def test_outgrown_survivors_go_through_the_retry(gpu_library, use_graph, chunks):
    from dataclasses import replace

    library, spec, case = lattice_case(side=3, viscosity=4e5, speed=1000.0)
    tight = replace(spec, contacts_per_particle=24)
    settings = dict(filter_margin=8e-3, use_graph=use_graph)
    ample, grown = (build(Engine, library, s, case, **settings) for s in (spec, tight))
    for e in (ample, grown):
        e.initialize()
    room, lapsed = grown.survivor_capacity, 0
    for steps in chunks:
        before, retried = ample.state(), bool(grown.capacity_retries)
        for e in (ample, grown):
            e.advance(steps)
        if grown.capacity_retries and not retried:
            assert lapsed > 0 and ample.capacity_retries == []
            assert int(ample.read("work", np.uint32, (64,))[W_SURVIVORS]) > room
            # The retry restores the state before the chunk: so does its peer.
            ample = build(Engine, library, spec, case, **settings)
            ample.restore(before, grown.step - steps)
            ample.advance(steps)
        lapsed = max(lapsed, int(ample.read("work", np.uint32, (64,))[W_LAPSED]))
    assert [r["flags"] for r in grown.capacity_retries] == [32]
    a, b = ample.state(), grown.state()
    assert a["contacts"] == b["contacts"] > 0
    for key, value in a.items():
        if isinstance(value, np.ndarray):
            assert value.tobytes() == b[key].tobytes(), key
