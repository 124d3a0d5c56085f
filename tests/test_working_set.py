"""The device bytes a layout states against those an engine holds."""

import pytest

from sand_atlas_dem_gb300.engine import CELL_LIST_BYTES, DISTANCE_GRID
from sand_atlas_dem_gb300.model import HostLayout
from tests.specimens import build, lattice_case, walled_lattice


def layout(geometry=None):
    library, spec, case = lattice_case(side=3) if geometry is None else walled_lattice(geometry)[:3]
    return HostLayout(library, spec, case["positions"], case["cell"], case["ids"], case["scales"]), library, spec, case


def test_lists_and_certificates_are_counted():
    h = layout()[0]
    lists = len(h.library.shapes) * CELL_LIST_BYTES * DISTANCE_GRID**3
    survivors = 4 * h.contact_capacity
    total = h.estimated_bytes()
    assert total > lists + (48 + 32 + 16) * survivors  # certificates, hit records, slots
    assert total - h.estimated_bytes(filter_margin=0.0) == lists - 16


@pytest.mark.gpu
@pytest.mark.parametrize("geometry,settings", [(None, {}), (None, dict(filter_margin=0.0)), ("mesh", {}), ("sdf", {})])
def test_the_estimate_is_what_the_engine_holds(gpu_library, geometry, settings):
    from sand_atlas_dem_gb300.engine import Engine

    h, library, spec, case = layout(geometry)
    e = build(Engine, library, spec, case, **settings)
    groups = (e.buffers, *e.sides, e.backups, e.history_backup)
    held = sum(buffer.tensor.numel() for group in groups for buffer in group.values())
    assert h.estimated_bytes(**settings) == e.estimated_bytes == held
