"""The nodes a grain may have with the SDF geometry (16-bit counts per virtual lane)."""

from types import SimpleNamespace

import pytest

from sand_atlas_dem_gb300.engine import check_lane_counts


def layout(nodes, contacts):
    return SimpleNamespace(library=SimpleNamespace(shapes=[SimpleNamespace(samples=range(n)) for n in nodes]),
                           contact_capacity=contacts)


@pytest.mark.parametrize("nodes,contacts", [([512], 1 << 24), ([3001, 2_097_120], 1 << 30), ([5_000_000], 65_535)])
def test_counts_that_fit(nodes, contacts):
    check_lane_counts(layout(nodes, contacts))


@pytest.mark.parametrize("nodes,contacts", [([100, 2_097_121], 1 << 20), ([5_000_000], 65_536)])
def test_counts_that_could_overflow_are_refused(nodes, contacts):
    with pytest.raises(ValueError, match="65,536"):
        check_lane_counts(layout(nodes, contacts))
