"""The value block of a native call follows the engine's settings (no GPU)."""

import numpy as np
import pytest

from sand_atlas_dem_gb300.engine import Engine
from sand_atlas_dem_gb300.model import CONFIG_ORDER


class Layout:
    def config_values(self, config):
        return np.array([float(config[k]) for k in CONFIG_ORDER])


def engine():
    e = Engine.__new__(Engine)
    e.layout, e.culler, e.tuning, e._value_cache = Layout(), None, {}, {}
    e.leaf_words, e.candidate_capacity, e.specimens, e.survivor_capacity = 1, 100, 1, 400
    e.distance_grid, e.filter_margin = True, 1e-3
    return e


@pytest.mark.parametrize("name,value,place", [("distance_grid", False, -2), ("filter_margin", 2e-3, -1),
                                              ("survivor_capacity", 800, -3)])
def test_a_changed_setting_reaches_the_next_call(name, value, place):
    e, config = engine(), {k: float(i) for i, k in enumerate(CONFIG_ORDER)}
    block, n = e._values(config)
    assert n == len(block) and e._values(config)[0] is block
    before = list(block)
    setattr(e, name, value)
    after = list(e._values(config)[0])
    assert after[place] == float(value) != before[place]
    assert [i for i in range(n) if before[i] != after[i]] == [n + place]


def test_the_block_is_by_name():
    e = engine()
    a = {k: float(i) for i, k in enumerate(CONFIG_ORDER)}
    swapped = {CONFIG_ORDER[1]: a[CONFIG_ORDER[0]], CONFIG_ORDER[0]: a[CONFIG_ORDER[1]],
               **{k: a[k] for k in CONFIG_ORDER[2:]}}
    assert list(e._values(a)[0])[:2] == [0.0, 1.0] and list(e._values(swapped)[0])[:2] == [1.0, 0.0]
