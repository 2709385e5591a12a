"""Results and inputs whose copies are split over host threads: sizes around the threshold and the slot
size, where a part can be empty or end inside a slot. Tables go up and come back whole."""
import numpy as np
import pytest

from tomostar_b200 import location as loc
from tomostar_b200.synthetic import regular_grid

pytestmark = pytest.mark.gpu

MB = 1 << 18  # floats


@pytest.mark.parametrize("floats", [3 * 3 * 2, MB * 2 - 18, MB * 2, MB * 2 + 18, MB * 9 + 36, MB * 33 - 54])
def test_tables_round_trip(solver, floats):
    n = 18  # nodes per table
    g = regular_grid(3, 3, 2, 1.0)
    count = max(1, floats // n)
    tabs = np.random.default_rng(floats).random((count, n), np.float32)
    with loc.Tables.upload(solver, g, tabs) as t:
        assert np.array_equal(t.copy(), tabs)
        assert np.array_equal(t.copy(count // 2, count - count // 2), tabs[count // 2:])
