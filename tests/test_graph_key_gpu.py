"""A captured solve is replayed for the same job only: another mode or settle tolerance on the same grid, seeds and
buffers is another job. Each solve under capture equals the one without (fields, evaluations, rounds)."""
import itertools

import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_mode_and_tolerance_are_part_of_the_job(precision):
    g = regular_grid(40, 33, 18, 1.0)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 7, 9, 5)))
    lon, lat = km_to_geo(g, np.array([3.0, 30.0]), np.array([20.0, 5.0]), 1.0)
    seeds = [point_source(g, s, float(a), float(b), 4.0) for a, b in zip(lon, lat)]

    def result(e, mode, tol):
        f = e.solve(g, s, seeds, mode=mode, tol=tol, precision=precision)
        return f, e.last_stats_struct.node_updates, list(e.last_stats_struct.rounds)

    jobs = list(itertools.product((L.MODE_FAST, L.MODE_ENGINE), (1e-3, 1e-7)))
    with EikonalCuda.create(0, 64) as e:
        want = {j: result(e, *j) for j in jobs}
        assert len({w[1] for w in want.values()}) == 4  # the four jobs differ
        e.set_graph(True)
        for j in jobs + jobs[::-1]:
            before = e.graph_replays
            for replays in (0, 1):  # captured, then replayed
                f, updates, rounds = result(e, *j)
                assert np.array_equal(f, want[j][0]) and (updates, rounds) == want[j][1:], j
                assert j == jobs[-1] or e.graph_replays == before + replays
