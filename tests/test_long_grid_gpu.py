"""A grid of more than 1,024 tiles along x (32,800 nodes; earlier libraries took up to 65,536 with a 64-node tile),
and the first size beyond the queue's words."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


def problem(nx):
    g = regular_grid(nx, 2, 2, 0.01)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 0.07, 0.09, 0.05)))
    x = np.linspace(0.02, 0.98, 25) * (nx - 1) * 0.01
    lon, lat = km_to_geo(g, x, 0 * x, 0.01)
    idx, t = zip(*(point_source(g, s, float(a), float(b), 0.0) for a, b in zip(lon, lat)))
    return g, s, [(np.concatenate(idx), np.concatenate(t))]


def test_more_than_1024_tiles_equal_plain():
    g, s, seeds = problem(32800)
    with EikonalCuda.create(0, 64) as e:
        for prec in (64, 32):
            want = e.solve(g, s, seeds, mode=L.MODE_PLAIN, precision=prec)
            for tile in (0, 5):
                L.check(L.load().ts_engine_set_tile(e.handle, prec, tile), e)
                assert np.array_equal(e.solve(g, s, seeds, precision=prec), want)


def test_beyond_the_tile_table_is_refused():
    g, s, seeds = problem(65537)
    with EikonalCuda.create(0, 64) as e:
        ok, why = e.try_solve(g, s, seeds, np.empty((1, g.count)))
        assert not ok and "too large" in why
