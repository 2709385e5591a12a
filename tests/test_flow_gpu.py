"""Tiles started by their neighbours: chains of tiles along one axis, plates, blocks of tiles with a partial
last one, several fields of different lengths of solve in one launch, and a settle tolerance that ends rounds
early. The engine's rule equals the plain per-plane path to the bit, with the same evaluations whatever
fields share the launch."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu

DIMS = [(20, 10, 6), (225, 5, 4), (4, 130, 6), (6, 10, 75), (97, 49, 5), (34, 6, 41), (67, 50, 26)]


@pytest.mark.parametrize("dims", DIMS)
def test_tile_order_equals_plain(dims):
    g = regular_grid(*dims, 1.0)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 7, 5, 4)))
    seeds = []
    for fx, fy, fz in ((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), (0.4, 0.7, 0.3)):
        lon, lat = km_to_geo(g, fx * (dims[0] - 1), fy * (dims[1] - 1), 1.0)
        seeds.append(point_source(g, s, float(lon), float(lat), fz * g.max_depth_km))
    with EikonalCuda.create(0, 64) as e:
        for prec in (64, 32):
            L.check(L.load().ts_engine_set_tile(e.handle, prec, 0), e)  # the tiled engine whatever the size
            for tol in (1e-7, 1e-3):
                want = e.solve(g, s, seeds, mode=L.MODE_PLAIN, precision=prec, tol=tol)
                got = e.solve(g, s, seeds, mode=L.MODE_ENGINE, precision=prec, tol=tol)
                together = e.last_stats_struct.node_updates
                assert np.array_equal(got, want), (prec, tol)
                alone = 0
                for q in range(len(seeds)):
                    assert np.array_equal(e.solve(g, s, seeds[q:q + 1], precision=prec, tol=tol)[0], want[q])
                    alone += e.last_stats_struct.node_updates
                assert alone == together
