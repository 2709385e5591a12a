"""Grids whose boxes do not fill the cluster of the resident solver (7, 6 and 4 boxes in 8 blocks, 15 in 16): the blocks
without a box take part in every round's end. Against the CPU oracle (FP64: the reference's rule and the fast
mode's) and the plain per-plane path (FP32)."""
import numpy as np
import pytest

from oracle import oracle as O
from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(12, 42, 11), (64, 13, 21), (90, 13, 13), (110, 21, 74), (64, 60, 37)])
def test_spare_blocks(dims):
    g = regular_grid(*dims, 1.0)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 7, 9, 5)))
    lon, lat = km_to_geo(g, 0.3 * dims[0], 0.7 * dims[1], 1.0)
    seeds = [point_source(g, s, float(lon), float(lat), 0.4 * g.max_depth_km), point_source(g, s, g.min_lon, g.min_lat, 0.0)]
    og = O.Grid.of(g)
    with EikonalCuda.create(0, 64) as e:
        exact = e.solve(g, s, seeds)
        fast = e.solve(g, s, seeds, mode=L.MODE_FAST)
        paired = e.solve(g, s, seeds, precision=32)
        assert np.array_equal(paired, e.solve(g, s, seeds, precision=32, mode=L.MODE_PLAIN))
    for f, (idx, t) in enumerate(seeds):
        assert np.array_equal(exact[f], O.relax(og, s, idx, t)[0])
        assert np.array_equal(fast[f], O.relax_wake(og, s, idx, t, L.WAKE_REL, causal=True)[0])
