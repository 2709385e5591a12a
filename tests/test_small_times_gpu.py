"""FP64 fields whose times' squares underflow (slowness of about 1e-156 to 1e-162 s/km; the
others are on either side of the line below which a node forms its roots): the choice of a node's terms
is the reference's to the bit there too, in the resident solver, the tiled engine and the plain path."""
import numpy as np
import pytest

from oracle import oracle as O
from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-119, 1e-122, 1e-155, 1e-160, 1e-161])
@pytest.mark.parametrize("dims", [(20, 18, 14), (34, 34, 18)])
def test_terms_are_the_references(dims, scale):
    g = regular_grid(*dims, 1.0)
    s = scale / (vp_linear(g) * (1 + checkerboard(g, 7, 9, 5)))
    lon, lat = km_to_geo(g, 8.3, 7.7, 1.0)
    seeds = [point_source(g, s, float(lon), float(lat), 3.1)]
    want = O.relax(O.Grid.of(g), s, *seeds[0])[0]
    with EikonalCuda.create(0, 64) as e:
        assert np.array_equal(e.solve(g, s, seeds)[0], want)
        assert np.array_equal(e.solve(g, s, seeds, mode=L.MODE_PLAIN)[0], want)
        L.check(L.load().ts_engine_set_tile(e.handle, 64, 1), e)
        assert np.array_equal(e.solve(g, s, seeds)[0], want)
