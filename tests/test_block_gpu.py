"""The engine's block tiles (32 x 16 x 8 and 32 x 16 x 16 nodes) at their edges: one node more or less
than a tile on each axis, thin grids, variable depth spacing, seeds on a tile face. The engine's rule
equals the plain per-plane path to the bit in both precisions; the two shapes give the same fields,
evaluations and rounds in the fast mode."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2), (31, 15, 7), (32, 16, 8), (33, 17, 9), (64, 16, 17), (65, 33, 33), (3, 40, 20), (70, 2, 19),
        (97, 18, 2)]


@pytest.fixture(scope="module")
def engine():
    s = EikonalCuda.create(0, 64)
    yield s
    s.close()


def shape(s, sid):
    for prec in (64, 32):
        L.check(L.load().ts_engine_set_tile(s.handle, prec, sid), s)


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("variable", [False, True])
def test_tile_edges(engine, dims, variable):
    depth = np.concatenate([[0.0], np.cumsum(1.04 ** np.arange(dims[2] - 1))]) if variable else None
    g = regular_grid(*dims, 1.0, depth)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 9, 6, 5)))
    seeds = []
    for x, y, z in ((0.0, 0.0, 0.0), (min(32.0, dims[0] - 1.0), min(15.5, dims[1] - 1.0), 0.5 * g.max_depth_km)):
        lon, lat = km_to_geo(g, x, y, 1.0)
        seeds.append(point_source(g, s, float(lon), float(lat), z))
    for prec in (64, 32):
        plain = engine.solve(g, s, seeds, mode=L.MODE_PLAIN, precision=prec)
        fast = []
        for sid, *_ in L.engine_shapes():
            shape(engine, sid)
            assert np.array_equal(engine.solve(g, s, seeds, mode=L.MODE_ENGINE, precision=prec), plain), (prec, sid)
            f = engine.solve(g, s, seeds, mode=L.MODE_FAST, precision=prec)
            st = engine.last_stats_struct
            fast.append((f, st.node_updates, list(st.rounds)))
        for f, updates, rounds in fast[1:]:
            assert np.array_equal(f, fast[0][0]) and updates == fast[0][1] and rounds == fast[0][2]


def test_earlier_shape_ids_are_accepted(engine):
    g = regular_grid(20, 20, 12, 1.0)
    s = 1 / vp_linear(g)
    seeds = [point_source(g, s, g.min_lon, g.min_lat, 3.0)]
    want = engine.solve(g, s, seeds)
    for sid in range(11):
        shape(engine, sid)
        assert np.array_equal(engine.solve(g, s, seeds), want)
    assert L.load().ts_engine_set_tile(engine.handle, 64, 11) == L.TS_E_ARG
    assert L.load().ts_engine_set_tile(engine.handle, 64, -1) == L.TS_E_ARG


@pytest.mark.parametrize("layered", [False, True])
def test_ties_equal_the_oracle(engine, layered):
    """Constant and layered media on a square grid: candidates whose roots equal a neighbour's time to
    the last bits, where the choice of the terms is decided by the formed roots."""
    from oracle import oracle as O

    g = regular_grid(34, 34, 18, 1.0)
    s = np.full(g.count, 0.2)
    if layered:
        s.reshape(g.shape)[9:] = 0.125
    seeds = [point_source(g, s, *map(float, km_to_geo(g, 16.0, 16.0, 1.0)), 8.0),
             point_source(g, s, g.min_lon, g.min_lat, 0.0)]
    for sid, *_ in L.engine_shapes():
        shape(engine, sid)
        got = engine.solve(g, s, seeds, mode=L.MODE_ENGINE, precision=64)
        for f, (idx, t) in enumerate(seeds):
            want = O.relax(O.Grid.of(g), s, idx, t)
            assert np.array_equal(got[f], (want[0] if isinstance(want, tuple) else want).reshape(-1))
