"""The resident solver (small grids, a block cluster per field) against the tiled engine: the same bits,
node evaluations and rounds at the edges of its range (one block, several, the largest boxes, rows and
levels that leave a short last box), in both precisions and both modes."""

import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair():
    auto, engine = EikonalCuda.create(0, 64), EikonalCuda.create(0, 64)
    for prec in (64, 32):
        L.check(L.load().ts_engine_set_tile(engine.handle, prec, 0), engine)  # a chosen shape is the engine's
    yield auto, engine
    auto.close()
    engine.close()


def problem(dims, n_fields, variable, seed):
    depth = None
    if variable:
        depth = np.concatenate([[0.0], np.cumsum(1.03 ** np.arange(dims[2] - 1))])
    g = regular_grid(*dims, 1.0, depth)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 7, 9, 5)))
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(0, dims[0] - 1, n_fields), rng.uniform(0, dims[1] - 1, n_fields)
    lon, lat = km_to_geo(g, x, y, 1.0)
    z = rng.uniform(0, 0.6, n_fields) * g.max_depth_km
    return g, s, [point_source(g, s, *p) for p in zip(lon, lat, z)]


# 2x2x2 and thin grids; 416 rows in one block; 417 (two blocks); short last boxes; 16 blocks; many fields.
DIMS = [((2, 2, 2), 1), ((3, 3, 50), 2), ((22, 20, 16), 3), ((20, 26, 16), 1), ((20, 139, 3), 1), ((33, 47, 25), 2),
        ((61, 61, 31), 1), ((63, 59, 37), 2), ((12, 80, 60), 1), ((24, 24, 24), 40)]


@pytest.mark.parametrize("dims,n_fields", DIMS)
@pytest.mark.parametrize("variable", [False, True])
def test_equals_the_engine(pair, dims, n_fields, variable):
    auto, engine = pair
    g, s, seeds = problem(dims, n_fields, variable, sum(dims))
    for prec in (64, 32):
        for mode in (L.MODE_ENGINE, L.MODE_FAST):
            a = auto.solve(g, s, seeds, mode=mode, precision=prec)
            sa = (auto.last_stats_struct.node_updates, list(auto.last_stats_struct.rounds))
            b = engine.solve(g, s, seeds, mode=mode, precision=prec)
            sb = (engine.last_stats_struct.node_updates, list(engine.last_stats_struct.rounds))
            assert np.array_equal(a, b), (prec, mode)
            assert sa == sb


def test_uneven_grids_in_one_launch(pair):
    auto, engine = pair
    probs = [problem(d, 1, v, q) for q, (d, v) in
             enumerate([((40, 31, 18), False), ((9, 64, 20), True), ((25, 12, 40), False)])]
    args = ([p[0] for p in probs], [p[1] for p in probs], [0, 1, 2, 1], [p[2][0] for p in probs] + [probs[1][2][0]])
    for prec in (64, 32):
        got = auto.solve_multi(*args, mode=L.MODE_FAST, precision=prec)
        want = engine.solve_multi(*args, mode=L.MODE_FAST, precision=prec)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_refusal_and_cancel(pair):
    auto, _ = pair
    g, s, seeds = problem((30, 30, 20), 2, False, 1)
    ok, why = auto.try_solve(g, s, seeds, np.empty((2, g.count)), max_rounds=1)
    assert not ok and "not settled after 1 rounds" in why
    auto.cancel()
    try:
        with pytest.raises(L.TsError) as e:
            auto.solve(g, s, seeds)
        assert e.value.code == L.TS_E_CANCELLED
    finally:
        auto.cancel(False)
    assert np.isfinite(auto.solve(g, s, seeds)).all()
