"""Both solvers under both rules against the CPU oracle, each on a context of its own whatever other tests have
chosen: the tiled engine at the edges of its tile, the resident solver with one block and with clusters; and a
batch of the inversion step's fields against the fields alone."""
import numpy as np
import pytest

from oracle import oracle as O
from tomostar_b200 import _lib as L
from tomostar_b200 import synthetic as syn
from tomostar_b200.eikonal import EikonalCuda, point_source

pytestmark = pytest.mark.gpu


def check(e, dims, variable):
    depth = np.concatenate([[0.0], np.cumsum(1.04 ** np.arange(dims[2] - 1))]) if variable else None
    g = syn.regular_grid(*dims, 1.0, depth)
    s = 1 / (syn.vp_linear(g) * (1 + syn.checkerboard(g, 9, 6, 5)))
    seeds = []
    for x, y, z in ((0.0, 0.0, 0.0), (min(32.0, dims[0] - 1.0), min(15.5, dims[1] - 1.0), 0.5 * g.max_depth_km)):
        lon, lat = syn.km_to_geo(g, x, y, 1.0)
        seeds.append(point_source(g, s, float(lon), float(lat), z))
    og = O.Grid.of(g)
    exact = e.solve(g, s, seeds, mode=L.MODE_ENGINE, precision=64)
    fast = e.solve(g, s, seeds, mode=L.MODE_FAST, precision=64)
    evals = e.last_stats_struct.node_updates
    for f, (idx, t) in enumerate(seeds):
        assert np.array_equal(exact[f], O.relax(og, s, idx, t)[0])
        want, ok, _, n = O.relax_wake(og, s, idx, t, L.WAKE_REL, causal=True)
        assert ok and np.array_equal(fast[f], want)
        evals -= n
    assert evals == 0  # every evaluation that the rule asks for, and no other


@pytest.mark.parametrize("variable", [False, True])
@pytest.mark.parametrize("dims", [(2, 2, 2), (31, 15, 7), (32, 16, 8), (33, 17, 9), (64, 16, 17), (65, 33, 33), (3, 40, 20),
                                  (70, 2, 19), (97, 18, 2)])
def test_tile_edges(dims, variable):
    with EikonalCuda.create(0, 64) as e:
        L.check(L.load().ts_engine_set_scheduler(e.handle, 1), e)
        check(e, dims, variable)


@pytest.mark.parametrize("variable", [False, True])
@pytest.mark.parametrize("dims", [(2, 2, 2), (22, 20, 16), (20, 26, 16),  # one block
                                  (20, 139, 3), (33, 47, 25), (61, 61, 31), (12, 80, 60)])  # 8 and 16
def test_resident(dims, variable):
    with EikonalCuda.create(0, 64) as e:
        check(e, dims, variable)


@pytest.mark.parametrize("mode", [L.MODE_ENGINE, L.MODE_FAST])
def test_batch_equals_fields_alone(mode):
    p = syn.inversion_step_121()
    seeds = [point_source(p.grid, p.slowness[0], *p.stations[q]) for q in range(6)]
    with EikonalCuda.create(0, 64) as e:
        together = e.solve(p.grid, p.slowness[0], seeds, precision=64, mode=mode)
        for q in (0, 3, 5):
            assert np.array_equal(together[q], e.solve(p.grid, p.slowness[0], seeds[q:q + 1], precision=64, mode=mode)[0])
