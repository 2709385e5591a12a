"""Which solver a context takes: its own choice, the tiled engine when that is chosen, its own choice again after
ts_engine_set_scheduler(0). (The two tell themselves apart by the tile visits they count: the resident solver's are
eight per round and box.) The autotuner keeps the faster of the two."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


def problem(dims):
    g = regular_grid(*dims, 1.0)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 7, 9, 5)))
    return g, s, [point_source(g, s, 0.5 * (g.min_lon + g.max_lon), g.min_lat, 3.0)]


@pytest.fixture
def ctx():
    with EikonalCuda.create(0, 64) as e:
        yield e


def resident(e, precision=64):
    e.solve(*problem((22, 20, 16)), precision=precision)
    st = e.last_stats_struct
    return st.tile_visits == 8 * sum(st.rounds)  # one box


def test_the_choice_can_be_taken_back(ctx):
    lib = L.load()
    assert resident(ctx) and resident(ctx, 32)
    for tile in (0, 6):
        L.check(lib.ts_engine_set_tile(ctx.handle, 64, tile), ctx)
        assert not resident(ctx) and resident(ctx, 32)
        L.check(lib.ts_engine_set_scheduler(ctx.handle, 0), ctx)
        assert resident(ctx) and resident(ctx, 32)
    L.check(lib.ts_engine_set_scheduler(ctx.handle, 1), ctx)
    assert not resident(ctx) and not resident(ctx, 32)
    L.check(lib.ts_engine_set_scheduler(ctx.handle, 0), ctx)
    assert resident(ctx) and resident(ctx, 32)


@pytest.mark.parametrize("chosen_before", [False, True])
def test_autotune_keeps_the_faster(ctx, chosen_before):
    if chosen_before:
        L.check(L.load().ts_engine_set_tile(ctx.handle, 64, 0), ctx)
    g, s, seeds = problem((22, 20, 16))
    tile, scheduler, ms = ctx.autotune([g], [s], [0], seeds, repeats=3)
    assert ms[(tile, scheduler)] == min(ms.values()) and len(ms) == 2
    assert resident(ctx) == (scheduler == 0) and resident(ctx, 32)
    # Given to another context it is the same choice.
    with EikonalCuda.create(0, 64) as other:
        L.check(L.load().ts_engine_set_tile(other.handle, 64, tile), other)
        L.check(L.load().ts_engine_set_scheduler(other.handle, scheduler), other)
        assert resident(other) == (scheduler == 0)


def test_autotune_of_an_engine_job_leaves_the_choice_open(ctx):
    g, s, seeds = problem((81, 81, 41))
    tile, scheduler, ms = ctx.autotune([g], [s], [0], seeds)
    assert scheduler == 0 and len(set(ms.values())) == 1 and np.isfinite(list(ms.values())).all()
    assert resident(ctx)
