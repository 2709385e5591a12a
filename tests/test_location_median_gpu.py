"""The warp search's weighted median at the sizes where its picks per lane change (32, 64, 96, 128) and
with what a selection can get wrong: equal residuals, zero weights, all weights zero, weights at the
ends of the exact range, picks whose table holds no time. With Geiger off everything equals the oracle
to the bit."""
import numpy as np
import pytest

from oracle import oracle as O
from tomostar_b200 import location as loc
from tomostar_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

COUNTS = [4, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129]


@pytest.fixture(scope="module")
def job_tables(solver):
    job = syn.relocation_small()
    tables = loc.Tables.build(solver, job.grid, job.slowness, job.table_source, job.table_phase)
    tabs = tables.copy()
    tabs[3, : tabs.shape[1] // 2] = np.inf  # one table without times in half of the grid
    tables.close()
    up = loc.Tables.upload(solver, job.grid, tabs)
    yield job, up, tabs
    up.close()


@pytest.mark.parametrize("weights", ["quality", "some zero", "all zero", "range ends"])
def test_pick_counts(solver, job_tables, weights):
    job, tables, tabs = job_tables
    rng = np.random.default_rng(7)
    table, sec, w, corr, off = [], [], [], [], [0]
    for e, n in enumerate(COUNTS):
        tb = rng.integers(0, len(tabs), n)
        node = rng.integers(0, tabs.shape[1])
        t = tabs[tb, node].astype(np.float64)
        t[~np.isfinite(t)] = 5.0
        s = t + rng.normal(0, 0.05, n)
        s[n // 2:] = np.round(s[n // 2:], 1)  # picks repeated on one table share residuals
        tb[n // 2:] = tb[n // 2]
        table.append(tb)
        sec.append(s)
        w.append({"quality": rng.choice([1.0, 0.75, 0.5, 0.25], n),
                  "some zero": rng.choice([1.0, 0.0, 0.25], n),
                  "all zero": np.zeros(n),
                  "range ends": rng.choice([2.0 ** -24, 262143.5, 1.0], n)}[weights])
        corr.append(np.zeros(n))
        off.append(off[-1] + n)
    args = (np.array(off, np.int32), np.concatenate(table).astype(np.int32), np.concatenate(sec), np.concatenate(w),
            np.concatenate(corr))
    start = job.start[: len(COUNTS)]
    tsta = job.table_source[:, :2]
    kw = dict(max_geiger_iterations=0)
    dev = loc.locate(solver, tables, start, *args, tsta, loc.LocatorSettings(**kw))
    ora, res = O.locate_many(O.Grid.of(job.grid), tabs, tsta, O.LocatorSettings(**kw), start, *args)
    for f in ("t0", "lon", "lat", "depth_km", "used", "rejected", "status"):
        assert np.array_equal(dev.locations[f], ora[f]), f
    assert np.array_equal(dev.residuals, res, equal_nan=True)
