"""What a context keeps between calls (field buffers of a table build, memory of freed tables) is there for any call
that needs it: on a device with 3 GB left, a call that fits only with that memory is not refused, batches and
suggestions count it."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200 import location as loc
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import regular_grid, vp_linear

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def short():
    """A context on a device whose memory is taken but for 3 GB, and a call that tells what is left."""
    import torch

    with EikonalCuda.create(0, 64) as e:
        g = regular_grid(200, 200, 100, 1.0)
        s = 1 / vp_linear(g)
        seeds = [point_source(g, s, g.min_lon, g.min_lat, 3.0)]
        build(e, g, s, 1).close()  # the context's own buffers
        torch.cuda.init()
        free = torch.cuda.mem_get_info()[0]
        hold = torch.empty(free - 3000 * MB, dtype=torch.uint8, device="cuda")
        yield e, g, s, seeds, lambda: torch.cuda.mem_get_info()[0]
        del hold
        torch.cuda.empty_cache()


def build(e, g, s, n):
    lon = np.linspace(g.min_lon, g.max_lon, n + 2)[1:-1]
    src = np.stack([lon, np.full(n, g.min_lat), np.zeros(n)], axis=1)
    return loc.Tables.build(e, g, s[None, :], src, np.zeros(n, np.int32))


def uploaded(e, n_bytes):
    g = regular_grid(64, 64, 64, 1.0)
    return loc.Tables.upload(e, g, np.zeros((n_bytes // (4 * g.count), g.count), np.float32))


def test_kept_field_buffers_make_room(short):
    e, g, s, seeds, left = short
    fields = 20
    with build(e, g, s, fields):
        before = left()
        kept = fields * 8 * 228 * g.ny * g.nz  # rows of 224 nodes and 4 of halo
        with uploaded(e, before + kept // 2) as t:
            assert t.count * 4 * 64 ** 3 > before
    # ... and are allocated again by the next build.
    with build(e, g, s, fields) as t:
        one = np.asarray(e.solve(g, s, [point_source(g, s, float(np.linspace(g.min_lon, g.max_lon, 22)[3]), g.min_lat, 0.0)],
                                 output=np.empty((1, g.count), np.float32)))
        assert np.array_equal(t.copy(2, 1)[0], one[0])


def test_freed_tables_count_as_free(short):
    e, g, s, seeds, left = short
    suggested = e.suggest_batch(g.count)
    uploaded(e, 2200 * MB).close()
    assert left() < 1200 * MB  # (idle in the context's pool)
    assert e.suggest_batch(g.count) >= suggested - 2
    with build(e, g, s, 25) as t:
        assert t.stats.launches == 1  # 0.9 GB of field buffers in one batch


def test_output_staging_is_cut_to_the_room(short):
    e, g, s, seeds, left = short
    n = int((left() - 200 * MB) // (8 * 228 * g.ny * g.nz))
    got = e.solve(g, s, seeds * n, output=np.empty((n, g.count), np.float32), mode=L.MODE_FAST)
    assert np.array_equal(got[0], got[n - 1]) and np.isfinite(got[n // 2]).all()
