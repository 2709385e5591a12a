"""More fields than the device has room for at once: solved in runs that fit, with the fields that each has alone. A
device whose memory is taken but for 3 GB."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import regular_grid, vp_linear

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module")
def short():
    import torch

    with EikonalCuda.create(0, 64) as e:
        g = regular_grid(33, 300, 100, 1.0)
        s = 1 / vp_linear(g)
        x, y = np.linspace(g.min_lon, g.max_lon, 7)[1:-1], np.linspace(g.min_lat, g.max_lat, 11)[1:-1]
        seeds = [point_source(g, s, float(x[k % 5]), float(y[k % 9]), 3.0) for k in range(5)]
        alone = [e.solve(g, s, [sd], mode=L.MODE_FAST)[0].astype(np.float32) for sd in seeds]
        torch.cuda.init()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - 3000 * MB, dtype=torch.uint8, device="cuda")
        yield e, g, s, seeds, alone
        del hold
        torch.cuda.empty_cache()


@pytest.mark.parametrize("locked", [False, True])
@pytest.mark.parametrize("multi", [False, True])
def test_more_fields_than_room(short, locked, multi):
    e, g, s, seeds, alone = short
    n = 251  # rows of 68 values for 33 nodes: 4 GB of field buffers
    sets = [seeds[k % 5] for k in range(n)]
    if multi:
        if locked:
            pytest.skip("solve_multi makes its own output")
        out = e.solve_multi([g], [s], [0] * n, sets, out_dtype=np.float32, mode=L.MODE_FAST)
    else:
        import torch

        out = torch.empty((n, g.count), dtype=torch.float32, pin_memory=locked).numpy()
        e.solve(g, s, sets, output=out, mode=L.MODE_FAST)
    for k in range(n):
        assert np.array_equal(out[k], alone[k % 5]), k


def test_unsettled_part_is_refused(short):
    e, g, s, seeds, _ = short
    ok, why = e.try_solve(g, s, [seeds[k % 5] for k in range(251)], np.empty((251, g.count), np.float32), max_rounds=1)
    assert not ok and "not settled" in why
