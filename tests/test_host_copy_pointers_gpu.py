"""Device and page-locked memory where a call takes an array: copied as it is, whatever the size (the threads that
split copies of pageable memory must not touch a device address)."""
import ctypes as C

import numpy as np
import pytest

from tomostar_b200 import location as loc
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import checkerboard, km_to_geo, regular_grid, vp_linear

pytestmark = pytest.mark.gpu


def at(tensor, dtype, shape):
    """An array over a tensor's memory (never read or written on the host)."""
    return np.frombuffer((C.c_char * (tensor.numel() * tensor.element_size())).from_address(tensor.data_ptr()), dtype).reshape(shape)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("dims", [(20, 18, 10), (81, 81, 41)])  # below and above the size of a split copy
def test_device_memory_in_and_out(dims, precision):
    import torch

    g = regular_grid(*dims, 1.0)
    s = 1 / (vp_linear(g) * (1 + checkerboard(g, 7, 9, 5)))
    lon, lat = km_to_geo(g, 5.0, 7.0, 1.0)
    seeds = [point_source(g, s, float(lon), float(lat), 2.0)]
    with EikonalCuda.create(0, 64) as e:
        want = e.solve(g, s, seeds, precision=precision)  # (makes the copy threads' streams at the larger size)
        for device in ("cuda", "cpu"):
            out = torch.zeros(g.count, dtype=torch.float64, device=device, pin_memory=device == "cpu")
            slow = torch.from_numpy(s.copy()).to(device)
            ok, why = e.try_solve(g, at(slow, np.float64, -1), seeds, at(out, np.float64, (1, -1)), precision=precision)
            assert ok, why
            assert np.array_equal(out.cpu().numpy(), want[0])


def test_tables_to_device_memory():
    import torch

    g = regular_grid(32, 32, 16, 1.0)
    tabs = np.random.default_rng(2).random((40, g.count), np.float32)
    up = torch.from_numpy(tabs).cuda()
    with EikonalCuda.create(0, 64) as e, loc.Tables.upload(e, g, tabs) as first:
        first.copy()
        with loc.Tables.upload(e, g, at(up, np.float32, tabs.shape)) as t:
            assert np.array_equal(t.copy(), tabs)
