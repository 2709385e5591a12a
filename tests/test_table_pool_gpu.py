"""Resident tables of more than a quarter of the device's memory leave the pool of the ray calls alone: what a call
frees stays there for the next one, as without tables."""
import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200 import location as loc
from tomostar_b200 import synthetic as syn
from tomostar_b200.eikonal import EikonalCuda
from tomostar_b200.rays import RayKernels

pytestmark = pytest.mark.gpu


def held_after_a_call(table_bytes):
    """Device memory that a context holds after a forward step whose rows have been freed (tables apart)."""
    import torch

    p = syn.inversion_step_121()
    with EikonalCuda.create(0, 64) as e:
        g = syn.regular_grid(128, 128, 64, 1.0)
        one = np.zeros((int(4.6e9) // (4 * g.count), g.count), np.float32)
        tables = [loc.Tables.upload(e, g, one) for _ in range(-(-table_bytes // one.nbytes))]
        rk = RayKernels(p.inv, p.grid, e)
        before = torch.cuda.mem_get_info()[0]
        rk.compute(p.slowness, p.stations, p.events, np.concatenate([p.arrivals] * 20), precision=64, mode=L.MODE_FAST)
        rk.compute(p.slowness, p.stations, p.events, p.arrivals[:10], precision=64, mode=L.MODE_FAST)
        held = before - torch.cuda.mem_get_info()[0]
        for t in tables:
            t.close()
    return held


def test_rows_pool_beside_large_tables():
    import torch

    quarter = torch.cuda.get_device_properties(0).total_memory // 4
    held_after_a_call(0)
    alone = held_after_a_call(0)
    beside = held_after_a_call(quarter + (1 << 30))
    assert abs(beside - alone) <= 64 << 20, (alone, beside)
