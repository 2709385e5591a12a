"""Results into memory whose pages are there, not there and partly there, around the sizes at which a copy is split
over threads (2 MB) and at which it is split whatever the pages (24 MB)."""
import ctypes as C
import mmap

import numpy as np
import pytest

from tomostar_b200 import _lib as L
from tomostar_b200 import location as loc
from tomostar_b200.eikonal import EikonalCuda
from tomostar_b200.synthetic import regular_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb", [1900, 2049, 2600, 23 * 1024 + 900, 24 * 1024 + 4])
def test_pages(kb):
    g = regular_grid(4, 4, 16, 1.0)  # tables of 1 kB
    tabs = np.random.default_rng(kb).random((kb, g.count), np.float32)
    with EikonalCuda.create(0, 64) as e, loc.Tables.upload(e, g, tabs) as t:
        for share in (0.0, 0.4, 1.0):
            m = mmap.mmap(-1, tabs.nbytes)
            out = np.frombuffer(m, np.float32)
            out[: int(share * out.size)] = -1
            assert L.load().ts_tables_copy(t.handle, 0, kb, out.ctypes.data_as(C.POINTER(C.c_float))) == 0
            assert np.array_equal(out.reshape(tabs.shape), tabs)
            del out
            m.close()
