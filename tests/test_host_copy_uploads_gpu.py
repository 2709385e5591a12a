"""Uploads of a context of their own until well past the amount at which they are split over threads (256 MB in all):
each batch of tables comes back as it went up, from pageable and page-locked memory."""
import numpy as np
import pytest

from tomostar_b200 import location as loc
from tomostar_b200.eikonal import EikonalCuda
from tomostar_b200.synthetic import regular_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("locked", [False, True])
def test_uploads_add_up(locked):
    import torch

    g = regular_grid(4, 4, 16, 1.0)  # tables of 1 kB
    rng = np.random.default_rng(1)
    with EikonalCuda.create(0, 64) as e:
        for kb in (60 * 1024, 2049, 60 * 1024 + 3, 60 * 1024 + 1, 60 * 1024, 30 * 1024 + 1, 3000):
            tabs = rng.random((kb, g.count), np.float32)
            if locked:
                tabs = torch.from_numpy(tabs).pin_memory().numpy()
            with loc.Tables.upload(e, g, tabs) as t:
                for first in range(0, kb, 1500):  # below the size of a split copy
                    n = min(1500, kb - first)
                    assert np.array_equal(t.copy(first, n), tabs[first:first + n])
