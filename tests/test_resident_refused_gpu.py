"""A device that does not take the resident solver's launch (no room for the cluster, or the launch refused): the
tiled engine solves the job. The refusals come from a stand-in for the CUDA runtime's call in a child process."""
import os
import subprocess
import sys

import numpy as np
import pytest

from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.synthetic import regular_grid, vp_linear

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKES = {
    "no_room": "int cudaOccupancyMaxActiveClusters(int* n, const void* f, const void* c) { *n = 0; count(); return 0; }",
    "query_fails": "int cudaOccupancyMaxActiveClusters(int* n, const void* f, const void* c) { count(); return 1; }",
    "launch_refused": "int cudaLaunchKernelExC(const void* c, const void* f, void** a) { count(); return 701; }",
}
COUNT = """#include <stdio.h>
#include <stdlib.h>
static void count(void) { FILE* f = fopen(getenv("FAKE_CALLS"), "a"); if (f) { fputc('x', f); fclose(f); } }
"""
CHILD = """
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from tests.test_resident_refused_gpu import problem
from tomostar_b200.eikonal import EikonalCuda
with EikonalCuda.create(0, 64) as e:
    np.save(sys.argv[2], np.concatenate([e.solve(*problem()), e.solve(*problem(), precision=32)]))
"""


def problem():
    g = regular_grid(61, 61, 31, 1.0)
    s = 1 / vp_linear(g)
    return g, s, [point_source(g, s, g.min_lon, g.min_lat, 3.0), point_source(g, s, g.max_lon, g.min_lat, 0.0)]


@pytest.mark.parametrize("fake", FAKES)
def test_the_engine_takes_the_job(fake, tmp_path):
    src, so, out, calls = (str(tmp_path / n) for n in ("fake.c", "fake.so", "out.npy", "calls"))
    with open(src, "w") as f:
        f.write(COUNT + FAKES[fake])
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, src], check=True)
    subprocess.run([sys.executable, "-c", CHILD, ROOT, out], check=True, timeout=300, cwd=ROOT,
                   env=dict(os.environ, LD_PRELOAD=so, FAKE_CALLS=calls))
    assert os.path.getsize(calls) == 2  # both solves met the refusal
    with EikonalCuda.create(0, 64) as e:
        want = np.concatenate([e.solve(*problem()), e.solve(*problem(), precision=32)])
    assert np.array_equal(np.load(out), want)
