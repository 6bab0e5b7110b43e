"""Rows of an x-pass tile that do not fit and are cut down."""
import numpy as np
import pytest

from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, rows", [(512, 6), (512, 12), (1024, 10), (270, 14)])
def test_cut_tiles_stay_even(gpu_lib, nx, rows):
    """A tile takes its rows two by two: whatever is left of it, every row of
    the box is transformed, to the same bits."""
    ref = None
    for r in (2, rows):
        g = SamGpu(nx=nx, ny=12, nz=6, i_strat=1, vis=1e-3, dt0=0.01, buoy_fac_z=1.0, lapse=1.0, i_cfl=1, cfl0=0.5)
        g.init_random(3)
        g.set_tiles(x_rows=r)
        g.step(1)
        got = g.download(), np.array([g.stats()["dt"]])
        ref = ref or got
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
        g.close()
