"""The shortest lines with compile-time stages against the oracle."""
import numpy as np
import pytest

import oracle as O
from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, tol", [(64, 1e-13), (32, 1e-5)])
@pytest.mark.parametrize("n", [6, 8, 9, 10, 12, 15, 16])
def test_short_lines(gpu_lib, precision, tol, n):
    """One resident RK stage with lines of 8 to 15 points, and the lengths on
    either side of them, along each direction, at the bars of the per-routine
    and the FP32 comparisons (both relative to the largest value)."""
    for axis in range(3):
        d = [20, 18, 24]
        d[axis] = n
        if d[0] % 2:
            continue
        cfg = dict(nx=d[0], ny=d[1], nz=d[2], i_strat=1, vis=1e-2, pr=0.7, dt0=0.01, buoy_fac_z=1.0, lapse=1.0, i_cfl=1,
                   cfl0=0.5)
        g, o = SamGpu(precision=precision, **cfg), O.Oracle(**cfg)
        u = o.init_random(7)
        g.upload(u)
        r = o.wave(o.d.lr)
        o.stage(u, r, 1)
        g.stage(1)
        ug = g.download()
        m = o.d.nz_min
        assert np.abs(ug[:m] - u[:m]).max() < tol * np.abs(u[:m]).max(), axis
        assert abs(g.stats()["dt"] - o.stats()["dt"]) < tol * o.stats()["dt"], axis
        g.close()
