"""Lines longer than the compile-time lengths against the oracle, at the sizes
where the register budget of their kernels changes."""
import numpy as np
import pytest

import oracle as O
from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, tol", [(64, 1e-13), (48, 1e-13), (32, 1e-5)])
@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_long_lines(gpu_lib, precision, tol, axis):
    """One resident RK stage with 384, 400, 640, 648 or 1024 points along one
    direction, at the bars of the per-routine and the FP32 comparisons (both
    relative to the largest value)."""
    for n in (384, 400, 640, 648, 1024):
        d = dict(nx=8, ny=10, nz=12)
        d["n" + axis] = n
        cfg = dict(i_strat=1, vis=1e-2, pr=0.7, dt0=0.01, buoy_fac_z=1.0, lapse=1.0, i_cfl=1, cfl0=0.5, **d)
        g, o = SamGpu(precision=precision, **cfg), O.Oracle(**cfg)
        u = o.init_random(7)
        g.upload(u)
        r = o.wave(o.d.lr)
        o.stage(u, r, 1)
        g.stage(1)
        ug = g.download()
        m = o.d.nz_min
        assert np.abs(ug[:m] - u[:m]).max() < tol * np.abs(u[:m]).max(), n
        assert abs(g.stats()["dt"] - o.stats()["dt"]) < tol * o.stats()["dt"], n
        g.close()
