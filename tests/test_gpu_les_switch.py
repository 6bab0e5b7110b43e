"""Closures switched on, changed and off on one solver: the pencil buffers grow
once and stay."""
import numpy as np
import pytest

from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_closures_after_one_another(gpu_lib, precision):
    """Each model's step from the same state gives the same bits whatever models
    ran before it."""
    cfg = dict(nx=32, ny=24, nz=20, precision=precision, i_strat=1, buoy_fac_z=1.0, lapse=1.0, vis=1e-3, dt0=1e-3)
    g = SamGpu(**cfg)
    g.init_random(3)
    u0 = g.download()
    seen = {}
    for model in (0, 1, 3, 2, 0, 3, 1, 2):
        g.set_les(model, c_smag=0.03, pr_t=0.7)
        g.upload(u0)
        g.set_tstep(1, 1e-3, 0.0)
        g.step(1)
        u = g.download()
        assert np.array_equal(seen.setdefault(model, u), u), model
    g.close()
