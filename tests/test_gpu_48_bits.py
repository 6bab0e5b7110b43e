"""The 48-bit form runs the FP64 form's kernels."""
import numpy as np
import pytest

from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, strat", [((24, 16, 32), 1), ((256, 12, 10), 1), ((30, 27, 320), 0)])
def test_48_bits_are_fp64s(gpu_lib, dims, strat):
    """The same bits in the state, the pressure's field and the statistics after
    two CFL steps and a single stage."""
    out = []
    for precision in (48, 64):
        g = SamGpu(nx=dims[0], ny=dims[1], nz=dims[2], precision=precision, i_strat=strat, buoy_fac_z=1.0 * strat,
                   lapse=1.0 * strat, vis=1e-3, i_cfl=1, cfl0=0.5)
        g.init_random(3)
        g.step(2)
        g.stage(1)
        u, r = g.download(with_r=True)
        st = g.stats()
        out.append((u, r[:g.nz_min], np.concatenate([[st["dt"], st["energy"]], st["u_max"], st["u_var"]])))
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
