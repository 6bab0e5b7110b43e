"""The learned closure's coefficients belong to points: the fused FP32 x pass of
256-point lines with coefficients that vary from point to point."""
import numpy as np
import pytest

import closure as CL
import oracle as O
from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


def second_stage(cfg, params, u0, sched):
    """Stage 1, which takes the coefficients (none: no closure), then stage 2
    with the x pass in another schedule: (U, R, the coefficients)."""
    g = SamGpu(precision=32, **cfg)
    g.upload(u0)
    coef = None
    if params is not None:
        g.mlp_set(params)
        # (the invariants asked for before the closure is switched on)
        coef = g.mlp_forward(g.closure_inputs()[0]).reshape(g.nz, g.ny, g.nx, 2)
        g.set_les(3)
    g.stage(1)
    g.set_fft_schedule([0, 0, sched, 0, 0])
    g.stage(2)
    u, r = g.download(with_r=True)
    m = g.nz_min
    g.close()
    return u[:m], r[:m, ..., :4], coef


@pytest.mark.parametrize("ny", [4, 8, 9, 10, 15])
def test_varying_coefficients_on_256_point_lines(gpu_lib, ny):
    """Fused kernel (4-row tiles: whole, with one, two or three rows left)
    against the general kernel, on the same state and the same coefficients.
    Both add the same terms to the same products and differ by the rounding of
    two transforms: 64 roundings of the largest value, as with equal
    coefficients.  Neighbours in each direction differ by a twentieth of the
    coefficient at least, and the closure's part of R is a thousand times the
    bar, so a coefficient of another point would show."""
    cfg = dict(nx=256, ny=ny, nz=8, i_strat=1, buoy_fac_z=1.0, lapse=1.0, vis=1e-4, i_cfl=1, cfl0=0.5)
    u0 = O.Oracle(**cfg).init_random(7, 0, 1.0, 0, 0.1)
    p = CL.init_params(2)
    p[CL.OFF_W3:CL.OFF_B3] *= 10
    (u, r, coef), (ur, rr, _) = (second_stage(cfg, p, u0, s) for s in (0, 1))
    bar = 64 * 2.0 ** -24
    for f in range(4):
        assert np.abs(u[..., f] - ur[..., f]).max() <= bar * np.abs(ur[..., f]).max(), f
        assert np.abs(r[..., f] - rr[..., f]).max() <= bar * np.abs(rr[..., f]).max(), f
    none = second_stage(cfg, None, u0, 0)[1]
    for axis in (0, 1, 2):
        assert np.abs(coef - np.roll(coef, 1, axis)).mean() > 0.05 * coef.mean(), axis
    for f in range(4):
        assert np.abs(r[..., f] - none[..., f]).max() > 1000 * bar * np.abs(rr[..., f]).max(), f
