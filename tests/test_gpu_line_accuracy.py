"""Accuracy of the FP64 form's x pass and of its long lines, whose products and
transforms run in 64-bit fixed point (sam_gb300/csrc/fx64.cuh), against
extended precision."""
import numpy as np
import pytest

from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu

LD, CLD = np.longdouble, np.clongdouble
ULP = 2.0 ** -53


@pytest.mark.parametrize("n", [128, 256, 512])
def test_mean_of_a_square_has_no_bias(gpu_lib, n):
    """u = v = f(x) (1 + cos y): the mode (0, 1, 0) of rhs.f's u v is the mean
    of f^2, whose transforms along y and z (four points) are sums alone.  Three
    results are rounded to FP64 on its way, each by at most 2^-53 of it and by
    0.58 of that in the rms; f's own errors and the products' are 1 / sqrt(n) of
    one line's.  One trial's error is therefore about 2^-53 in the rms, the mean
    of 128 trials 0.09, and 0.4 is more than four times that."""
    g = SamGpu(nx=n, ny=4, nz=4, dt0=0.01)
    err = []
    for t in range(128):
        rng = np.random.default_rng(t)
        a = rng.standard_normal(g.nx_min) + 1j * rng.standard_normal(g.nx_min)
        a[0] = a[0].real
        a *= 2.0 ** rng.uniform(0, 1)
        u = g.wave(g.lu)
        for f in (0, 1):
            u[0, :3, :, f] = np.array([1.0, 0.5, 0.5])[:, None] * a
        g.upload(u)
        g.stage(1)
        got = -g.download(with_r=True)[1][0, 1, 0, 0].imag
        e = a.astype(CLD)
        ref = e[0].real ** 2 + 2 * (e[1:].real ** 2 + e[1:].imag ** 2).sum()
        err.append(float((got - ref) / ref) / ULP)
    g.close()
    assert abs(np.mean(err)) < 0.4, (np.mean(err), np.std(err))
