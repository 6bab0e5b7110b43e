"""x_deriv and y_deriv of long lines against the oracle, at the bar of the
per-routine comparisons."""
import numpy as np
import pytest

import oracle as O
from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 320, 324, 512, 1000, 1024])
def test_plane_derivatives_of_long_lines(gpu_lib, n):
    """Eight pairs of lines take 48 KB of shared memory and more from about 300
    points on."""
    rng = np.random.default_rng(n)
    for dims in ((n, 24), (24, n)):
        g, o = SamGpu(nx=dims[0], ny=dims[1], nz=4), O.Oracle(nx=dims[0], ny=dims[1], nz=4)
        f = np.asfortranarray(rng.standard_normal(dims))
        for got, ref in ((g.x_deriv(f), o.x_deriv(f)), (g.y_deriv(f), o.y_deriv(f))):
            assert np.abs(got - ref).max() < 1e-13 * np.abs(ref).max()
        g.close()
