"""The range of dm.f's coefficient on the GPU, whose test filter runs on
integers under a power of two per tile."""
import numpy as np
import pytest

from sam_gb300 import SamGpu
from test_gpu_les import velocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 5, 3), (40, 9, 15)])
def test_dynamic_coefficient_of_the_largest_fields(gpu_lib, dims):
    """Velocity times 2^k in a box 2^(k + 5) as large: every difference, product
    and sum of dm.f is the same times a power of two, L_ij by 2^2k and M_ij by
    2^-10, and the coefficient by 2^(2 k + 10), to the bit.  u_i u_j comes to
    2^1018 (k = 508), its 27-point sums past the largest number, while every
    filtered value, sum and the coefficient itself stay below it."""
    nx, ny, nz = dims
    u = velocity(nx, ny, nz, 2)
    ref = SamGpu(nx=nx, ny=ny, nz=nz, xl=1.0, yl=1.3, zl=0.7).dm(u)[1]
    assert ref != 0.0
    for k in (-400, 0, 480, 500, 503, 506, 508):
        s = 2.0 ** (k + 5)
        g = SamGpu(nx=nx, ny=ny, nz=nz, xl=s, yl=1.3 * s, zl=0.7 * s)
        assert g.dm(u * 2.0 ** k)[1] == np.ldexp(ref, 2 * k + 10), k
        g.close()
