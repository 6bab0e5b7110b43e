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


def wave_numbers(m):
    k = (m - 1) // 2
    return np.concatenate([np.arange(0, k + 1), np.arange(-k, 0)])


def stored(f, axis, m):
    k, n = (m - 1) // 2, f.shape[axis]
    return np.take(f, np.concatenate([np.arange(0, k + 1), np.arange(n - k, n)]), axis)


def padded(f, axis, n):
    m = f.shape[axis]
    out = np.zeros(f.shape[:axis] + (n,) + f.shape[axis + 1:], f.dtype)
    np.moveaxis(out, axis, 0)[wave_numbers(m)] = np.moveaxis(f, axis, 0)
    return out


def forward(g, p):
    f = np.fft.rfft(p, axis=2, norm="forward")[..., :g.nx_min]
    f = stored(np.fft.fft(f, axis=1, norm="forward"), 1, g.ny_min)
    return stored(np.fft.fft(f, axis=0, norm="forward"), 0, g.nz_min)


def inverse(g, f):
    f = np.fft.ifft(padded(f, 0, g.nz), axis=0, norm="forward")
    f = np.fft.ifft(padded(f, 1, g.ny), axis=1, norm="forward")
    h = np.zeros(f.shape[:2] + (g.nx // 2 + 1,), f.dtype)
    h[..., :g.nx_min] = f
    h[..., 0] = h[..., 0].real
    return np.fft.irfft(h, n=g.nx, axis=2, norm="forward")


def rhs(g, p, real):
    """rhs.f without stratification, of the physical fields p, in the arithmetic of `real`."""
    p = [q.astype(real) for q in p]
    k = [np.arange(g.nx_min)[None, None, :].astype(real), wave_numbers(g.ny_min)[None, :, None].astype(real),
         wave_numbers(g.nz_min)[:, None, None].astype(real)]
    r = [-1j * sum(k[b] * forward(g, p[a] * p[b]) for b in range(3)) for a in range(3)]
    q = sum(k[a] * r[a] for a in range(3)) / np.maximum(k[0] ** 2 + k[1] ** 2 + k[2] ** 2, real(1e-10))
    return [r[a] - k[a] * q for a in range(3)]


def distance(a, b):
    return float(np.sqrt(sum((np.abs(x - y) ** 2).sum() for x, y in zip(a, b)) / sum((np.abs(y) ** 2).sum() for y in b)))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [270, 512, 768, 1000, 1024])
def test_rhs_of_long_lines_against_fp64(gpu_lib, n, axis):
    """The resident right-hand side with long lines along one direction is no
    further from extended precision than FP64 arithmetic (numpy's transforms),
    in the 2-norm; a quarter is left for the order of FP64's sums.  White and
    steep spectra: r is a derivative, so a steep one shows the noise of a
    product line where the line itself is small."""
    dims = [12, 10, 10]
    dims[axis] = n
    g = SamGpu(nx=dims[0], ny=dims[1], nz=dims[2], dt0=0.01)
    k_sq = (np.arange(g.nx_min)[None, None, :] ** 2 + wave_numbers(g.ny_min)[None, :, None] ** 2 +
            wave_numbers(g.nz_min)[:, None, None] ** 2)
    for slope in (0.0, -11 / 12):
        rng = np.random.default_rng(n)
        u = g.wave(3)
        for f in range(3):
            u[:g.nz_min, ..., f] = forward(g, rng.standard_normal((g.nz, g.ny, g.nx))) * (1.0 + k_sq) ** slope
        u *= 2.0 ** rng.uniform(0, 1)
        g.upload(u)
        g.stage(1)
        got = g.download(with_r=True)[1]
        got = [got[:g.nz_min, ..., f] for f in range(3)]
        ref = rhs(g, [inverse(g, u[:g.nz_min, ..., f].astype(CLD)) for f in range(3)], LD)
        fp64 = rhs(g, [inverse(g, u[:g.nz_min, ..., f]) for f in range(3)], np.float64)
        assert distance(got, ref) <= 1.25 * distance(fp64, ref), slope
    g.close()


@pytest.mark.parametrize("n", [12, 64, 250, 256, 320, 512])
def test_rhs_of_given_fields_keeps_small_products(gpu_lib, n):
    """sam_gpu_rhs on physical arrays where u is 1e-18 of itself wherever v is
    not zero: r_1 at kx = 0 is -i ky times the mean of u v over x, a product of
    normal numbers that FP64 keeps to its last bits beside u u of order one.
    Bar as above."""
    g = SamGpu(nx=n, ny=10, nz=10)
    rng = np.random.default_rng(n)
    uu = g.phys(g.lr)
    uu[..., :2] = rng.standard_normal(uu.shape[:3] + (2,))
    uu[: n // 2, ..., 1] = 0.0
    uu[n // 2:, ..., 0] *= 1e-18
    p = [uu[..., f].transpose(2, 1, 0).copy() for f in range(3)]
    got = g.rhs(uu)[:g.nz_min, 1:, 0, 0]
    ref, fp64 = (rhs(g, p, real)[0][:, 1:, 0] for real in (LD, np.float64))
    assert distance([got], [ref]) <= 1.25 * distance([fp64], [ref])
    g.close()
