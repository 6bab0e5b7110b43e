"""Accuracy and exceptional lines of the FP64 form's line transforms, which run
in 64-bit fixed point (sam_gb300/csrc/fx64.cuh), against extended precision.

Bar: the relative error of a line in the 2-norm, rms over the lines, within
0.8 sqrt(log2 n) 2^-53 (and at least 2^-53): the error model of an FP64
radix-2 transform, whose log2 n levels each round every value once by 0.4 to
0.8 units of 2^-53 in the rms."""
import numpy as np
import pytest

import oracle as O
from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu

LENGTHS = [2, 3, 4, 5, 6, 8, 9, 15, 16, 25, 30, 32, 45, 48, 64, 81, 96, 125, 128, 135, 162, 200, 243, 256, 320, 500, 512,
           540, 1024]


def lines(kind, n, m, rng):
    z = rng.standard_normal((n, m)) + 1j * rng.standard_normal((n, m))
    k = np.minimum(np.arange(n), n - np.arange(n))[:, None]
    if kind == "steep":
        return z * (1.0 + k) ** (-5 / 3)
    if kind == "smooth":
        return z * np.exp(-0.3 * k)
    if kind == "single":
        return z * (k == (1 if n >= 4 else 0))
    if kind == "range":
        return z * 10.0 ** rng.uniform(-30, 0, (n, m))
    return z


def solver(n):
    return SamGpu(nx=4, ny=16, nz=n, n_dealias=0)


def stored(g, full):
    """The stored z modes 0 .. k, -k .. -1 of full lines (n, m) as u(Nze, Ny_min, Nx_min, 1)."""
    n, km = g.nz, (g.nz_min - 1) // 2
    u = np.zeros((n, g.ny_min, g.nx_min, 1), dtype=np.complex128, order="F")
    keep = np.concatenate([full[:km + 1], full[n - km:]], 0) if km else full[:1]
    u[:g.nz_min, :, :, 0] = keep.reshape(g.nz_min, g.ny_min, g.nx_min)
    return u


def padded(g, u):
    n, km = g.nz, (g.nz_min - 1) // 2
    x = np.zeros((n,) + u.shape[1:3], dtype=np.clongdouble)
    x[:km + 1] = u[:km + 1, :, :, 0]
    if km:
        x[n - km:] = u[km + 1:2 * km + 1, :, :, 0]
    return x


def inverse(g, u):
    return np.moveaxis(g.z_trans_b(u, 1)[..., 0], 2, 0)


def line_errors(got, ref):
    scale = np.sqrt((np.abs(ref) ** 2).sum(0))
    return np.sqrt((np.abs(got - ref) ** 2).sum(0))[scale > 0] / scale[scale > 0]


def bar(n):
    return 2.0 ** -53 * max(1.0, 0.8 * np.sqrt(np.log2(n)))


@pytest.mark.parametrize("n", LENGTHS)
def test_transforms_against_extended_precision(gpu_lib, n):
    g = solver(n)
    rng = np.random.default_rng(n)
    m = g.ny_min * g.nx_min
    for kind in ("white", "steep", "smooth", "single", "range"):
        u = stored(g, lines(kind, n, m, rng))
        ref = np.fft.ifft(padded(g, u), axis=0, norm="forward")
        err = line_errors(inverse(g, u), ref)
        assert np.sqrt((err ** 2).mean()) < bar(n), (kind, "inverse")
        f = np.zeros((n, g.ny_min, g.nx_min, 1), dtype=np.complex128, order="F")
        f[..., 0] = lines(kind, n, m, rng).reshape(n, g.ny_min, g.nx_min)
        full = np.fft.fft(f[..., 0].astype(np.clongdouble), axis=0, norm="forward")
        km = (g.nz_min - 1) // 2
        ref = np.concatenate([full[:km + 1], full[n - km:]], 0) if km else full[:1]
        norm = np.sqrt((np.abs(full) ** 2).sum(0))
        got = g.z_trans_f(f.copy(order="F"), 1)[:g.nz_min, ..., 0]
        err = np.sqrt((np.abs(got - ref) ** 2).sum(0)) / norm
        assert np.sqrt((err ** 2).mean()) < bar(n), (kind, "forward")
    g.close()


@pytest.mark.parametrize("n", [30, 64, 243, 256, 512])
def test_scaling_by_powers_of_two_is_exact(gpu_lib, n):
    """One scale per line: a line times 2^k gives the same integers, so the
    results are the same times 2^k, down to and including lines of subnormals
    and up to the largest numbers."""
    g = solver(n)
    u = stored(g, lines("smooth", n, g.ny_min * g.nx_min, np.random.default_rng(1)))
    ref = inverse(g, u)
    for k in (-900, -500, -1, 3, 500, 900, 1005):
        assert np.array_equal(inverse(g, u * 2.0 ** k), ref * 2.0 ** k), k
    tiny = inverse(g, u * 2.0 ** -1030)
    assert np.abs(tiny - ref * 2.0 ** -1030).max() <= n * 2.0 ** -1074  # inputs and results rounded to subnormals
    # results beyond the largest number are infinities, as in FP64
    assert not np.isfinite(inverse(g, np.where(u != 0, 1.0, 0.0) * 1.7e308)).all()
    g.close()


@pytest.mark.parametrize("n", [30, 64, 256, 512])
def test_exceptional_lines(gpu_lib, n):
    """Zeros stay zeros; an infinity or a NaN spoils its own line and no other."""
    g = solver(n)
    u = stored(g, lines("white", n, g.ny_min * g.nx_min, np.random.default_rng(2)))
    u[:, 1, 0, 0] = 0.0
    ref = inverse(g, u)
    assert not ref[:, 1, 0].any()
    for bad in (np.inf, -np.inf, np.nan):
        v = u.copy(order="F")
        v[2, 0, 0, 0] = complex(1.0, bad)
        got = inverse(g, v)
        line = got[:, 0, 0]
        assert not (np.isfinite(line.real) | np.isfinite(line.imag)).any()
        got[:, 0, 0] = ref[:, 0, 0]
        assert np.array_equal(got, ref)
    g.close()


COMPILED = sorted(2 ** a * 3 ** b * 5 ** c for a in range(9) for b in range(6) for c in range(4)
                  if 16 <= 2 ** a * 3 ** b * 5 ** c <= 256)


@pytest.mark.parametrize("precision, tol", [(64, 1e-13), (32, 1e-5)])
@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_every_compiled_length(gpu_lib, precision, tol, axis):
    """One resident RK stage on boxes with each length that has compile-time
    stages along one direction, against the oracle at the bars of the
    per-routine and the FP32 comparisons (both relative to the largest value)."""
    for n in COMPILED:
        if axis == "x" and n % 2:
            continue
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
        so, sg = o.stats(), g.stats()
        assert abs(sg["dt"] - so["dt"]) < tol * so["dt"], n
        np.testing.assert_allclose(sg["u_var"][:4], so["u_var"][:4], rtol=max(tol, 1e-12))
        g.close()


@pytest.mark.parametrize("pr", [1.0, 0.4])
def test_damping_of_single_modes(gpu_lib, pr):
    """Integrating factors exp(-x), x = nu k^2 dt, from nearly one to far below
    a half, where the epilogue changes from u + u (e - 1) to u e: no flow, so
    each mode of T is damped alone.  Bar, per mode and relative to it: the
    three stages' exponents carry four roundings of relative size 2^-53 each
    (nu dt, the two parts of k^2, their product), which the exponential turns
    into 4 x 2^-53, and each stage rounds its factors, their join and the
    product (four more)."""
    cfg = dict(nx=24, ny=20, nz=32, i_strat=1, vis=0.5, pr=pr, dt0=0.15, i_cfl=0)
    g = SamGpu(**cfg)
    u = g.wave(4)
    rng = np.random.default_rng(3)
    m, my, mx = g.nz_min, g.ny_min, g.nx_min
    u[:m, :, 1:, 3] = rng.standard_normal((m, my, mx - 1)) + 1j * rng.standard_normal((m, my, mx - 1))
    g.upload(u)
    g.step(1)
    got = g.download()
    k = [np.concatenate([np.arange(0, q // 2 + 1), np.arange(-(q // 2), 0)]) for q in (m, my)]
    k_sq = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + np.arange(1, mx)[None, None, :] ** 2
    x = np.longdouble(0.5) / np.longdouble(pr) * np.longdouble(0.15) * k_sq
    ref = u[:m, :, 1:, 3] * np.exp(-x)
    assert (np.abs(got[:m, :, 1:, 3] - ref) <= (12 + 4 * x) * 2.0 ** -53 * np.abs(ref)).all()
    g.close()


@pytest.mark.parametrize("nx, ny", [(16, 9), (64, 32), (90, 27), (128, 16), (250, 12)])
@pytest.mark.parametrize("les", [0, 1])
def test_product_lines_do_not_depend_on_the_tile(gpu_lib, nx, ny, les):
    """A product line is formed, transformed and stored by one team whatever
    the tile's rows and the scratch lines (fewer than the teams, or one for
    each): the same bits, tiles cut by Ny and an odd last row included."""
    ref = None
    for rows, group in ((8, 9), (2, 1), (4, 2), (16, 9), (16, 1)):
        g = SamGpu(nx=nx, ny=ny, nz=8, i_strat=1, vis=1e-3, dt0=0.01, buoy_fac_z=1.0, lapse=1.0, i_cfl=1, cfl0=0.5)
        g.init_random(3)
        if les:
            g.set_les(1, c_smag=0.03, pr_t=0.7)
        g.set_tiles(x_rows=rows, x_group=group)
        g.step(2)
        got = g.download(), np.array([g.stats()["dt"]])
        ref = ref or got
        for a, b in zip(got, ref):
            assert np.array_equal(a, b), (rows, group)
        g.close()
