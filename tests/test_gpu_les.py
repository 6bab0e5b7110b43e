"""Parity of the subgrid-model routines (filter.f, sm.f, dm.f) and get_mean.f
on the GPU against the oracle's restatements."""
import numpy as np
import pytest

import closure as CL
import oracle as O
from sam_gb300 import SamGpu

pytestmark = pytest.mark.gpu


def periodic_fill(a):
    """periodicity.f:7-32: halo planes 0 and n+1 from the periodic images,
    x first, then y, then z."""
    a[0], a[-1] = a[-2], a[1]
    a[:, 0], a[:, -1] = a[:, -2], a[:, 1]
    if a.ndim >= 3:
        a[:, :, 0], a[:, :, -1] = a[:, :, -2], a[:, :, 1]
    return a


def relerr(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 12, 10), (24, 20, 32)])
def test_filter(gpu_lib, dims):
    nx, ny, nz = dims
    g, o = SamGpu(nx=nx, ny=ny, nz=nz), O.Oracle(nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(4)
    f_bar = np.asfortranarray(rng.standard_normal((nx + 2, ny + 2, 6, 3)))  # halos arbitrary: used as given in y
    assert relerr(g.filter(f_bar, 6), o.filter(f_bar, 6)) < 1e-14


def velocity(nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    u = np.zeros((nx + 2, ny + 2, nz + 2, 3), order="F")
    x = np.arange(nx + 2)[:, None, None] * 2 * np.pi / nx
    y = np.arange(ny + 2)[None, :, None] * 2 * np.pi / ny
    z = np.arange(nz + 2)[None, None, :] * 2 * np.pi / nz
    u[..., 0] = np.sin(x) * np.cos(2 * y) * np.cos(z) + 0.3 * rng.standard_normal((nx + 2, ny + 2, nz + 2))
    u[..., 1] = np.cos(3 * x) * np.sin(y) + 0.3 * rng.standard_normal((nx + 2, ny + 2, nz + 2))
    u[..., 2] = np.sin(2 * z + x) + 0.3 * rng.standard_normal((nx + 2, ny + 2, nz + 2))
    for c in range(3):
        u[..., c] = periodic_fill(u[..., c].copy())
    return np.asfortranarray(u)


@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 12, 10), (32, 32, 32)])
def test_smagorinsky(gpu_lib, dims):
    nx, ny, nz = dims
    cfg = dict(nx=nx, ny=ny, nz=nz, xl=1.0, yl=1.3, zl=0.7, c_smag=0.0289)
    g, o = SamGpu(**cfg), O.Oracle(**cfg)
    u = velocity(nx, ny, nz, 1)
    vt_o, vt_g = o.sm(u), g.sm(u)
    assert relerr(vt_g, vt_o) < 1e-13


@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 12, 10), (32, 32, 32)])
def test_dynamic_smagorinsky(gpu_lib, dims):
    nx, ny, nz = dims
    cfg = dict(nx=nx, ny=ny, nz=nz, xl=1.0, yl=1.3, zl=0.7)
    g, o = SamGpu(**cfg), O.Oracle(**cfg)
    u = velocity(nx, ny, nz, 2)
    vt_o, c_o = o.dm(u)
    vt_g, c_g = g.dm(u)
    assert abs(c_g - c_o) <= 1e-12 * abs(c_o)
    assert relerr(vt_g, vt_o) < 1e-12


@pytest.mark.parametrize("dims", [(8, 5, 3), (40, 9, 15), (64, 16, 2)])
def test_dynamic_coefficient_of_scaled_and_local_fields(gpu_lib, dims):
    """The test filter runs on integers under a power of two per tile (32 x 8 x
    2 points) and in FP64 where a tile has none to offer.  Powers of two leave
    every rounding of both where it is, so the coefficient does not change by
    a bit; a field that is zero but for one corner, and tiles cut by the box,
    against the oracle at the per-routine bar; NaN stays NaN."""
    nx, ny, nz = dims
    cfg = dict(nx=nx, ny=ny, nz=nz, xl=1.0, yl=1.3, zl=0.7)
    g, o = SamGpu(**cfg), O.Oracle(**cfg)
    u = velocity(nx, ny, nz, 2)
    c = g.dm(u)[1]
    assert abs(c - o.dm(u)[1]) <= 1e-12 * abs(c)
    for k in (-60, -1, 7, 60):
        assert g.dm(u * 2.0 ** k)[1] == c, k
    for tiny in (0.0, 1e-300):  # below 2^-959 the sums are taken in FP64
        v = u * tiny
        v[1:4, 1:4, 1:3] = u[1:4, 1:4, 1:3]
        for n in range(3):
            v[..., n] = periodic_fill(v[..., n].copy())
        cv, co = g.dm(v)[1], o.dm(v)[1]
        assert abs(cv - co) <= 1e-12 * abs(co), tiny
    w = u.copy(order="F")
    w[2, 2, 2, 1] = np.nan
    assert np.isnan(g.dm(w)[1])


@pytest.mark.parametrize("i_remove", [0, 1])
def test_get_mean(gpu_lib, i_remove):
    cfg = dict(nx=16, ny=12, nz=40, i_strat=1, buoy_fac_z=1.0, lapse=1.0)
    g, o = SamGpu(**cfg), O.Oracle(**cfg)
    u = o.init_random(8)
    # a mean temperature profile with a jump-like slope in the kx = ky = 0 column
    u[1:6, 0, 0, 3] += np.array([0.3 - 0.2j, 0.1 + 0.05j, -0.04j, 0.02, 0.01j])
    fo = np.asfortranarray(u[..., 3].copy())
    fg = np.asfortranarray(u[..., 3].copy())
    um_o, j_o = o.get_mean(fo, i_remove)
    um_g, j_g = g.get_mean(fg, i_remove)
    assert relerr(um_g[: 40], um_o[: 40]) < 1e-13
    # the jump is a difference of extrapolated profile values: compare it on
    # the scale of the profile, not of itself
    assert abs(j_g - j_o) <= 1e-13 * np.abs(um_o).max()
    assert relerr(fg[: o.d.nz_min, 0, 0], fo[: o.d.nz_min, 0, 0]) < 1e-13


LES_CASES = [(1, 0), (1, 1), (2, 0), (2, 1)]


@pytest.mark.parametrize("model,strat", LES_CASES)
def test_coupled_closure_matches_oracle(gpu_lib, model, strat):
    """Smagorinsky (model 1) and dynamic Smagorinsky (model 2) coupled into
    the RK3 step: the GPU run against the oracle's restatement, several CFL
    steps, per field to 1e-12; the coefficient in use agrees too."""
    cfg = dict(nx=24, ny=16, nz=32, i_strat=strat, buoy_fac_z=1.0 * strat, lapse=1.0 * strat, vis=1e-4,
               i_cfl=1, cfl0=0.5)
    g, o = SamGpu(**cfg), O.Oracle(**cfg)
    u = o.init_random(7, 0, 1.0, 0, 0.1)
    r = o.wave(o.d.lr)
    g.upload(u)
    g.set_les(model, c_smag=0.03, pr_t=0.7)
    o.set_les(model, c_smag=0.03, pr_t=0.7)
    o.steps(u, r, 4)
    g.step(4)
    ug = g.download()
    for n in range(o.d.lu):
        assert relerr(ug[..., n], u[..., n]) <= 1e-12, n
    assert abs(g.les_coef() - o.les_coef()) <= 1e-12 * abs(o.les_coef())
    assert o.les_coef() > 0


def test_coupled_closure_stages_and_fp32(gpu_lib):
    """Single stages (sam_gpu_stage) with the dynamic closure, then the FP32
    bulk form of the same run within its tolerance."""
    cfg = dict(nx=32, ny=32, nz=32, i_strat=1, buoy_fac_z=1.0, lapse=1.0, vis=1e-4, dt0=0.01)
    g, o = SamGpu(**cfg), O.Oracle(**cfg)
    u = o.init_random(2, 0, 1.0, 0, 0.1)
    u0 = u.copy(order="F")
    r = o.wave(o.d.lr)
    g.upload(u)
    g.set_les(2, pr_t=1.0)
    o.set_les(2, pr_t=1.0)
    for nrk in (1, 2, 3):
        o.stage(u, r, nrk)
        g.stage(nrk)
        ug, rg = g.download(with_r=True)
        m = o.d.nz_min  # rows above Nz_min of r are unspecified (z_trans_f.f)
        for n in range(o.d.lu):
            assert relerr(ug[:m, ..., n], u[:m, ..., n]) <= 1e-12, (nrk, n)
            assert relerr(rg[:m, ..., n], r[:m, ..., n]) <= 1e-12, (nrk, n)
    g32 = SamGpu(precision=32, **cfg)
    g32.upload(u0)
    g32.set_les(2, pr_t=1.0)
    g32.step(1)
    u32 = g32.download()
    for n in range(o.d.lu):
        assert relerr(u32[..., n], u[..., n]) <= 2e-5, n


@pytest.mark.parametrize("precision,model", [(64, 1), (64, 2), (32, 1), (32, 3)])
@pytest.mark.parametrize("strat,ny", [(1, 8), (1, 9), (0, 2), (0, 10)])
def test_closure_on_256_point_lines(gpu_lib, precision, model, strat, ny):
    """The fused x passes of 256-point lines with a closure (tiles of 4 rows:
    whole, with one or two rows left, both numbers of products) against
    the general kernel, which the Stockham schedule takes.  Both add the same
    terms to the same products; they differ by the rounding of two transforms
    of 256 points (log2 n + 2 roundings each way at most, all fields of one
    size), so one stage agrees to 64 roundings of the largest value; the three
    stages of a step to 256.  The learned closure's network is all zeros here:
    its coefficient is then the same at every point for both kernels."""
    cfg = dict(nx=256, ny=ny, nz=8, i_strat=strat, buoy_fac_z=1.0 * strat, lapse=1.0 * strat, vis=1e-4, i_cfl=1, cfl0=0.5)
    eps = 2.0 ** -53 if precision == 64 else 2.0 ** -24
    u0 = O.Oracle(**cfg).init_random(7, 0, 1.0, 0, 0.1)
    out = []
    for sched in (0, 1):
        g = SamGpu(precision=precision, **cfg)
        g.upload(u0)
        if model == 3:
            g.mlp_set(np.zeros(CL.N_PARAMS, np.float32))
        g.set_les(model, c_smag=0.03, pr_t=0.7)
        g.set_fft_schedule([0, 0, sched, 0, 0])
        g.stage(1)
        a = g.download()
        g.stage(2)
        g.stage(3)
        out.append((a, g.download(), g.stats()["dt"]))
        g.close()
    (a, b, dt), (ar, br, dtr) = out
    for n in range(4 if strat else 3):
        assert relerr(a[..., n], ar[..., n]) <= 64 * eps, n
        assert relerr(b[..., n], br[..., n]) <= 256 * eps, n
    assert abs(dt - dtr) <= 64 * eps * dtr


def test_closure_off_restores_reference_products(gpu_lib):
    cfg = dict(nx=16, ny=16, nz=16, vis=1e-3)
    g = SamGpu(**cfg)
    g.init_taylor_green()
    u0 = g.download()
    g.set_les(1, c_smag=0.05)
    g.step(1)
    assert g.les_coef() > 0
    g.set_les(0)
    g.upload(u0)
    g.step(2)
    g2 = SamGpu(**cfg)
    g2.upload(u0)
    g2.step(2)
    assert np.array_equal(g.download(), g2.download())
    with pytest.raises(Exception, match="EINVAL"):
        g.set_les(4)
