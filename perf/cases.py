"""The measured cases: what a user of this library has it do, through its
public entry points, and what one pass of each takes.

A pass of a resident run is what a driver does between two output times:
set_tstep, upload of the wave-space state from pinned host memory, a number of
RK3 steps, download.  The library holds one context per process (as sam.f's
COMMON blocks do), so the states of one case share the solver; it is kept
between the states of that case and rebuilt when another case runs.

Single-precision runs return their state in single precision (on the GPU,
where a post-processing program would take it up): the state carries no more.
"""
import ctypes
import math
import os

import numpy as np
import torch

import sam_gb300
from sam_gb300 import SamGpu
from sam_gb300.sam_gpu import SamEnsemble, load_library

MLP_FILE = os.path.join(os.path.dirname(sam_gb300.__file__), "data", "closure_mlp.npz")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # Taylor-Green vortex at 64^3, FP64, no stratification: the smallest
        # validation run, launch- and latency-bound
        dict(name="tg_64_fp64", kind="run", nx=64, ny=64, nz=64, precision=64, strat=False, init="tg", cfl=False, steps=10),
        # stratified decaying turbulence at 128^3, FP64 drop-in form, with the
        # shell spectra a driver writes at each output time
        dict(name="strat_128_fp64", kind="run", nx=128, ny=128, nz=128, precision=64, strat=True, init="random", cfl=True,
             steps=10, spectra=True),
        # gravity-wave packet at 256^3, FP64: the headline workload
        dict(name="packet_256_fp64", kind="run", nx=256, ny=256, nz=256, precision=64, strat=True, init="packet", cfl=True,
             steps=4),
        # lengths with factors 3 and 5 and odd lengths: boxes fitted to a
        # domain's aspect ratio rather than to a power of two
        dict(name="ragged_fp64", kind="run", nx=120, ny=135, nz=162, precision=64, strat=True, init="random", cfl=True,
             steps=4),
        # the FP32 bulk form of the headline workload, and an ordinary 128^3 run
        dict(name="packet_256_fp32", kind="run", nx=256, ny=256, nz=256, precision=32, strat=True, init="packet", cfl=True,
             steps=20),
        dict(name="strat_128_fp32", kind="run", nx=128, ny=128, nz=128, precision=32, strat=True, init="random", cfl=True,
             steps=40),
        # the double-float form of the headline workload
        dict(name="packet_256_dd", kind="run", nx=256, ny=256, nz=256, precision=48, strat=True, init="packet", cfl=True,
             steps=8),
        # large-eddy simulation at 256^3: dm.f's dynamic coefficient in FP64,
        # the learned closure in FP32
        dict(name="les_dynamic_256_fp64", kind="run", nx=256, ny=256, nz=256, precision=64, strat=True, init="random",
             cfl=True, steps=2, les=2),
        dict(name="les_learned_256_fp32", kind="run", nx=256, ny=256, nz=256, precision=32, strat=True, init="random",
             cfl=True, steps=8, les=3),
        # sam.f's stage loop with the per-routine drop-ins on its own host arrays
        dict(name="dropin_stage_96", kind="dropin", nx=96, ny=80, nz=72, precision=64, strat=True, init="random", cfl=True),
        # an ensemble of uneven members (FP32, learned closure on the larger ones)
        dict(name="ensemble", kind="ensemble", n32=8, n64=8, n96=4, n128=1, steps=8),
        # training the closure on minibatches of 8192 points
        dict(name="closure_train", kind="train", samples=65536, steps=16, batch=8192),
    ]


def smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


SIZES = [n for n in range(24, 257) if smooth(n)]


def draw(rng):
    """One more case of the same ranges: grids of 24 to 256 points a side
    (even in x, factors 2, 3 and 5), every precision form, the closures."""
    def side(n, even=False):
        lo, hi = n / 1.4, min(256.0, n * 1.4)
        return rng.choice([m for m in SIZES if lo <= m <= hi and not (even and m % 2)])

    kind = rng.choices(["fp64", "fp32", "dd", "dyn", "learned", "dropin", "ensemble", "train"],
                       [6, 4, 2, 2, 2, 2, 1, 1])[0]
    if kind == "train":
        return dict(kind="train", samples=int(2 ** rng.uniform(13, 17)), steps=rng.randint(2, 24),
                    batch=rng.choice([1000, 2048, 4096, 8192]))
    if kind == "ensemble":
        return dict(kind="ensemble", n32=rng.randint(1, 12), n64=rng.randint(0, 8), n96=rng.randint(0, 3),
                    n128=rng.randint(0, 1), steps=rng.randint(2, 8))
    top = {"dropin": 128, "dyn": 192, "learned": 256}.get(kind, 256)
    n = math.exp(rng.uniform(math.log(32), math.log(top)))
    c = dict(kind="run", nx=side(n, even=True), ny=side(n), nz=side(n), precision={"fp32": 32, "learned": 32, "dd": 48}.get(kind, 64),
             strat=rng.random() < 0.8, init=rng.choice(["random", "packet"]), cfl=True, steps=rng.randint(1, 4))
    if kind == "dropin":
        c["kind"] = "dropin"
        del c["steps"]
    elif kind in ("dyn", "learned"):
        c["les"] = 2 if kind == "dyn" else 3
        c["strat"] = True
        c["steps"] = min(c["steps"], 2)
    return c


# ---------------------------------------------------------------- the physics
def config(case):
    """The library's configuration of a case (box [0, 2 pi]^3)."""
    packet = case["init"] == "packet"
    n_bv = 2.0 if packet else 1.0
    vis = 1e-4 if packet or case.get("les") else (1 / 400 if case["init"] == "tg" else 1 / 800)
    cfg = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], i_strat=int(case["strat"]), i_cfl=int(case["cfl"]), cfl0=0.5,
               vis=vis, pr=1.0, dt0=0.01 if case["init"] == "tg" else 1e-3, precision=case["precision"])
    if case["strat"]:
        cfg.update(buoy_fac_z=n_bv * n_bv, lapse=1.0)
    return cfg


def members(case):
    """The configurations of the ensemble's members, each with its own
    stratification and viscosity; the closure on 96^3 and 128^3."""
    out = []
    for n, key in ((32, "n32"), (64, "n64"), (96, "n96"), (128, "n128")):
        for m in range(case[key]):
            out.append(dict(kind="run", nx=n, ny=n, nz=n, precision=32, strat=True, init="random", cfl=True,
                            steps=case["steps"], les=3 if n >= 96 else 0, n_bv=0.5 + 3.5 * ((m * 7 + n) % 11) / 10))
    return out


def member_config(c):
    cfg = config(c)
    cfg.update(buoy_fac_z=c["n_bv"] ** 2, vis=0.08 / c["nx"])
    return cfg


def dims(case):
    kx, ky, kz = (int((n - 0.1) / 3.0) for n in (case["nx"], case["ny"], case["nz"]))
    return kx, ky, kz, kx + 1, 2 * ky + 1, 2 * kz + 1, (4 if case["strat"] else 3), (9 if case["strat"] else 6)


def waves(k, device):
    """Signed wave numbers of 2 k + 1 stored modes: 0 .. k, -k .. -1."""
    return torch.cat([torch.arange(0, k + 1), torch.arange(-k, 0)]).to(device=device, dtype=torch.float64)


def wave_numbers(case, device="cuda"):
    kx, ky, kz = dims(case)[:3]
    return (torch.arange(0, kx + 1, device=device, dtype=torch.float64)[:, None, None], waves(ky, device)[None, :, None],
            waves(kz, device)[None, None, :])


def take(f, k, dim):
    """The 2 k + 1 stored modes of a full transform along dim."""
    n = f.shape[dim]
    return torch.cat([f.narrow(dim, 0, k + 1), f.narrow(dim, n - k, k)], dim)


def to_wave(phys, case):
    """Physical fields [n, x, y, z] to the stored modes [n, kx, ky, kz], scaled by 1 / (Nx Ny Nz)."""
    kx, ky, kz = dims(case)[:3]
    f = torch.fft.rfft(phys, dim=1, norm="forward").narrow(1, 0, kx + 1)
    f = take(torch.fft.fft(f, dim=2, norm="forward"), ky, 2)
    return take(torch.fft.fft(f, dim=3, norm="forward"), kz, 3)


def put(f, k, n, dim):
    shape = list(f.shape)
    shape[dim] = n - 2 * k - 1
    return torch.cat([f.narrow(dim, 0, k + 1), torch.zeros(shape, dtype=f.dtype, device=f.device), f.narrow(dim, k + 1, k)],
                     dim)


def to_phys(wave, case):
    """The stored modes to physical fields (unscaled); kx = 0 keeps its real part."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kx, ky, kz = dims(case)[:3]
    f = torch.fft.ifft(put(wave, kz, nz, 3), dim=3, norm="forward")
    f = torch.fft.ifft(put(f, ky, ny, 2), dim=2, norm="forward")
    f[:, 0] = f[:, 0].real.to(f.dtype)
    return torch.fft.irfft(f, n=nx, dim=1, norm="forward")


def project(u, case):
    """The solenoidal part of the first three fields."""
    k = wave_numbers(case)
    k_sq = (k[0] ** 2 + k[1] ** 2 + k[2] ** 2).clamp_min(1e-10)
    div = (k[0] * u[0] + k[1] * u[1] + k[2] * u[2]) / k_sq
    for n in range(3):
        u[n] -= k[n] * div
    return u


def start(case, seed):
    """The initial modes [n, kx, ky, kz] of a run, on the GPU, from the seed:
    a random solenoidal field with E(k) ~ k^4 exp(-2 (k/4)^2) at rms 1 (T at a
    tenth of it), a Gaussian-enveloped wave k = (8, 0, 16) of amplitude 0.05
    with 1 % noise, or the Taylor-Green vortex with 1 % noise."""
    kx, ky, kz, mx, my, mz, lu, lr = dims(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + nx * 10007 + ny * 101 + nz)
    noise = torch.randn((lu, nx, ny, nz), generator=g, device="cuda", dtype=torch.float64)
    x, y, z = (torch.arange(n, device="cuda", dtype=torch.float64) * (2 * math.pi / n) for n in (nx, ny, nz))
    if case["init"] == "random":
        u = to_wave(noise, case)
        del noise
        k = wave_numbers(case)
        k_sq = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
        u *= k_sq * torch.exp(-k_sq / 16)
        u = project(u, case)
        w = torch.full((mx, 1, 1), 2.0, device="cuda", dtype=torch.float64)
        w[0] = 1.0
        rms = torch.stack([(w * (u[n].real ** 2 + u[n].imag ** 2)).sum() for n in range(lu)])
        u[:3] /= torch.sqrt(rms[:3].sum() / 3)
        if lu == 4:
            u[3] *= 0.1 / torch.sqrt(rms[3])
        return u
    if case["init"] == "tg":
        phys = 0.01 * noise
        phys[0] += torch.sin(x)[:, None, None] * torch.cos(y)[None, :, None] * torch.cos(z)[None, None, :]
        phys[1] -= torch.cos(x)[:, None, None] * torch.sin(y)[None, :, None] * torch.cos(z)[None, None, :]
    else:
        phys = 5e-4 * noise
        k1, k3 = min(8, kx), min(16, kz)
        s = math.pi / 4
        env = (torch.exp(-((x - math.pi) / s) ** 2 / 2)[:, None, None] * torch.exp(-((y - math.pi) / s) ** 2 / 2)[None, :, None] *
               torch.exp(-((z - math.pi) / s) ** 2 / 2)[None, None, :])
        arg = k1 * x[:, None, None] + k3 * z[None, None, :]
        phys[0] += 0.05 * env * torch.cos(arg)
        phys[2] -= 0.05 * env * torch.cos(arg) * (k1 / max(k3, 1))
        if lu == 4:
            phys[3] += 0.02 * env * torch.sin(arg)
    u = to_wave(phys, case)
    return project(u, case)


# ------------------------------------------------------------- states, passes
_kept = {"key": None, "solver": None}


def solver(case):
    """The process's solver for this case (one context per process)."""
    key = repr(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "spectra", "samples", "batch")))
    if _kept["key"] != key or SamGpu._live is not _kept["solver"]:
        _kept["key"] = _kept["solver"] = None
        if case["kind"] == "ensemble":
            mem = members(case)
            s = SamEnsemble([member_config(c) for c in mem])
            for c, m in zip(mem, s.members):
                if c["les"]:
                    m.mlp_set(np.load(MLP_FILE)["params"])
                    m.set_les(c["les"])
        elif case["kind"] == "train":
            s = SamGpu(nx=16, ny=16, nz=16, i_strat=1, precision=32)
        else:
            s = SamGpu(**config(case))
            if case.get("les") == 3:
                s.mlp_set(np.load(MLP_FILE)["params"])
            if case.get("les"):
                s.set_les(case["les"])
        _kept["key"], _kept["solver"] = key, s
    return _kept["solver"]


def host_wave(case, pinned=True):
    """A pinned host array in the reference's layout u(Nze, Ny_min, Nx_min, Lu):
    (the torch tensor [n, kx, ky, kz], its Fortran-ordered numpy view)."""
    kx, ky, kz, mx, my, mz, lu, lr = dims(case)
    t = torch.zeros((lu, mx, my, case["nz"]), dtype=torch.complex128, pin_memory=pinned)
    return t, t.numpy().transpose(3, 2, 1, 0)


def loaded(case, seed):
    t, a = host_wave(case)
    u = start(case, seed)
    full = torch.zeros(t.shape, dtype=t.dtype, device="cuda")
    full[..., :u.shape[3]] = u
    t.copy_(full)
    return {"in_t": t, "in": a}


def prepare(case, seed):
    s = {"case": dict(case)}
    if case["kind"] == "run":
        s.update(loaded(case, seed))
        s["out_t"], s["out"] = host_wave(case)
        solver(case)
    elif case["kind"] == "ensemble":
        s["members"] = []
        for i, c in enumerate(members(case)):
            m = {"case": c, **loaded(c, seed * 1000 + i)}
            m["out_t"], m["out"] = host_wave(c)
            s["members"].append(m)
        solver(case)
    elif case["kind"] == "dropin":
        kx, ky, kz, mx, my, mz, lu, lr = dims(case)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        t, _ = host_wave(case, pinned=False)
        t[..., :mz] = start(case, seed).cpu()
        s["u"] = t.numpy()
        s["blocks"] = np.zeros((lu, nz, mx, my), dtype=np.complex128)
        s["uu"] = np.zeros((lu, nz, ny, nx))  # sam.f's uu: planes of modes, then the physical fields
        s["r"] = np.zeros((lr + 1, mx, my, nz), dtype=np.complex128)
        s["u_sav"] = np.ascontiguousarray(t.numpy()[2:4, ..., :mz])
        s["isymm"] = np.zeros(lu, dtype=np.int32)
        solver(case)
    else:
        s["features"], s["target"], s["params"] = training_data(case, seed)
        solver(case)
    return s


def single(t):
    return t.to("cuda").to(torch.complex64)


def run_resident(g, case, s):
    cfg = config(case)
    g.set_tstep(1, cfg["dt0"], 0.0)
    g.upload(s["in"])
    g.step(case["steps"])
    g.download(out=s["out"])
    st = g.stats()
    out = {"u": s["out_t"], "time": st["time"], "dt": st["dt"], "energy": st["energy"], "u_max": st["u_max"]}
    if case.get("spectra"):
        out["ek"] = g.spectra()["ek"]
    if case["precision"] == 32:
        out["u"] = single(s["out_t"])
        for k in ("time", "dt", "energy", "u_max"):
            out[k] = np.asarray(out[k], dtype=np.float32)
    return out


def run(state):
    case = state["case"]
    g = solver(case)
    if case["kind"] == "run":
        return run_resident(g, case, state)
    if case["kind"] == "ensemble":
        for m, s in zip(g.members, state["members"]):
            m.set_tstep(1, 1e-3, 0.0)
            m.upload(s["in"])
        g.step(case["steps"])
        out = []
        for m, s in zip(g.members, state["members"]):
            m.download(out=s["out"])
            out.append(single(s["out_t"]))
        return out
    if case["kind"] == "dropin":
        lib = load_library()
        lu = len(state["u"])

        def p(a):
            return a.ctypes.data_as(ctypes.c_void_p)

        def ck(rc):
            if rc != 0:
                raise RuntimeError(lib.sam_gpu_error_string().decode())

        u, blocks, uu, r = (p(state[k]) for k in ("u", "blocks", "uu", "r"))
        sym = p(state["isymm"])
        ck(lib.sam_gpu_set_tstep(1, 1e-3, 0.0))
        ck(lib.sam_gpu_z_trans_b(u, blocks, lu, sym, None, None, None))
        ck(lib.sam_gpu_x2z_decomp(blocks, uu, lu, uu))
        ck(lib.sam_gpu_xy_trans_b(uu, uu, lu, None))
        ck(lib.sam_gpu_rhs(uu, uu, r, p(state["u_sav"]) if case["strat"] else None, None))
        st = g.stats()
        return {"phys": state["uu"], "r": state["r"], "dt": st["dt"], "u_max": st["u_max"]}
    g.mlp_set(state["params"])
    hist = g.mlp_train(state["features"], state["target"], case["steps"], batch=case["batch"])
    return {"loss": hist, "params": g.mlp_get(), "coef": g.mlp_forward(state["features"])}


def work(case):
    """One pass's algorithmic bytes (each pass's pencils read and written once,
    the copies of the state to and from the host) and operations (5 n log2 n a
    complex line of the pruned line sets; the network's products)."""
    if case["kind"] == "ensemble":
        parts = [work(c) for c in members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if case["kind"] == "train":
        n = min(case["batch"], case["samples"]) * case["steps"]
        per = 12 * 64 + 64 * 64 + 64 * 2
        return {"bytes": case["samples"] * (12 * 4 + 2 * 4 + 2 * 4), "flops": 2.0 * per * (3 * n + case["samples"])}
    kx, ky, kz, mx, my, mz, lu, lr = dims(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nin = lu + (lr if case.get("les") else 0)
    es = 8 if case["precision"] == 32 else 16
    line = {n: 5 * n * math.log2(n) for n in (nx, ny, nz)}
    a, b, c, d, w = mx * my * nz, mx * ny * nz, mx * ny * nz, mx * my * nz, mx * my * mz
    one_b = es * (lu * w + 2 * nin * a + 2 * nin * b + 2 * lr * c + 2 * lr * d + (4 * lu + 1) * w)
    one_f = (nin + lr) * (mx * my * line[nz] + mx * nz * line[ny] + ny * nz * line[nx] / 2)
    if case["kind"] == "dropin":
        return {"bytes": 16.0 * (lu * w + lr * c + 2 * lr * d + (lu + 1) * w) + 16.0 * lu * nx * ny * nz, "flops": one_f}
    n, extra = case["steps"], 0.0
    if case.get("les") == 3:  # the network, once a step
        extra = 2.0 * (12 * 64 + 64 * 64 + 64 * 2) * nx * ny * nz * n
    if case.get("les") == 2:  # the test filters of dm.f, once a step
        extra = 21.0 * 12 * nx * ny * nz * n
    return {"bytes": 3.0 * n * one_b + 2 * 16.0 * lu * w, "flops": 3.0 * n * one_f + extra}


# ------------------------------------------- the same results in 64 bits, torch
def derivatives(u, case, vorticity):
    """Physical strain (S11 S12 S22 S13 S23 S33), temperature gradient and vorticity."""
    k = wave_numbers(case)
    pairs = [(0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2)]
    f = [0.5j * (k[b] * u[a] + k[a] * u[b]) for a, b in pairs] + [1j * k[a] * u[3] for a in range(3)]
    if vorticity:
        f += [1j * (k[(a + 1) % 3] * u[(a + 2) % 3] - k[(a + 2) % 3] * u[(a + 1) % 3]) for a in range(3)]
    p = torch.cat([to_phys(q[None], case) for q in f])
    return p[:6], p[6:9], p[9:]


def strain_norm(s):
    return torch.sqrt(2 * (s[0] ** 2 + s[2] ** 2 + s[5] ** 2 + 2 * (s[1] ** 2 + s[3] ** 2 + s[4] ** 2)))


def dynamic_coefficient(u, case):
    """dm.f's volume-averaged C delta^2 of the physical velocity, clipped at 0."""
    h = [2 * math.pi / n for n in (case["nx"], case["ny"], case["nz"])]
    ub = [0.5 * (u[c] + torch.roll(u[c], 1, c)) for c in range(3)]

    def diff(f, c):
        return (torch.roll(f, -1, c) - torch.roll(f, 1, c)) / h[c]

    def filt(f):
        for c in (2, 1, 0):
            f = (torch.roll(f, -1, c) + 4 * f + torch.roll(f, 1, c)) / 6
        return f

    ip, jp, fact = (0, 1, 2, 0, 1, 0), (0, 1, 2, 1, 2, 2), (1, 1, 1, 2, 2, 2)
    s = [0.25 * (diff(ub[i], j) + diff(ub[j], i)) if i != j else 0.5 * diff(ub[i], i) for i, j in zip(ip, jp)]
    mag = torch.sqrt(2 * sum(w * q * q for w, q in zip(fact, s)))
    sh = [filt(q) for q in s]
    mag_h = torch.sqrt(2 * sum(w * q * q for w, q in zip(fact, sh)))
    uh = [filt(q) for q in ub]
    num = den = 0.0
    for c in range(6):
        m = -filt(mag * s[c]) + 4 * mag_h * sh[c]
        lij = filt(ub[ip[c]] * ub[jp[c]]) - uh[ip[c]] * uh[jp[c]]
        num = num + fact[c] * float((lij * m).sum())
        den = den + fact[c] * float((m * m).sum())
    v = -0.5 * num / den
    return v if v > 0 else 0.0


def bf(x):
    return x.to(torch.bfloat16).to(torch.float64)


def network(p, x):
    """The closure's network with its BF16 weights and activations: (C, h1, h2, o)."""
    w1, b1, w2, b2, w3, b3 = torch.split(p, [768, 64, 4096, 64, 128, 2])
    h1 = bf(torch.relu(x @ bf(w1.view(64, 12)).T + b1))
    h2 = bf(torch.relu(h1 @ bf(w2.view(64, 64)).T + b2))
    o = h2 @ bf(w3.view(2, 64)).T + b3
    return 0.02 * torch.nn.functional.softplus(o), h1, h2, o


def learned_coefficients(u, case, cfg, dsq):
    s, g, w = derivatives(u, case, True)
    eps, bz = 1e-30, cfg["buoy_fac_z"]
    n2, nu = bz * cfg["lapse"], max(cfg["vis"], 1e-12)
    m = [[s[0], s[1], s[3]], [s[1], s[2], s[4]], [s[3], s[4], s[5]]]
    s2 = strain_norm(s) ** 2
    sn = torch.sqrt(s2)
    tr3 = sum(m[i][k] * m[k][j] * m[j][i] for i in range(3) for j in range(3) for k in range(3))
    wsw = sum(w[i] * m[i][j] * w[j] for i in range(3) for j in range(3))
    gsg = sum(g[i] * m[i][j] * g[j] for i in range(3) for j in range(3))
    w2, g2 = (w * w).sum(0), (g * g).sum(0)
    wn, gn, inv = torch.sqrt(w2), torch.sqrt(g2), 1 / (s2 + eps)
    f = [torch.log1p(w2 * inv), tr3 / (s2 * sn + eps), wsw / (sn * w2 + eps), torch.log1p(abs(n2) * inv),
         torch.asinh(bz * g[2] * inv), torch.log1p(abs(bz) * torch.sqrt(g[0] ** 2 + g[1] ** 2) * inv), s[5] / (sn + eps),
         w[2] / (sn + wn + eps), gsg / (sn * g2 + eps), (w * g).sum(0) / (wn * gn + eps), torch.log1p(sn * dsq / nu),
         4 * (s[3] ** 2 + s[4] ** 2) * inv]
    x = bf(torch.stack(f, -1).reshape(-1, 12))
    del f, s, g, w
    p = torch.from_numpy(np.load(MLP_FILE)["params"].astype(np.float64)).cuda()
    c = torch.cat([network(p, q)[0] for q in torch.split(x, 1 << 21)])
    return c.reshape(case["nx"], case["ny"], case["nz"], 2)


def rhs64(u, case, cfg, cds, coef, dsq):
    """The projected right-hand side and the physical velocity (rhs.f)."""
    phys = to_phys(u, case)
    k = wave_numbers(case)
    pairs = [(0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2)] + ([(0, 3), (1, 3), (2, 3)] if case["strat"] else [])
    sub = None
    if case.get("les"):
        s, g, _ = derivatives(u, case, False)
        mag = strain_norm(s)
        nu, kap = (cds * mag, cds * mag) if coef is None else (coef[..., 0] * dsq * mag, coef[..., 1] * dsq * mag)
        sub = [-2 * nu * q for q in s] + [-kap * q for q in g]
    t = []
    for m, (a, b) in enumerate(pairs):
        q = phys[a] * phys[b]
        if sub is not None:
            q = q + sub[m]
        t.append(to_wave(q[None], case)[0])
    r = [-1j * (k[0] * t[a] + k[1] * t[b] + k[2] * t[c]) for a, b, c in ((0, 1, 3), (1, 2, 4), (3, 4, 5))]
    if case["strat"]:
        r[2] = r[2] + cfg["buoy_fac_z"] * u[3]
        r.append(-1j * (k[0] * t[6] + k[1] * t[7] + k[2] * t[8]) - cfg["lapse"] * u[2])
    k_sq = (k[0] ** 2 + k[1] ** 2 + k[2] ** 2).clamp_min(1e-10)
    pr = -1j * (k[0] * r[0] + k[1] * r[1] + k[2] * r[2]) / k_sq
    for n in range(3):
        r[n] = r[n] - 1j * k[n] * pr
    return torch.stack(r), pr, phys


def steps64(case, cfg, u):
    """The run's steps in 64 bits: (u, statistics of the last step)."""
    kx, ky, kz = dims(case)[:3]
    k = wave_numbers(case)
    k_sq = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    gamma, zeta = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)
    dsq = (2 * math.pi) ** 2 / (case["nx"] * case["ny"] * case["nz"]) ** (2 / 3)
    dt, time, r = cfg["dt0"], 0.0, None
    cds, coef, st = 0.0, None, {}
    for _ in range(case["steps"]):
        for n in range(3):
            if n == 0 and case.get("les") == 2:
                cds = dynamic_coefficient(to_phys(u[:3], case), case)
            if n == 0 and case.get("les") == 3:
                coef = learned_coefficients(u, case, cfg, dsq)
            new, _, phys = rhs64(u, case, cfg, cds, coef, dsq)
            if n == 0:
                u_max = phys.abs().amax((1, 2, 3))
                if case["cfl"]:
                    dt = cfg["cfl0"] * math.sqrt(3.0) / float(max(u_max[0] * kx, u_max[1] * ky, u_max[2] * kz))
                var = (phys ** 2).mean((1, 2, 3)) - phys.mean((1, 2, 3)) ** 2
                st = {"u_max": u_max, "energy": 0.5 * float(var[:3].sum())}
            del phys
            if n > 0:
                u = u + zeta[n] * dt * r
            u = (u + gamma[n] * dt * new) * torch.exp(-cfg["vis"] * (gamma[n] + zeta[n]) * dt * k_sq)
            r = new
        time += dt
    um = np.zeros(4)
    um[:len(st["u_max"])] = st["u_max"].cpu().numpy()
    return u, {"time": time, "dt": dt, "energy": st["energy"], "u_max": um}


def padded(u, case):
    full = torch.zeros(u.shape[:3] + (case["nz"],), dtype=u.dtype, device=u.device)
    full[..., :u.shape[3]] = u
    return full


def exact(case, seed):
    if case["kind"] == "train":
        return train64(case, seed)
    if case["kind"] == "ensemble":
        return [padded(steps64(c, member_config(c), start(c, seed * 1000 + i))[0], c) for i, c in enumerate(members(case))]
    cfg = config(case)
    u = start(case, seed)
    if case["kind"] == "dropin":
        kx, ky, kz, mx, my, mz, lu, lr = dims(case)
        r, p, phys = rhs64(u, case, cfg, 0.0, None, 0.0)
        out = torch.zeros((lr + 1, mx, my, case["nz"]), dtype=torch.complex128, device="cuda")
        out[:lu, ..., :mz] = r
        out[lu, ..., :mz] = p
        u_max = phys.abs().amax((1, 2, 3))
        um = np.zeros(4)
        um[:lu] = u_max.cpu().numpy()
        dt = 0.5 * math.sqrt(3.0) / float(max(u_max[0] * kx, u_max[1] * ky, u_max[2] * kz))
        return {"phys": phys.permute(0, 3, 2, 1).cpu().numpy(), "r": out, "dt": dt, "u_max": um}
    u, st = steps64(case, cfg, u)
    out = {"u": padded(u, case), **st}
    if case.get("spectra"):
        k = wave_numbers(case)
        shell = (torch.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2) + 0.5).to(torch.int64)
        e = (u[:3].real ** 2 + u[:3].imag ** 2).sum(0)
        e[1:] *= 2
        kx, ky, kz = dims(case)[:3]
        ek = torch.zeros(int(math.sqrt(kx * kx + ky * ky + kz * kz) + 0.5) + 1, dtype=torch.float64, device="cuda")
        ek.index_add_(0, shell.reshape(-1), e.reshape(-1))
        out["ek"] = ek.cpu().numpy()
    return out


# ------------------------------------------------------------ closure training
def training_data(case, seed):
    """Invariants of the closure's range, smooth targets with scatter, and He-style initial weights."""
    rng = np.random.default_rng(seed)
    n = case["samples"]
    x = rng.standard_normal((n, 12)).astype(np.float32)
    x[:, [0, 3, 5, 10]] = np.abs(x[:, [0, 3, 5, 10]]) * 1.5  # the logarithms are non-negative
    y = np.stack([0.02 + 0.01 * np.tanh(x[:, 0] - x[:, 3]), 0.02 + 0.01 * np.tanh(x[:, 1] + 0.5 * x[:, 10])], 1)
    y = (y + 0.003 * rng.standard_normal((n, 2))).astype(np.float32)
    p = np.zeros(5122, dtype=np.float32)
    p[:768] = rng.standard_normal(768) * math.sqrt(2 / 12)
    p[832:4928] = rng.standard_normal(4096) * math.sqrt(2 / 64)
    p[4992:5120] = rng.standard_normal(128) * 0.1 / 8
    return x, y, p


def train64(case, seed):
    x, y, p = (torch.from_numpy(a).cuda().to(torch.float64) for a in training_data(case, seed))
    x = bf(x)
    n = min(case["batch"], case["samples"])
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), []
    for s in range(case["steps"]):
        at = (s % (case["samples"] // n)) * n
        xs, ys = x[at:at + n], y[at:at + n]
        c, h1, h2, o = network(p, xs)
        e = c - ys
        loss.append(0.5 * float((e * e).sum()) / n)
        w2, w3 = bf(p[832:4928].view(64, 64)), bf(p[4992:5120].view(2, 64))
        do = e / n * 0.02 * torch.sigmoid(o)
        d2 = (do @ w3) * (h2 > 0)
        d1 = (d2 @ w2) * (h1 > 0)
        g = torch.cat([(d1.T @ xs).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), (do.T @ h2).reshape(-1), do.sum(0)])
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * math.sqrt(1 - 0.999 ** (s + 1)) / (1 - 0.9 ** (s + 1)) * m / (torch.sqrt(v) + 1e-8)
    return {"loss": np.array(loss), "params": p, "coef": network(p, x)[0]}
