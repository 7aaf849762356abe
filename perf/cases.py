"""The work a user of this package has it do, as cases that can be timed: single RK3 steps of channels of
every kind and size through GpuChannel / GpuBatch, the batched plane transforms, the statistics, and a
step whose state lives in host memory. Inputs are seeded velocity fields with the full decaying spectrum
of a developed flow (divergence-free, laminar mean), made on the GPU."""
import functools
import math

import numpy as np
import torch

from rnl_multiblock_nofft_gb300.native import GpuBatch, GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.triads import TriadLists
from rnl_multiblock_nofft_gb300.workloads import ensemble_params, re_tau_params

# retained modes per direction; the transforms run on 3/2 as many points (24 ... 1152)
MODES = (16, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768)


def _step(name, form, nx, nz, ny, period=0, points=0, height=6.0, re_tau=180.0, core_nx=0, core_nz=0, ctpress=0):
    """One RK3 step. period/points/height: square posts (grid points, wall units; 0: smooth walls);
    core_nx/core_nz: a coarser core band; ctpress 1: constant pressure gradient instead of flow rate."""
    c = dict(kind="step", form=form, nx=nx, nz=nz, ny=ny, period=period, points=points, height=height, re_tau=re_tau,
             core_nx=core_nx, core_nz=core_nz, ctpress=ctpress)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's own run size, smooth walls: the smallest channel a user steps, where launches count
        _step("small_fp64", "fp64", 32, 32, 153),
        _step("small_mixed", "mixed", 32, 32, 153),
        # the textured channel the throughput figures are quoted on, in both forms
        _step("textured_fp64", "fp64", 256, 256, 301, period=16, points=8),
        _step("textured_mixed", "mixed", 256, 256, 301, period=16, points=8),
        # ragged multiblock channel in the plain form: unequal lengths in x and z, a coarser core band
        _step("multiblock_fp64", "fp64", 192, 96, 129, period=12, points=5, height=8.0, core_nx=96, core_nz=48),
        # the large multiblock channel (production size of the mixed form)
        _step("multiblock_mixed", "mixed", 768, 384, 385, period=24, points=12, re_tau=550.0, core_nx=384, core_nz=192),
        # a parameter study: independent channels of uneven sizes, Re_tau and posts advanced by one graph
        dict(kind="ensemble", form="mixed", channels=16, draw_seed=2000, name="ensemble_mixed"),
        # the as-run nonlinear term of the reference (triad lists) at its own size
        dict(kind="triads", form="fp64", nx=32, nz=32, ny=153, name="triads_fp64"),
        # plane transforms of a post-processing program, each direction
        dict(kind="planes_inverse", nx=256, nz=256, planes=64, name="planes_inverse"),
        dict(kind="planes_forward", nx=96, nz=192, planes=40, name="planes_forward"),
        # an output step of a running simulation: statistics of the state, read back
        dict(kind="stats", form="fp64", nx=128, nz=96, ny=129, period=12, points=6, height=6.0, name="stats_fp64"),
        # a host program that keeps the state in its own (page-locked) arrays: in, one step, out
        dict(kind="host", form="mixed", nx=128, nz=96, ny=201, name="host_mixed"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def sizes(most, lo=16, hi=768):
        while True:
            nx, nz, ny = rng.choice([n for n in MODES if lo <= n <= hi]), rng.choice([n for n in MODES if lo <= n <= hi]), log_int(48, 385)
            if nx <= 8 * nz and nz <= 8 * nx and nx * nz * ny <= most:
                return nx, nz, ny

    def posts(nx, nz):
        gx, gz = 3 * nx // 2, 3 * nz // 2  # the reference also wants gx to be a multiple of the tiles in z
        fits = [d for d in range(8, 25) if gx % d == 0 and gz % d == 0 and gx % (gz // d) == 0]
        if not fits or nx * nz > 192 * 192 or rng.random() < 0.35:  # (long post lists take long to build)
            return 0, 0, 6.0
        period = rng.choice(fits)
        return period, rng.randint(max(2, period // 4), 2 * period // 3), round(rng.uniform(5.0, 10.0), 2)

    form = rng.choice(("fp64", "mixed"))
    most = 256 * 256 * 301 if form == "fp64" else 512 * 384 * 301
    kind = rng.choice(("step", "step", "step", "step", "multiblock", "ensemble", "planes_inverse", "planes_forward", "stats", "host", "triads"))
    if kind == "step":
        nx, nz, ny = sizes(most)
        period, points, height = posts(nx, nz)
        return _step(None, form, nx, nz, ny, period, points, height, round(rng.uniform(120, 400), 1), ctpress=rng.randint(0, 1))
    if kind == "multiblock":
        while True:
            nx, nz, ny = sizes(most // 2, lo=32)
            if ny >= 65:
                break
        period, points, height = posts(nx, nz)
        return _step(None, form, nx, nz, ny, period, points, height, round(rng.uniform(120, 400), 1), core_nx=nx // 2, core_nz=nz // 2)
    if kind == "ensemble":
        return dict(kind="ensemble", form=form, channels=rng.randint(3, 16), draw_seed=rng.randint(1, 10000))
    if kind == "triads":
        return dict(kind="triads", form=form, nx=rng.choice((16, 32)), nz=rng.choice((16, 32)), ny=2 * rng.randint(24, 76) + 1)
    if kind == "stats":
        nx, nz, ny = sizes(192 * 192 * 200)
        period, points, height = posts(nx, nz)
        return dict(kind="stats", form=form, nx=nx, nz=nz, ny=ny, period=period, points=points, height=height)
    if kind == "host":
        nx, nz, ny = sizes(128 * 128 * 201)
        return dict(kind="host", form=form, nx=nx, nz=nz, ny=ny)
    nx, nz, _ = sizes(512 * 512 * 48, hi=512)
    return dict(kind=kind, nx=nx, nz=nz, planes=min(log_int(1, 96), 64))


# --------------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------------
DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")


@functools.lru_cache(maxsize=64)
def _setup(nx, nz, ny, period, points, height, re_tau, core_nx, core_nz, ctpress):
    """The grid, metrics and post lists of a channel: what a program builds once for a geometry."""
    kw = dict(posts=True, post_period=period, post_points=points, post_height_plus=height) if period else {}
    p = re_tau_params(nx, ny, re_tau=re_tau, flpress=ctpress, Nz=nz, **kw)
    if core_nx:
        p.Ngalx, p.Ngalz = (p.Ngalx[0], 3 * core_nx // 2), (p.Ngalz[0], 3 * core_nz // 2)
    return build_setup(p)


@functools.lru_cache(maxsize=4)
def _triads(nx, nz, ny):
    return TriadLists.complete(_setup(nx, nz, ny, 0, 0, 6.0, 180.0, 0, 0, 0))


@functools.lru_cache(maxsize=8)
def _ensemble(n, seed):
    return [build_setup(p) for p in ensemble_params(n, seed)]


def _setup_of(c):
    return _setup(c["nx"], c["nz"], c["ny"], c.get("period", 0), c.get("points", 0), c.get("height", 6.0),
                  c.get("re_tau", 180.0), c.get("core_nx", 0), c.get("core_nz", 0), c.get("ctpress", 0))


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def _fields(s, seed):
    """u1, u2, u3 [level][N2][N1/2+1] complex128: parabolic mean and a divergence-free perturbation whose spectrum
    decays over all modes; the short columns of a multiblock channel live in their wall bands alone."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    n1h, n2, nu, nv = s.N1 // 2 + 1, s.N2, s.nyu, s.nyv
    yu, yv, th = _t(s.yu), _t(s.yv), _t(s.dthdyu * s.ddthetavi)
    k1x, k1z = _t(s.k1x)[None, :], _t(s.k1z)[:, None]
    i = torch.arange(n1h, device=DEV)[None, :]
    r = torch.arange(n2, device=DEV)[:, None]
    kz = torch.where(r < n2 // 2, r, r - n2)
    amp = torch.exp(-torch.sqrt((i * i + kz * kz).double()) / max(3.0, s.N1 / 12, s.N2 / 12))
    amp = torch.where((r == n2 // 2) | ((i == 0) & (kz <= 0)), torch.zeros_like(amp), amp)
    rnd = torch.randn((2, 2, n2, n1h), generator=gen, dtype=torch.float64, device=DEV)
    cv, cp = (torch.complex(rnd[q, 0], rnd[q, 1]) * amp for q in (0, 1))
    for q in (cv, cp):  # kx = 0: rows kz and -kz are conjugates of one another
        half = torch.arange(1, n2 // 2, device=DEV)
        q[n2 - half, 0] = q[half, 0].conj()
    cp[n2 // 2 + 1:, 0] *= -1
    k2 = k1x * k1x + k1z * k1z
    k2 = torch.where(k2 == 0, torch.ones_like(k2), k2)

    def perturbation(ev, eu):
        d = torch.zeros(nu, dtype=torch.float64, device=DEV)
        d[1:-1] = (ev[1:] - ev[:-1]) * th[1:-1]
        d, eu = d[:, None, None], eu[:, None, None]
        return (1j * (k1x / k2) * cv) * d + (k1z * cp) * eu, cv * ev[:, None, None], (1j * (k1z / k2) * cv) * d - (k1x * cp) * eu

    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    ev = torch.where(yv.abs() <= 1, (1 - yv * yv) ** 2, zero)
    ev[0] = ev[-1] = 0
    eu = torch.where(yu.abs() <= 1, (1 - yu * yu) ** 2, zero)
    u1, u2, u3 = perturbation(ev, eu / float(max(s.N1, s.N2) / 4))
    energy = sum(float((x[x.shape[0] // 2].abs() ** 2).sum()) for x in (u1, u2, u3))
    scale = 0.05 / math.sqrt(2 * energy / 3)
    for x in (u1, u2, u3):
        x *= scale
    if s.multiblock:
        short = _t(~s.is_long()).reshape(n2, n1h)
        for x in (u1, u2, u3):
            x[:, short] = 0
        for b in (1, 3):
            (ulo, uhi), (vlo, vhi) = s.band_levels(b, 2), s.band_levels(b, 1)
            lv, lu = torch.arange(nv, device=DEV), torch.arange(nu, device=DEV)
            ev = torch.where((lv >= vlo) & (lv <= vhi), (yv - yv[vlo]) ** 2 * (yv[vhi] - yv) ** 2, zero)
            eu = torch.where((lu > ulo) & (lu < uhi), ((yu - yv[vlo]) * (yv[vhi] - yu)).clamp(min=0) ** 2, zero)
            a = perturbation(0.4 * scale * ev / ev.max(), 0.05 * scale * eu / eu.max())
            for x, y, lo, hi in zip((u1, u2, u3), a, (ulo + 1, vlo, ulo + 1), (uhi, vhi + 1, uhi)):
                x[lo:hi] += torch.where(short, y[lo:hi], 0)
            inner, ghost, w = (uhi - 1, uhi, -s.gw[0, 1]) if b == 1 else (ulo + 1, ulo, -s.gw[2, 0])
            u1[ghost, short] = w * u1[inner, short]
            u3[ghost, short] = w * u3[inner, short]
    u1[:, 0, 0] = torch.where(yu.abs() <= 1, 1.5 * (1 - yu * yu), zero).to(u1.dtype)
    for x, w in ((u1, s.gw_bc_u1), (u3, s.gw_bc_u3)):
        x[0], x[-1] = w * x[1], w * x[-2]
    return u1, u2, u3


class _Memory:
    """Device memory of a channel, which a tensor on it keeps alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 2}


def _views(g, s):
    """The device-resident state of a channel, u1, u2, u3, p [level][N2][N1/2+1], as tensors on its own memory."""
    levels = (s.nyu, s.nyv, s.nyu, s.nyu - 2)
    return [torch.view_as_complex(torch.as_tensor(_Memory(g, ptr, (n, s.N2, s.N1 // 2 + 1, 2))))
            for ptr, n in zip(g.device_state(), levels)]


def _channel(s, form, seed, triads=None):
    """A channel with its state on the device and its scalars set: what a running simulation holds."""
    g = GpuChannel(s, form, triads)
    views = _views(g, s)
    for v, x in zip(views, _fields(s, seed)):
        v.copy_(x)
    views[3].zero_()
    torch.cuda.synchronize()
    g.set_scalars(t=0.0, dt=0.0, dti=0.0, dtc=0.0, mpgx=s.p.mpgx, iter=0, QxT=0.0)
    return g, views


def _planes(case, seed):
    """Spectral planes of a developed flow: decaying spectrum, mean mode of order one."""
    nx, nz, n = case["nx"], case["nz"], case["planes"]
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.view_as_complex(torch.randn((n, nz, nx // 2 + 1, 2), generator=gen, dtype=torch.float64, device=DEV))
    kz = torch.arange(nz, device=DEV)
    kz = torch.minimum(kz, nz - kz)[:, None].double()
    kx = torch.arange(nx // 2 + 1, device=DEV)[None, :].double()
    x = x * torch.exp(-torch.sqrt(kx * kx + kz * kz) / max(3.0, nx / 12, nz / 12))
    x[:, 0, 0] = 1 + torch.rand(n, generator=gen, dtype=torch.float64, device=DEV)
    return x


def _points(case, seed):
    """Physical planes of order one with fluctuations at every wavelength."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    shape = (case["planes"], 3 * case["nz"] // 2, 3 * case["nx"] // 2)
    return 1 + 0.3 * torch.randn(shape, generator=gen, dtype=torch.float64, device=DEV)


@functools.lru_cache(maxsize=8)
def _transformer(nx, nz):
    """The handle a program that only transforms planes keeps: a channel with scratch for 64 planes or more."""
    return GpuChannel(_setup(nx, nz, 81, 0, 0, 6.0, 180.0, 0, 0, 0), "fp64")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        setups = _ensemble(case["channels"], case["draw_seed"])
        made = [_channel(s, case["form"], seed + 1000 * i) for i, s in enumerate(setups)]
        return dict(kind=kind, batch=GpuBatch([g for g, _ in made]), out=[v for _, v in made])
    if kind == "planes_inverse":
        x = _planes(case, seed)
        torch.cuda.synchronize()
        out = torch.empty((case["planes"], 3 * case["nz"] // 2, 3 * case["nx"] // 2), dtype=torch.float64, device=DEV)
        return dict(kind=kind, g=_transformer(case["nx"], case["nz"]), x=x, out=out, n=case["planes"])
    if kind == "planes_forward":
        x = _points(case, seed)
        torch.cuda.synchronize()
        out = torch.empty((case["planes"], case["nz"], case["nx"] // 2 + 1), dtype=torch.complex128, device=DEV)
        return dict(kind=kind, g=_transformer(case["nx"], case["nz"]), x=x, out=out, n=case["planes"])
    s = _setup_of(case)
    if kind == "host":
        g = GpuChannel(s, case["form"])

        def pinned():
            return [torch.empty(sh, dtype=torch.complex128, pin_memory=True).numpy() for sh in g.shapes]

        state, out = pinned(), pinned()
        fields = list(_fields(s, seed))
        fields.append(torch.zeros((s.nyu - 2, s.N2, s.N1 // 2 + 1), dtype=torch.complex128, device=DEV))
        for h, x in zip(state, fields):
            torch.from_numpy(h).copy_(x.reshape(x.shape[0], -1).T.contiguous())
        g.upload_state(*state)
        g.set_scalars(t=0.0, dt=0.0, dti=0.0, dtc=0.0, mpgx=s.p.mpgx, iter=0, QxT=0.0)
        return dict(kind=kind, g=g, state=state, out=out)
    g, views = _channel(s, case["form"], seed, _triads(case["nx"], case["nz"], case["ny"]) if kind == "triads" else None)
    return dict(kind=kind, g=g, out=views)


def run(st):
    kind = st["kind"]
    if kind in ("step", "triads"):
        st["g"].step()
        return st["out"]
    if kind == "ensemble":
        st["batch"].step()
        return st["out"]
    if kind == "planes_inverse":
        st["g"].four_to_phys(st["x"].data_ptr(), st["out"].data_ptr(), st["n"])
        return st["out"]
    if kind == "planes_forward":
        st["g"].phys_to_four(st["x"].data_ptr(), st["out"].data_ptr(), st["n"])
        return st["out"]
    if kind == "stats":
        st["g"].stats_accumulate()
        plane, cond, n = st["g"].stats()
        pressure, cond_pw = st["g"].stats_pw()
        out = dict(velocity=plane[:9], vorticity=plane[9:], pressure=pressure, count=n, spectra=st["g"].spectra(), slip=st["g"].slip())
        return dict(out, cond=cond, cond_pw=cond_pw) if cond is not None else out
    st["g"].upload_state_async(*st["state"])
    st["g"].step()
    st["g"].download_state_async(st["out"])
    st["g"].synchronize()
    return st["out"], st["g"].scalars()


# --------------------------------------------------------------------------------------------------
# the work of one pass
# --------------------------------------------------------------------------------------------------
def _step_work(s, triads=False):
    """The state in and out once (complex128); flops of the transforms (5 N log2 N a complex line, x lines real),
    the products, and the solves of three substeps."""
    n1h, n2 = s.N1 // 2 + 1, s.N2
    if s.multiblock:
        wall = sum(s.band_levels(b, 2)[1] - s.band_levels(b, 2)[0] - 1 for b in (1, 3))
        parts = [(wall, s.N1, s.N2, s.G1, s.G2), (s.nyu - 2 - wall, s.N1c, s.N2c, s.G1c, s.G2c)]
    else:
        parts = [(s.nyu - 2, s.N1, s.N2, s.G1, s.G2)]
    points = sum(lev * (a // 2 + 1) * b for lev, a, b, _, _ in parts)
    flops = 0.0
    for lev, a, b, ga, gb in parts:
        line = (a // 2 + 1) * 5 * gb * math.log2(gb) + gb * 2.5 * ga * math.log2(ga)
        flops += lev * ((6 + 6) * line + 6 * ga * gb)
    if triads:  # nine products of every mode with every mode, 8 flops a term
        flops = (s.nyu - 2) * 9 * 8 * 0.75 * (s.N1 * n1h * s.N2 * n2)
    return {"bytes": 16.0 * 8 * points, "flops": 3 * (flops + 150.0 * points)}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        w = [_step_work(s) for s in _ensemble(case["channels"], case["draw_seed"])]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind.startswith("planes"):
        nx, nz, n = case["nx"], case["nz"], case["planes"]
        gx, gz = 3 * nx // 2, 3 * nz // 2
        return {"bytes": n * (16.0 * nz * (nx // 2 + 1) + 8.0 * gx * gz),
                "flops": n * ((nx // 2 + 1) * 5 * gz * math.log2(gz) + gz * 2.5 * gx * math.log2(gx))}
    s = _setup_of(case)
    w = _step_work(s, kind == "triads")
    if kind == "stats":  # the state in, six inverse transforms, the sums
        return {"bytes": w["bytes"] / 2, "flops": w["flops"] / 6}
    return w


# --------------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# --------------------------------------------------------------------------------------------------
def _to_points(x, gx, gz):
    """Spectral planes [..., N2, N1/2+1] -> physical [..., gz, gx], unscaled; Im of x-mode 0 is ignored."""
    n2 = x.shape[-2]
    a = torch.zeros((*x.shape[:-2], gz, x.shape[-1]), dtype=x.dtype, device=x.device)
    a[..., :n2 // 2, :] = x[..., :n2 // 2, :]
    a[..., gz - n2 // 2:, :] = x[..., n2 // 2:, :]
    return torch.fft.irfft(torch.fft.ifft(a, dim=-2, norm="forward"), n=gx, dim=-1, norm="forward")


def _to_modes(f, n1, n2):
    x = torch.fft.fft(torch.fft.rfft(f, dim=-1, norm="forward")[..., :n1 // 2 + 1], dim=-2, norm="forward")
    return torch.cat([x[..., :n2 // 2, :], x[..., f.shape[-2] - n2 // 2:, :]], dim=-2)


def _thomas(lower, diag, upper, rhs):
    """Solves the tridiagonal systems of every column; lists of per-level coefficients, rhs [level][...] in place."""
    n = rhs.shape[0]
    inv, up = 1.0 / diag[0], []
    rhs[0] *= inv
    for j in range(1, n):
        up.append(upper[j - 1] * inv)
        inv = 1.0 / (diag[j] - lower[j] * up[-1])
        rhs[j] = (rhs[j] - lower[j] * rhs[j - 1]) * inv
    for j in range(n - 2, -1, -1):
        rhs[j] -= up[j] * rhs[j + 1]


def _interpolated(s, u1, u2, u3):
    """v at the centres of the interior u levels, u and w at the interior v levels."""
    yu, yv = _t(s.yu)[:, None, None], _t(s.yv)[:, None, None]
    vc = ((yu[1:-1] - yv[:-1]) * u2[1:] + (yv[1:] - yu[1:-1]) * u2[:-1]) / (yv[1:] - yv[:-1])
    a, b = (yv[1:-1] - yu[1:-2]) / (yu[2:-1] - yu[1:-2]), (yu[2:-1] - yv[1:-1]) / (yu[2:-1] - yu[1:-2])
    return vc, a * u1[2:-1] + b * u1[1:-2], a * u3[2:-1] + b * u3[1:-2]


def _exact_step(s, seed, mpgx):
    u1, u2, u3 = _fields(s, seed)
    n1, n2, g1, g2, nu, nv, off, dd, p = s.N1, s.N2, s.G1, s.G2, s.nyu, s.nyv, s.dny, s.ddthetavi, s.p
    pr = torch.zeros((nu - 2, n2, n1 // 2 + 1), dtype=torch.complex128, device=DEV)
    ikx, ikz = 1j * _t(s.k1x)[None, :], 1j * _t(s.k1z)[:, None]
    kk = _t(s.k2x)[None, :] + _t(s.k2z)[:, None]
    thu, thv, yv = _t(s.dthdyu)[:, None, None], _t(s.dthdyv)[:, None, None], _t(s.yv)
    du, dv = _t(s.dyu2i)[:, :, None, None], _t(s.dyv2i)[:, :, None, None]
    old = [torch.zeros_like(u1), torch.zeros_like(u2), torch.zeros_like(u3)]
    dy = yv[off + 1:off + s.nn + 2] - yv[off:off + s.nn + 1]
    inside = slice(off + 1, off + s.nn + 2)
    flow = float((dy * u1[inside, 0, 0].real).sum())
    ju, jv = range(1, nu - 1), range(1, nv - 1)
    block = max(1, int(2e8) // (g1 * g2))
    for k in range(3):
        a, b, c, d, g = s.aRK[k], s.bRK[k], s.cRK[k], s.dRK[k], s.gRK[k]
        vc, uf, wf = _interpolated(s, u1, u2, u3)
        x = [torch.zeros_like(q) for q in (u1, u2, u3)]
        uv, vv, wv = torch.zeros_like(u2), torch.zeros_like(u1), torch.zeros_like(u2)
        most, phys = [0.0, 1e-6, 0.0], {}
        forced = range(1, off + 2), range(nv - 1 - off, nu - 1)

        def der(e, f):
            q = ikx * e + ikz * f
            q[..., n2 // 2, :] = 0
            return q

        for q0 in range(1, nu - 1, block):
            q1 = min(q0 + block, nu - 1)
            fu, fv, fw = (_to_points(z, g1, g2) for z in (u1[q0:q1], vc[q0 - 1:q1 - 1], u3[q0:q1]))
            most[0], most[2] = max(most[0], float(fu.abs().max())), max(most[2], float(fw.abs().max()))
            uu, uw, ww = (_to_modes(z, n1, n2) for z in (fu * fu, fu * fw, fw * fw))
            vv[q0:q1] = _to_modes(fv * fv, n1, n2)
            x[0][q0:q1], x[2][q0:q1] = der(uu, uw), der(uw, ww)
            for q in range(q0, q1):
                if off and any(q in z for z in forced):
                    phys[0, q], phys[2, q] = fu[q - q0].clone(), fw[q - q0].clone()
        for q0 in range(1, nv - 1, block):
            q1 = min(q0 + block, nv - 1)
            fu, fv, fw = (_to_points(z, g1, g2) for z in (uf[q0 - 1:q1 - 1], u2[q0:q1], wf[q0 - 1:q1 - 1]))
            most[1] = max(most[1], float((fv.abs().amax(dim=(1, 2)) * thv[q0:q1, 0, 0]).max()))
            uv[q0:q1], wv[q0:q1] = _to_modes(fu * fv, n1, n2), _to_modes(fw * fv, n1, n2)
            x[1][q0:q1] = der(uv[q0:q1], wv[q0:q1])
            for q in range(q0, q1):
                if off and any(q in z for z in forced):
                    phys[1, q] = fv[q - q0].clone()
        if k == 0:  # the wall-normal limit is never set by the reference
            cfl = min(1 / (p.alp * (n1 // 2) * most[0]), 1 / (p.bet * (n2 // 2) * most[2]))
            dt = min(2.5 * s.dtv, p.CFL * cfl)
        x[0][1:-1] += (uv[1:] - uv[:-1]) * thu[1:-1] * dd
        x[2][1:-1] += (wv[1:] - wv[:-1]) * thu[1:-1] * dd
        x[1][1:-1] += (vv[2:-1] - vv[1:-2]) * thv[1:-1] * dd
        rhs = []
        for u, z, o, m, grad in ((u1, x[0], old[0], du, -d * ikx * pr), (u2, x[1], old[1], dv, -d * dd * thv[1:-1] * (pr[1:] - pr[:-1])),
                                 (u3, x[2], old[2], du, -d * ikz * pr)):
            lap = m[0, 1:-1] * u[:-2] + (kk + m[1, 1:-1]) * u[1:-1] + m[2, 1:-1] * u[2:]
            r = torch.zeros_like(u)
            r[1:-1] = a / p.Re * lap - c * o[1:-1] + grad - g * z[1:-1]
            rhs.append(r)
        rhs[0][1:-1, 0, 0] -= d * mpgx
        old = x
        if off and p.ib_enable:
            rows = [list(range(1, off + 1)) + list(range(nu - 1 - off, nu - 1)), list(range(1, off + 1)) + list(range(nv - 1 - off, nv - 1))]
            for f, (grid, lev) in enumerate(((2, rows[0]), (1, rows[1]), (2, rows[0]))):
                points, weight = s.list_ib[grid].astype(np.int64), s.A_ib[grid]
                for q in lev:
                    at = points[:, 2] + off == q
                    e, w = _t(points[at]), _t(weight[at])
                    plane = _to_points(rhs[f][q], g1, g2)
                    refs = e[:, 5] + off
                    goal = torch.zeros(len(w), dtype=torch.float64, device=DEV)
                    for rq in set(refs.tolist()):
                        sel = refs == rq
                        goal[sel] = w[sel] * phys[f, rq][e[sel, 4] - 1, e[sel, 3] - 1]
                    plane[e[:, 1] - 1, e[:, 0] - 1] = p.Kib / dt * (goal - phys[f, q][e[:, 1] - 1, e[:, 0] - 1])
                    rhs[f][q] = _to_modes(plane, n1, n2)
        beta = b * dt / p.Re
        for u, r, m, w0, w1 in ((u1, rhs[0], du, s.gw[1, 0], s.gw[1, 1]), (u2, rhs[1], dv, 0.0, 0.0), (u3, rhs[2], du, s.gw[1, 0], s.gw[1, 1])):
            r[1:-1] = u[1:-1] + dt * r[1:-1]
            one = torch.ones_like(kk)
            n = u.shape[0]
            lower = [0.0] + [-beta * m[0, j] for j in range(1, n - 1)] + [w1]
            diag = [one] + [1 - beta * (m[1, j] + kk) for j in range(1, n - 1)] + [one]
            upper = [w0] + [-beta * m[2, j] for j in range(1, n - 1)] + [0.0]
            _thomas(lower, diag, upper, r)
            u.copy_(r)
        if p.flpress == 0:  # flow-rate correction of the mean mode
            n = s.nn + 3
            one = torch.ones((), dtype=torch.float64, device=DEV)
            r = torch.full((n,), -d * dt, dtype=torch.float64, device=DEV)
            r[0] = r[-1] = 0
            m = du[:, off:off + n, 0, 0]
            _thomas([0.0] + [-beta * m[0, j] for j in range(1, n - 1)] + [s.gw[1, 1]], [one] + [1 - beta * m[1, j] for j in range(1, n - 1)] + [one],
                    [s.gw[1, 0]] + [-beta * m[2, j] for j in range(1, n - 1)] + [0.0], r)
            more = (flow - float((dy * u1[inside, 0, 0].real).sum())) / float((dy * r[1:-1]).sum())
            mpgx += more
            u1[off:off + n, 0, 0] += more * r
        psi = (ikx * u1[1:-1] + ikz * u3[1:-1] + dd * thu[1:-1] * (u2[1:] - u2[:-1])) / (dt * (a + b))
        psi[0, 0, 0] = 0
        n = nu - 2
        tu, tv = dd * thu[1:-1, 0, 0], dd * thv[:, 0, 0]
        lower = [0.0] + [tu[j] * tv[j] * torch.ones_like(kk) for j in range(1, n)]
        upper = [tu[j] * tv[j + 1] * torch.ones_like(kk) for j in range(n - 1)] + [0.0]
        diag = [kk - tu[j] * ((tv[j] if j else 0.0) + (tv[j + 1] if j < n - 1 else 0.0)) for j in range(n)]
        diag[0][0, 0] = 1.0 / (s.yu[2 + off] - s.yu[1 + off]) ** 2
        upper[0][0, 0] = 0.0
        _thomas(lower, diag, upper, psi)
        pr += psi
        f = dt * (a + b)
        u1[1:-1] -= f * ikx * psi
        u3[1:-1] -= f * ikz * psi
        u2[1:-1] -= f * dd * thv[1:-1] * (psi[1:] - psi[:-1])
        u2[0] = u2[-1] = 0
        for u, w in ((u1, s.gw_bc_u1), (u3, s.gw_bc_u3)):
            u[0], u[-1] = w * u[1], w * u[-2]
    return [u1, u2, u3, pr]


def exact(case, seed):
    kind = case["kind"]
    if kind == "planes_inverse":
        return _to_points(_planes(case, seed), 3 * case["nx"] // 2, 3 * case["nz"] // 2)
    if kind == "planes_forward":
        return _to_modes(_points(case, seed), case["nx"], case["nz"])
    if kind == "ensemble":
        return [_exact_step(s, seed + 1000 * i, s.p.mpgx) for i, s in enumerate(_ensemble(case["channels"], case["draw_seed"]))]
    s = _setup_of(case)
    if kind == "triads" or s.multiblock:
        return None  # list convolutions and the two-resolution channel: minutes in plain torch
    if kind == "stats":
        u1, u2, u3 = _fields(s, seed)
        vc, uf, wf = _interpolated(s, u1, u2, u3)
        plane = torch.zeros((9, s.nyu), dtype=torch.float64, device=DEV)
        for j in range(s.nyu - 2):
            u, v, w = (_to_points(z, s.G1, s.G2) for z in (u1[j + 1], vc[j], u3[j + 1]))
            plane[:6, j + 1] = torch.stack([z.sum() for z in (u, u * u, w, w * w, u * v, u * w)])
        for j in range(s.nyv - 2):
            v, w = (_to_points(z, s.G1, s.G2) for z in (u2[j + 1], wf[j]))
            plane[6:, j + 1] = torch.stack([z.sum() for z in (v, v * v, v * w)])
        spectra = {q: (x.abs() ** 2).reshape(x.shape[0], -1).T.contiguous() for q, x in (("U", u1), ("V", u2), ("W", u3))}
        return dict(velocity=plane, spectra=spectra)
    out = _exact_step(s, seed, s.p.mpgx)
    if kind == "host":  # the host layout: [column][level]
        return [x.reshape(x.shape[0], -1).T.contiguous() for x in out], {}
    return out
