"""Timing cases: the work a program gives this library, through its public entry points.

Each case is a dict of plain values.  "kind" names the way the library is used:

    run       a device-resident run between two outputs: kmm_run over `steps` time steps, then the
              restart records (the mixed form: single-precision copies of them) read back;
    ensemble  kmm_ensemble_run over several channels of different grids;
    host      kmm_run_host: the state lives in the host program's page-locked arrays;
    linear    a host time loop that calls the routines one by one: `steps` implicit stages under a
              frozen forcing (a Stokes run), then the fields read back;
    nonlinear such a loop's vcw3dp (dealiased u x omega and -u.grad c);
    xyzfft    kmm_xyzfft_noalloc on the caller's device arrays.

Inputs are made from the seed: a mean profile plus divergence-free random modes that vanish at the
walls, random low modes for the scalar, uniform particles.  The time steps are small enough that a
run continued over many passes stays far from CFL 1.
"""
import math

import numpy as np
import torch

from polymer_dns_b200 import abi, inputs, runtime

PI = math.pi
COMPILED = (32, 64, 96, 128)
RAGGED_XZ = (24, 40, 48, 60, 72, 80, 100, 108, 120, 144, 160)   # 3/2 grids off the compiled lengths too
RAGGED_Y = (24, 36, 40, 48, 54, 60, 72, 80, 100, 120, 144, 160)


def listed():
    return [
        # the smallest runs: a parameter scan of a short laminar channel at constant flow rate,
        # where launches and host round trips count
        dict(name="run 32^3 fluid", kind="run", nx=32, ny=32, nz=32, precision=0, scalar=0, polymer=0, ib=0,
             npart=0, flow_rate=1.0, scheme=0, steps=50),
        # the Re_tau = 180 production run: scalar and 100,000 tracers
        dict(name="run 128^3 scalar", kind="run", nx=128, ny=128, nz=128, precision=0, scalar=1, polymer=0, ib=0,
             npart=100000, flow_rate=0.0, scheme=1, steps=40),
        # the same run in the mixed form
        dict(name="run 128^3 scalar mixed", kind="run", nx=128, ny=128, nz=128, precision=1, scalar=1, polymer=0,
             ib=0, npart=100000, flow_rate=0.0, scheme=1, steps=40),
        # a grid chosen by resolution and not by power of two, Euler tracers
        dict(name="run 80x61x60 scalar", kind="run", nx=80, ny=60, nz=60, precision=0, scalar=1, polymer=0, ib=0,
             npart=5000, flow_rate=0.0, scheme=0, steps=20),
        # drag reduction around a body: FENE-P polymer, scalar, Goldstein cylinder, tracers
        dict(name="run 128^3 polymer body", kind="run", nx=128, ny=128, nz=128, precision=0, scalar=1, polymer=1,
             ib=1, npart=100000, flow_rate=0.0, scheme=1, steps=6),
        # polymer channel without a body, mixed form
        dict(name="run 96^3 polymer mixed", kind="run", nx=96, ny=96, nz=96, precision=1, scalar=1, polymer=1, ib=0,
             npart=0, flow_rate=0.0, scheme=0, steps=12),
        # the largest: the Re_tau = 395 grid with a scalar
        dict(name="run 384x257x384 scalar", kind="run", nx=384, ny=256, nz=384, precision=0, scalar=1, polymer=0,
             ib=0, npart=0, flow_rate=0.0, scheme=0, steps=3),
        # six uneven channels of a Reynolds-number study advanced together
        dict(name="ensemble of 6", kind="ensemble", members="64x64x64,64x64x64,96x96x96,96x96x96,128x128x96,128x128x96",
             precision=0, npart=20000, steps=10),
        # a host program that keeps its arrays and steps on the device
        dict(name="host 64^3 scalar", kind="host", nx=64, ny=64, nz=64, precision=0, scalar=1, npart=10000, steps=8),
        # a host loop that calls the routines: implicit stage, then the nonlinear stage
        dict(name="linear 128x129x96", kind="linear", nx=128, ny=128, nz=96, steps=5),
        dict(name="nonlinear 96^3", kind="nonlinear", nx=96, ny=96, nz=96, scalar=1),
        # one initial field transformed in a program that owns its device memory
        dict(name="xyzfft 64x97x64", kind="xyzfft", nx=64, ny=96, nz=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most, compiled=False):
    """(nx, ny, nz) with at most `most` points: compiled lengths, or a mix with any others."""
    while True:
        if compiled or rng.random() < 0.5:
            g = [rng.choice(COMPILED) for _ in range(3)]
        else:
            g = [rng.choice(COMPILED + RAGGED_XZ), rng.choice(COMPILED + RAGGED_Y), rng.choice(COMPILED + RAGGED_XZ)]
        if g[0] * g[1] * g[2] <= most:
            return g


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["ensemble", "host", "linear", "nonlinear", "xyzfft"])
    if kind == "ensemble":
        grids = ["%dx%dx%d" % tuple(_grid(rng, 128 * 128 * 96, compiled=True)) for _ in range(rng.randint(2, 6))]
        return dict(kind=kind, members=",".join(grids), precision=rng.randint(0, 1), npart=_log_int(rng, 500, 20000),
                    steps=rng.randint(4, 12))
    if kind == "host":
        nx, ny, nz = _grid(rng, 96 ** 3, compiled=True)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=0, scalar=rng.randint(0, 1),
                    npart=_log_int(rng, 100, 20000), steps=rng.randint(3, 10))
    if kind in ("linear", "nonlinear"):
        nx, ny, nz = _grid(rng, 128 ** 3)
        case = dict(kind=kind, nx=nx, ny=ny, nz=nz)
        case["scalar" if kind == "nonlinear" else "steps"] = rng.randint(0, 1) if kind == "nonlinear" else rng.randint(2, 6)
        return case
    if kind == "xyzfft":
        while True:
            nx, ny, nz = _grid(rng, 128 ** 3)
            if (ny + 1) * nz * nx <= 4 * 1024 * 1024:
                return dict(kind=kind, nx=nx, ny=ny, nz=nz)
    precision = int(rng.random() < 0.35)
    polymer = int(rng.random() < 0.35)
    nx, ny, nz = _grid(rng, 128 ** 3, compiled=precision == 1)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, scalar=1 if polymer else rng.randint(0, 1),
                polymer=polymer, ib=int(polymer and rng.random() < 0.5),
                npart=rng.choice([0, _log_int(rng, 100, 200000)]), flow_rate=0.0, scheme=rng.randint(0, 1),
                steps=rng.randint(4, 10) if polymer else rng.randint(10, 40))


# ---------------------------------------------------------------- inputs
def _params(case, nx, ny, nz, npart):
    re, r_tau = 2800.0, 180.0
    polymer, ib = case.get("polymer", 0), case.get("ib", 0)
    # (random fields of the nonlinear kind have wall values of order one: dt enters its CFL number only)
    dt = 0.0005 if polymer else 1e-8 if case.get("kind") == "nonlinear" else 0.002
    kw = dict(nx=nx, ny=ny, nz=nz, dt=dt, re=re, r_tau=r_tau, xl=4 * PI, zl=4 * PI / 3, npart=npart, ap=1e-3,
              tracer_scheme=case.get("scheme", 1), precision=case.get("precision", 0),
              flow_rate=case.get("flow_rate", 0.0))
    if case.get("scalar", 1):
        kw.update(scalar_on=1, diff=1.0, scalar_bc=1, scalar_q=1.0)
    if polymer:
        kw.update(polymer_on=1, zlmax=30.0, tpoly=20.0, qbeta=0.9, diffpoly=1.0 / (re * 1e-3))
    if ib:
        kw.update(gain=400.0 * dt, ugain=40.0, ib_spread_all=1)
    return abi.default_params(**kw)


def _modes(p, seed, kmax=4, nmode=48):
    """(u, v, w, c) on the (nx, nz, nyp) grid (the reference's Fortran layout), on the GPU."""
    rng = np.random.default_rng(seed)
    kx = rng.integers(0, kmax + 1, nmode)
    kz = rng.integers(-kmax, kmax + 1, nmode)
    kz[(kx == 0) & (kz == 0)] = 1
    ph, amp, c0, c1 = (torch.as_tensor(a, device="cuda") for a in (
        rng.uniform(0, 2 * PI, nmode), rng.standard_normal(nmode), rng.standard_normal(nmode),
        0.5 * rng.standard_normal(nmode)))
    y = torch.as_tensor(inputs.grid_y(p.ny, p.yl) / (p.yl / 2.0), device="cuda")
    a = 2 * PI / p.xl * torch.as_tensor(kx, device="cuda", dtype=torch.float64)
    b = 2 * PI / p.zl * torch.as_tensor(kz, device="cuda", dtype=torch.float64)
    x = torch.arange(p.nx, device="cuda", dtype=torch.float64) * (p.xl / p.nx)
    z = torch.arange(p.nz, device="cuda", dtype=torch.float64) * (p.zl / p.nz)
    t = a[:, None, None] * x[None, :, None] + b[:, None, None] * z[None, None, :] + ph[:, None, None]
    cs, sn = torch.cos(t).reshape(nmode, -1), torch.sin(t).reshape(nmode, -1)
    E, dE = (1 - y ** 2) ** 2, -4 * y * (1 - y ** 2)
    P = c0[:, None] + c1[:, None] * y
    f, df = amp[:, None] * E * P, amp[:, None] * (dE * P + E * c1[:, None])
    half = nmode // 2
    one = torch.arange(nmode, device="cuda") < half     # psi1: u = psi_y, v = -psi_x; psi2: w = psi_y, v = -psi_z

    def field(wave, prof):
        return (wave.T @ prof).reshape(p.nx, p.nz, p.ny + 1)

    u = field(cs * one[:, None], df)
    w = field(cs * ~one[:, None], df)
    v = field(sn, f * torch.where(one, a, b)[:, None])
    s = 0.1 / float(torch.sqrt((u * u + v * v + w * w).mean()))
    if p.flow_rate > 0:
        mean = 1.5 * (1 - y ** 2)
    else:
        mean = torch.as_tensor(p.r_tau / p.re * inputs.reichardt((1 - np.abs(y.cpu().numpy())) * p.r_tau), device="cuda")
    c = field(cs, amp[:, None] * (1 - y ** 2) * P) * 0.2
    return s * u + mean, s * v, s * w, c


def _host(t):
    return t.contiguous().cpu().numpy().reshape(-1)


def _context(case, nx, ny, nz, npart, seed):
    """A channel at its initial state."""
    p = _params(case, nx, ny, nz, npart)
    ctx = runtime.KmmContext(p)
    u, v, w, c = _modes(p, seed)
    for name, t in (("INITU", u), ("INITV", v), ("INITW", w)) + ((("INITSCL", c),) if p.scalar_on else ()):
        ctx.upload(name, _host(t))
    if npart:
        for name, a in zip(("XPART", "YPART", "ZPART"),
                           inputs.uniform_particles(npart, p.xl, p.yl, p.zl, p.ap, seed + 1)):
            ctx.upload(name, a)
    if case.get("ib", 0):
        ctx.upload("IMATRIX", inputs.cylinder_imatrix(nx, ny, nz, p.xl, p.yl))
    ctx.initial()
    ctx.call("sync")
    return ctx


def _shape(p, name):
    """C-order shape of a field's host array (the reference's Fortran shape reversed)."""
    return tuple(reversed(abi.field_shape(abi.FIELD[name], p.nx, p.ny, p.nz, p.npart)))


def _pinned(p, name):
    kind, _ = abi.field_kind(abi.FIELD[name])
    return torch.empty(_shape(p, name), dtype=torch.complex128 if kind in ("spectral", "wall") else torch.float64,
                       pin_memory=True)


def _records(p):
    names = ["V", "OMY", "FN", "GN", "U0", "W0"]
    if p.scalar_on:
        names += ["SCALAR"]
    if p.polymer_on:
        names += ["C11", "C12", "C33"]
    if p.npart:
        names += ["XPART", "YPART", "ZPART"]
    return names


def _random_spectral(p, n, seed):
    """n decaying random spectral fields with the symmetries a real field has."""
    rng = torch.Generator(device="cuda")
    rng.manual_seed(int(seed))
    nxh, nz, nyp = p.nx // 2, p.nz, p.ny + 1
    ky = torch.arange(nyp, device="cuda", dtype=torch.float64)
    kz = torch.minimum(torch.arange(nz, device="cuda"), nz - torch.arange(nz, device="cuda")).double()
    kx = torch.arange(nxh, device="cuda", dtype=torch.float64)
    decay = torch.exp(-0.15 * ky[None, None, :] - 0.2 * kz[None, :, None] - 0.2 * kx[:, None, None])
    out = []
    for _ in range(n):
        a = torch.randn((nxh, nz, nyp), dtype=torch.complex128, device="cuda", generator=rng) * decay
        a[0, 0] = a[0, 0].real.to(a.dtype)
        a[0, nz // 2 + 1:] = torch.flip(a[0, 1:nz // 2], [0]).conj()
        a[:, nz // 2] = 0
        out.append(a)
    return out


def _routine_fields(case, seed):
    """(params, {field: device tensor}) of the routine-by-routine kinds."""
    p = _params(dict(case, precision=0), case["nx"], case["ny"], case["nz"], 0)
    if case["kind"] == "linear":
        names = ["V", "OMY", "FN", "FNM1", "GN", "GNM1", "SCALAR", "SCN", "SCNM1"]
    else:
        names = ["U", "V", "W", "OMX", "OMY", "OMZ"] + (["SCLX", "SCLY", "SCLZ"] if p.scalar_on else [])
    f = dict(zip(names, _random_spectral(p, len(names), seed)))
    for k in ("FN", "FNM1", "GN", "GNM1", "SCN", "SCNM1"):
        if k in f:
            f[k] *= 1e-2
    return p, f


# ---------------------------------------------------------------- a pass
def prepare(case, seed):
    kind = case["kind"]
    if kind == "xyzfft":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        p = _params(dict(scalar=0), nx, ny, nz, 0)
        u = _modes(p, seed)[0].contiguous()
        return dict(kind=kind, phys=u, dims=(nx, ny, nz),
                    spec=torch.empty((nx // 2, nz, ny + 1), dtype=torch.complex128, device="cuda"))
    if kind == "ensemble":
        ctxs, out = [], []
        for m, g in enumerate(case["members"].split(",")):
            nx, ny, nz = (int(s) for s in g.split("x"))
            c = _context(dict(case, scalar=1), nx, ny, nz, case["npart"], seed + 100 * m)
            c.run(2)
            ctxs.append(c)
            names = ("V", "SCALAR", "XPART")
            out.append({k: _pinned(c.params, k) for k in names})
        return dict(kind=kind, ctxs=ctxs, out=out, steps=case["steps"], mixed=case["precision"] == 1)
    if kind in ("linear", "nonlinear"):
        p, f = _routine_fields(case, seed)
        ctx = runtime.KmmContext(p)
        for k, t in f.items():
            ctx.upload(k, _host(t))
        if kind == "linear":
            ctx.call("gfcn")
        names = ("V", "OMY", "SCALAR", "U") if kind == "linear" else ("FN", "GN", "OMZ") + (("SCN",) if p.scalar_on else ())
        ctx.call("sync")
        return dict(kind=kind, ctx=ctx, p=p, out={k: _pinned(p, k) for k in names}, steps=case.get("steps", 1))
    ctx = _context(case, case["nx"], case["ny"], case["nz"], case["npart"], seed)
    p = ctx.params
    if kind == "host":
        names = ["V", "FN", "FNM1", "OMY", "GN", "GNM1", "U0", "H1N", "H1NM1", "W0", "H3N", "H3NM1"]
        names += ["SCALAR", "SCN", "SCNM1"] if p.scalar_on else []
        names += ["XPART", "YPART", "ZPART", "UPART", "VPART", "WPART"]
        out = {k: _pinned(p, k) for k in names}
        for k, t in out.items():
            ctx.download_ptr(k, t.data_ptr(), t.numel() * t.element_size())
            ctx.bind_host(k, t.data_ptr(), t.numel() * t.element_size())
        return dict(kind=kind, ctx=ctx, out=out, steps=case["steps"])
    return dict(kind=kind, ctx=ctx, out={k: _pinned(p, k) for k in _records(p)}, steps=case["steps"],
                mixed=p.precision == 1)


def _read(ctx, out, single=False):
    for k, t in out.items():
        ctx.download_ptr(k, t.data_ptr(), t.numel() * t.element_size())
    if single:   # what a mixed-precision run keeps of its fields
        return {k: t.to(torch.complex64 if t.is_complex() else torch.float32) for k, t in out.items()}
    return out


def run(state):
    kind = state["kind"]
    if kind == "run":
        state["ctx"].run(state["steps"])
        return _read(state["ctx"], state["out"], state["mixed"])
    if kind == "host":
        state["ctx"].run_host(state["steps"])
        return state["out"]
    if kind == "ensemble":
        status = runtime.ensemble_run(state["ctxs"], state["steps"])
        if any(status):
            raise RuntimeError("ensemble member status %r" % (status,))
        return [_read(c, o, state["mixed"]) for c, o in zip(state["ctxs"], state["out"])]
    if kind == "xyzfft":
        nx, ny, nz = state["dims"]
        st = runtime.xyzfft_noalloc(state["phys"].data_ptr(), state["spec"].data_ptr(), nx, ny, nz)
        if st:
            raise RuntimeError("kmm_xyzfft_noalloc returned %d" % st)
        return state["spec"]
    ctx, p = state["ctx"], state["p"]
    if kind == "nonlinear":
        ctx.call("vcw3dp")
        return _read(ctx, state["out"])
    g = p.re / (p.dt * p.theta)
    for _ in range(state["steps"]):
        ctx.call("phirhs", "SCALAR", "SCN", "SCNM1", p.diff)
        ctx.call("penta", "SCALAR", p.re * p.diff / (p.dt * p.theta), 0, 1.0, 0.0, 1.0, 0.0)
        ctx.call("phi_from_v")
        ctx.call("phirhs", "V", "FN", "FNM1", 1.0)
        ctx.call("solve", "V", g, 0)
        ctx.call("solve", "V", 0.0, 0)
        ctx.call("phirhs", "OMY", "GN", "GNM1", 1.0)
        ctx.call("influence")
        ctx.call("penta", "OMY", g, 0, 1.0, 0.0, 1.0, 0.0)
        for name in ("V", "OMY", "SCALAR"):
            ctx.call("norm", name)
        ctx.call("veloc")
        ctx.call("vort")
        ctx.call("gradscl")
    return _read(ctx, state["out"])


# ---------------------------------------------------------------- work
def _step_work(nx, ny, nz, scalar, polymer, npart):
    """Bytes and operations of one time step: its field passes at 16 bytes a mode (velocity 28, scalar
    13, polymer 108), 264 bytes a particle; the transforms of its fields at 5 n log2 n a length."""
    nyp, mx, mz, nxh = ny + 1, 3 * nx // 2, 3 * nz // 2, nx // 2
    nspec = nyp * nz * nxh
    byts = 16.0 * nspec * (28 + 13 * scalar + 108 * polymer) + 264.0 * npart
    fields = 6 + 3 + scalar * 4 + polymer * 60
    ylines, zlines, xlines = nz * nxh, nyp * nxh, nyp * mz
    flops = fields * (ylines * 5.0 * ny * math.log2(2 * ny) + zlines * 5.0 * mz * math.log2(mz) +
                      xlines * 2.5 * mx * math.log2(mx))
    flops += nspec * 60.0 * (2 + scalar + 6 * polymer)
    return byts, flops


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        byts = flops = 0.0
        for g in case["members"].split(","):
            b, f = _step_work(*(int(s) for s in g.split("x")), 1, 0, case["npart"])
            byts, flops = byts + b * case["steps"], flops + f * case["steps"]
        return {"bytes": byts, "flops": flops}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nspec = (ny + 1) * nz * nx // 2
    if kind == "xyzfft":
        n = (ny + 1) * nz * nx
        return {"bytes": 16.0 * n, "flops": 2.5 * n * math.log2(2.0 * ny * nz * nx)}
    if kind == "linear":
        # a stage: 9 fields and the two Green's functions read; 3 solved fields, u, w, two vorticities and
        # three scalar derivatives written; 4 fields read back at the end
        return {"bytes": 16.0 * nspec * ((9 + 2 + 3 + 2 + 2 + 3) * case["steps"] + 4),
                "flops": 300.0 * nspec * case["steps"]}
    if kind == "nonlinear":
        nin, nout = (9, 4) if case["scalar"] else (6, 3)
        _, flops = _step_work(nx, ny, nz, case["scalar"], 0, 0)
        return {"bytes": 16.0 * nspec * (nin + 2 * nout), "flops": flops}
    b, f = _step_work(nx, ny, nz, case["scalar"], case.get("polymer", 0), case["npart"])
    if kind == "host":   # every bound field crosses the host link both ways each step
        b += 2 * (16.0 * nspec * (6 + 3 * case["scalar"]) + 48.0 * case["npart"])
    return {"bytes": b * case["steps"], "flops": f * case["steps"]}


# ---------------------------------------------------------------- 64-bit reference values
def _dct1(a):
    """sum over the even extension (FFTW's REDFT00) along the last axis."""
    ext = torch.cat([a, torch.flip(a[..., 1:-1], [-1])], dim=-1)
    return torch.fft.fft(ext, dim=-1)[..., :a.shape[-1]]


def _exact_xyzfft(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    u = _modes(_params(dict(scalar=0), nx, ny, nz, 0), seed)[0].to(torch.complex128)
    a = _dct1(u) / ny
    a[..., 0] /= 2
    a[..., -1] /= 2
    return torch.fft.fft(torch.fft.fft(a, dim=0)[: nx // 2] / nx, dim=1) / nz


def _exact_nonlinear(case, seed):
    p, f = _routine_fields(case, seed)
    ny, nz, nxh, mx, mz = p.ny, p.nz, p.nx // 2, 3 * p.nx // 2, 3 * p.nz // 2
    half = nz // 2

    def phys(a):
        a = a.clone()
        a[..., 1:-1] *= 0.5
        b = _dct1(a)
        s = torch.zeros((mx // 2 + 1, mz, ny + 1), dtype=torch.complex128, device="cuda")
        s[:nxh, :half] = b[:, :half]
        s[:nxh, mz - half:] = b[:, half:]
        s = torch.fft.ifft(s, dim=1) * mz
        s[0] = s[0].real.to(s.dtype)
        return torch.fft.irfft(s, n=mx, dim=0) * mx

    def spec(h):
        s = torch.fft.fft(torch.fft.rfft(h, dim=0)[:nxh], dim=1) / (mx * mz)
        s = _dct1(torch.cat([s[:, :half], s[:, mz - half:]], dim=1)) / ny
        s[..., 0] /= 2
        s[..., -1] /= 2
        return s

    U = {k: phys(a) for k, a in f.items()}
    dpdx = -2.0 / p.yl * (2.0 * p.r_tau / (p.yl * p.re)) ** 2
    out = {"GN": spec(U["V"] * U["OMZ"] - U["W"] * U["OMY"] - dpdx),
           "FN": spec(U["W"] * U["OMX"] - U["U"] * U["OMZ"]),
           "OMZ": spec(U["U"] * U["OMY"] - U["V"] * U["OMX"])}
    if p.scalar_on:
        out["SCN"] = spec(p.scalar_q - U["U"] * U["SCLX"] - U["V"] * U["SCLY"] - U["W"] * U["SCLZ"])
    return out


def _cheb_der(a, dyde):
    """d/dy along the last axis: D_i = sum over m > i, m - i odd, of 2 m a_m, D_0 halved."""
    n = a.shape[-1]
    m = torch.arange(n, device="cuda")
    D = torch.where((m[None, :] > m[:, None]) & ((m[None, :] - m[:, None]) % 2 == 1), 2.0 * m[None, :], 0.0).double()
    D[0] *= 0.5
    return (a @ D.T.to(a.dtype)) * dyde


def _exact_advance(p, x, fn, fnm1, var):
    """The CN / AB2 step of one field with zero Dirichlet values: phirhs, the tau solve, norm."""
    N, nz, nxh, th, dyde = p.ny, p.nz, p.nx // 2, p.theta, 2.0 / p.yl
    wx = torch.arange(nxh, device="cuda").double() * (2 * PI / p.xl)
    j = torch.arange(nz, device="cuda").double()
    wz = torch.where(j < nz // 2, j, j - nz) * (2 * PI / p.zl)
    k2 = wx[:, None] ** 2 + wz[None, :] ** 2
    d2 = _cheb_der(_cheb_der(x, dyde), dyde)
    r = -p.re * var / (p.dt * th) * x - p.re * var / (2 * th) * (3.0 * fn - fnm1)
    r = r + (1 - th) * k2[:, :, None] * x / th - (1 - th) * d2 / th
    B = torch.zeros((N + 1, N + 1), dtype=torch.float64)
    for n in range(2, N + 1):   # integrated twice; modes N-1 and N of the right-hand side are dropped
        B[n, n - 2] = (2.0 if n == 2 else 1.0) / (4.0 * n * (n - 1))
        if n <= N - 2:
            B[n, n] = -1.0 / (2.0 * (n * n - 1))
        if n + 2 <= N - 2:
            B[n, n + 2] = 1.0 / (4.0 * n * (n + 1))
    B = B.cuda()
    top = torch.ones(N + 1, dtype=torch.float64, device="cuda")
    bot = torch.where(torch.arange(N + 1, device="cuda") % 2 == 0, 1.0, -1.0).double()
    eye = torch.diag(torch.cat([torch.zeros(2), torch.ones(N - 1)]).double()).cuda() * dyde ** 2
    out = torch.empty_like(x)
    for i in range(nxh):
        A = eye[None] - (k2[i] + p.re * var / (p.dt * th))[:, None, None] * B[None]
        A[:, 0], A[:, 1] = top, bot
        s = r[i] @ B.T.to(r.dtype)
        s[:, :2] = 0
        sol = torch.linalg.solve(A, torch.stack([s.real, s.imag], dim=-1))
        out[i] = torch.complex(sol[..., 0], sol[..., 1])
    # norm: the kx = 0 plane made Hermitian in kz, the Nyquist kz zeroed
    m = 0.5 * (out[0, 1:nz // 2] + torch.flip(out[0, nz // 2 + 1:], [0]).conj())
    out[0, 1:nz // 2] = m
    out[0, nz // 2 + 1:] = torch.flip(m, [0]).conj()
    out[0, 0] = out[0, 0].real.to(out.dtype)
    out[:, nz // 2] = 0
    return out


def _exact_linear(case, seed):
    p, f = _routine_fields(case, seed)
    om, sc = f["OMY"], f["SCALAR"]
    for _ in range(case["steps"]):
        om = _exact_advance(p, om, f["GN"], f["GNM1"], 1.0)
        sc = _exact_advance(p, sc, f["SCN"], f["SCNM1"], p.diff)
    return {"V": None, "U": None, "OMY": om, "SCALAR": sc}


def exact(case, seed):
    kind = case["kind"]
    if kind == "xyzfft":
        return _exact_xyzfft(case, seed)
    if kind == "nonlinear":
        return _exact_nonlinear(case, seed)
    if kind == "linear":
        return _exact_linear(case, seed)
    return None   # whole time steps: the scheme itself, over many steps
