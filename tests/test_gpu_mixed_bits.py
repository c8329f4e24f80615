"""Mixed-precision runs repeat bit for bit: from one state on every way a step can be launched, and the routines that form
their initial state are the general sequences (cderiv, then the pointwise terms) bit for bit."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, runtime
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu

STATE = ("V", "OMY", "FN", "GN", "U0", "W0", "SCALAR", "SCN")


@pytest.mark.parametrize("polymer", [0, 1])
@pytest.mark.parametrize("grid", [(32, 32, 32), (64, 96, 32)])
def test_runs_repeat(grid, polymer):
    kw = dict(polymer_on=1, zlmax=30.0, tpoly=20.0, qbeta=0.9, diffpoly=0.3) if polymer else {}
    p = kc.cfg_small(*grid, dt=0.001, precision=1, scalar_on=1, diff=1.0, scalar_bc=1, **kw)
    fields = kc.initial_fields(p)
    out = []
    for how in ("run", "again", "steps", "kernels", "ensemble"):
        with runtime.KmmContext(p) as c, runtime.KmmContext(p) as d:
            c.call("set_option", abi.OPT_GRAPH, 0 if how == "kernels" else 1)
            for x in (c, d):
                kc.load_initial(x, p, fields, 0.1 * fields[0])
                x.initial()
            if how == "ensemble":
                assert runtime.ensemble_run([c, d], 4) == [0, 0]
            elif how == "steps":
                for _ in range(4):
                    c.step()
            else:
                c.run(4)
            out.append({k: c.download(k) for k in STATE})
    for o in out[1:]:
        for k in STATE:
            assert np.array_equal(o[k], out[0][k]), k


def _i(k, a):
    """i k a with the products rounded singly."""
    return -k * a.imag + 1j * (k * a.real)


@pytest.mark.parametrize("grid", [(32, 32, 32), (64, 96, 32)])
def test_routines_are_the_general_sequences(grid):
    p = kc.cfg_small(*grid, precision=1, scalar_on=1, diff=1.0)
    rng = np.random.default_rng(5)
    f = {k: kc.random_spectral(rng, p) for k in ("U", "V", "W", "SCALAR")}
    with runtime.KmmContext(p) as c:
        c.upload("SCALAR", np.ones_like(f["SCALAR"]))
        c.call("gradscl")
        kx, kz = c.download("SCLX").imag, c.download("SCLZ").imag
        d = {}
        for k, a in f.items():
            c.upload(k, a)
            c.call("cderiv", k, "T1")
            d[k] = c.download("T1")
        c.call("gradscl")
        c.call("vort")
        want = {"SCLX": _i(kx, f["SCALAR"]), "SCLY": d["SCALAR"], "SCLZ": _i(kz, f["SCALAR"]),
                "OMZ": _i(kx, f["V"]) - d["U"], "OMX": d["W"] - _i(kz, f["V"])}
        for k, a in want.items():
            assert np.array_equal(c.download(k), a), k
        c.call("cderiv", "V", "T1")
        c.call("cderiv", "T1", "T2")
        d2 = c.download("T2")
        c.call("phi_from_v")
        w2 = kx * kx + kz * kz
        phi = (d2.real - w2 * f["V"].real) + 1j * (d2.imag - w2 * f["V"].imag)
        assert np.array_equal(c.download("V"), phi)


@pytest.mark.parametrize("ny", [32, 64, 96, 128])
def test_column_solves_do_not_depend_on_the_precision(ny):
    """The fused column kernels solve in FP64 in both precisions: one step from one state leaves the same bits, whatever
    register budget each instance is compiled for."""
    out = []
    for precision in (0, 1):
        p = kc.cfg_small(32, ny, 32, dt=0.001, precision=precision, scalar_on=1, diff=1.0, scalar_bc=1)
        rng = np.random.default_rng(5)
        with runtime.KmmContext(p) as c:
            fields = kc.initial_fields(p)
            kc.load_initial(c, p, fields, 0.1 * fields[0])
            c.initial()
            for k in ("V", "OMY", "FN", "FNM1", "GN", "GNM1", "SCALAR", "SCN", "SCNM1"):
                c.upload(k, kc.random_spectral(rng, p))
            c.call("step", allow=(abi.ERR_CFL,))
            out.append({k: c.download(k) for k in ("V", "OMY", "SCALAR")})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
