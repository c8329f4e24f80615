"""The forms that mixed-precision contexts use where FP64 ones take a faster route with another rounding: the
initial transform with one line per transform, and the general column operators."""
import numpy as np
import pytest

from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu

TOL = 1e-12   # a routine


@pytest.fixture(scope="module")
def rt():
    from polymer_dns_b200 import build, runtime
    build.build()
    return runtime


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import pyoracle
    pyoracle.build()
    return pyoracle


@pytest.mark.parametrize("nx,ny,nz", [(32, 32, 32), (32, 96, 64), (128, 64, 32), (64, 128, 96)])
def test_routines_of_a_mixed_context(rt, oracle_mod, nx, ny, nz):
    p = kc.cfg_small(nx, ny, nz, scalar_on=1, diff=1.0, precision=1)
    g, o = rt.KmmContext(p), oracle_mod.Oracle(kc.cfg_small(nx, ny, nz, scalar_on=1, diff=1.0))
    rng = np.random.default_rng(ny)

    def put(name, a):
        g.upload(name, a)
        o.set(name, a)

    def both(*call, check):
        g.call(*call)
        o.call(*call)
        for name in check:
            assert kc.rel_err(g.download(name), o.get(name)) <= TOL, (call, name)

    put("INITU", rng.standard_normal((nx, nz, ny + 1)))
    both("xyzfft", "U", "INITU", check=("U",))
    for name in ("V", "W", "OMY", "FN", "FNM1", "SCALAR"):
        put(name, kc.random_spectral(rng, p))
    for name in ("U0", "W0"):
        put(name, rng.standard_normal(ny + 1) * np.exp(-0.3 * np.arange(ny + 1)))
    both("gfcn", check=("GF1", "DENOM"))
    both("influence", check=("V", "C1", "C2"))
    both("vort", check=("OMX", "OMZ"))
    both("gradscl", check=("SCLX", "SCLY", "SCLZ"))
    both("phirhs", "SCALAR", "FN", "FNM1", 0.7, check=("SCALAR",))
    both("phi_from_v", check=("V",))
    put("V", kc.random_spectral(rng, p))
    both("veloc", check=("U", "W", "V"))
