"""phirhs, phi, veloc, vort, gradscl and the influence-matrix correction in their one-pass forms at every
blocked ny and at ny of the warp-per-column form, against the oracle."""
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


@pytest.mark.parametrize("theta", [0.5, 1.0])
@pytest.mark.parametrize("ny", [24, 32, 60, 64, 96, 128, 256])
def test_column_ops(rt, oracle_mod, ny, theta):
    p = kc.cfg_small(8, ny, 12, theta=theta, scalar_on=1, diff=1.0)
    g, o = rt.KmmContext(p), oracle_mod.Oracle(p)
    rng = np.random.default_rng(ny)

    def put(name, a):
        g.upload(name, a)
        o.set(name, a)

    for name in ("U", "V", "W", "OMY", "FN", "FNM1", "SCALAR", "BCTOP", "BCBOT"):
        put(name, kc.random_spectral(rng, p) if name[:2] != "BC" else np.ones((p.nz, p.nx // 2), complex))
    for name in ("U0", "W0"):
        put(name, rng.standard_normal(p.ny + 1) * np.exp(-0.3 * np.arange(p.ny + 1)))

    def both(*call, check):
        g.call(*call)
        o.call(*call)
        for name in check:
            assert kc.rel_err(g.download(name), o.get(name)) <= TOL, (call, name)

    both("gfcn", check=("GF1", "DENOM"))
    both("vort", check=("OMX", "OMZ"))
    both("gradscl", check=("SCLX", "SCLY", "SCLZ"))
    both("phirhs", "SCALAR", "FN", "FNM1", 0.7, check=("SCALAR",))
    assert not g.download("BCTOP").any() and not g.download("BCBOT").any()
    put("V", kc.random_spectral(rng, p))
    both("influence", check=("V", "C1", "C2"))
    put("V", kc.random_spectral(rng, p))
    both("phi_from_v", check=("V",))
    put("V", kc.random_spectral(rng, p))
    both("veloc", check=("U", "W", "V"))
