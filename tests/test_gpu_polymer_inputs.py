"""The polymer step's reduced inputs (six conformation components and their gradients, the scalar only where beta
depends on it) and q_ij formed from the stress coefficients (constant beta) or transformed (beta of the scalar)."""
import numpy as np
import pytest

from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu

TOL = 1e-10   # a run


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


@pytest.mark.parametrize("itarget", [0, 1, 2])
@pytest.mark.parametrize("grid", [(32, 32, 32), (20, 36, 12)])
def test_polymer_steps(rt, oracle_mod, grid, itarget):
    p = kc.cfg_small(*grid, scalar_on=1, polymer_on=1, diff=1.0, scalar_bc=1, scalar_q=1.0, zlmax=30.0, tpoly=20.0,
                     qbeta=0.9, diffpoly=1000.0, itarget=itarget, alpha_poly=0.7)
    fields = kc.initial_fields(p, amp=0.05, seed=4)
    g, o = rt.KmmContext(p), oracle_mod.Oracle(p)
    for c in (g, o):
        kc.load_initial(c, p, fields, 0.1 + np.abs(fields[0]))
        assert c.initial() == 0
        assert c.run(4) == 0
    # (the diagonal q_ii = zb (f c_ii - 1) cancels to 1e-3 of its terms here; it takes the same path)
    for name in ("V", "OMY", "FN", "GN", "SCALAR", "C11", "C12", "C13", "C22", "C23", "C33", "C23N", "STR12N",
                 "QP12", "QP13", "QP23"):
        assert kc.rel_err(g.download(name), o.get(name)) <= TOL, name
