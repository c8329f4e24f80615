"""The diagonal polymer stresses: q_ii = zb (f c_ii - 1) cancels, so its error is measured against the terms it is made
of."""
import numpy as np
import pytest

from polymer_dns_b200 import runtime
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import pyoracle
    pyoracle.build()
    return pyoracle


@pytest.mark.parametrize("itarget", [0, 2])
def test_diagonal_stresses(oracle_mod, itarget):
    p = kc.cfg_small(32, 32, 32, scalar_on=1, polymer_on=1, diff=1.0, scalar_bc=1, scalar_q=1.0, zlmax=30.0, tpoly=20.0,
                     qbeta=0.9, diffpoly=1000.0, itarget=itarget, alpha_poly=0.7)
    fields = kc.initial_fields(p, amp=0.05, seed=4)
    g, o = runtime.KmmContext(p), oracle_mod.Oracle(p)
    for c in (g, o):
        kc.load_initial(c, p, fields, 0.1 + np.abs(fields[0]))
        assert c.initial() == 0
        assert c.run(4) == 0
    zb = (1.0 - p.qbeta) / (p.re * p.qbeta * p.tpoly)
    for m in ("11", "22", "33"):
        q, want = g.download("QP" + m), o.get("QP" + m)
        # a run's 1e-10 of f c_ii, whose mean mode is near 1 (beta of the scalar: zb grows as 1 / beta - 1)
        scale = zb if itarget == 0 else np.abs(want).max() / max(np.abs(o.get("STR%sN" % m)).max(), 1e-300)
        assert np.abs(q - want).max() <= 1e-10 * scale * (1.0 + np.abs(o.get("STR%sN" % m)).max()), m
