"""The x stage with one block per row (mx = 576, no polymer or body) against the oracle: three field pairs, and five with
a scalar and tracers."""
import numpy as np
import pytest

from polymer_dns_b200 import inputs, runtime
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu

TOL = 1e-10   # a run


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import pyoracle
    pyoracle.build()
    return pyoracle


# mz = 24 and 18 rows of 576 points; 576 is no multiple of the 160 threads of five pairs
@pytest.mark.parametrize("scalar,npart,flow_select,scalar_q", [(0, 0, 1, 0.0), (0, 40, 0, 0.0), (1, 0, 1, 0.0), (1, 40, 1, 0.7),
                                                               (1, 0, 0, 0.7)])
@pytest.mark.parametrize("grid", [(384, 32, 16), (384, 20, 12)])
def test_rows_of_576(oracle_mod, grid, scalar, npart, flow_select, scalar_q):
    kw = dict(scalar_on=1, diff=1.0, scalar_bc=1, scalar_q=scalar_q) if scalar else {}
    p = kc.cfg_small(*grid, dt=0.002, npart=npart, ap=1e-3, flow_select=flow_select, **kw)
    fields = kc.initial_fields(p, amp=0.05, seed=6)
    g, o = runtime.KmmContext(p), oracle_mod.Oracle(p)
    for c in (g, o):
        kc.load_initial(c, p, fields, 0.1 + 0.2 * np.abs(fields[0]) if scalar else None)
        if npart:
            for name, a in zip(("XPART", "YPART", "ZPART"), inputs.uniform_particles(npart, p.xl, p.yl, p.zl, p.ap, 5)):
                (c.upload if c is g else c.set)(name, a)
        assert c.initial() == 0
        assert c.run(3) == 0
    names = ["V", "OMY", "FN", "GN", "U0", "W0", "UP3D", "VP3D", "WP3D"]
    names += ["SCALAR", "SCN"] if scalar else []
    names += ["XPART", "YPART", "ZPART", "UPART", "VPART"] if npart else []
    for name in names:
        assert kc.rel_err(g.download(name), o.get(name)) <= TOL, name
    sg, so = g.stats(), o.stats()
    assert abs(sg.cflmax - so.cflmax) <= TOL * so.cflmax and abs(sg.umax - so.umax) <= TOL * so.umax
