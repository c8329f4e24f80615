"""Grids off the compiled lengths: the warp-per-column solves on cached tables at the smallest, ordinary
and largest ny of each register layout, and both step paths at every x register layout they gained."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, inputs
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu

ROUTINE_TOL = 1e-12   # the bars of the compiled lengths: a routine, a whole run of a few steps
RUN_TOL = 1e-10


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


@pytest.mark.parametrize("ny", [8, 30, 36, 60, 80, 100, 120, 144, 160, 180, 270])
def test_warp_column_solves(rt, oracle_mod, ny):
    p = kc.cfg_small(6, ny, 8)   # 24 columns: a last block with none to spare; nxh = 3
    g, o = rt.KmmContext(p), oracle_mod.Oracle(p)
    rng = np.random.default_rng(ny)

    def put(name, a):
        g.upload(name, a)
        o.set(name, a)

    def wall():
        return rng.standard_normal((p.nz, p.nx // 2)) + 1j * rng.standard_normal((p.nz, p.nx // 2))

    for gv in (p.re / (p.dt * p.theta), 0.0):
        put("WRKC", kc.random_spectral(rng, p, hermitian=False))
        put("BCTOP", wall())
        put("BCBOT", wall())
        g.call("solve", "WRKC", gv, 0)
        o.call("solve", "WRKC", gv, 0)
        assert kc.rel_err(g.download("WRKC"), o.get("WRKC")) <= ROUTINE_TOL
    for bc in ((1.0, 0.0, 1.0, 0.0), (0.0, 1.0, 0.0, 1.0), (1.0, 0.3, 0.7, 0.5)):
        put("WRKC", kc.random_spectral(rng, p, hermitian=False))
        put("BCTOP", wall())
        put("BCBOT", wall())
        g.call("penta", "WRKC", 2800.0, 0, *bc)
        o.call("penta", "WRKC", 2800.0, 0, *bc)
        assert kc.rel_err(g.download("WRKC"), o.get("WRKC")) <= ROUTINE_TOL


@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("grid", [(24, 24, 24), (80, 36, 20), (144, 16, 12), (160, 20, 12), (12, 160, 24), (20, 100, 40)])
def test_steps_match_oracle(rt, oracle_mod, grid, fused):
    p = kc.cfg_small(*grid, dt=1e-3, scalar_on=1, diff=1.0, scalar_bc=1, scalar_q=0.5, npart=50)
    fields = kc.initial_fields(p, amp=0.1, kmax=2, seed=31)
    parts = inputs.uniform_particles(p.npart, p.xl, p.yl, p.zl, p.ap, 7)
    g, o = rt.KmmContext(p), oracle_mod.Oracle(p)
    g.call("set_option", abi.OPT_FUSED, fused)
    for c, put in ((g, g.upload), (o, o.set)):
        kc.load_initial(c, p, fields, np.zeros_like(fields[0]))
        for name, a in zip(("XPART", "YPART", "ZPART"), parts):
            put(name, a)
        assert c.initial() == 0
    for _ in range(3):
        assert g.step() == 0
        assert o.step() == 0
    for name in ("V", "OMY", "FN", "GN", "U0", "W0", "SCALAR", "SCN", "XPART", "YPART"):
        assert kc.rel_err(g.download(name), o.get(name)) <= RUN_TOL, name
