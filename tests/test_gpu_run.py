"""kmm_run and kmm_ensemble_run enqueue a step once the one before has reported: the results, the step
counter and a stop status must be those of single steps, each waited for."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, inputs
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from polymer_dns_b200 import build, runtime
    build.build()
    return runtime


def _ctx(rt, p, amp=0.1, seed=3, graph=1):
    g = rt.KmmContext(p)
    g.call("set_option", abi.OPT_GRAPH, graph)
    fields = kc.initial_fields(p, amp=amp, seed=seed)
    kc.load_initial(g, p, fields, np.zeros_like(fields[0]) if p.scalar_on else None)
    for name, a in zip(("XPART", "YPART", "ZPART"), inputs.uniform_particles(p.npart, p.xl, p.yl, p.zl, p.ap, 5)):
        if p.npart:
            g.upload(name, a)
    g.call("initial", allow=(abi.ERR_CFL,))
    return g


@pytest.mark.parametrize("grid,npart,graph", [((32, 32, 32), 100, 1), ((32, 32, 32), 0, 0), ((40, 40, 20), 100, 1)])
def test_run_equals_steps(rt, grid, npart, graph):
    p = kc.cfg_small(*grid, scalar_on=1, diff=1.0, scalar_bc=1, scalar_q=0.5, npart=npart)
    a, b = _ctx(rt, p, graph=graph), _ctx(rt, p, graph=graph)
    a.run(7)
    for _ in range(7):
        b.step()
    sa, sb = a.stats(), b.stats()
    assert (sa.it, sa.cflmax, sa.umax) == (sb.it, sb.cflmax, sb.umax)
    for name in ["V", "OMY", "FN", "FNM1", "GN", "U0", "SCALAR", "SCN"] + (["XPART", "UPART"] if npart else []):
        assert np.array_equal(a.download(name), b.download(name)), name


def test_run_stops_at_the_failing_step(rt):
    """The time step of a run far beyond CFL 1: the first step reports it and no other follows."""
    p = kc.cfg_small(32, 32, 32, dt=0.5)
    a, b = _ctx(rt, p), _ctx(rt, p)
    assert a.call("run", 5, allow=(abi.ERR_CFL,)) == abi.ERR_CFL
    assert b.call("step", allow=(abi.ERR_CFL,)) == abi.ERR_CFL
    assert a.stats().it == b.stats().it == 1
    for name in ("V", "FN", "GN", "U0"):
        assert np.array_equal(a.download(name), b.download(name)), name


def test_many_ensembles_in_turn(rt):
    """Nine ensembles of two (more parent graphs than the cache keeps) advanced in turn, against single runs."""
    p = kc.cfg_small(32, 32, 32)
    sets = [[_ctx(rt, p, seed=10 * e + m) for m in range(2)] for e in range(9)]
    for _ in range(2):
        for s in sets:
            assert rt.ensemble_run(s, 3) == [0, 0]
    for e in (0, 8):
        for m in range(2):
            lone = _ctx(rt, p, seed=10 * e + m)
            lone.run(6)
            assert sets[e][m].stats().it == 6
            for name in ("V", "OMY", "FN"):
                assert np.array_equal(sets[e][m].download(name), lone.download(name)), (e, m, name)
