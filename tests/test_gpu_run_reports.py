"""Runs that overlap a step with the next one's launch: the flow-rate correction, and a wait that ran out behind a step's
report (found by the host through the injection; no device wait runs out)."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, runtime
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu

NAMES = ("V", "OMY", "FN", "GN", "U0", "W0")


def _ctx(seed=3, **kw):
    p = kc.cfg_small(32, 32, 32, **kw)
    c = runtime.KmmContext(p)
    kc.load_initial(c, p, kc.initial_fields(p, amp=0.1, seed=seed))
    assert c.initial() == 0
    return c


def _same(a, b):
    for k in NAMES:
        assert np.array_equal(a.download(k), b.download(k)), k
    sa, sb = a.stats(), b.stats()
    assert (sa.it, sa.cflmax, sa.umax, sa.dpdx) == (sb.it, sb.cflmax, sb.umax, sb.dpdx)


def _bind(c):
    """Host arrays as the home of the prognostic fields."""
    home = {k: np.asfortranarray(c.download(k)) for k in ("V", "FN", "FNM1", "OMY", "GN", "GNM1", "U0", "H1N", "H1NM1",
                                                          "W0", "H3N", "H3NM1")}
    for k, a in home.items():
        c.bind_host(k, a.ctypes.data, a.nbytes)
    return home


def _advance(how, c, other, n, allow=()):
    if how == "run":
        return c.call("run", n, allow=allow)
    if how == "host":
        return c.run_host(n, allow=allow)
    st = runtime.ensemble_run([c, other], n)
    assert st[1] == abi.OK and (st[0] == abi.OK or st[0] in allow)
    return st[0]


@pytest.mark.parametrize("how", ["run", "host", "ensemble"])
def test_constant_flow_rate(how):
    a, b, other = (_ctx(flow_rate=1.05, seed=s) for s in (3, 3, 4))
    home = _bind(a) if how == "host" else None
    assert _advance(how, a, other, 7) == 0
    for _ in range(7):
        b.step()
    _same(a, b)
    assert a.stats().dpdx != _ctx(flow_rate=0.0).stats().dpdx
    del home


# the looks of a run of three steps: each step's report, then the end of the run
@pytest.mark.parametrize("look", [1, 2, 4])
@pytest.mark.parametrize("how", ["run", "host", "ensemble"])
def test_late_timeout(how, look):
    a, b, other = _ctx(), _ctx(), _ctx(seed=4)
    home = _bind(a) if how == "host" else None
    for c in (a, b):
        _advance(how if c is a else "run", c, other, 3)   # graphs captured
    a.call("inject", abi.INJECT_LATE, look)
    assert _advance(how, a, other, 3, allow=(abi.ERR_TIMEOUT,)) == abi.ERR_TIMEOUT
    done = min(look, 3)
    assert a.stats().it == 3 + done and a.stats().status == abi.ERR_TIMEOUT
    assert _advance(how, a, other, 2) == abi.OK   # reported once, the context is usable
    b.run(done + 2)
    _same(a, b)
    del home
