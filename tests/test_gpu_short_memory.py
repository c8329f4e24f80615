"""Device memory that runs out while tables and buffers are built on first use (reported by the host-side injection,
nothing is really exhausted): the forms that need no such memory run, and the next build starts afresh."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, runtime
from tests.kmm_cases import cfg_small, initial_fields, load_initial, rel_err

pytestmark = pytest.mark.gpu

NAMES = ("V", "OMY", "FN", "GN", "U0", "W0")


def _run(grid, fail, fused=1, how="run", **kw):
    p = cfg_small(*grid, dt=0.002, **kw)
    with runtime.KmmContext(p) as c:
        c.call("set_option", abi.OPT_FUSED, fused)
        fields = initial_fields(p, kmax=3)
        load_initial(c, p, fields)
        c.initial()
        c.call("inject", abi.INJECT_NOMEM, fail)
        if how == "ensemble":
            assert runtime.ensemble_run([c], 2) == [abi.OK]
        else:
            c.run(2)
        first = {k: c.download(k) for k in NAMES}
        c.call("inject", abi.INJECT_NOMEM, 0)
        c.call("set_option", abi.OPT_FUSED, 1)
        c.run(1)
        return first, {k: c.download(k) for k in NAMES}


# the fused step's one allocation, and with mixed precision the second of its three twiddle tables
@pytest.mark.parametrize("grid,precision,fail", [((32, 32, 32), 0, 1), ((40, 24, 12), 0, 1), ((32, 32, 32), 1, 1),
                                                 ((32, 32, 32), 1, 3)])
def test_fused_step_without_memory_is_the_routine_step(grid, precision, fail):
    want, _ = _run(grid, 0, fused=0, precision=precision)
    _, after = _run(grid, 0, precision=precision)
    for how in ("run", "ensemble"):
        got, got_after = _run(grid, fail, how=how, precision=precision)
        for k in NAMES:
            assert np.array_equal(got[k], want[k]), (how, k)
            # the two paths' rounding over 3 steps: FP64, or (FN's floor at this grid) FP32
            assert rel_err(got_after[k], after[k]) < (1e-3 if precision else 1e-9), (how, k)


# the rj rows, the corner factors, a canonical table and the tables kept
@pytest.mark.parametrize("ny", [32, 36])
@pytest.mark.parametrize("fail", [1, 2, 4, 8, 10])
def test_solves_without_memory_for_tables(ny, fail):
    p = cfg_small(24, ny, 12)
    rng = np.random.default_rng(7)
    x = rng.standard_normal((ny + 1, 12, 12)) + 1j * rng.standard_normal((ny + 1, 12, 12))
    got = []
    for n in (0, fail):
        with runtime.KmmContext(p) as c:
            c.call("inject", abi.INJECT_NOMEM, n)
            out = []
            for _ in range(4):   # the failing call, and calls that may build again
                c.upload("V", x)
                c.call("solve", "V", 50.0, 0)
                out.append(c.download("V"))
                c.upload("OMY", x)
                c.call("penta", "OMY", 50.0, 0, 1.0, 0.0, 1.0, 0.0)
                out.append(c.download("OMY"))
            got.append(out)
    for a, b in zip(*got):
        assert np.abs(a).max() > 0.0
        assert rel_err(b, a) < 1e-10   # tabled and table-free solves of one tau system


def test_tables_only_for_configurations_that_come_back():
    """ny without blocked kernels: a solve builds its tau tables at the third call with one g, and a changing g none."""
    p = cfg_small(24, 36, 12)
    rng = np.random.default_rng(8)
    x = rng.standard_normal((37, 12, 12)) + 1j * rng.standard_normal((37, 12, 12))
    with runtime.KmmContext(p) as c:
        def solve(g):
            c.upload("V", x)
            n = c.launch_count()
            c.call("solve", "V", g, 0)
            return c.launch_count() - n, c.download("V")

        assert [solve(10.0 + m)[0] for m in range(20)] == [1] * 20
        same = [solve(5.0) for _ in range(4)]
        assert [n for n, _ in same] == [1, 1, 3, 1]   # tables, their reciprocals, the solve
        assert np.array_equal(same[0][1], same[1][1]) and np.array_equal(same[2][1], same[3][1])
        assert rel_err(same[2][1], same[0][1]) < 1e-10
