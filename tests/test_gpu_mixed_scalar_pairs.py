"""A mixed-precision step's scalar terms have the same bits with a polymer that exerts no force (beta = 1) as without
one: the x transforms carry two fields each, so the input fields must keep their places in the pairs."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, runtime
from tests.kmm_cases import cfg_small, initial_fields, load_initial

pytestmark = pytest.mark.gpu


STATE = ("V", "OMY", "FN", "FNM1", "GN", "GNM1", "U0", "W0", "H1N", "H1NM1", "H3N", "H3NM1", "SCALAR", "SCN", "SCNM1")


@pytest.mark.parametrize("grid", [(32, 32, 32), (64, 96, 32)])
def test_scalar_bits_do_not_depend_on_the_polymer(grid):
    out = []
    for polymer in (0, 1):
        kw = dict(polymer_on=1, zlmax=30.0, tpoly=20.0, qbeta=1.0, diffpoly=0.3) if polymer else {}
        p = cfg_small(*grid, dt=0.001, precision=1, scalar_on=1, diff=1.0, scalar_bc=1, **kw)
        fields = initial_fields(p)
        with runtime.KmmContext(p) as c:
            c.call("set_option", abi.OPT_FUSED, 0)
            c.call("set_option", abi.OPT_DERIVED_INPUTS, 0)   # inputs in the list's own order
            load_initial(c, p, fields, 0.1 * fields[0])
            c.initial()
            if out:   # the initial nonlinear terms are formed by another x stage with polymer: start from the same
                for k, a in state.items():
                    c.upload(k, a)
            state = {k: c.download(k) for k in STATE}
            for _ in range(3):
                c.step()
            out.append({k: c.download(k) for k in STATE})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
