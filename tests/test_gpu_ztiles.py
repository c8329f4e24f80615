"""The z transforms' CTA tiles (two kx by two y) and their split over blocks: an odd number of kx (the
last tile clipped), and grids on either side of the field-splitting rule, against plain loads."""
import numpy as np
import pytest

from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from polymer_dns_b200 import build, runtime
    build.build()
    return runtime


@pytest.mark.parametrize("grid,scalar,prec", [((54, 32, 64), 1, 0), ((54, 64, 128), 0, 0),   # 27 kx
                                              ((32, 32, 64), 1, 0),     # 136 tiles: one field per block
                                              ((64, 64, 32), 1, 0),     # 528 tiles: two
                                              ((128, 64, 32), 1, 0),    # 1056 tiles: all four
                                              ((128, 64, 32), 0, 0), ((128, 64, 32), 1, 1)])
def test_tiles_match_plain_loads(rt, grid, scalar, prec):
    """Same FFTs and operation order on both sides, so the states agree to the rounding of fused
    multiply-adds after 4 steps: 1e-13 relative in FP64, 1e-5 with FP32 intermediates."""
    kw = dict(scalar_on=scalar, diff=1.0, scalar_bc=1, scalar_q=0.5) if scalar else {}
    p = kc.cfg_small(*grid, precision=prec, **kw)
    fields = kc.initial_fields(p, amp=0.1, seed=21)
    sc = np.zeros_like(fields[0]) if scalar else None
    state = []
    for ztma in (1, 0):
        g = rt.KmmContext(p)
        g.call("set_option", 4, ztma)
        kc.load_initial(g, p, fields, sc)
        assert g.initial() == 0
        assert g.run(4) == 0
        state.append({n: g.download(n) for n in ["V", "OMY", "FN", "GN", "U0", "W0"] + (["SCALAR", "SCN"] if scalar else [])})
        g.close()
    for name, a in state[0].items():
        e = kc.rel_err(a, state[1][name])
        assert e <= (1e-13 if prec == 0 else 1e-5), (name, e)
