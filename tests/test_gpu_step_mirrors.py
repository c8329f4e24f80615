"""The mirrors a step leaves current on grids with a run-time length in x or y: the fused step's u, w, omega_x,
dc/dy, c1, c2 and 3/2-grid velocities against the routine step's."""
import numpy as np
import pytest

from polymer_dns_b200 import abi, runtime
from tests.kmm_cases import cfg_small, initial_fields, load_initial, rel_err

pytestmark = pytest.mark.gpu

# nyp = 25 (one coefficient a lane), 161 (six) and 33 (blocked columns); mx = 60, 30, 108 and 240
GRIDS = [(40, 24, 12), (20, 160, 12), (72, 32, 12), (160, 20, 8)]


@pytest.mark.parametrize("scalar", [0, 1])
@pytest.mark.parametrize("grid", GRIDS)
def test_mirrors_after_a_run(grid, scalar):
    nx, ny, nz = grid
    p = cfg_small(nx, ny, nz, dt=0.002, **(dict(scalar_on=1, diff=1.0, scalar_bc=1, scalar_q=1.0) if scalar else {}))
    fields = initial_fields(p, kmax=3)
    scl = 0.1 * fields[0] if scalar else None
    names = ["U", "W", "OMX", "C1", "C2", "UP3D", "VP3D", "WP3D"] + (["SCLY"] if scalar else [])
    got = []
    for fused in (1, 0):
        with runtime.KmmContext(p) as c:
            c.call("set_option", abi.OPT_FUSED, fused)
            load_initial(c, p, fields, scl)
            c.initial()
            c.run(2)
            got.append({k: c.download(k) for k in names})
    for k in names:
        assert np.abs(got[1][k]).max() > 0.0, k
        # two steps of FP64 rounding; c1 and c2 divide by the wall derivatives' determinant
        assert rel_err(got[0][k], got[1][k]) < 1e-9, k


@pytest.mark.parametrize("grid", GRIDS)
def test_wall_rows_are_zero_after_a_step(grid):
    p = cfg_small(*grid, dt=0.002)
    with runtime.KmmContext(p) as c:
        load_initial(c, p, initial_fields(p, kmax=3))
        c.initial()
        for k in ("BCTOP", "BCBOT"):
            c.upload(k, np.ones_like(c.download(k)))
        c.run(1)
        for k in ("BCTOP", "BCBOT"):
            assert not c.download(k).any(), k
