"""The tracers' interpolation cells where the cheap estimate of the lookup ends: positions on either side of
every cell boundary, in each direction, against the oracle's expressions."""
import numpy as np
import pytest

from polymer_dns_b200 import inputs
from tests import kmm_cases as kc

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("ny", [8, 64, 128, 1000])
@pytest.mark.parametrize("eps", [1e-13, 1e-11, 1e-8, 1e-4])   # inside and outside the estimate's margins
def test_cells_beside_every_boundary(rt, oracle_mod, ny, eps):
    nx, nz = 20, 12
    base = dict(nx=nx, ny=ny, nz=nz)
    p0 = kc.cfg_small(**base)
    y = inputs.grid_y(ny)[1:-1]
    x = np.arange(1, 30) * p0.xl / 30
    z = np.arange(1, 18) * p0.zl / 18
    n = 2 * (len(x) + len(y) + len(z))
    rng = np.random.default_rng(ny)
    P = np.stack([rng.uniform(0, p0.xl, n), rng.uniform(-0.99, 0.99, n), rng.uniform(0, p0.zl, n)])
    row = 0
    for d, b in ((0, x), (1, y), (2, z)):
        for s in (-1, 1):
            P[d, row:row + len(b)] = b * (1 + s * eps) if d != 1 else b + s * eps * (1 - b * b)
            row += len(b)
    p = kc.cfg_small(npart=n, **base)
    g, o = rt.KmmContext(p), oracle_mod.Oracle(p)
    for name, a in zip(("XPART", "YPART", "ZPART"), P):
        g.upload(name, a)
        o.set(name, a)
    assert np.array_equal(g.tracer_cells(), o.tracer_cells())
