"""A run's host thread sleeps between its looks at the step's report where the device's scheduling flag asks for it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, sys, time
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
dev = ctypes.c_int()
assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuDevicePrimaryCtxSetFlags_v2(dev, 4) == 0   # CU_CTX_SCHED_BLOCKING_SYNC
sys.path.insert(0, %r)
from polymer_dns_b200 import runtime
from tests.kmm_cases import cfg_small, initial_fields, load_initial
p = cfg_small(128, 128, 128, dt=0.001)
c = runtime.KmmContext(p)
load_initial(c, p, initial_fields(p))
c.initial()
c.run(5)
t, u = time.perf_counter(), time.process_time()
c.run(400)
print("share", (time.process_time() - u) / (time.perf_counter() - t))
c.close()
"""


def test_blocking_flag_frees_the_core():
    out = subprocess.run([sys.executable, "-c", CHILD % ROOT], cwd=ROOT, capture_output=True, text=True, timeout=240)
    assert out.returncode == 0, out.stderr[-2000:]
    share = float(out.stdout.split("share")[1])
    # a polling thread uses the whole core; a sleeping one the launches and one look in 20 us or more
    assert share < 0.5, share
