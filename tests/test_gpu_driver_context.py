"""Flux calls on host arrays in a context that the caller made by the driver API (not the device's primary one):
they run in it and leave it current.  In a process of its own."""
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
import set_b200 as S
n = 60000   # arrays of 0.5 to 3.8 MB: several threads
rng = np.random.default_rng(1)
nrm = np.eye(3)[rng.integers(0, 3, n)]
q = [np.c_[rng.uniform(0.5, 2, n), rng.normal(size=(n, 3)), rng.uniform(0.5, 2, n), rng.normal(size=(n, 3))] for _ in range(2)]
first = S.chlld_batch(3, nrm, q[0], q[1])
cuda = ctypes.CDLL("libcuda.so.1")
dev, own, now = ctypes.c_int(), ctypes.c_void_p(), ctypes.c_void_p()
assert cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cuda.cuCtxCreate_v2(ctypes.byref(own), 0, dev) == 0
for _ in range(2):
    again = S.chlld_batch(3, nrm, q[0], q[1])
    assert all((a == b).all() for a, b in zip(first, again))
    assert cuda.cuCtxGetCurrent(ctypes.byref(now)) == 0 and now.value == own.value
print("ok")
"""


def test_flux_calls_in_a_driver_context():
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]
