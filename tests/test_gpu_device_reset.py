"""Flux calls on host arrays keep pinned slots and a memory pool between calls; a caller's device reset ends
both, and the calls after it allocate anew.  In a process of its own, which holds nothing else on the device."""
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
S.lib()
path = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l)   # the library's own runtime
cudart = ctypes.CDLL(path)
n = 60000   # arrays of 0.5 to 3.8 MB: several slots
rng = np.random.default_rng(1)
nrm = np.eye(3)[rng.integers(0, 3, n)]
q = [np.c_[rng.uniform(0.5, 2, n), rng.normal(size=(n, 3)), rng.uniform(0.5, 2, n), rng.normal(size=(n, 3))] for _ in range(2)]
first = S.chlld_batch(3, nrm, q[0], q[1])
for _ in range(3):
    assert cudart.cudaDeviceReset() == 0
    for _ in range(2):
        again = S.chlld_batch(3, nrm, q[0], q[1])
        assert all((a == b).all() for a, b in zip(first, again))
print("ok")
"""


def test_flux_calls_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]
