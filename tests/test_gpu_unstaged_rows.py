"""Host rows where no pinned slot can be had (a fake cudaHostAlloc that refuses them, in a process of its own): the
driver's copies give what the staged ones give, for contiguous, pitched and renumbered rows both ways."""
import os
import shutil
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

FAKE = """
#define _GNU_SOURCE
#include <dlfcn.h>
static int calls;
int cudaHostAlloc(void** p, unsigned long n, unsigned flags) {
    if (n < 256 * 1024) {   /* a handle's pinned mirror */
        void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
        return rt ? ((int (*)(void**, unsigned long, unsigned))dlsym(rt, "cudaHostAlloc"))(p, n, flags) : 2;
    }
    calls++;
    *p = 0;
    return 2;
}
int refused(void) { return calls; }
"""

SCRIPT = """
import ctypes, hashlib, os, sys
sys.path.insert(0, {root!r})
import numpy as np
import set_b200 as S
from set_b200 import facelist as FL
h = hashlib.sha256()
rng = np.random.default_rng(1)
n = 60000
nrm = np.eye(3)[rng.integers(0, 3, n)]
q = [np.c_[rng.uniform(0.5, 2, n), rng.normal(size=(n, 3)), rng.uniform(0.5, 2, n), rng.normal(size=(n, 3))] for _ in range(2)]
for a in S.chlld_batch(3, nrm, q[0], q[1]):
    h.update(a.tobytes())
desc = S.cart_desc((41, 40, 39), dt_init=1e-4)
cp = S.fill_lism(desc, S.lism_ic(seed=2, pert_amp=0.05))
with S.Solver(desc, cell_par=cp) as s:
    s.step(2, S.step_opts())
    h.update(s.conserved().tobytes())
    h.update(np.ascontiguousarray(s.get_state()[0][:, :8]).tobytes())
m = FL.box_facelist((30, 28, 26), stretch=0.3, permute_seed=3, seed=1)
par = FL.fl_params(r_src=0.2, dt_init=1e-4)
with FL.FaceListSolver(m, FL.lism_cellpar(m, seed=2, params=par), par) as s:
    s.step(2, S.step_opts())
    h.update(s.conserved().tobytes())
    h.update(np.ascontiguousarray(s.get_state()[0][:, :8]).tobytes())
fake = os.environ.get("LD_PRELOAD")
print(ctypes.CDLL(fake).refused() if fake else 0, h.hexdigest())
"""


def run(preload=None):
    env = dict(os.environ)
    env.pop("LD_PRELOAD", None)
    if preload:
        env["LD_PRELOAD"] = str(preload)
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
    refused, digest = r.stdout.split()[-2:]
    return int(refused), digest


@pytest.mark.skipif(shutil.which("gcc") is None, reason="builds the fake with gcc")
def test_rows_without_pinned_slots(tmp_path):
    src, lib = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    refused, digest = run(lib)
    assert refused > 0
    assert digest == run()[1]
