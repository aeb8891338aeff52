"""Flux calls on arrays in pinned memory, which the driver copies itself: the results of pageable arrays, and
no slower than those (arrays handed over as 8-byte rows took four times as long; 1.5 times is the limit here,
0.4 was measured)."""
import ctypes as C
import time

import numpy as np
import pytest

import set_b200 as S

pytestmark = pytest.mark.gpu


def run(arrays):
    p = [a.ctypes.data_as(C.POINTER(C.c_int32 if a.dtype == np.int32 else C.c_double)) for a in arrays]
    best = 1e9
    for _ in range(6):
        t = time.perf_counter()
        assert S.lib().setb_chlld_batch(len(arrays[0]), 3, 0, 0, p[0], None, *p[1:]) == 0
        best = min(best, time.perf_counter() - t)
    return best


def test_pinned_arrays():
    import torch
    n = 100000
    rng = np.random.default_rng(5)
    q = [np.c_[rng.uniform(0.5, 2, n), rng.normal(size=(n, 3)), rng.uniform(0.5, 2, n), rng.normal(size=(n, 3))]
         for _ in range(2)]
    pageable = [np.eye(3)[rng.integers(0, 3, n)], q[0], q[1], np.zeros((n, 8)), np.zeros((n, 3)), np.zeros(n, np.int32)]
    pageable = [np.ascontiguousarray(a) for a in pageable]
    keep = [torch.from_numpy(a).pin_memory() for a in pageable]
    pinned = [t.numpy() for t in keep]
    t0, t1 = run(pageable), run(pinned)
    for a, b in zip(pageable, pinned):
        np.testing.assert_array_equal(a, b)
    assert t1 <= 1.5 * t0
