"""A batch's march length: one that the caller sets is the one that runs, whatever its members, the tuner
keeps a length that it has timed, and the batch reports what runs.  With fewer work items than SMs the
reported grid is the number of items, which shows the length that ran."""
import numpy as np
import pytest

import set_b200 as S

pytestmark = pytest.mark.gpu

NZ = 41


def batch(precision):
    b = S.Batch(2, precision=precision)
    slot = b.add(S.cart_desc((20, 7, NZ), dt_init=1e-3), S.lism_ic(seed=3), S.step_opts(precision=precision))
    return b, slot


@pytest.mark.parametrize("precision", [0, 1])
def test_the_length_that_is_set_runs(precision):
    want = None
    for lz in (1, 2, 8, 40, 41, 1 << 20):
        b, slot = batch(precision)
        with b:
            b.set_tiling(lz)
            assert b.info()["lz"] == min(lz, NZ)
            b.step(2)
            chunks = -(-NZ // min(lz, NZ))
            assert b.info()["grid"] == -(-NZ // -(-NZ // chunks))   # chunks as even as they come
            u = b.conserved(slot)
        want = u if want is None else want
        np.testing.assert_array_equal(u, want)


def test_the_tuned_length_runs():
    b, slot = batch(1)
    with b:
        own = b.info()["lz"]
        t = b.tune(reps=2)
        runs = b.info()["lz"]
        assert runs == min(t["lz"], NZ) or (t["lz"] == 32 and runs == own)
        b.step(1)
        chunks = -(-NZ // runs)
        assert b.info()["grid"] == -(-NZ // -(-NZ // chunks))
