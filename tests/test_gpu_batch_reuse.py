"""A batch's memory in use again: a solve admitted where a retired one of another shape lay (the same
footprint, so the same addresses, its tensor maps among them) takes the same steps as in a new batch."""
import numpy as np
import pytest

import set_b200 as S

pytestmark = pytest.mark.gpu

SHAPES = [(64, 48, 40), (40, 64, 48), (48, 40, 64), (80, 32, 48)]   # 122880 cells each


def solve(batch, shape, precision, steps):
    opts = S.step_opts(precision=precision)
    slot = batch.add(S.cart_desc(shape, dt_init=1e-3), S.lism_ic(seed=3, pert_amp=0.05), opts)
    batch.step(steps)
    u = batch.conserved(slot)
    batch.remove(slot)
    return u


@pytest.mark.parametrize("precision", [0, 1])
def test_a_solve_in_a_retired_solves_memory(precision):
    want = []
    for shape in SHAPES:
        with S.Batch(1, precision=precision) as b:
            want.append(solve(b, shape, precision, 3))
    with S.Batch(1, precision=precision) as b:
        for _ in range(2):
            for shape, u in zip(SHAPES, want):
                np.testing.assert_array_equal(solve(b, shape, precision, 3), u)
