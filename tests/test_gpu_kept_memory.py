"""Device memory that the library keeps between calls stays within its stated bounds."""
import numpy as np
import pytest

import set_b200 as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes():
    """Without a synchronisation: it would make the pools return what they hold above their bounds."""
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("first,second", [((64, 64, 64), (160, 160, 160)), ((120, 120, 120), (64, 64, 64))])
def test_a_batch_and_what_it_keeps_stay_within_its_budget(first, second):
    """Solves of one size fill the budget and retire, solves of another fill it again: live and kept memory
    together take no more of the device than the budget and one unit of the pool's growth (32 MB), at every
    admission and after the last solve has gone."""
    budget = 1000 * 10 ** 6
    o = S.step_opts(precision=1)
    free_bytes()
    with S.Batch(64, precision=1, hbm_budget=budget) as b:
        before = free_bytes()
        for shape in (first, second, first):
            slots = []
            while (s := b.try_add(S.cart_desc(shape, dt_init=1e-3), S.lism_ic(seed=1), o)) is not None:
                slots.append(s)
                assert before - free_bytes() <= budget + 32 * MB
            b.step(1)
            b.sync()
            assert len(slots) == budget // (b.info()["bytes_used"] // len(slots))
            for s in slots:
                b.remove(s)
            b.sync()
            assert before - free_bytes() <= budget + 32 * MB


def test_kept_memory_does_not_stand_in_the_way_of_a_solver():
    """A batch that keeps 3.4 GB of a retired solve, the device filled but for 2 GB: a handle of 3.0 GB is
    still created, steps, and the batch goes on."""
    import torch
    o = S.step_opts(precision=1)
    big = S.cart_desc((272, 272, 272))   # 168 B a cell in a batch
    with S.Batch(2, precision=1) as b:
        s = b.add(big, S.lism_ic(seed=1), o)
        b.step(1)
        b.remove(s)
        b.sync()
        filler = torch.empty(free_bytes() - (2 << 30), dtype=torch.uint8, device="cuda")
        desc = S.cart_desc((288, 288, 288))   # 128 B a cell
        with S.Solver(desc, ic=S.lism_ic(seed=1)) as solver:
            assert solver.step(1, S.step_opts()) > 0
        del filler
        torch.cuda.empty_cache()
        s = b.add(big, S.lism_ic(seed=1), o)
        b.step(1)
        assert b.status(s).steps == 1


def test_flux_calls_keep_64_mb():
    """A call of 1.5 million faces (372 MB on the device) after one of a few: 64 MB may stay, and one unit of
    the pool's growth (32 MB)."""
    def call(n):
        q = np.tile([1.0, 0.1, 0.2, 0.3, 1.0, 0.5, 0.4, 0.3], (n, 1))
        return S.chlld_batch(3, np.tile([1.0, 0.0, 0.0], (n, 1)), q, q)
    call(10)
    before = free_bytes()
    call(1500000)
    assert before - free_bytes() <= 96 * MB
