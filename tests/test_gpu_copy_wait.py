"""With a wait limit of one check, every plane copy is issued right before its wait, so the waits of the
march itself run out and the second wait delivers the plane: the state is the one of a normal run."""
import numpy as np
import pytest

import set_b200 as S
from set_b200.slab import SlabSolver, _DeviceArray

pytestmark = pytest.mark.gpu

SHAPE = (1024, 88, 64)   # 32 x 8 columns: marches of all 64 planes
HEAD_WORDS, TIMEOUTS = 13, 12   # clock (48 bytes) and counters; the last counter: waits that ran out


def test_every_wait_of_a_march_runs_out_and_recovers():
    import torch
    desc = S.cart_desc(SHAPE, dt_init=1e-3)
    cp = S.fill_lism(desc, S.lism_ic(seed=5, pert_amp=0.05))
    o = S.step_opts()
    out, waits = [], []
    for limit in (0, -1):
        with SlabSolver(desc, 0, SHAPE[2], cp) as s:
            S.lib().setb_set_copy_wait(s.h, limit)
            s.stage(1, o)
            s.stage(2, o)
            out.append(s.conserved())
            head = s.dt_tensor().data_ptr()
            words = torch.as_tensor(_DeviceArray(head, (HEAD_WORDS,), (1,)), device="cuda").clone()
            waits.append(int(words.view(torch.int64)[TIMEOUTS]))
    np.testing.assert_array_equal(out[0], out[1])
    # the warp that issues a copy cannot find it landed: 32 lanes of 64 planes, 256 columns, two stages
    assert waits[0] == 0 and waits[1] >= 2 * 256 * 64 * 32
