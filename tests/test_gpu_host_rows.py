"""Transfers between pageable host memory and the device (rows staged by a team of threads) against
the driver's own copies from and to pinned memory: the same bytes, at row counts around a staging
slot (8192 rows of 64 bytes), with odd row pitches, renumbered, and from several threads at once."""
import threading

import numpy as np
import pytest

import set_b200 as S
from set_b200 import facelist as FL

pytestmark = pytest.mark.gpu


def pinned(shape):
    import torch
    return torch.zeros(shape, dtype=torch.float64).pin_memory().numpy()


def random_state(n, seed):
    rng = np.random.default_rng(seed)
    cp = rng.uniform(0.5, 2.0, (n, 16))
    return cp


@pytest.mark.parametrize("shape", [(1, 1, 1), (63, 65, 2), (64, 64, 2), (91, 9, 10), (64, 64, 4), (129, 64, 63)])
def test_cartesian_rows_match_pinned_copies(shape):
    n = shape[0] * shape[1] * shape[2]
    cp = random_state(n, 5)
    cp_pinned = pinned((n, 16))
    cp_pinned[:] = cp
    desc = S.cart_desc(shape, r_src=0.0)
    with S.Solver(desc, cell_par=cp) as a, S.Solver(desc, cell_par=cp_pinned) as b:
        np.testing.assert_array_equal(a.conserved(), b.conserved())
        out, out_pinned = np.full((n, 16), -7.0), pinned((n, 16))
        a.get_state(out)
        a.get_state(out_pinned)
        np.testing.assert_array_equal(out[:, :8], out_pinned[:, :8])
        assert (out[:, 8:] == -7.0).all()
        a.set_state(random_state(n, 6))
        b.set_state(random_state(n, 6))
        np.testing.assert_array_equal(a.conserved(), b.conserved())
        u = pinned((8,) + shape[::-1])
        S.lib().setb_get_conserved(a.h, S._p(u))
        np.testing.assert_array_equal(a.conserved(), u)


@pytest.mark.parametrize("shape", [(3, 2, 1), (32, 32, 8), (40, 33, 29)])
def test_renumbered_rows_round_trip(shape):
    m = FL.box_facelist(shape, permute_seed=3, seed=1)
    n = FL.box_facelist(shape, seed=1)
    cp = random_state(n.n_cell, 8)
    key = lambda x: np.lexsort((x[:, 0], x[:, 1], x[:, 2]))
    im, i0 = key(m.cell_center), key(n.cell_center)
    cpm = np.zeros_like(cp)
    cpm[im] = cp[i0]
    par = FL.fl_params(r_src=0.0)
    with FL.FaceListSolver(n, cp, par) as a, FL.FaceListSolver(m, cpm, par) as b:
        np.testing.assert_array_equal(a.conserved()[:, i0], b.conserved()[:, im])
        np.testing.assert_array_equal(a.get_state()[0][i0], b.get_state()[0][im])


def test_threads_and_flux_batches_at_once():
    """Solvers and flux batches on four threads share the staging slots."""
    n = 40000
    rng = np.random.default_rng(2)
    nrm = np.eye(3)[rng.integers(0, 3, n)]
    q = [np.c_[rng.uniform(0.5, 2, n), rng.normal(size=(n, 3)), rng.uniform(0.5, 2, n), rng.normal(size=(n, 3))]
         for _ in range(2)]
    want = S.chlld_batch(3, nrm, q[0], q[1])[0]
    desc = S.cart_desc((64, 48, 40), r_src=0.0)
    cps = [random_state(64 * 48 * 40, 20 + k) for k in range(4)]
    bad = []

    def work(k):
        with S.Solver(desc, cell_par=cps[k]) as s:
            first = s.get_state()[0]
            for _ in range(4):
                s.set_state(cps[k])
                if not (s.get_state()[0] == first).all():
                    bad.append(("state", k))
                if not (S.chlld_batch(3, nrm, q[0], q[1])[0] == want).all():
                    bad.append(("flux", k))

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
