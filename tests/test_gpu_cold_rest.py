"""Pressureless, field-free cells at rest in some directions (velocity components of exactly 0), one Euler
step at first order: the faces between such sides have no wave-fan region where neither side reaches the
other, are reported as the oracle reports them and carry no flux.  Densities are powers of two and velocities
multiples of 2^-12, so every pressure is recovered exactly; cells within 1e-11 (test_gpu_stage_tiles.py)."""
import numpy as np
import pytest

import oracle as O
import set_b200 as S
from set_b200 import facelist as FL
from tests.test_gpu_parity import oracle_opts, oracle_problem
from tests.test_gpu_stage_tiles import random_cells

pytestmark = pytest.mark.gpu

SHAPE = (12, 11, 10)


def cells():
    cp = random_cells(SHAPE, "none", 91)
    rng = np.random.default_rng(92)
    n = len(cp)
    cp[:, 0] = np.exp2(np.round(np.log2(cp[:, 0])))
    cp[:, 1:4] = np.round(cp[:, 1:4] * 4096) / 4096
    cp[:, 1:4][rng.uniform(size=(n, 3)) < 0.4] = 0.0
    cp[rng.uniform(size=n) < 0.6, 4] = 0.0
    return cp


def compare(U, n_wave, Uo, n_wave_o):
    assert n_wave == n_wave_o > 0
    for v in range(5):
        assert np.abs(U[v] - Uo[v]).max() <= 1e-11 * np.abs(Uo[v]).max()


@pytest.mark.parametrize("n_state", [2, 3])
def test_cartesian(n_state):
    cp = cells()
    inflow = S.lism_prim(bmag=0.0)
    desc = S.cart_desc(SHAPE, inflow=inflow, r_src=0.0, dt_init=1e-3)
    o = S.step_opts(n_state=n_state, scheme=1, order=1)
    g, _ = oracle_problem(desc, S.lism_ic(lism=inflow, seed=1))
    Uo = O.cellpar_to_cons(cp, SHAPE[::-1])
    _, do = O.run(g, oracle_opts(o), Uo, 1)
    with S.Solver(desc, cell_par=cp) as s:
        s.step(1, o, check=False)
        compare(s.conserved(), s.status().n_wave_err, Uo, do.n_wave_err)


@pytest.mark.parametrize("n_state", [2, 3])
def test_face_list(n_state):
    cp = cells()
    m = FL.box_facelist(SHAPE, permute_seed=4, seed=1, stretch=0.0, sides={a + b: 2 for a in "xyz" for b in "-+"})
    par = FL.fl_params(r_src=0.0, dt_init=1e-3)
    Uo = O.cellpar_to_cons(cp, (m.n_cell,)).reshape(8, -1).copy()
    _, do, _ = O.fl_run(O.facelist(m, par), O.make_opts(n_state, 1, 1, 0.4), Uo, 1)
    with FL.FaceListSolver(m, cp, par) as s:
        s.step(1, S.step_opts(n_state=n_state, scheme=1, order=1), check=False)
        compare(s.conserved(), s.status().n_wave_err, Uo, do.n_wave_err)
