"""A cell without a valid state (its pressure is no number, of either sign bit) in a uniform flow, one Euler
step: the faces that the oracle finds to have no wave-fan region are found and carry no flux, and every
other face carries what it carries there, so the count, the cells that turn invalid and the rest of the
state (1e-11 of each variable's largest magnitude, as in test_gpu_stage_tiles.py) are the oracle's."""
import numpy as np
import pytest

import oracle as O
import set_b200 as S
from set_b200 import facelist as FL
from tests.test_gpu_parity import oracle_opts, oracle_problem

pytestmark = pytest.mark.gpu

SHAPE = (12, 11, 10)
FLOWS = [(8.0, 0.3, 0.2), (-8.0, 0.3, 0.2), (0.1, 0.3, 0.2)]


def compare(U, n_wave, Uo, n_wave_o):
    assert n_wave == n_wave_o > 0
    np.testing.assert_array_equal(np.isnan(U).any(0), np.isnan(Uo).any(0))
    for v in range(8):
        scale = np.nanmax(np.abs(Uo[v]))
        assert np.nanmax(np.abs(U[v] - Uo[v])) <= 1e-11 * max(scale, 1e-300), v


def cells(n_state, u, value):
    inflow = S.lism_prim(bmag=0.0 if n_state == 2 else 1.0, u=u)
    cp = np.zeros((int(np.prod(SHAPE)), 16))
    cp[:, :8] = inflow
    cp[6 + SHAPE[0] * (5 + SHAPE[1] * 5), 4] = value
    return inflow, cp


@pytest.mark.parametrize("value", [np.nan, -np.nan])
@pytest.mark.parametrize("u", FLOWS)
@pytest.mark.parametrize("n_state,order", [(3, 1), (2, 1), (3, 2), (2, 2)])
def test_cartesian(n_state, order, u, value):
    inflow, cp = cells(n_state, u, value)
    desc = S.cart_desc(SHAPE, inflow=inflow, r_src=0.0, dt_init=1e-4)
    o = S.step_opts(n_state=n_state, scheme=1, order=order)
    g, _ = oracle_problem(desc, S.lism_ic(lism=inflow, seed=1))
    Uo = O.cellpar_to_cons(cp, SHAPE[::-1])
    _, do = O.run(g, oracle_opts(o), Uo, 1)
    with S.Solver(desc, cell_par=cp) as s:
        s.step(1, o, check=False)
        compare(s.conserved(), s.status().n_wave_err, Uo, do.n_wave_err)


@pytest.mark.parametrize("value", [np.nan, -np.nan])
@pytest.mark.parametrize("u", FLOWS)
@pytest.mark.parametrize("n_state,order", [(3, 1), (2, 1), (3, 2), (2, 2)])
def test_face_list(n_state, order, u, value):
    _, cp = cells(n_state, u, value)
    m = FL.box_facelist(SHAPE, permute_seed=4, seed=1, stretch=0.2, sides={"y-": 2, "x-": 2, "x+": 2})
    at = np.lexsort((m.cell_center[:, 0], m.cell_center[:, 1], m.cell_center[:, 2]))
    par = FL.fl_params(r_src=0.0, dt_init=1e-4)
    cpm = np.zeros_like(cp)
    cpm[at] = cp
    Uo = O.cellpar_to_cons(cpm, (m.n_cell,)).reshape(8, -1).copy()
    _, do, _ = O.fl_run(O.facelist(m, par), O.make_opts(n_state, order, 1, 0.4), Uo, 1)
    with FL.FaceListSolver(m, cpm, par) as s:
        s.step(1, S.step_opts(n_state=n_state, scheme=1, order=order), check=False)
        compare(s.conserved(), s.status().n_wave_err, Uo, do.n_wave_err)
