"""Faces counted by the step's diagnostics are counted once, wherever the tiles of the grid meet: a face on the
seam of two tiles is computed in both."""
import numpy as np
import pytest

import oracle as O
import set_b200 as S
from set_b200 import facelist as FL
from tests.test_gpu_parity import oracle_opts, oracle_problem
from tests.test_gpu_stage_tiles import random_cells

pytestmark = pytest.mark.gpu


def half_cold_cells(shape):
    """Half of the cells without pressure, densities and velocities that are recovered exactly
    (test_cold_cells_without_a_field of test_gpu_stage_tiles.py)."""
    cp = random_cells(shape, "none", 74)
    cold = np.random.default_rng(75).uniform(size=len(cp)) < 0.5
    cp[:, 0] = np.exp2(np.round(np.log2(cp[:, 0])))
    cp[:, 1:4] = np.round(cp[:, 1:4] * 4096) / 4096
    cp[cold, 4] = 0.0
    return cp


def oracle_count(desc, inflow, o, cp):
    g, _ = oracle_problem(desc, S.lism_ic(lism=inflow, seed=1))
    U = O.cellpar_to_cons(cp, (desc.nz, desc.ny, desc.nx))
    return O.run(g, oracle_opts(o), U, 1)[1].n_wave_err


@pytest.mark.parametrize("shape", [(70, 34, 21), (97, 44, 16)])   # mixed form: 7 and 15 tile rows on 148 SMs
@pytest.mark.parametrize("n_state", [2, 3])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_faces_of_invalid_cells(shape, n_state, precision):
    """Cells without a valid state in a subsonic uniform flow at first order: none of their faces has a
    wave-fan region.  On both sides of the seams of every form's tiles (32 columns; 7, 11 and 15 rows) and
    inside tiles: the oracle's count, and as many faces recomputed on the seams as inside."""
    nx, ny, nz = shape
    inflow = S.lism_prim(bmag=0.0 if n_state == 2 else 1.0, u=(0.1, 0.3, 0.2))
    o = S.step_opts(n_state=n_state, scheme=1, order=1, precision=precision)
    desc = S.cart_desc(shape, inflow=inflow, r_src=0.0, dt_init=1e-4)
    redo = []
    for columns in (((31, (6, 10, 14, 21)), (64, (7, 11, 15, 22))), ((12, (3, 8, 17, 25)), (50, (3, 8, 17, 25)))):
        cp = np.zeros((nx * ny * nz, 16))
        cp[:, :8] = inflow
        for k in (2, 7, 12):
            for i, rows in columns:
                for j in rows:
                    cp[i + nx * (j + ny * k), 4] = np.nan
        want = oracle_count(desc, inflow, S.step_opts(n_state=n_state, scheme=1, order=1), cp)
        assert want == 6 * 24
        with S.Solver(desc, cell_par=cp) as s:
            s.step(1, o, check=False)
            d = s.status()
        assert d.n_wave_err == want
        redo.append(d.n_fp64_redo)
    assert redo[0] == redo[1] and (redo[0] > 0) == (precision > 0)


@pytest.mark.parametrize("shape", [(64, 33, 8), (32, 11, 4), (96, 45, 7), (64, 28, 9)])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_faces_on_the_grid_s_end(shape, precision):
    """Grids that end where tiles end (11, 15 and 7 rows): the end faces are the last tiles' own."""
    nx, ny, nz = shape
    inflow = S.lism_prim(u=(0.1, 0.3, 0.2))
    cp = np.zeros((nx * ny * nz, 16))
    cp[:, :8] = inflow
    for i, j, k in ((nx - 1, ny - 1, nz - 1), (nx - 1, 5, 0), (3, ny - 1, nz // 2), (0, 0, nz - 1)):
        cp[i + nx * (j + ny * k), 4] = np.nan
    desc = S.cart_desc(shape, inflow=inflow, r_src=0.0, dt_init=1e-4)
    want = oracle_count(desc, inflow, S.step_opts(scheme=1, order=1), cp)
    with S.Solver(desc, cell_par=cp) as s:
        s.step(1, S.step_opts(scheme=1, order=1, precision=precision), check=False)
        assert s.status().n_wave_err == want == 24


@pytest.mark.parametrize("shape", [(33, 23, 9), (70, 34, 5)])
@pytest.mark.parametrize("n_state", [2, 3])
def test_cold_faces_without_a_region(shape, n_state):
    cp = half_cold_cells(shape)
    inflow = S.lism_prim(bmag=0.0)
    desc = S.cart_desc(shape, inflow=inflow, r_src=0.0, dt_init=2e-2 / max(shape))
    o = S.step_opts(n_state=n_state, scheme=1, order=1)
    want = oracle_count(desc, inflow, o, cp)
    with S.Solver(desc, cell_par=cp) as s:
        s.step(1, o, check=False)
        assert s.status().n_wave_err == want > 0


@pytest.mark.parametrize("n_state", [2, 3])
def test_cold_faces_of_a_face_list(n_state):
    """The same cells on a renumbered face list: the oracle's count and, as faces without a region have no
    flux in either program, its cells (1e-11, as test_gpu_facelist_paths.py)."""
    shape = (33, 23, 9)
    cp = half_cold_cells(shape)
    m = FL.box_facelist(shape, permute_seed=4, seed=1, stretch=0.0, sides={a + b: 2 for a in "xyz" for b in "-+"})
    par = FL.fl_params(r_src=0.0, dt_init=2e-2 / max(shape))
    Uo = O.cellpar_to_cons(cp, (m.n_cell,)).reshape(8, -1).copy()
    _, do, _ = O.fl_run(O.facelist(m, par), O.make_opts(n_state, 1, 1, 0.4), Uo, 1)
    with FL.FaceListSolver(m, cp, par) as s:
        s.step(1, S.step_opts(n_state=n_state, scheme=1, order=1), check=False)
        U, d = s.conserved(), s.status()
    assert d.n_wave_err == do.n_wave_err > 0
    for v in range(5):
        assert np.abs(U[v] - Uo[v]).max() <= 1e-11 * np.abs(Uo[v]).max()
