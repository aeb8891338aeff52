"""The mixed form's two tile shapes.

15 rows (the shape of 128^3 and 384^3): grids that take it on 148 SMs, one row short of and on the edge of
its tiles, with ragged columns, against the oracle (tolerances of test_gpu_stage_tiles.py: 1e-6, dt 1e-5);
7 rows: test_gpu_stage_tiles.py.  Both shapes give the same cells the same bits, and slabs of a grid take
its shape whatever their own extents would make them choose."""
import numpy as np
import pytest

import set_b200 as S
from set_b200 import slab as SL
from tests.test_gpu_stage_tiles import one_step, random_cells

pytestmark = pytest.mark.gpu

ROWS_15 = [(97, 29, 16), (65, 44, 16), (128, 45, 12), (640, 29, 3), (481, 15, 7), (1601, 15, 2)]


@pytest.mark.parametrize("shape", ROWS_15)
@pytest.mark.parametrize("n_state,field,scheme,order", [(3, "all", 2, 2), (3, "part", 1, 1), (2, "none", 2, 2)])
def test_fifteen_rows_step_on_every_region(shape, n_state, field, scheme, order):
    err, dt = one_step(shape, n_state, field, 0, 1, 83, scheme, order)
    assert err <= 1e-6 and dt <= 1e-5


@pytest.mark.parametrize("shape,pad_y", [((97, 29, 16), 2), ((65, 44, 16), 5), ((481, 15, 7), 1)])
@pytest.mark.parametrize("n_state,order", [(3, 1), (3, 2), (2, 2)])
def test_shapes_agree_bitwise(shape, pad_y, n_state, order):
    """The same cells behind copies of their first row (what the zero-gradient boundary shows them anyway),
    which make the rows fit the other shape better."""
    nx, ny, nz = shape
    field = "all" if n_state == 3 else "none"
    cp = random_cells(shape, field, 84).reshape(nz, ny, nx, 16)
    out = []
    for a in (cp, np.pad(cp, ((0, 0), (pad_y, 0), (0, 0), (0, 0)), mode="edge")):
        n = a.shape[2::-1]
        desc = S.cart_desc(n, lo=(0.0, 0.0, 0.0), hi=tuple(m / 64.0 for m in n), r_src=0.0, dt_init=1e-4)
        with S.Solver(desc, cell_par=np.ascontiguousarray(a).reshape(-1, 16)) as s:
            s.step(1, S.step_opts(n_state=n_state, scheme=1, order=order, precision=1), check=False)
            out.append(s.conserved())
    np.testing.assert_array_equal(out[0], out[1][:, :, pad_y:])


@pytest.mark.parametrize("shape,parts,n_state", [((64, 15, 50), 3, 3), ((160, 15, 20), 2, 2)])
def test_mixed_slabs_of_a_fifteen_row_grid(shape, parts, n_state):
    lism = S.lism_prim() if n_state == 3 else S.lism_prim(bmag=0.0)
    desc = S.cart_desc(shape, inflow=lism, r_src=0.3, rho_src=20.0, dt_init=1e-4)
    cp = S.fill_lism(desc, S.lism_ic(lism=lism, seed=7, pert_amp=0.05))
    o = S.step_opts(n_state=n_state, precision=1)
    with S.Solver(desc, cell_par=cp) as g, SL.LocalSlabs(desc, parts, cp) as ls:
        g.step(8, o)
        ls.step(8, o)
        np.testing.assert_array_equal(g.conserved(), ls.conserved())
        assert g.get_state()[1] == ls.get_state()[1]
