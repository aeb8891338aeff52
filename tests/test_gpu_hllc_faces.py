"""The plain form's HLLC with a field in part of the domain: a face's flux depends on its own two states
alone, not on the faces that share its warp, so cells get the same bits whatever the seams of the tiles or
the numbering of the cells and faces."""
import numpy as np
import pytest

import set_b200 as S
from set_b200 import facelist as FL
from tests.test_gpu_stage_tiles import random_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("pad_x,pad_y", [(7, 0), (0, 4), (19, 9)])
def test_cartesian_flux_does_not_depend_on_the_tile(order, pad_x, pad_y):
    """The same cells with copies of the first column and row set before them (what the zero-gradient
    boundary shows them anyway): the seams of the tiles lie elsewhere.  The last column of a tile is left
    out, as it sums its fluxes in another order."""
    nx, ny, nz, h = 75, 29, 5, 1.0 / 64.0
    cp = random_cells((nx, ny, nz), "part", 81).reshape(nz, ny, nx, 16)
    padded = np.pad(cp, ((0, 0), (pad_y, 0), (pad_x, 0), (0, 0)), mode="edge")
    out = []
    for a in (cp, padded):
        n = a.shape[2::-1]
        desc = S.cart_desc(n, lo=(0.0, 0.0, 0.0), hi=tuple(h * m for m in n), r_src=0.0, dt_init=1e-4)
        with S.Solver(desc, cell_par=np.ascontiguousarray(a).reshape(-1, 16)) as s:
            s.step(1, S.step_opts(n_state=2, scheme=1, order=order), check=False)
            out.append(s.conserved())
    i = np.arange(nx)
    keep = (i % 32 != 31) & ((i + pad_x) % 32 != 31)
    np.testing.assert_array_equal(out[0][..., keep], out[1][:, :, pad_y:, pad_x:][..., keep])


@pytest.mark.parametrize("order,scheme", [(1, 1), (2, 2)])
def test_renumbered_face_list(order, scheme):
    a = FL.box_facelist((14, 12, 10), stretch=0.4, seed=2)
    b = FL.box_facelist((14, 12, 10), stretch=0.4, seed=2, permute_seed=17)
    key = lambda x: np.lexsort((x[:, 0], x[:, 1], x[:, 2]))
    ia, ib = key(a.cell_center), key(b.cell_center)
    cpa = random_cells((14, 12, 10), "part", 82)
    cpb = np.zeros_like(cpa)
    cpb[ib] = cpa[ia]
    par = FL.fl_params(r_src=0.0, dt_init=1e-3)
    o = S.step_opts(n_state=2, order=order, scheme=scheme)
    with FL.FaceListSolver(a, cpa, par) as x, FL.FaceListSolver(b, cpb, par) as y:
        x.step(3, o, check=False)
        y.step(3, o, check=False)
        np.testing.assert_array_equal(x.conserved()[:, ia], y.conserved()[:, ib])
