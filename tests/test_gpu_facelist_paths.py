"""Face lists on general normals and on states that select every wave-fan region.

The box mesh is rotated as a whole, so no normal is aligned with an axis; cell states are random
(far subsonic to supersonic both ways; no field, a field in part of the cells, a field everywhere).
Every solver and wave-speed estimate takes one step against the oracle's face-list driver.

Tolerance, relative to each variable's largest magnitude: 1e-11 (a face flux agrees to 1e-10 of its
largest component at worst, where a star denominator cancels, and a step moves a cell by at most
dt/h < 0.1 of a flux).
"""
import numpy as np
import pytest

import oracle as O
import set_b200 as S
from set_b200 import facelist as FL
from tests.test_gpu_stage_tiles import random_cells

pytestmark = pytest.mark.gpu

WALLS = {k: 2 for k in ("x-", "x+", "y-", "y+", "z-", "z+")}


def rotated_mesh(shape, seed):
    m = FL.box_facelist(shape, stretch=0.5, permute_seed=seed, sides=WALLS, seed=seed)
    q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(3, 3)))
    for name in ("cell_center", "gran_center", "gran_normal"):
        setattr(m, name, np.ascontiguousarray(getattr(m, name) @ q.T))
    return m


@pytest.mark.parametrize("n_state,n_disc,field,order,scheme",
                         [(3, 0, "all", 2, 2), (3, 0, "part", 1, 1), (2, 0, "none", 2, 2), (2, 0, "part", 2, 1),
                          (3, 1, "all", 2, 2), (3, 2, "part", 2, 1), (2, 1, "none", 1, 2), (1, 0, "all", 2, 2),
                          (0, 0, "all", 2, 1)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (9, 7, 5), (16, 11, 3)])
def test_facelist_step_on_every_region(shape, n_state, n_disc, field, order, scheme):
    m = rotated_mesh(shape, 3)
    params = FL.fl_params(r_src=0.0, dt_init=2e-2 / max(shape))
    cp = random_cells(shape, field, 61)
    om = O.facelist(m, params)
    Uo = O.cellpar_to_cons(cp, (m.n_cell,)).reshape(8, -1).copy()
    ck, _, _ = O.fl_run(om, O.make_opts(n_state, order, scheme, 0.4, n_disc), Uo, 1)
    with FL.FaceListSolver(m, cp, params) as s:
        s.step(1, S.step_opts(n_state=n_state, n_disc=n_disc, order=order, scheme=scheme))
        U, d = s.conserved(), s.status()
    for v in range(8):
        assert np.abs(U[v] - Uo[v]).max() <= 1e-11 * max(np.abs(Uo[v]).max(), 1e-300), v
    assert abs(d.dt_next - ck.dt_next) <= 1e-12 * ck.dt_next


@pytest.mark.parametrize("scheme", [1, 2])
def test_facelist_steps_split_over_calls_and_edits_between_them(scheme):
    """The cell update leaves the next stage's primitive state behind; the first stage of a call forms
    it anew, so calls may be split anywhere and the resident state may be edited between them."""
    import torch
    from set_b200.slab import _DeviceArray
    m = rotated_mesh((9, 8, 7), 5)
    params = FL.fl_params(r_src=0.2, rho_src=5.0, v_src=2.0, dt_init=1e-3)
    cp = FL.lism_cellpar(m, seed=2, params=params)
    o = S.step_opts(scheme=scheme)
    with FL.FaceListSolver(m, cp, params) as a, FL.FaceListSolver(m, cp, params) as b:
        a.step(5, o)
        for n in (1, 3, 1):
            b.step(n, o)
        np.testing.assert_array_equal(a.conserved(), b.conserved())
        for s in (a, b):   # double the energy in place
            ptr, vs, _, _ = s.state_view()
            view = torch.as_tensor(_DeviceArray(ptr, (8, m.n_cell), (vs, 1)), device="cuda")
            view[4] *= 2.0
            torch.cuda.synchronize()
        with FL.FaceListSolver(m, cp, params) as c:   # the edited state on a fresh handle, same clock
            c.copy_from(a)
            a.step(2, o)
            b.step(2, o)
            c.step(2, o)
            np.testing.assert_array_equal(a.conserved(), b.conserved())
            np.testing.assert_array_equal(a.conserved(), c.conserved())
