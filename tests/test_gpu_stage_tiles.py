"""The stage kernels on states that select every wave-fan region, at the edges of their tiles.

One step from random cell states (normal velocities from far subsonic to supersonic both ways, so
the faces select FL, L*, L**, R**, R* and FR; no field, a field in part of the cells, a field
everywhere), on grids one cell short of, equal to and one cell past the tile rows of the plain
(11), delta (11) and mixed (15) forms and the 32 columns, on single cells, rows and planes, and on
z extents that end chunks unevenly.

Tolerance against the oracle, relative to each variable's largest magnitude: plain 1e-11 (a face
flux agrees to 1e-10 of its largest component at worst, where a star denominator cancels
(test_gpu_parity.py), and a step moves a cell by at most dt/h < 0.1 of a flux); delta and mixed
1e-6 (FP32 rounding 6e-8 of a flux of up to ~10 times the state, dt/h < 0.1).
"""
import numpy as np
import pytest

import oracle as O
import set_b200 as S
from tests.test_gpu_parity import oracle_opts, oracle_problem

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 10, 3), (31, 11, 2), (32, 12, 9), (33, 14, 5), (65, 15, 17), (30, 16, 33), (40, 23, 12)]


def random_cells(shape, field, seed):
    rng = np.random.default_rng(seed)
    n = shape[0] * shape[1] * shape[2]
    cp = np.zeros((n, 16))
    cp[:, 0] = np.exp(rng.uniform(-1.0, 1.0, n))
    cp[:, 1:4] = rng.normal(size=(n, 3)) * np.exp(rng.uniform(-2.0, 1.5, n))[:, None]
    cp[:, 4] = np.exp(rng.uniform(-1.0, 1.5, n))
    if field != "none":
        cp[:, 5:8] = rng.normal(size=(n, 3)) * np.exp(rng.uniform(-2.0, 1.0, n))[:, None]
    if field == "part":   # warps with and without a field, and mixed ones
        cp[rng.uniform(size=n) < 0.7, 5:8] = 0.0
        cp[: n // 3, 5:8] = 0.0
    return cp


def one_step(shape, n_state, field, n_disc, precision, seed, scheme=2, order=2):
    inflow = S.lism_prim(bmag=0.0 if field == "none" else 1.0)
    desc = S.cart_desc(shape, inflow=inflow, dt_init=2e-2 / max(shape))
    o = S.step_opts(n_state=n_state, n_disc=n_disc, precision=precision, scheme=scheme, order=order)
    cp = random_cells(shape, field, seed)
    g, _ = oracle_problem(desc, S.lism_ic(lism=inflow, seed=1))
    Uo = O.cellpar_to_cons(cp, shape[::-1])
    ck, _ = O.run(g, oracle_opts(o), Uo, 1)
    with S.Solver(desc, cell_par=cp) as s:
        s.step(1, o)
        U, d = s.conserved(), s.status()
    err = [np.abs(U[v] - Uo[v]).max() / max(np.abs(Uo[v]).max(), 1e-300) for v in range(8)]
    return max(err), abs(d.dt_next - ck.dt_next) / ck.dt_next


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("n_state,field", [(3, "all"), (3, "part"), (2, "none"), (2, "part")])
def test_plain_step_on_every_region(shape, n_state, field):
    err, dt = one_step(shape, n_state, field, 0, 0, 71)
    assert err <= 1e-11 and dt <= 1e-12


@pytest.mark.parametrize("n_state,n_disc,scheme,order", [(3, 1, 2, 2), (3, 2, 1, 1), (2, 1, 1, 2), (2, 2, 2, 1),
                                                         (1, 0, 2, 2), (0, 0, 1, 1)])
def test_plain_step_other_estimates_and_solvers(n_state, n_disc, scheme, order):
    err, dt = one_step((33, 23, 9), n_state, "part", n_disc, 0, 72, scheme, order)
    assert err <= 1e-11 and dt <= 1e-12


@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 14, 5), (33, 15, 9), (65, 16, 17), (40, 31, 12)])
@pytest.mark.parametrize("precision", [1, 2])
def test_mixed_forms_step_on_every_region(shape, precision):
    err, dt = one_step(shape, 3, "all", 0, precision, 73)
    assert err <= 1e-6 and dt <= 1e-5


@pytest.mark.parametrize("n_state", [2, 3])
def test_cold_cells_without_a_field(n_state):
    """Half of the cells without pressure: sides of zero sound speed that collide, recede (star density
    0; the fan of two such sides has no contact speed, so the face has no region unless it lies outside)
    and face warm ones.  Densities are powers of two and velocities multiples of 2^-12, so every pressure
    is recovered exactly and both programs see the same zeros.  Faces without a region have no flux in
    either program, so all cells agree to the tolerance above (a face between two chunks of the z march
    is counted by both chunks, so the count is at least the oracle's)."""
    shape = (33, 23, 9)
    cp = random_cells(shape, "none", 74)
    cold = np.random.default_rng(75).uniform(size=len(cp)) < 0.5
    cp[:, 0] = np.exp2(np.round(np.log2(cp[:, 0])))
    cp[:, 1:4] = np.round(cp[:, 1:4] * 4096) / 4096
    cp[cold, 4] = 0.0
    inflow = S.lism_prim(bmag=0.0)
    desc = S.cart_desc(shape, inflow=inflow, r_src=0.0, dt_init=2e-2 / max(shape))
    o = S.step_opts(n_state=n_state, scheme=1, order=1)
    g, _ = oracle_problem(desc, S.lism_ic(lism=inflow, seed=1))
    Uo = O.cellpar_to_cons(cp, shape[::-1])
    _, do = O.run(g, oracle_opts(o), Uo, 1)
    with S.Solver(desc, cell_par=cp) as s:
        s.step(1, o, check=False)
        U, d = s.conserved(), s.status()
    assert d.n_wave_err >= do.n_wave_err > 0
    for v in range(5):
        assert np.abs(U[v] - Uo[v]).max() <= 1e-11 * np.abs(Uo[v]).max()
