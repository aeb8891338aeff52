"""Steps captured into a CUDA graph on the handle's stream and replayed: the bits of steps run directly (chained
launches become edges of the graph, a tensor map travels with its kernel's parameters)."""
import ctypes as C

import numpy as np
import pytest

import set_b200 as S
from set_b200 import facelist as FL

pytestmark = pytest.mark.gpu


def compare(make, opts, n):
    import torch
    with make() as direct, make() as captured:
        for s in (direct, captured):   # modules and the compensation
            s.step(1, opts)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(captured.stream())):
            assert S.lib().setb_step(captured.h, n, C.byref(opts), None) == 0
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        direct.step(3 * n, opts)
        np.testing.assert_array_equal(direct.conserved(), captured.conserved())
        assert direct.status().time_all == captured.status().time_all


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("scheme", [1, 2])
def test_cartesian(precision, scheme):
    compare(lambda: S.Solver(S.cart_desc((70, 34, 21), dt_init=1e-4), ic=S.lism_ic(seed=1)),
            S.step_opts(precision=precision, scheme=scheme), 2)


@pytest.mark.parametrize("scheme", [1, 2])
def test_face_list(scheme):
    m = FL.box_facelist((12, 10, 8), stretch=0.3, permute_seed=1, seed=1)
    par = FL.fl_params(r_src=0.2, dt_init=1e-4)
    cp = FL.lism_cellpar(m, seed=2, params=par)
    compare(lambda: FL.FaceListSolver(m, cp, par), S.step_opts(scheme=scheme), 2)
