"""Multigrid solves on a stream of their own: nothing they need waits in the legacy default stream."""
import pytest
import torch

import gmg
import inputs

pytestmark = pytest.mark.gpu


def test_first_solve_while_the_default_stream_is_busy():
    # the captured cycle's state is set up in the first solve, and is cleared before it is used
    dims, nrhs = (8, 8, 8, 8), 3
    w = gmg.WilsonClover(dims, -0.05, 1.0, antiperiodic=True)
    w.set_gauge(inputs.smooth_gauge(dims, inputs.rng(stream=301), 0.3))
    b = torch.from_numpy(inputs.gaussian_field((4096, nrhs, 12), inputs.rng(stream=777))).cuda()
    its = []
    for busy in (False, True):
        mg = gmg.MultiGrid(w, nrhs, nlevels=3, block=((2, 2, 2, 2), (2, 2, 2, 2)), nvec=(6, 6), setup_iters=30,
                           prec="f32", graph=1)
        mg.setup()
        x, r = torch.zeros_like(b), torch.zeros_like(b)
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        if busy:
            torch.cuda._sleep(1_000_000_000)
        with torch.cuda.stream(side):
            it, rr = mg.solve(b, x, tol=1e-10, maxiter=300)
            w.M(x, r)
            r = b - r
            true = (torch.linalg.vector_norm(r, dim=(0, 2)) / torch.linalg.vector_norm(b, dim=(0, 2))).max()
        torch.cuda.synchronize()
        assert rr <= 1e-10 and true.item() <= 2e-10, (it, rr, true.item())
        assert mg.graphs() == (1, 0)
        its.append(it)
    assert abs(its[0] - its[1]) <= 1, its
