"""The coarse levels' one-kernel solver steps, and the separate kernels they replace
where a Krylov basis is longer than they take, in captured and host-driven solves:
every right-hand side reaches 1e-10 by its recomputed true residual."""
import pytest
import torch

import gmg
import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs,nvec,kw", [
    (1, (5, 7), {}),                                            # one right-hand side, odd vector counts
    (3, (6, 6), dict(coarsest_restart=40, coarsest_iters=45)),  # basis of 40: separate kernels on the coarsest level
    (5, (8, 4), dict(wrapper_iters=3, coarsest_restart=4)),     # several short cycles per solve
])
@pytest.mark.parametrize("graph", [0, 1])
def test_solves_reach_1e10(nrhs, nvec, kw, graph):
    dims = (8, 8, 8, 8)
    w = gmg.WilsonClover(dims, -0.05, 1.0, antiperiodic=True)
    w.set_gauge(inputs.smooth_gauge(dims, inputs.rng(stream=301), 0.3))
    mg = gmg.MultiGrid(w, nrhs, nlevels=3, block=((2, 2, 2, 2), (2, 2, 2, 2)), nvec=nvec, setup_iters=30, prec="f32",
                       graph=graph, **dict(dict(coarsest_iters=30, wrapper_iters=6), **kw))
    mg.setup()
    b = torch.from_numpy(inputs.gaussian_field((4096, nrhs, 12), inputs.rng(stream=770 + nrhs))).cuda()
    for _ in range(2):  # the second solve replays what the first captured
        x = torch.zeros_like(b)
        it, rr = mg.solve(b, x, tol=1e-10, maxiter=300)
        r = torch.zeros_like(b)
        w.M(x, r)
        r = b - r
        true = (torch.linalg.vector_norm(r, dim=(0, 2)) / torch.linalg.vector_norm(b, dim=(0, 2))).max().item()
        assert rr <= 1e-10 and true <= 2e-10, (it, rr, true)
    if graph:
        assert mg.graphs()[1] == 0
