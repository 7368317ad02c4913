"""The coarse-operator constructions' workspace, kept in the aggregation."""
import numpy as np
import pytest
import torch

import gmg
import inputs

pytestmark = pytest.mark.gpu


def test_constructions_on_two_streams():
    # over the Wilson-clover operator (asynchronous) and over a coarse stencil of its 12
    # components, from one aggregation on two streams: the second uses the workspace after the first
    fd, cd, N = (8, 8, 8, 8), (4, 4, 4, 4), 12
    w = gmg.WilsonClover(fd, -0.1, 1.0, antiperiodic=1)
    w.set_gauge(inputs.hot_gauge(fd, inputs.rng(stream=900)))
    fine = gmg.CoarsenedMatrix(fd, 12)
    fine.set_links(inputs.random_links(fd, 12, inputs.rng(stream=901)))
    ag = gmg.Aggregation(fd, cd, 12, N)
    ag.set_basis(inputs.gaussian_field((N, 4096, 12), inputs.rng(stream=902)))
    got = []
    for busy in (False, True):
        a, b = gmg.CoarsenedMatrix(cd, N), gmg.CoarsenedMatrix(cd, N)
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            if busy:
                torch.cuda._sleep(200_000_000)
            a.CoarsenOperator(ag, w)
            if not busy:
                torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            b.CoarsenOperator(ag, fine)
        torch.cuda.synchronize()
        got.append((a.get_links(), b.get_links()))
    for x, y in zip(*got):
        assert np.array_equal(x, y)


def test_large_workspace_is_given_back():
    # two fields of 64 vectors of 12 components on 16^4 sites: 1.6 GB during the construction
    fd, cd, dof, N = (16, 16, 16, 16), (4, 4, 4, 4), 12, 64
    V = 65536
    links = torch.view_as_complex(torch.randn((9, V, dof, dof, 2), dtype=torch.float64, device="cuda"))
    fine = gmg.CoarsenedMatrix(fd, dof)
    fine.set_links(links)
    ag = gmg.Aggregation(fd, cd, dof, N)
    ag.set_basis(torch.view_as_complex(torch.randn((N, V, dof, 2), dtype=torch.float64, device="cuda")))
    out = gmg.CoarsenedMatrix(cd, N)
    out.set_links(np.zeros((9, 256, N, N)))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    out.CoarsenOperator(ag, fine)
    taken = free - torch.cuda.mem_get_info()[0]
    first = out.get_links()
    assert taken < 1 << 30, taken
    out.CoarsenOperator(ag, fine)
    assert np.array_equal(out.get_links(), first)


def test_batch_change_frees_the_workspace():
    fd, cd, N = (16, 16, 16, 16), (4, 4, 4, 4), 16
    w = gmg.WilsonClover(fd, -0.1, 1.0, antiperiodic=1)
    w.set_gauge(inputs.smooth_gauge(fd, inputs.rng(stream=905), 0.3))
    ag = gmg.Aggregation(fd, cd, 12, N)
    ag.set_basis(torch.view_as_complex(torch.randn((N, 65536, 12, 2), dtype=torch.float64, device="cuda")))
    cm = gmg.CoarsenedMatrix(cd, N)
    cm.CoarsenOperator(ag, w)
    first = cm.get_links()
    free = torch.cuda.mem_get_info()[0]
    ag.set_coarsen_batch(4)
    assert torch.cuda.mem_get_info()[0] - free > 300 << 20  # two fields of 201 MB
    cm.CoarsenOperator(ag, w)
    # other batches, other widths of the products: rounding only
    assert np.abs(cm.get_links() - first).max() < 1e-11 * np.abs(first).max()
