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
