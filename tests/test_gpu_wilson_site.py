"""The Wilson-clover site kernel (few right-hand sides) and its rearranged copies of the links and the clover."""
import pytest
import torch

import gmg
import inputs

pytestmark = pytest.mark.gpu

DT = {"f64": torch.complex128, "f32": torch.complex64}
DIMS = (4, 6, 4, 3)
V = 288


def _handle(gauge_stream, kernel="site", dims=DIMS):
    w = gmg.WilsonClover(dims, -0.1, 1.0, antiperiodic=1)
    w.set_gauge(inputs.hot_gauge(dims, inputs.rng(stream=gauge_stream)))
    if kernel:
        w.set_kernel(kernel)
    return w


def _field(prec, nrhs, stream, v=V):
    return torch.from_numpy(inputs.gaussian_field((v, nrhs, 12), inputs.rng(stream=stream))).cuda().to(DT[prec])


def _captured(w, x, out):
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        w.M(x, out)
    return g


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_captured_apply_follows_set_gauge(prec, nrhs):
    x = _field(prec, nrhs, 870)
    w = _handle(871)
    out = torch.zeros_like(x)
    w.M(x, out)  # builds the copies: the graph holds the site kernel on them
    g = _captured(w, x, out)
    w.set_gauge(inputs.hot_gauge(DIMS, inputs.rng(stream=872)))
    out.zero_()
    g.replay()
    ref = torch.zeros_like(x)
    _handle(872).M(x, ref)
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
