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


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_copies_of_a_lost_timing_are_freed(prec):
    # the copies stay allocated only where the site kernel is what later calls run
    def run(dims):
        w, v = _handle(873, None, dims), dims[0] * dims[1] * dims[2] * dims[3]
        x = _field(prec, 7, 874, v)
        out = torch.zeros_like(x)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        w.M(x, out)
        torch.cuda.synchronize()
        return w, w.tuned_kernel(prec, 7), free - torch.cuda.mem_get_info()[0]

    run((4, 4, 4, 4))  # loads the kernels
    dims = (20, 24, 20, 24)
    copies = 230400 * 72 * (16 if prec == "f64" else 8)
    w, kernel, taken = run(dims)
    print(kernel, taken, copies)
    assert taken < copies / 4 if kernel != "site" else taken >= copies, (kernel, taken)


def _offset(prec, nrhs, stream, entries):
    """A field whose first entry lies `entries` complex numbers into an aligned buffer."""
    x = _field(prec, nrhs, stream)
    buf = torch.zeros(x.numel() + entries, dtype=x.dtype, device="cuda")
    buf[entries:] = x.reshape(-1)
    return buf[entries:].view(x.shape)


# squared relative deviation: sums of about 100 terms, rounded in the field's precision
TOL = {"f64": 1e-28, "f32": 1e-12}


def _oracle(x, op, gauge_stream):
    import oracle as orc
    U = inputs.hot_gauge(DIMS, inputs.rng(stream=gauge_stream))
    return orc.wilson_clover(DIMS, U, orc.clover_build(DIMS, U, 1.0), -0.1, 1, x.cpu().numpy().astype("complex128"), op)


def _deviation(ref, got):
    import oracle as orc
    return orc.rel_dev_sq(ref, got.cpu().numpy().astype("complex128"))


@pytest.mark.parametrize("prec,entries", [("f64", 0), ("f64", 1), ("f32", 0), ("f32", 1), ("f32", 2)])
@pytest.mark.parametrize("nrhs", [1, 3, 7])
@pytest.mark.parametrize("op", ["M", "Mdag", "Mdiag"])
def test_field_alignments(prec, entries, nrhs, op):
    import oracle as orc
    x, out = _offset(prec, nrhs, 875, entries), _offset(prec, nrhs, 876, entries)
    getattr(_handle(877), op)(x, out)
    assert _deviation(_oracle(x, {"M": orc.OP_M, "Mdag": orc.OP_MDAG, "Mdiag": orc.OP_MDIAG}[op], 877), out) < TOL[prec]


@pytest.mark.parametrize("prec,entries,nrhs", [("f64", 0, 1), ("f32", 0, 2), ("f32", 1, 2), ("f32", 1, 5), ("f32", 1, 9)])
def test_first_call_in_a_capture(prec, entries, nrhs):
    # no copies, and nothing timed: whatever runs has to take these fields
    import oracle as orc
    x, out = _offset(prec, nrhs, 878, entries), _offset(prec, nrhs, 879, entries)
    w = _handle(880, None)
    g = _captured(w, x, out)
    g.replay()
    torch.cuda.synchronize()
    assert _deviation(_oracle(x, orc.OP_M, 880), out) < TOL[prec]


def test_choices_by_alignment():
    # a choice made for fields of 8-byte alignment, where few kernels apply, is not the aligned fields' one
    dims = (16, 16, 16, 8)
    w = _handle(881, None, dims)
    x = _field("f32", 12, 882, 32768)
    buf = torch.zeros(2 * x.numel() + 1, dtype=x.dtype, device="cuda")
    lo, hi = buf[1:x.numel() + 1].view(x.shape), buf[x.numel() + 1:].view(x.shape)
    w.M(lo, hi)
    assert w.tuned_kernel("f32", 12) == "quad"
    w.M(x, torch.zeros_like(x))
    assert w.tuned_kernel("f32", 12) == "tile"


def test_choices_by_kind_of_operator():
    # the site kernel wins Mdiag by far more than M: one's choice is not the other's
    dims = (16, 16, 16, 16)
    x = _field("f32", 6, 883, 65536)
    out = torch.zeros_like(x)
    w = _handle(884, None, dims)
    w.Mdiag(x, out)
    assert w.tuned_kernel("f32", 6) == "auto"  # M's, not timed yet
    w.M(x, out)
    assert w.tuned_kernel("f32", 6) == "tile"


def test_small_lattice_times_the_staged_kernel():
    x = _field("f64", 24, 885, 256)  # 8.3 us staged, 18.5 us by tiles
    w = _handle(886, None, (4, 4, 4, 4))
    w.M(x, torch.zeros_like(x))
    assert w.tuned_kernel("f64", 24) == "staged"
