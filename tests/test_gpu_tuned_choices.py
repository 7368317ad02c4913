"""Launch choices found by timing are shared by handles of the same sizes."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import gmg
import inputs

pytestmark = pytest.mark.gpu


def _shape(cm, R):
    ctas, pps = ctypes.c_int(), ctypes.c_int()
    assert gmg.lib().gmg_coarse_tuned_shape(cm._h, R, 9, gmg.BF16, ctypes.byref(ctas), ctypes.byref(pps)) == 0
    return ctas.value, pps.value


def test_second_handle_takes_the_first_ones_choice():
    dims, N, R = (4, 2, 4, 2), 16, 7
    A = inputs.random_links(dims, N, inputs.rng(stream=760))
    x = torch.from_numpy(inputs.gaussian_field((64, R, N), inputs.rng(stream=761))).cuda().to(torch.complex64)
    got = []
    for _ in range(2):
        cm = gmg.CoarsenedMatrix(dims, N)
        cm.set_links(A)
        cm.prepare("bf16")
        assert _shape(cm, R) == (0, 0)  # nothing before the handle's first apply
        out = torch.zeros_like(x)
        cm.M(x, out, compute="bf16")
        got.append((_shape(cm, R), out))
    assert got[0][0] == got[1][0] != (0, 0)
    assert torch.equal(got[0][1], got[1][1])


def test_handles_of_several_threads():
    # first applies of equal lattices from four threads at once, each on its own handle and stream
    dims = (4, 4, 4, 6)
    U = inputs.hot_gauge(dims, inputs.rng(stream=762))
    x = torch.from_numpy(inputs.gaussian_field((384, 2, 12), inputs.rng(stream=763))).cuda()
    outs, errs = [None] * 4, []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                w = gmg.WilsonClover(dims, -0.1, 1.0, antiperiodic=True)
                w.set_gauge(U)
                outs[k] = torch.zeros_like(x)
                w.M(x, outs[k])
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errs.append(e)

    torch.cuda.synchronize()
    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs
    ref = outs[0].cpu().numpy()
    for o in outs[1:]:  # another variant sums in another order
        assert np.abs(o.cpu().numpy() - ref).max() < 1e-13
