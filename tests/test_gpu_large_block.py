"""Projection and promotion with one block of more than 2^28 components (8.6 GB of FP64 basis)."""
import pytest
import torch

import gmg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.complex128, torch.complex64])
def test_one_block_beyond_2_28_components(dt):
    fd, dof, N = (32, 32, 32, 33), 256, 2
    V = 32 * 32 * 32 * 33
    g = torch.Generator(device="cuda")
    g.manual_seed(17)
    B = torch.randn((N, V, dof), dtype=torch.complex128, device="cuda", generator=g)
    x = torch.randn((V, 1, dof), dtype=dt, device="cuda", generator=g)
    ag = gmg.Aggregation(fd, (1, 1, 1, 1), dof, N)
    ag.set_basis(B)
    y = torch.zeros((1, 1, N), dtype=dt, device="cuda")
    ag.ProjectToSubspace(x, y)
    x64 = x.reshape(-1).to(torch.complex128)
    ref = torch.stack([torch.vdot(b.reshape(-1), x64) for b in B])
    # 2.8e8 terms of size 1 (rounded to FP32 in basis and field, for FP32): sqrt of their number against the sum of it
    tol = 1e-11 if dt == torch.complex128 else 1e-5
    size = (V * dof) ** 0.5
    assert (y[0, 0].to(torch.complex128) - ref).abs().max().item() < tol * size
    c = torch.tensor([[[0.3 - 0.5j, 1.1 + 0.2j]]], dtype=dt, device="cuda")
    del x, x64
    out = torch.full((V, 1, dof), float("nan"), dtype=dt, device="cuda")
    ag.PromoteFromSubspace(c, out)
    c64 = c.to(torch.complex128)
    err = (out[:, 0].to(torch.complex128) - (B[0] * c64[0, 0, 0] + B[1] * c64[0, 0, 1])).abs().max().item()
    assert err < (1e-14 if dt == torch.complex128 else 1e-5)
    ag.__del__()
    del B, out
    torch.cuda.empty_cache()
