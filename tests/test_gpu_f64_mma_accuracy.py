"""Accuracy of the FP64 tensor-core kernels, and their launch shapes.

FP64 results differ from the oracle's by the order of their sums: a relative error of
1e-13 at most over sums of up to 3072 terms (1e-26 squared; one operand rounded to
FP32 would give 1e-15).  FP32 fields are widened, summed in FP64 and rounded once:
1e-7 relative on fields and 1e-7 on the FP32 copies of links and basis (1e-13 squared
with a margin of five; an operand in 16 bits would give 1e-6 at best).
"""
import numpy as np
import pytest
import torch

import gmg
import inputs
import oracle as orc

pytestmark = pytest.mark.gpu

TOL = {torch.complex128: 1e-26, torch.complex64: 1e-13}


def _dev(a, dt):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)


def _host(t):
    return t.cpu().numpy().astype(np.complex128)


@pytest.mark.parametrize("dt", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("dims,N,R", [
    ((2, 2, 2, 2), 24, 1),     # a handful of sites
    ((4, 4, 4, 4), 32, 32),    # a split into shares that would open a second wave of CTAs
    ((4, 4, 4, 4), 50, 1),     # two row chunks, one right-hand side
    ((4, 4, 3, 2), 34, 27),    # FP32: seven quads, narrower tiles
    ((4, 4, 2, 2), 50, 64),    # eight units per site
    ((4, 4, 6, 8), 26, 12),
    ((8, 8, 6, 8), 10, 40),    # one share; ten quads
])
@pytest.mark.parametrize("op", ["M", "Mdag", "Mdir"])
def test_stencil(dims, N, R, dt, op):
    r = inputs.rng(stream=910 + N + R)
    V = int(np.prod(dims))
    A = inputs.random_links(dims, N, r)
    x = inputs.gaussian_field((V, R, N), r)
    cm = gmg.CoarsenedMatrix(dims, N)
    cm.set_links(A)
    cm.prepare("f32")
    inp = _dev(x, dt)
    out = torch.full_like(inp, float("nan"))
    if op == "Mdir":
        cm.Mdir(inp, out, 2, -1)
        ref = orc.coarse_apply(dims, A, x, orc.OP_MDIR, point=gmg.lib().gmg_point_from_dir_disp(4, 1, 2, -1))
    else:
        getattr(cm, op)(inp, out)
        ref = orc.coarse_apply(dims, A, x, {"M": orc.OP_M, "Mdag": orc.OP_MDAG}[op])
    # the CUDA-core kernels (one right-hand side on few sites; whole 4 x 4 tiles of 28 right-hand
    # sides and more at nbasis 32 to 40) sum FP32 fields in FP32
    cuda_cores = dt == torch.complex64 and ((R == 1 and N <= 32) or (R >= 28 and 32 <= N <= 40 and R % 4 == N % 4 == 0))
    tol = 1e-11 if cuda_cores else TOL[dt]
    assert orc.rel_dev_sq(ref, _host(out)) < tol


@pytest.mark.parametrize("dt", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("fd,cd,dof,N,R", [
    ((8, 8, 8, 8), (2, 2, 2, 2), 12, 24, 12),   # K 3072
    ((4, 4, 8, 8), (2, 2, 4, 4), 12, 2, 1),     # six promotion items a block: CTAs of fewer warps
    ((8, 8, 8, 8), (4, 4, 4, 4), 12, 16, 16),
    ((4, 4, 6, 4), (2, 2, 2, 2), 12, 24, 5),    # blocks of 24 sites: nine items
    ((10, 6, 6, 6), (10, 6, 6, 1), 12, 60, 58),  # 360 blocks: promotion by chunks of right-hand sides, the last one partial
    ((8, 8, 5, 8), (8, 8, 5, 2), 10, 64, 61),
])
def test_project_and_promote(fd, cd, dof, N, R, dt):
    Vf, Vc = int(np.prod(fd)), int(np.prod(cd))
    r = inputs.rng(stream=920 + N + R)
    B = inputs.gaussian_field((N, Vf, dof), r)
    f = inputs.gaussian_field((Vf, R, dof), r)
    c = inputs.gaussian_field((Vc, R, N), r)
    ag = gmg.Aggregation(fd, cd, dof, N)
    ag.set_basis(B)
    got_c = torch.full((Vc, R, N), float("nan"), dtype=dt, device="cuda")
    got_f = torch.full((Vf, R, dof), float("nan"), dtype=dt, device="cuda")
    ag.ProjectToSubspace(_dev(f, dt), got_c)
    ag.PromoteFromSubspace(_dev(c, dt), got_f)
    assert orc.rel_dev_sq(orc.block_project(fd, cd, B, f), _host(got_c)) < TOL[dt]
    assert orc.rel_dev_sq(orc.block_promote(fd, cd, B, c), _host(got_f)) < TOL[dt]


def test_coarsenings():
    fd, cd, nvec = (6, 4, 4, 6), (2, 2, 2, 3), 5
    U = inputs.hot_gauge(fd, inputs.rng(stream=930))
    B = orc.chiral_double(inputs.gaussian_field((nvec, int(np.prod(fd)), 12), inputs.rng(stream=931)), 0.5)
    ag = gmg.Aggregation(fd, cd, 12, 2 * nvec)
    ag.set_basis(B)
    w = gmg.WilsonClover(fd, -0.1, 1.0, antiperiodic=1)
    w.set_gauge(U)
    cm = gmg.CoarsenedMatrix(cd, 2 * nvec)
    cm.CoarsenOperator(ag, w)
    ref = orc.coarsen_wilson(fd, cd, B, U, orc.clover_build(fd, U, 1.0), -0.1, 1, 0, variant=1)
    got = cm.get_links()
    for p in range(9):
        assert orc.rel_dev_sq(ref[p], got[p]) < 1e-26, p
    A = inputs.random_links(fd, 12, inputs.rng(stream=932))
    fine = gmg.CoarsenedMatrix(fd, 12)
    fine.set_links(A)
    cm.CoarsenOperator(ag, fine)
    ref, got = orc.coarsen_coarse(fd, cd, B, A, variant=1), cm.get_links()
    for p in range(9):
        assert orc.rel_dev_sq(ref[p], got[p]) < 1e-26, p
