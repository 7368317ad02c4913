"""FP64 tensor-core forms (complex products by mma.sync m8n8k4) against the FP64 oracle.

Sizes at the edges of the kernels' tiles: 8 rows, 4 right-hand sides, 4
contracted complex numbers, up to 5 row tiles and 4 right-hand-side quads per
warp.  FP64 results differ from the oracle's by the order of their sums only
(1e-15 relative squared deviation); FP32 fields are widened on load and rounded
once on store (1e-7, as the other FP32 tests).
"""
import numpy as np
import pytest
import torch

import gmg
import inputs
import oracle as orc

pytestmark = pytest.mark.gpu

TOL = {torch.complex128: 1e-15, torch.complex64: 1e-7}


def _dev(a, dt):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dt)


def _host(t):
    return t.cpu().numpy().astype(np.complex128)


@pytest.mark.parametrize("dt", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("dims,N,R", [
    ((2, 2, 2, 2), 2, 2),      # one partial tile in every direction
    ((3, 2, 5, 2), 8, 4),      # exactly one tile
    ((4, 3, 2, 3), 10, 17),    # remainders of rows, of k and of the quads; 5 quads in chunks
    ((2, 2, 2, 3), 40, 5),     # five row tiles
    ((2, 1, 2, 2), 42, 16),    # six row tiles: two row chunks
    ((2, 2, 2, 2), 66, 3),     # nine row tiles
    ((8, 6, 8, 8), 26, 1),     # one right-hand side on a large lattice
    ((8, 8, 6, 8), 12, 13),    # one warp per unit (no split over points)
])
@pytest.mark.parametrize("op", ["M", "Mdag", "Mdiag"])
def test_stencil(dims, N, R, dt, op):
    r = inputs.rng(stream=700 + N + R)
    V = int(np.prod(dims))
    A = inputs.random_links(dims, N, r)
    x = inputs.gaussian_field((V, R, N), r)
    cm = gmg.CoarsenedMatrix(dims, N)
    cm.set_links(A)
    cm.prepare("f32")
    ref = orc.coarse_apply(dims, A, x, {"M": orc.OP_M, "Mdag": orc.OP_MDAG, "Mdiag": orc.OP_MDIAG}[op])
    inp = _dev(x, dt)
    out = torch.full_like(inp, float("nan"))  # every entry is written
    getattr(cm, op)(inp, out)
    assert orc.rel_dev_sq(ref, _host(out)) < TOL[dt]


def test_stencil_active_list():
    dims, N = (4, 2, 3, 2), 18
    r = inputs.rng(stream=790)
    A = inputs.random_links(dims, N, r)
    x = inputs.gaussian_field((48, 9, N), r)
    cm = gmg.CoarsenedMatrix(dims, N)
    cm.set_links(A)
    inp = _dev(x, torch.complex128)
    out = torch.full_like(inp, 7.0)
    active = [8, 0, 3, 5, 1]
    cm.Mdag(inp, out, active=active)
    ref, got = orc.coarse_apply(dims, A, x, orc.OP_MDAG), _host(out)
    for q in range(9):
        if q in active:
            assert orc.rel_dev_sq(ref[:, q], got[:, q]) < 1e-15
        else:
            assert np.all(got[:, q] == 7.0)


@pytest.mark.parametrize("dt", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("fd,cd,dof,N,R", [
    ((4, 4, 4, 4), (2, 2, 2, 2), 12, 2, 1),     # partial tiles of rows and right-hand sides
    ((8, 8, 8, 4), (2, 2, 2, 1), 12, 8, 4),     # exactly one tile, few blocks
    ((6, 4, 6, 4), (2, 2, 2, 2), 10, 18, 7),    # dof not a multiple of 4, block sizes 3 and 2
    ((4, 4, 4, 2), (2, 2, 2, 2), 7, 5, 6),      # odd dof and nbasis; K = 56
    ((3, 3, 2, 2), (3, 3, 2, 2), 12, 3, 5),     # one site per block: fewer sites than warps
    ((8, 8, 8, 8), (4, 4, 4, 4), 12, 40, 21),   # five row tiles, six quads in chunks
    ((4, 4, 4, 4), (2, 2, 2, 2), 40, 48, 33),   # two row chunks, nine quads
    ((8, 8, 8, 8), (4, 8, 8, 8), 12, 24, 30),   # many small blocks
])
def test_project_and_promote(fd, cd, dof, N, R, dt):
    Vf, Vc = int(np.prod(fd)), int(np.prod(cd))
    r = inputs.rng(stream=710 + N + R)
    B = inputs.gaussian_field((N, Vf, dof), r)
    f = inputs.gaussian_field((Vf, R, dof), r)
    c = inputs.gaussian_field((Vc, R, N), r)
    ag = gmg.Aggregation(fd, cd, dof, N)
    ag.set_basis(B)
    got_c = torch.full((Vc, R, N), float("nan"), dtype=dt, device="cuda")  # every entry is written
    got_f = torch.full((Vf, R, dof), float("nan"), dtype=dt, device="cuda")
    ag.ProjectToSubspace(_dev(f, dt), got_c)
    ag.PromoteFromSubspace(_dev(c, dt), got_f)
    assert orc.rel_dev_sq(orc.block_project(fd, cd, B, f), _host(got_c)) < TOL[dt]
    assert orc.rel_dev_sq(orc.block_promote(fd, cd, B, c), _host(got_f)) < TOL[dt]


@pytest.mark.parametrize("fd,cd,nvec,batch", [
    ((6, 4, 4, 6), (2, 2, 2, 2), 5, 0),   # block sizes 3 and 2, nbasis 10
    ((6, 4, 6, 4), (3, 2, 3, 1), 3, 4),   # odd coarse extents and one of 1, batches of 4 and 2
    ((4, 6, 4, 4), (4, 3, 2, 2), 9, 0),   # block extent 1: every site on a face; 144 sites, nbasis 18
])
def test_coarsen_wilson_edges(fd, cd, nvec, batch):
    U = inputs.hot_gauge(fd, inputs.rng(stream=730 + nvec))
    h = inputs.gaussian_field((nvec, int(np.prod(fd)), 12), inputs.rng(stream=740 + nvec))
    B = orc.chiral_double(h, 0.5)
    ag = gmg.Aggregation(fd, cd, 12, 2 * nvec)
    ag.set_basis(B)
    ag.set_coarsen_batch(batch)
    w = gmg.WilsonClover(fd, -0.1, 1.0, antiperiodic=1)
    w.set_gauge(U)
    cm = gmg.CoarsenedMatrix(cd, 2 * nvec)
    cm.CoarsenOperator(ag, w)
    ref = orc.coarsen_wilson(fd, cd, B, U, orc.clover_build(fd, U, 1.0), -0.1, 1, 0, variant=1)
    got = cm.get_links()
    for p in range(9):
        assert orc.rel_dev_sq(ref[p], got[p]) < 1e-15, p


def test_coarsen_coarse_edges():
    fd, cd, dof, nvec = (6, 4, 4, 2), (3, 2, 2, 1), 10, 4  # odd coarse extents, site dof not a multiple of 4
    r = inputs.rng(stream=750)
    A = inputs.random_links(fd, dof, r)
    B = orc.chiral_double(inputs.gaussian_field((nvec, int(np.prod(fd)), dof), r), 0.5)
    fine = gmg.CoarsenedMatrix(fd, dof)
    fine.set_links(A)
    ag = gmg.Aggregation(fd, cd, dof, 2 * nvec)
    ag.set_basis(B)
    cm = gmg.CoarsenedMatrix(cd, 2 * nvec)
    cm.CoarsenOperator(ag, fine)
    ref = orc.coarsen_coarse(fd, cd, B, A, variant=1)
    got = cm.get_links()
    for p in range(9):
        assert orc.rel_dev_sq(ref[p], got[p]) < 1e-15, p
