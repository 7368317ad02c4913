"""Block orthonormalisation by FP64 MMAs against the oracle's Gram-Schmidt.

Sizes at the edges of the kernels' tiles: 8 vectors a tile and 4 to 32 values of k a
step (Gram matrix, four and eight warps a block), 128 columns a chunk (substitution,
several CTAs a block and several blocks a CTA).  Both forms give the same
basis up to rounding; two passes of a well-conditioned Gaussian panel leave 1e-13
relative at most (1e-24 squared, as the other tests of this operation).
"""
import numpy as np
import pytest

import gmg
import inputs
import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fd,cd,dof,N", [
    ((2, 2, 2, 2), (2, 2, 1, 1), 1, 2),      # K 4: one step
    ((2, 2, 2, 2), (1, 2, 1, 1), 3, 5),      # K 24
    ((3, 2, 4, 2), (1, 1, 2, 1), 3, 8),      # K 72; exactly one Gram tile
    ((3, 3, 2, 2), (1, 1, 1, 1), 1, 9),      # K 36, one block; one vector in the second Gram tile
    ((6, 4, 4, 4), (2, 2, 2, 2), 5, 16),     # K 120
    ((4, 4, 4, 4), (1, 2, 2, 1), 3, 17),     # K 192
    ((6, 4, 2, 2), (2, 2, 1, 1), 7, 25),     # K 168
    ((8, 8, 8, 4), (1, 1, 2, 1), 2, 33),     # K 2048: a block's chunks over several CTAs
    ((6, 6, 8, 8), (3, 3, 4, 8), 8, 7),      # 288 blocks, K 64
    ((8, 8, 6, 8), (4, 8, 3, 8), 13, 39),    # 768 blocks (four warps each), K 52
])
def test_orthonormalise(fd, cd, dof, N):
    B0 = inputs.gaussian_field((N, int(np.prod(fd)), dof), inputs.rng(stream=800 + N))
    ag = gmg.Aggregation(fd, cd, dof, N)
    ag.set_basis(B0)
    assert np.array_equal(ag.get_basis(), B0)
    ag.Orthogonalise(passes=2)
    assert orc.rel_dev_sq(orc.block_orthonormalise(fd, cd, B0, passes=2), ag.get_basis()) < 1e-24
    assert ag.CheckOrthogonal() < 1e-13
