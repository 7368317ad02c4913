"""The Gram kernel's half tile (33 to 36 basis vectors) against the oracle's Gram-Schmidt.

One to four vectors in the last tile, values of k short of a step and of a warp's share,
with four and with eight warps a block; two passes of a well-conditioned Gaussian panel
leave 1e-13 relative at most (1e-24 squared, as the other tests of this operation).
"""
import numpy as np
import pytest

import gmg
import inputs
import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fd,cd,dof,N", [
    ((8, 8, 8, 4), (1, 1, 2, 1), 2, 33),     # K 2048, two blocks
    ((4, 4, 4, 4), (2, 2, 2, 2), 3, 34),     # K 48
    ((6, 4, 4, 2), (2, 2, 2, 1), 13, 35),    # K 312
    ((8, 8, 6, 8), (4, 8, 3, 8), 13, 36),    # 768 blocks (four warps each), K 52
])
def test_orthonormalise(fd, cd, dof, N):
    B0 = inputs.gaussian_field((N, int(np.prod(fd)), dof), inputs.rng(stream=940 + N))
    ag = gmg.Aggregation(fd, cd, dof, N)
    ag.set_basis(B0)
    ag.Orthogonalise(passes=2)
    assert orc.rel_dev_sq(orc.block_orthonormalise(fd, cd, B0, passes=2), ag.get_basis()) < 1e-24
    assert ag.CheckOrthogonal() < 1e-13
