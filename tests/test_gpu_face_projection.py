"""The face projections of the Wilson coarsening (half-spinors, two sites a turn).

Faces of one site and of other odd counts, where the last turn has one site only,
every direction and both of a lattice's small and large block counts, against the
oracle's full-spinor construction: FP64 sums in another order (1e-15 relative
squared deviation, as the other construction tests).
"""
import numpy as np
import pytest

import gmg
import inputs
import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fd,cd,nvec", [
    ((4, 3, 2, 3), (2, 3, 2, 3), 2),      # blocks of two sites: faces of one and of two
    ((6, 6, 6, 2), (2, 2, 2, 2), 5),      # faces of 9
    ((4, 6, 6, 6), (2, 2, 2, 2), 9),      # faces of 27 and 18
    ((12, 6, 12, 9), (6, 6, 6, 9), 7),    # 1944 blocks: the units of a block in one CTA
])
@pytest.mark.parametrize("apbc", [0, 1])
def test_faces(fd, cd, nvec, apbc):
    U = inputs.hot_gauge(fd, inputs.rng(stream=830 + nvec))
    B = orc.chiral_double(inputs.gaussian_field((nvec, int(np.prod(fd)), 12), inputs.rng(stream=840 + nvec)), 0.5)
    ag = gmg.Aggregation(fd, cd, 12, 2 * nvec)
    ag.set_basis(B)
    w = gmg.WilsonClover(fd, -0.1, 1.0, antiperiodic=apbc)
    w.set_gauge(U)
    cm = gmg.CoarsenedMatrix(cd, 2 * nvec)
    cm.CoarsenOperator(ag, w)
    ref = orc.coarsen_wilson(fd, cd, B, U, orc.clover_build(fd, U, 1.0), -0.1, apbc, 0, variant=1)
    got = cm.get_links()
    for p in range(9):
        assert orc.rel_dev_sq(ref[p], got[p]) < 1e-15, p
