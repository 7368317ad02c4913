"""Block orthonormalisation at the limits of the range."""
import numpy as np
import pytest

import gmg
import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 9, 40, 44])  # one to five tiles of the tensor-core Gram kernel, and the other path
def test_check_reports_a_vector_whose_norm_overflows(N):
    fd, cd, dof = (4, 4, 4, 2), (2, 2, 2, 1), 12
    r = inputs.rng(stream=890 + N)
    B = np.zeros((N, 128, dof), dtype=np.complex128)
    ag = gmg.Aggregation(fd, cd, dof, N)
    # the last vector shares no site component with the others: only its own norm shows it
    B[:N - 1, :, :6] = inputs.gaussian_field((max(N - 1, 1), 128, 6), r)[:N - 1]
    B[N - 1, :, 6:] = inputs.gaussian_field((1, 128, 6), r)[0]
    ag.set_basis(B)
    ag.Orthogonalise(passes=2)
    B = ag.get_basis()
    assert ag.CheckOrthogonal() < 1e-13
    B[N - 1] *= 1e200 * (1 + 1j)
    ag.set_basis(B)
    assert ag.CheckOrthogonal() == np.inf
