"""Filtered eigenpairs where the block Gram and rotation kernels end inside a tile of rows.

Dimensions with the remainders 0, 2, 3, 4 and 6 of 8 rows (the rotation's tile; the
Gram takes 4), blocks of 8 and of 16 vectors. The filtered
mode's FP64 phase accepts residuals of 1e-10 max(|lambda|, 1); eigenvalues of a
Hermitian operator are then within 1e-9 of the dense ones.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sector", [(18, 9, 0, 1), (19, 8, 0, None), (17, 8, 0, None), (18, 8, 0, None),
                                    (19, 9, 0, 1), (19, 7, 0, None), (18, 9, 9, None), (18, 7, 0, None)])
@pytest.mark.parametrize("pairs", [2, 9])
def test_filtered_pairs_against_dense(sector, pairs):
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    sites, up, momentum, parity = sector
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), heisenberg_terms(sites, delta=1.3, j2=0.2))
    h = op.to_scipy().toarray()
    got = op.eigsh(pairs, mode="filtered", tolerance=1e-10, seed=2, eigenvectors=True)
    assert got.converged
    np.testing.assert_allclose(got.eigenvalues, np.linalg.eigvalsh(h)[:pairs], atol=1e-9)
    x = got.eigenvectors
    assert np.max(np.abs(x.conj() @ x.T - np.eye(pairs))) < 1e-9
    assert max(np.linalg.norm(h @ v - e * v) for e, v in zip(got.eigenvalues, x)) < 1e-9 * sites
