"""Projected eigenproblems with very small couplings stay unitary.

Dense solves of matrix-free chains whose couplings are 1e-156 and 1e-158 times
the usual ones, in real and complex sectors of 4 to 70 rows: squares of the
matrix elements are subnormal or zero there, and only the rotations' phases and
angles keep the eigenvectors orthonormal. 100 sweeps of 69 rounds of rotations
with unit determinant to a few eps each bound the loss by 100 * 69 * 4 eps =
6e-12.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-150, 1e-156, 1e-158])
@pytest.mark.parametrize("sites,up,momentum", [(8, 4, 1), (8, 4, 0), (10, 5, 1), (12, 4, 1), (12, 5, 2), (8, 4, None)])
def test_small_couplings(sites, up, momentum, scale):
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    terms = [(word, [(scale * c, at) for c, at in pairs]) for word, pairs in heisenberg_terms(sites, delta=0.7, j2=0.3)]
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum), terms, storage="matrix_free")
    assert 3 < op.dim <= 78
    k = min(3, op.dim - 1)
    got = op.eigsh(k, eigenvectors=True)
    x = got.eigenvectors
    assert np.max(np.abs(x.conj() @ x.T - np.eye(k))) < 6e-12
