"""The projected eigenproblems (device Jacobi) at the edges of their sizes.

Complete spectra of small sectors through the dense path of eigsh, against
numpy on the assembled matrix: odd and even sizes, real and complex, the
largest that fit shared memory and the first beyond. Eigenvalues of a
backward-stable solver differ by a small multiple of eps |H| (here |H| < 10);
1e-12 is that with room for the size.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (sites, up, momentum, parity): dimension 2, 3, 25 and 26 (complex), 31, 70, 77 and 80 (complex: the
# shared-memory limit is 78), 80 and 112 to 126 (real: the limit is 112)
SECTORS = [(4, 2, 0, 1), (6, 3, 0, None), (10, 5, 3, None), (10, 5, 2, None), (12, 6, 0, 1), (8, 4, None, None),
           (12, 6, 1, None), (12, 6, 2, None), (12, 6, 0, None), (16, 2, None, None), (9, 4, None, None)]


@pytest.mark.parametrize("sector", SECTORS)
def test_dense_spectrum(sector):
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    sites, up, momentum, parity = sector
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), heisenberg_terms(sites, delta=0.7, j2=0.3))
    h = op.to_scipy().toarray()
    want = np.linalg.eigvalsh(h)
    k = max(1, op.dim - 1)
    r = op.eigsh(k, eigenvectors=True, tolerance=1e-10)
    assert np.max(np.abs(r.eigenvalues - want[:k])) < 1e-12
    v = r.eigenvectors
    assert np.max(np.abs(v.conj() @ v.T - np.eye(k))) < 1e-11
    assert np.max(np.linalg.norm(v @ h.T - r.eigenvalues[:, None] * v, axis=1)) < 1e-11


def test_thick_restart_complex_sector(oracle):
    from qmbed_b200 import GpuBasis, GpuOperator
    terms = oracle.heisenberg_terms(18, delta=0.8)
    op = GpuOperator(GpuBasis(18, up=9, momentum=5), terms)
    ref = oracle.Operator.build(oracle.Basis(18, up=9, momentum=5), terms)
    for m in (21, 32):
        got = op.eigsh(3, krylov_dimension=m, tolerance=1e-11, seed=4).eigenvalues
        want = ref.eigsh(3, krylov_dimension=m, tolerance=1e-11, seed=4).eigenvalues
        assert np.max(np.abs(got - want) / np.abs(want)) < 1e-10
