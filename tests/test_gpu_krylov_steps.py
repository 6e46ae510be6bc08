"""Fused and queued Gram-Schmidt steps of the FP64 Krylov solvers.

A Lanczos basis and thick-restart eigenpairs over sectors at the edges of the
fused step's slabs (128 rows a block up to 18 944 rows, then 256, 512, 1024;
separate launches beyond 151 552, which take one, two and three elements a
thread: pairs of rows, rows of odd dimensions, complex rows), dimensions below a
slab, real and complex, with panels from one column on. Tolerances: two Gram-Schmidt
passes leave the basis orthonormal to a few eps per column (1e-13 for up to 60
columns, the run ended at norms of 1e-4); projections of H are exact to 1e-13 |H|; eigenpairs are asked for
with residuals of 1e-10.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# sites, up, momentum -> dimension
SECTORS = [(3, 1, None), (5, 2, None), (9, 4, None), (10, 4, None), (16, 8, None), (20, 10, 3), (17, 8, None),
           (18, 9, None), (19, 9, None), (20, 10, None)]
LARGE = [(21, 10, None), (22, 11, None), (28, 9, 0), (27, 10, 0), (26, 13, 3)]  # 246 675 and 312 455 rows are odd


def _operator(sites, up, momentum):
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    return GpuOperator(GpuBasis(sites, up=up, momentum=momentum), heisenberg_terms(sites, delta=0.7, j2=0.3))


@pytest.mark.parametrize("sector", SECTORS + LARGE)
def test_lanczos_basis(sector):
    from qmbed_b200.lanczos import LanczosBasis
    op = _operator(*sector)
    rng = np.random.default_rng(sum(filter(None, sector)))
    start = rng.standard_normal(op.dim) + (0.0 if op.is_real else 1j * rng.standard_normal(op.dim))
    basis = LanczosBasis(op, start, min(60 if sector in SECTORS else 12, op.dim), 1e-4)
    q, m = basis.to_numpy(), basis.krylov_dimension
    assert m >= (2 if op.dim < 100 else 30 if sector in SECTORS else 12)
    assert np.max(np.abs(q.conj() @ q.T - np.eye(m))) < 1e-13
    projected = q.conj() @ (op.to_scipy() @ q.T)
    t = np.diag(basis.diagonal) + np.diag(basis.off_diagonal, 1) + np.diag(basis.off_diagonal, -1)
    assert np.max(np.abs(projected - t)) < 1e-13 * 2.0 * sector[0]


@pytest.mark.parametrize("sector", [s for s in SECTORS if s[0] >= 9])
def test_thick_restart_eigenpairs(sector):
    op = _operator(*sector)
    h = op.to_scipy()
    got = op.eigsh(4, krylov_dimension=24, eigenvectors=True, tolerance=1e-10, seed=3,
                   max_iterations=4000)
    assert got.converged
    x = got.eigenvectors
    assert np.max(np.abs(x.conj() @ x.T - np.eye(4))) < 1e-13
    for value, vector in zip(got.eigenvalues, x):
        assert np.linalg.norm(h @ vector - value * vector) < 1e-9
    if op.dim < 2000:
        np.testing.assert_allclose(got.eigenvalues, np.linalg.eigvalsh(h.toarray())[:4], atol=1e-11 * sector[0])
