"""Lanczos decompositions whose tolerance lies below the fixed 1e-14 of the step kernels.

A diagonal operator and a start vector of three basis states with a trace of a
fourth: the Krylov space is exhausted after three steps but for that trace, so
the third norm is beta_2 = trace |prod (l_d - l_i)| / (|v| beta_0 beta_1), set
here to 6e-15. With a tolerance of 1e-15 the run goes on, and its fourth column
is the trace's state: sums of at most four terms of size |H| <= 1 leave up to
4e-16 of other directions in a vector of 6e-15. Every run must give the same
bytes, whatever lies in the memory its columns take. Sectors: the fused step
(12,870 rows) and the separate launches (184,756 rows), real and complex starts.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(sites, cplx):
    from qmbed_b200 import GpuBasis, GpuOperator
    rng = np.random.default_rng(sites)
    fields = rng.uniform(0.2, 1.0, sites) / sites
    op = GpuOperator(GpuBasis(sites, up=sites // 2), [("z", [(float(h), (i,)) for i, h in enumerate(fields)])])
    energies = op.to_scipy().diagonal().real
    order = np.argsort(energies)
    at = order[[0, op.dim // 3, (2 * op.dim) // 3, op.dim - 1]]
    lam = energies[at]
    amp = np.array([0.7, 1.0, 0.8])
    # beta_0 and beta_1 of the three states
    q = amp / np.linalg.norm(amp)
    w = lam[:3] * q
    w = w - (q @ w) * q
    beta0 = np.linalg.norm(w)
    p = w / beta0
    w = lam[:3] * p
    w = w - (p @ w) * p - beta0 * q
    beta1 = np.linalg.norm(w - q * (q @ w))
    trace = 6e-15 * np.linalg.norm(amp) * beta0 * beta1 / abs(np.prod(lam[3] - lam[:3]))
    start = np.zeros(op.dim, np.complex128 if cplx else np.float64)
    start[at] = np.append(amp, trace)
    if cplx:
        start[at] *= np.exp(1j * np.array([0.3, 1.1, -0.4, 2.0]))
    return op, start, at, lam


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("sites", [16, 20])
def test_norms_between_the_tolerance_and_the_kernels_floor(sites, cplx):
    from qmbed_b200.lanczos import LanczosBasis
    op, start, at, lam = _case(sites, cplx)
    rng = np.random.default_rng(7)
    first = None
    for _ in range(3):
        # another run leaves its columns in the memory that the next one takes
        other = rng.standard_normal(op.dim) + (1j * rng.standard_normal(op.dim) if cplx else 0.0)
        LanczosBasis(op, other, 4, 1e-15).close()
        basis = LanczosBasis(op, start, 4, 1e-15)
        assert basis.krylov_dimension == 4
        q = basis.to_numpy()
        got = (basis.diagonal.tobytes(), basis.off_diagonal.tobytes(), q.tobytes())
        basis.close()
        assert 5e-15 < basis.off_diagonal[2] < 7e-15
        assert np.max(np.abs(np.linalg.norm(q, axis=1) - 1.0)) < 1e-13
        assert abs(q[3, at[3]]) > 0.95 and abs(basis.diagonal[3] - lam[3]) < 0.1 * np.max(np.abs(lam))
        assert first is None or got == first
        first = got
