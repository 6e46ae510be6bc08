"""What Lanczos runs throw away of the steps they queue ahead, in kernel launches.

A step takes 2 launches in the fused sectors and 5 in the larger ones (4 more
when its second pass is the host's, 1 when the host scales the next column).
Runs that end early may have queued eight steps at first, and make the one that
ends them again; runs whose every step the queue leaves short must go step by
step. 30 launches are allowed for the upload, the norms and the read-back.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(sites, size=1.0, offset=0.0):
    from qmbed_b200 import GpuBasis, GpuOperator
    fields = np.random.default_rng(sites).uniform(0.2, 1.0, sites) / sites
    terms = [("z", [(size * float(h), (i,)) for i, h in enumerate(fields)])]
    return GpuOperator(GpuBasis(sites, up=sites // 2), terms + ([("I", [(offset, (0,))])] if offset else []))


def _launches(op, start, m, tolerance):
    from qmbed_b200 import engine
    from qmbed_b200.lanczos import LanczosBasis
    LanczosBasis(op, start, m, tolerance).close()
    before = engine.launch_count()
    basis = LanczosBasis(op, start, m, tolerance)
    return engine.launch_count() - before, basis


@pytest.mark.parametrize("sites,per_step", [(16, 2), (20, 5)])
def test_a_run_that_ends_early(sites, per_step):
    op = _operator(sites)
    start = np.zeros(op.dim)
    start[[3, op.dim // 2, op.dim - 5]] = [0.6, -1.0, 0.8]
    launches, basis = _launches(op, start, 100, 1e-12)
    assert basis.krylov_dimension == 3
    assert launches <= (8 + 1) * per_step + 30


@pytest.mark.parametrize("sites,per_step", [(16, 3), (20, 10)])
def test_a_run_whose_columns_the_host_scales(sites, per_step):
    """Energies of 1e-15 to 9e-15: every norm is below the step kernels' floor, and none near the tolerance.

    Twelve columns: plain 64-bit arithmetic keeps their norms between 2e-16 and
    1e-15. 2^50 H is the same operator to the bit, with norms that the kernels scale by
    themselves: the columns must be the same bytes, the coefficients 2^50 times.
    """
    start = np.random.default_rng(1).standard_normal(_operator(sites).dim)
    launches, basis = _launches(_operator(sites, 8e-15, 5e-15), start, 12, 1e-25)
    assert basis.krylov_dimension == 12 and np.all(basis.off_diagonal <= 8e-15)
    assert launches <= (12 + 8) * per_step + 30
    scaled = _launches(_operator(sites, 8e-15 * 2.0 ** 50, 5e-15 * 2.0 ** 50), start, 12, 1e-25)[1]
    assert np.array_equal(scaled.to_numpy(), basis.to_numpy())
    assert np.array_equal(scaled.diagonal, basis.diagonal * 2.0 ** 50)
    assert np.array_equal(scaled.off_diagonal, basis.off_diagonal * 2.0 ** 50)
