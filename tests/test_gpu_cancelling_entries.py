"""Stored rows in which transitions to one column cancel: the column is not in the row.

An infinite input reaches exactly the rows whose stored entry (of the row lists
that to_scipy() assembles) is not zero, and the diagonal's row. Sectors whose
characters change sign under parity, at k = pi, and complex ones.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sites,up,momentum,parity,j2", [(12, 6, 6, -1, 0.5), (12, 6, 6, 1, 0.5), (12, 6, 0, -1, 0.5),
                                                        (10, 5, 5, -1, 1.0), (14, 7, 7, -1, 0.3), (12, 4, 4, None, 0.5),
                                                        (12, 6, 3, None, 1.0), (9, 4, None, -1, 0.5)])
def test_infinite_entries(sites, up, momentum, parity, j2):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), heisenberg_terms(sites, delta=0.6, j2=j2))
    h = op.to_scipy().tocsc()
    cplx = not op.is_real
    dtype = torch.complex128 if cplx else torch.float64
    for c in range(op.dim):
        x = torch.ones(op.dim, device="cuda", dtype=dtype)
        x[c] = float("inf")
        y = torch.empty_like(x)
        op.apply_device(x, y, complex_vectors=cplx)
        reached = np.zeros(op.dim, bool)
        reached[h.indices[h.indptr[c]:h.indptr[c + 1]]] = True
        got = ~np.isfinite(y.cpu().numpy())
        got[c] = reached[c]  # the row's own product d x takes the infinity whatever d is
        assert np.array_equal(got, reached)
