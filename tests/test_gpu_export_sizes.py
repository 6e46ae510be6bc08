"""Sizes announced for an export against what the export returns.

Diagonal sums that cancel leave rounding of either side of the drop limit,
depending on the order they are added in: the order of the tiles is not that of
the row lists. The announced count is what a caller allocates by.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sector", [(14, 7, None, None), (16, 8, 0, None), (16, 8, 3, None), (18, 9, 0, 1)])
@pytest.mark.parametrize("j,delta,j2", [(1.0, 0.7, 0.5), (10.0, 0.7, 0.3), (33.3, 1.1, 0.77)])
def test_announced_count_is_the_exported_count(sector, j, delta, j2):
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    from qmbed_b200._lib import check, lib
    sites, up, momentum, parity = sector
    terms = heisenberg_terms(sites, j=j, delta=delta, j2=j * j2)
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), terms)
    announced, returned = ctypes.c_uint64(), ctypes.c_uint64()
    check(lib().qmbed_gpu_operator_export_csr(op.handle, ctypes.byref(announced), None, None, None))
    row_ptr = np.zeros(op.dim + 1, np.uint64)
    check(lib().qmbed_gpu_operator_export_csr(op.handle, ctypes.byref(returned), row_ptr.ctypes.data, None, None))
    assert announced.value == returned.value == row_ptr[-1]
