"""Row lists of operators held as tiles: assembled for an export or a scan, and gone afterwards.

26 sites at k = 3 (400,023 rows, 10 million entries): 42 MB of tiles, 280 MB as
rows with explicit values. 64 MB are left for the driver.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_exports_leave_nothing():
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(26, up=13, momentum=3), heisenberg_terms(26, delta=0.8))
    before = _free()
    row_ptr, cols, values = op.csr()
    assert before - _free() < (64 << 20)
    assert row_ptr[-1] == len(cols) == len(values)
    assert len(cols) - op.info()["nnz_offdiag"] == np.count_nonzero(cols == np.repeat(np.arange(op.dim), np.diff(row_ptr.astype(np.int64))))


@pytest.mark.parametrize("sector,cplx", [((14, 7, 3, None), True), ((14, 7, 0, 1), False), ((13, 6, None, -1), False)])
@pytest.mark.parametrize("storage", ["packed", "explicit"])
def test_the_count_before_an_export(sector, cplx, storage):
    """The sizes of the arrays: entries and nonzero diagonal values."""
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    sites, up, momentum, parity = sector
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), heisenberg_terms(sites, j2=0.5, delta=0.7),
                     storage=storage)
    row_ptr, cols, values = op.csr()
    assert op.is_real != cplx and row_ptr[-1] == len(cols)
    assert np.all(values != 0.0)  # every slot of the arrays was filled
    dense = op.to_scipy().toarray()
    assert np.max(np.abs(dense - dense.conj().T)) < 1e-13


def test_scans_of_packed_components():
    from qmbed_b200 import GpuBasis, GpuOperator
    from qmbed_b200.scan import j1j2_component_terms, j1j2_scan_points, scan_lowest
    points = j1j2_scan_points(3, seed=2)
    got = {}
    for storage in ("packed", "explicit"):
        basis = GpuBasis(18, up=9, momentum=2)
        ops = [GpuOperator(basis, terms, storage=storage) for terms in j1j2_component_terms(18)]
        if storage == "packed":
            # components without off-diagonal entries are real and stay packed: scans take explicit rows of those
            ops = [op if not op.is_real else GpuOperator(basis, terms, storage="explicit")
                   for op, terms in zip(ops, j1j2_component_terms(18))]
            assert any(op.info()["storage"] == 2 for op in ops)
        scan_lowest([ops], points, eigenpairs=2)
        before = _free()
        got[storage] = scan_lowest([ops], points, eigenpairs=2)[0]
        assert before - _free() < (64 << 20)
    np.testing.assert_allclose(got["packed"], got["explicit"], atol=1e-9)
