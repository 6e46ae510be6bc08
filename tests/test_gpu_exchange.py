"""The exchange kernel (matrix-free, nearest and next-nearest neighbours) against the general table kernel.

set_lookup("table_generic") runs the general kernel on the same image table,
which the parity tests hold against the oracle. Sizes: the smallest chains
(five sites: all wraps touch), odd ones, 31 to 34 sites (the 32-bit state word
ends at 32), the last partial step of four sites in every remainder; sectors
with and without states outside (k = pi, parity -1), complex characters; open
and periodic chains, bonds left out. Rows add at most 2 sites products, so
1e-14 |H| |x| (FP64) and 2e-6 (FP32) bound the two orders' difference.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(5, 2, 0, None), (6, 3, 0, 1), (7, 3, 2, None), (9, 4, 0, 1), (12, 6, 6, -1), (13, 6, 0, -1), (14, 7, 3, None),
         (16, 8, 8, 1), (18, 9, 0, None), (31, 4, 0, 1), (32, 4, 5, None), (33, 4, 0, 1), (34, 5, 17, -1), (34, 4, 3, None)]


def _terms(sites, delta, j2, periodic, field):
    from qmbed_b200 import heisenberg_terms
    terms = heisenberg_terms(sites, delta=delta, j2=j2, periodic=periodic)
    if field:
        terms.append(("z", [(field, (i,)) for i in range(sites)]))
    return terms


@pytest.mark.parametrize("j2,field", [(0.0, 0.0), (0.35, 0.2)])
@pytest.mark.parametrize("sector", CASES)
def test_against_the_general_table_kernel(sector, j2, field):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    sites, up, momentum, parity = sector
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), _terms(sites, 0.7, j2, True, field),
                     storage="matrix_free")
    size = 3.0 * sites * (1.0 + j2)
    for cplx in ([False, True] if op.is_real else [True]):
        for precision, tolerance in ((64, 1e-14), (32, 2e-6)):
            dtype = {(64, False): torch.float64, (32, False): torch.float32, (64, True): torch.complex128,
                     (32, True): torch.complex64}[precision, cplx]
            x = torch.randn(op.dim, device="cuda", dtype=dtype)
            y, ref = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
            op.set_lookup("auto")
            op.apply_device(x, y, precision=precision, complex_vectors=cplx)
            op.set_lookup("table_generic")
            op.apply_device(x, ref, precision=precision, complex_vectors=cplx)
            assert float((y - ref).norm()) <= tolerance * size * float(x.norm())


@pytest.mark.parametrize("j2", [0.0, 0.4])
def test_row_slabs_and_open_chains(j2):
    import ctypes

    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    from qmbed_b200._lib import check, lib
    op = GpuOperator(GpuBasis(15, up=7, parity=1), _terms(15, 1.2, j2, False, 0.0), storage="matrix_free")
    x = torch.randn(op.dim, device="cuda", dtype=torch.float64)
    ref = torch.empty_like(x)
    op.set_lookup("table_generic")
    op.apply_device(x, ref)
    op.set_lookup("auto")
    whole = torch.empty_like(x)
    op.apply_device(x, whole)
    assert float((whole - ref).norm()) <= 1e-14 * 60 * float(x.norm())
    for row0, rows in ((0, 1), (5, 33), (op.dim - 130, 130)):
        part = torch.full((rows,), float("nan"), device="cuda", dtype=torch.float64)
        check(lib().qmbed_gpu_operator_apply_rows_device(op.handle, 64, row0, rows, ctypes.c_void_p(x.data_ptr()),
                                                         ctypes.c_void_p(part.data_ptr()), None))
        assert torch.equal(part, whole[row0:row0 + rows])


def test_infinities_and_alignment():
    """An infinite entry reaches the rows that hold its column and no other; vectors off their own alignment work."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    basis = GpuBasis(14, up=7, momentum=0, parity=1)
    op = GpuOperator(basis, heisenberg_terms(14, delta=0.3, j2=0.2), storage="matrix_free")
    h = GpuOperator(basis, heisenberg_terms(14, delta=0.3, j2=0.2)).to_scipy()
    x = torch.ones(op.dim, device="cuda", dtype=torch.float64)
    x[3] = float("inf")
    y = torch.empty_like(x)
    op.apply_device(x, y)
    assert np.array_equal(~torch.isfinite(y).cpu().numpy(), np.asarray(h[:, [3]].todense()).ravel() != 0)
    buf = torch.randn(2 * op.dim + 1, device="cuda", dtype=torch.float64)
    odd, even = torch.empty_like(buf[1:]), torch.empty_like(buf[1:])
    op.apply_device(buf[1:], odd, complex_vectors=True)
    op.apply_device(buf[1:].clone(), even, complex_vectors=True)
    assert float((odd - even).norm()) <= 1e-14 * 60 * float(buf.norm())


@pytest.mark.parametrize("momentum,parity,j2", [(0, 1, 0.0), (15, -1, 0.3), (4, None, 0.0)])
def test_a_table_beyond_the_l2(momentum, parity, j2):
    """30 sites: an image table of 620 MB, so the kernel's longer steps, here with a last step of six sites."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(30, up=15, momentum=momentum, parity=parity), heisenberg_terms(30, delta=0.6, j2=j2),
                     storage="matrix_free")
    for precision, tolerance in ((64, 1e-14), (32, 2e-6)):
        cplx = not op.is_real
        dtype = {(64, False): torch.float64, (32, False): torch.float32, (64, True): torch.complex128,
                 (32, True): torch.complex64}[precision, cplx]
        x = torch.randn(op.dim, device="cuda", dtype=dtype)
        y, ref = torch.empty_like(x), torch.empty_like(x)
        op.set_lookup("auto")
        op.apply_device(x, y, precision=precision, complex_vectors=cplx)
        op.set_lookup("table_generic")
        op.apply_device(x, ref, precision=precision, complex_vectors=cplx)
        assert float((y - ref).norm()) <= tolerance * 120 * float(x.norm())
