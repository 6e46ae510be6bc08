"""Exchange kernels that need more than 48 KB of shared memory (matrix-free J1-J2, many up spins).

Several variants of the kernel on one sector size take the same amount of
shared memory: real and complex vectors on a real sector, parity +1 and -1.
Each has to be set up for it by itself. Reference and tolerance as in the
exchange kernel's other tests: the general kernel on the same table, 1e-14
(FP64) and 2e-6 (FP32) of |H| |x|.
"""

import pytest

pytestmark = pytest.mark.gpu


def _operator(sites, up, momentum, parity):
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    return GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity),
                       heisenberg_terms(sites, delta=0.8, j2=0.4), storage="matrix_free")


def _check(op, sites, precision, cplx):
    import torch
    dtype = {(64, False): torch.float64, (32, False): torch.float32, (64, True): torch.complex128,
             (32, True): torch.complex64}[precision, cplx]
    x = torch.randn(op.dim, device="cuda", dtype=dtype)
    y, ref = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
    op.set_lookup("auto")
    op.apply_device(x, y, precision=precision, complex_vectors=cplx)
    op.set_lookup("table_generic")
    op.apply_device(x, ref, precision=precision, complex_vectors=cplx)
    op.set_lookup("auto")
    assert float((y - ref).norm()) <= (1e-14 if precision == 64 else 2e-6) * 5.0 * sites * float(x.norm())


@pytest.mark.parametrize("sites,up", [(34, 31), (36, 32), (36, 29)])
def test_variants_of_one_size(sites, up):
    for parity in (1, -1):
        op = _operator(sites, up, 0, parity)
        for precision in (64, 32):
            for cplx in (False, True):
                _check(op, sites, precision, cplx)
    _check(_operator(sites, up, 3, None), sites, 64, True)
