"""The flip chain's products when a box copy does not arrive within its bounded wait.

A thread that gives up reads the words itself, so the output is complete and
the same bytes. QMBED_FLIP_WAIT_POLLS=0 makes every wait give up at once (the
copies then arrive as they would have). Boxes of 4 and 16 KB, group passes of
one and of two groups, every element size.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [None, "multi"])
@pytest.mark.parametrize("sites", [10, 13, 17, 18, 22])
def test_products_without_waiting(sites, passes, monkeypatch):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    terms = [("zz", [(0.7, (i, (i + 1) % sites)) for i in range(sites)]), ("x", [(0.3 + 0.01 * i, (i,)) for i in range(sites)])]
    op = GpuOperator(GpuBasis(sites), terms, storage="matrix_free")
    if passes:
        monkeypatch.setenv("QMBED_FLIP_PASSES", passes)
    for dtype, precision in ((torch.complex128, 64), (torch.float64, 64), (torch.complex64, 32), (torch.float32, 32)):
        x = torch.randn(op.dim, device="cuda", dtype=dtype)
        want, got = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
        monkeypatch.delenv("QMBED_FLIP_WAIT_POLLS", raising=False)
        op.apply_device(x, want, precision=precision, complex_vectors=dtype.is_complex)
        monkeypatch.setenv("QMBED_FLIP_WAIT_POLLS", "0")
        op.apply_device(x, got, precision=precision, complex_vectors=dtype.is_complex)
        assert torch.equal(got, want) and torch.isfinite(torch.view_as_real(want) if dtype.is_complex else want).all()
