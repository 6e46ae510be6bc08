"""A product over its own input takes its copy's memory from the pool's idle blocks where nothing else is free.

A thermal run on 28 sites leaves its panel of 575 MB in the pool; 16 MB are left
beside it, and the copy of a complex vector of 31 sites takes 78 MB.
"""

import pytest

pytestmark = pytest.mark.gpu


def test_a_copy_that_needs_the_pool():
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    from qmbed_b200.lanczos import ftlm_sample
    small = GpuOperator(GpuBasis(28, up=14, momentum=0, parity=1), heisenberg_terms(28))
    op = GpuOperator(GpuBasis(31, up=15, momentum=0, parity=1), heisenberg_terms(31))
    x = torch.randn(op.dim, device="cuda", dtype=torch.complex128)
    want = torch.empty_like(x)
    op.apply_device(x, want, complex_vectors=True)
    ftlm_sample(small, 1, [0.5], 100, seed=3)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), device="cuda", dtype=torch.uint8)
    try:
        op.apply_device(x, x, complex_vectors=True)
        torch.cuda.synchronize()
    finally:
        del filler
        torch.cuda.empty_cache()  # the other tests' memory
    assert torch.equal(x, want)
