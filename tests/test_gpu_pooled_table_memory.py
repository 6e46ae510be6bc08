"""Idle blocks of the pool count as free memory where a lookup table is refused for lack of it.

The image table of 30 sites at half filling takes 620 MB and asks for 1034 MB of
free memory. A thermal run on 28 sites leaves its panel of 575 MB in the pool; 800 MB
are left beside it.
"""

import pytest

pytestmark = pytest.mark.gpu


def test_a_table_that_needs_the_pool():
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    from qmbed_b200.lanczos import ftlm_sample
    op = GpuOperator(GpuBasis(28, up=14, momentum=0, parity=1), heisenberg_terms(28))
    basis = GpuBasis(30, up=15, momentum=0, parity=1)
    ftlm_sample(op, 1, [0.5], 100, seed=3)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (800 << 20), device="cuda", dtype=torch.uint8)
    try:
        free = GpuOperator(basis, heisenberg_terms(30), storage="matrix_free")
    finally:
        del filler
        torch.cuda.empty_cache()  # the other tests' memory
    assert free.lookup_info()["table_bytes"] > 0 and op.dim > 0
