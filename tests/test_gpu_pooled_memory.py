"""Device memory that calls leave behind: at most the pool's 1 GiB per device, given back when it is needed.

Handles of three 28-site sectors run thermal Lanczos with panels of 575 MB each,
a 22-site propagation takes 270 MB of vectors. What stays allocated while the
handles live is compared with what their own buffers take (measured in front of
the calls), with 256 MB to spare for the solvers' small buffers and the driver.
"""

import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30
SPARE = 256 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _thermal(op):
    from qmbed_b200.lanczos import ftlm_sample
    return ftlm_sample(op, 1, [0.5], 100, seed=3)


def _handles():
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    return [GpuOperator(GpuBasis(28, up=14, momentum=k, parity=p), heisenberg_terms(28, delta=d))
            for k, p, d in ((0, 1, 1.0), (14, -1, 1.0), (0, 1, 0.5))]


def test_what_calls_leave_behind():
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    _thermal(_handles()[0])  # the library's own setup
    start = _free()
    ops = _handles()
    sites = 22
    chain = GpuOperator(GpuBasis(sites), [("zz", [(0.5, (i, (i + 1) % sites)) for i in range(sites)]),
                                          ("x", [(0.4, (i,)) for i in range(sites)])], storage="matrix_free")
    before = _free()
    for op in ops:
        _thermal(op)
        op.eigsh(2, krylov_dimension=40, tolerance=1e-6)
    state = torch.zeros(1 << sites, device="cuda", dtype=torch.complex128)
    state[5] = 1.0
    chain.chebyshev_evolve_device(state, [0.1])
    del state
    assert before - _free() <= GIB + SPARE
    for op in ops:
        op.close()
    chain.close()
    assert start - _free() <= SPARE


def test_an_allocation_that_needs_the_pool():
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = _handles()[0]
    _thermal(op)  # leaves its panel of 575 MB in the pool
    other = GpuBasis(28, up=14, momentum=3)
    filler = torch.empty(_free() - (200 << 20), device="cuda", dtype=torch.uint8)
    try:
        rows = GpuOperator(other, heisenberg_terms(28))  # 1.4 million complex rows: 230 MB
    finally:
        del filler
        torch.cuda.empty_cache()  # the other tests' memory
    assert rows.info()["nnz_offdiag"] > 0 and op.dim > 0
