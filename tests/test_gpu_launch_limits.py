"""Kernels with more than 48 KB of shared memory, called with different sizes from several threads.

A kernel's limit on dynamic shared memory belongs to the process: a thread that
launches a smaller size must not lower it under another thread's launches.
"""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_threads(*jobs):
    errors = []

    def run(job):
        try:
            job()
        except Exception as error:  # noqa: BLE001 - reported below
            errors.append(error)

    threads = [threading.Thread(target=run, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_exchange_kernel_sizes():
    """36 sites with 32 up take 54 KB, 34 with 31 up 51 KB, the same kernel."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    large, small = (GpuOperator(GpuBasis(sites, up=up, momentum=0, parity=1), heisenberg_terms(sites, j2=0.3),
                                storage="matrix_free") for sites, up in ((36, 32), (34, 31)))

    def product(op):
        x = torch.ones(op.dim, device="cuda", dtype=torch.float64)
        y = torch.empty_like(x)
        op.apply_device(x, y)
        torch.cuda.synchronize()
        return y

    want = product(large)
    _in_threads(lambda: product(small))
    assert torch.equal(product(large), want)


def test_projected_eigenproblem_and_assembly_sizes():
    """Dense eigenproblems of two sizes (84 and 105 rows, below the dense limit of 128) on two threads."""
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms

    def solve(sites, up, count):
        op = GpuOperator(GpuBasis(sites, up=up), heisenberg_terms(sites, delta=0.4))
        want = np.linalg.eigvalsh(op.to_scipy().toarray())[:3]
        for _ in range(count):
            got = op.eigsh(3).eigenvalues
            assert np.max(np.abs(got - want)) < 1e-11

    def assemble(sites, j2, count):
        for _ in range(count):
            basis = GpuBasis(sites, up=sites // 2, momentum=0, parity=1)
            op = GpuOperator(basis, heisenberg_terms(sites, j2=j2))
            assert op.info()["nnz_offdiag"] > 0

    _in_threads(lambda: solve(9, 3, 400), lambda: solve(15, 2, 300))  # 84 and 105 rows
    _in_threads(lambda: assemble(26, 0.5, 40), lambda: assemble(22, 0.0, 80))
