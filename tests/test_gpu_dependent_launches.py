"""Products whose launch overlaps the end of the one before, in chains of dependent calls.

A product's blocks may become resident while the stream's previous kernel
drains; they wait before they read a vector. 300 products run back to back on
two vectors in turn (each reads what the one before wrote, and writes what that
one read) and must give the bytes of the same products with a synchronisation
after each, in vectors small enough to stay in the L1s and larger than all of
them together. Same kernels, same order of sums: equality is exact.
"""

import pytest

pytestmark = pytest.mark.gpu


def _chain(step, x, y, count, wait):
    import torch
    for _ in range(count):
        step(x, y)
        x, y = y, x
        if wait:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    return x


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("kind,sites", [("packed", 12), ("packed", 18), ("packed", 22), ("packed", 26),
                                        ("matrix_free", 14), ("matrix_free", 20), ("matrix_free", 26),
                                        ("block", 16), ("block", 24), ("flip", 13), ("flip", 16), ("flip", 20)])
@pytest.mark.parametrize("captured", [False, True])
def test_chains_of_products(kind, sites, precision, captured):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    dtype = torch.float64 if precision == 64 else torch.float32
    if kind == "flip":
        terms = [("zz", [(0.11, (i, (i + 1) % sites)) for i in range(sites)]), ("x", [(0.07, (i,)) for i in range(sites)])]
        op = GpuOperator(GpuBasis(sites), terms, storage="matrix_free")
    else:
        terms = [(word, [(0.08 * c, s) for c, s in pairs]) for word, pairs in heisenberg_terms(sites, delta=0.6)]
        op = GpuOperator(GpuBasis(sites, up=sites // 2, momentum=0, parity=1), terms,
                         storage="matrix_free" if kind == "matrix_free" else "packed")
    columns = 8 if kind == "block" else 1
    start = torch.randn(op.dim * columns, device="cuda", dtype=dtype)

    def step(x, y):
        stream = torch.cuda.current_stream().cuda_stream
        if kind == "block":
            op.apply_block_device(x, y, columns, precision=precision, alpha=0.9, beta=0.4, stream=stream)
        else:
            op.apply_device(x, y, precision=precision, stream=stream)

    x, y = start.clone(), torch.zeros_like(start)
    want = _chain(step, x, y, 300, True).clone()
    x, y = start.clone(), torch.zeros_like(start)
    if captured:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(5):
                step(x, y)
                step(y, x)
        for _ in range(30):
            graph.replay()
        torch.cuda.synchronize()
        got = x
    else:
        got = _chain(step, x, y, 300, False)
    assert torch.isfinite(want).all() and torch.equal(got, want)
