"""H.v of symmetry sectors with stored rows, the output over the input.

Such a call gives the bytes of the call with two vectors: the rows read a copy
of the input (in the stream's own memory, or in the allocation-free entry's
fixed array). Sectors of one tile, of a few, of the
four-warp and the one-warp split, real, complex rows and complex vectors.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["apply_device", "apply_device_noalloc"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("sites,momentum,parity", [(8, 0, 1), (14, 7, -1), (18, 0, 1), (18, 5, None), (24, 0, 1), (26, 3, None)])
def test_output_over_the_input(sites, momentum, parity, precision, entry):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(sites, up=sites // 2, momentum=momentum, parity=parity),
                     heisenberg_terms(sites, delta=0.7, j2=0.2))
    real = torch.float64 if precision == 64 else torch.float32
    for cplx in ([False, True] if op.is_real else [True]):
        x = torch.randn(op.dim * (2 if cplx else 1), device="cuda", dtype=real)
        want = torch.full_like(x, float("nan"))
        getattr(op, entry)(x, want, precision=precision, complex_vectors=cplx)
        getattr(op, entry)(x, x, precision=precision, complex_vectors=cplx)
        assert torch.equal(x, want)


@pytest.mark.parametrize("entry", ["apply_device", "apply_device_noalloc"])
def test_output_over_the_input_under_capture(entry):
    """After calls with two vectors only: the first call of the other kind may be a captured one."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(20, up=10, momentum=0, parity=1), heisenberg_terms(20, delta=0.4))
    start = torch.randn(op.dim, device="cuda", dtype=torch.float64)
    once, twice = torch.empty_like(start), torch.empty_like(start)
    getattr(op, entry)(start, once)
    getattr(op, entry)(once, twice)
    x = start.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        getattr(op, entry)(x, x, stream=torch.cuda.current_stream().cuda_stream)
    for want in (once, twice):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want)
