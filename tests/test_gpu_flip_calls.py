"""Flip-chain calls beside the plain product: refused outputs, first products under capture."""

import pytest

pytestmark = pytest.mark.gpu


def _chain(sites):
    from qmbed_b200 import GpuBasis, GpuOperator
    return GpuOperator(GpuBasis(sites), [("zz", [(0.4, (i, (i + 1) % sites)) for i in range(sites)]),
                                         ("x", [(0.2 + 0.01 * i, (i,)) for i in range(sites)])], storage="matrix_free")


def test_group_passes_refuse_their_input_as_output(monkeypatch):
    """Passes add to the output, so it cannot be the input; the one-launch form keeps its tile kernel for it."""
    import torch
    from qmbed_b200 import QmbedError
    op = _chain(18)
    x = torch.randn(op.dim, device="cuda", dtype=torch.float64)
    monkeypatch.setenv("QMBED_FLIP_PASSES", "multi")
    with pytest.raises(QmbedError, match="cannot write over"):
        op.apply_device(x, x)


@pytest.mark.parametrize("sites", [9, 18])
def test_first_product_of_an_element_size_under_capture(sites):
    """After one product of any kind, products of every kind can be captured (no allocation is left to make)."""
    import torch
    kinds = [(torch.float64, 64, False), (torch.complex128, 64, True), (torch.float32, 32, False),
             (torch.complex64, 32, True)]
    for warm in kinds:
        op, ref = _chain(sites), _chain(sites)
        x = torch.randn(op.dim, device="cuda").to(warm[0])
        op.apply_device(x, torch.empty_like(x), precision=warm[1], complex_vectors=warm[2])
        for dtype, precision, cplx in kinds:
            for offset in (0, 1):  # whole vectors, and views off the 16-byte boundary
                buf = torch.randn(op.dim + 1, device="cuda", dtype=dtype)
                x = buf[offset:offset + op.dim]
                out = torch.full((op.dim + 1,), float("nan"), device="cuda", dtype=dtype)
                y = out[offset:offset + op.dim]
                want = torch.empty(op.dim + 1, device="cuda", dtype=dtype)[offset:offset + op.dim]
                ref.apply_device(x, want, precision=precision, complex_vectors=cplx)
                graph = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(graph):
                    op.apply_device(x, y, precision=precision, complex_vectors=cplx,
                                    stream=torch.cuda.current_stream().cuda_stream)
                graph.replay()
                torch.cuda.synchronize()
                assert torch.equal(y, want)
