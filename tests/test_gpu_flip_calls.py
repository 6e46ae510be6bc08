"""Flip-chain calls beside the plain product: refused outputs."""

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
