"""Thermal runs refuse Krylov dimensions above 8192 before they take memory for them."""

import pytest

pytestmark = pytest.mark.gpu


def test_dimension_above_the_limit():
    from qmbed_b200 import GpuBasis, GpuOperator, QmbedError, heisenberg_terms
    from qmbed_b200.lanczos import ftlm_sample
    # 8192 columns of 4,850,640 rows would be 318 GB
    op = GpuOperator(GpuBasis(31, up=15, momentum=0, parity=1), heisenberg_terms(31), storage="matrix_free")
    with pytest.raises(QmbedError, match="above 8192"):
        ftlm_sample(op, 1, [1.0], 9000)
