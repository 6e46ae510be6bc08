"""The flip chain's box kernels against a plain 64-bit evaluation.

Sizes at the edges of the dispatch: chains shorter than a box, one box, boxes
of 4 KB and of 16 KB, with and without bits above the box, and forced group
passes of 3 to 9 bits and of two groups, for every element size (4, 8 and 16
bytes: 2, 1 and 0 state bits inside a 16-byte word). Diagonals with terms of
every span (inside a word, the lanes' bits, the box, above it, across all).
A value sums at most sites + 300 rounded products of size up to |c| |x|, so
(sites + 300) eps sum|c| |x| bounds its error; 1e-13 (FP64) and 2e-5 (FP32)
relative to sum|c| |x| hold that.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _terms(sites, kind):
    rng = np.random.default_rng(sites)
    x = [("x", [(float(c), (i,)) for i, c in enumerate(rng.uniform(0.3, 1.2, sites)) if kind != "gaps" or i % 3])]
    if kind == "all_to_all":
        return x + [("zz", [(float(rng.uniform(-1, 1)), (i, j)) for i in range(sites) for j in range(i)])]
    ring = [("zz", [(float(c), (i, (i + 1) % sites)) for i, c in enumerate(rng.uniform(-1, 1, sites))])]
    fields = [("z", [(float(c), (i,)) for i, c in enumerate(rng.uniform(-2, 2, sites))]),
              ("zzz", [(0.37, (0, sites // 2, sites - 1))]), ("I", [(0.21, (0,))])]
    return x + ring + fields


def _reference(sites, terms, x):
    """H x by state bits in 64 bits, and sum|c|."""
    import torch
    s = torch.arange(1 << sites, device="cuda")
    y, size = torch.zeros_like(x), 0.0
    for label, couplings in terms:
        for c, at in couplings:
            size += abs(c)
            if label == "x":
                y += c * x[s ^ (1 << at[0])]
            else:
                sign = torch.ones(1 << sites, device="cuda", dtype=torch.float64)
                for i in at if label != "I" else ():
                    sign = sign * (2.0 * ((s >> i) & 1) - 1.0)
                y += c * sign * x
    return y, size


@pytest.mark.parametrize("kind", ["chain", "all_to_all", "gaps"])
@pytest.mark.parametrize("sites", [3, 8, 9, 10, 11, 16, 17, 18, 19])
def test_box_action(sites, kind):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    terms = _terms(sites, kind)
    op = GpuOperator(GpuBasis(sites, normalization="pauli_cartesian"), terms, storage="matrix_free")
    gen = torch.Generator(device="cuda").manual_seed(sites)
    for dtype, precision, tolerance in ((torch.complex128, 64, 1e-13), (torch.float64, 64, 1e-13),
                                        (torch.complex64, 32, 2e-5), (torch.float32, 32, 2e-5)):
        wide = torch.complex128 if dtype.is_complex else torch.float64
        x = torch.randn(1 << sites, device="cuda", dtype=dtype, generator=gen)
        y = torch.full_like(x, float("nan"))
        op.apply_device(x, y, precision=precision, complex_vectors=dtype.is_complex)
        want, size = _reference(sites, terms, x.to(wide))
        assert float((y.to(wide) - want).norm()) <= tolerance * size * float(x.to(wide).norm())


@pytest.mark.parametrize("sites", [13, 14, 15, 19, 22])
@pytest.mark.parametrize("kind", ["chain", "all_to_all"])
def test_forced_group_passes(sites, kind, monkeypatch):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    monkeypatch.setenv("QMBED_FLIP_PASSES", "multi")
    terms = _terms(sites, kind)
    op = GpuOperator(GpuBasis(sites, normalization="pauli_cartesian"), terms, storage="matrix_free")
    for dtype, precision, tolerance in ((torch.complex128, 64, 1e-13), (torch.complex64, 32, 2e-5)):
        x = torch.randn(1 << sites, device="cuda", dtype=dtype)
        y = torch.full_like(x, float("nan"))
        op.apply_device(x, y, precision=precision, complex_vectors=True)
        want, size = _reference(sites, terms, x.to(torch.complex128))
        assert float((y.to(torch.complex128) - want).norm()) <= tolerance * size * float(x.to(torch.complex128).norm())


@pytest.mark.parametrize("sites", [12, 18])
def test_vectors_between_words(sites):
    """complex64 vectors that start in the middle of a 16-byte word."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    terms = _terms(sites, "chain")
    op = GpuOperator(GpuBasis(sites, normalization="pauli_cartesian"), terms, storage="matrix_free")
    buf = torch.randn((1 << sites) + 1, device="cuda", dtype=torch.complex64)
    out = torch.zeros_like(buf)
    op.apply_device(buf[1:], out[1:], precision=32, complex_vectors=True)
    want, size = _reference(sites, terms, buf[1:].to(torch.complex128))
    assert float((out[1:].to(torch.complex128) - want).norm()) <= 2e-5 * size * float(want.norm())
    assert complex(out[0]) == 0


@pytest.mark.parametrize("passes", ["", "multi"])
def test_fused_steps_in_a_propagation(passes, monkeypatch):
    """p and q of the Clenshaw step: the propagated state against the matrix exponential of a 13-site chain."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    if passes:
        monkeypatch.setenv("QMBED_FLIP_PASSES", passes)
    sites = 13
    terms = _terms(sites, "chain")
    op = GpuOperator(GpuBasis(sites, normalization="pauli_cartesian"), terms, storage="matrix_free")
    v = torch.randn(1 << sites, device="cuda", dtype=torch.complex128)
    v /= v.norm()
    state = v.clone()
    op.chebyshev_evolve_device(state, [0.15, 0.4], tolerance=1e-12)
    _, size = _reference(sites, terms, v)
    want, pieces = v, int(np.ceil(size * 0.4))
    for _ in range(pieces):
        term = want
        for order in range(1, 26):
            term = _reference(sites, terms, term)[0] * (-0.4j / (pieces * order))
            want = want + term
    assert float((state - want).norm()) < 1e-10
