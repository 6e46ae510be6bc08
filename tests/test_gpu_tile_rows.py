"""Stored rows in tiles of 32 against the row lists that to_scipy() assembles.

The two assemblies share no kernel: the row lists expand every product of a
row in one thread and sort, the tiles pop transitions by site pair. The sizes
sit at the edges of the tiles and of the dispatch (one row, 31 to 33 rows, a
partial last tile, four warps per tile or one, eight gathers in flight). A
row sums at most 64 products of rounded factors, so 64 eps |H| |x| bounds the
difference of two orders of summation; 1e-14 (FP64) and 2e-6 (FP32) relative
to |H| |x| hold that.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dm_terms(sites, delta, d):
    bonds = [(i, (i + 1) % sites) for i in range(sites)]
    return [("zz", [(delta, b) for b in bonds]), ("+-", [(0.5 + 0.5j * d, b) for b in bonds]),
            ("-+", [(0.5 - 0.5j * d, b) for b in bonds])]


def _disorder_terms(sites):
    rng = np.random.default_rng(3)
    j = rng.uniform(0.5, 1.5, sites)
    bonds = [(i, (i + 1) % sites) for i in range(sites)]
    return [("zz", [(0.7, b) for b in bonds]), ("z", [(0.1 * i, (i,)) for i in range(sites)]),
            ("xx", [(j[i], b) for i, b in enumerate(bonds)]), ("yy", [(j[i], b) for i, b in enumerate(bonds)])]


def _cases():
    from qmbed_b200 import heisenberg_terms, tfim_terms
    chain = lambda n, **k: heisenberg_terms(n, **k)
    return {
        "one_row": ((4, 0, 0, None), chain(4)),
        "two_rows": ((4, 2, 0, 1), chain(4, delta=0.6)),
        "31_rows": ((12, 6, 0, 1), chain(12, delta=0.6, j2=0.2)),
        "k_pi_negative_parity": ((14, 7, 7, -1), chain(14, delta=1.1)),
        "parity_only": ((13, 6, None, -1), chain(13, j2=0.4)),
        "complex_odd": ((13, 6, 4, None), chain(13, delta=0.9, j2=0.3)),
        "complex_divisors": ((12, 6, 2, None), chain(12, delta=0.9)),
        "dm_k0": ((12, 6, 0, None), _dm_terms(12, 0.8, 0.3)),
        "dm_no_symmetry": ((11, 5, None, None), _dm_terms(11, 0.8, 0.3)),
        "fixed_weight": ((14, 7, None, None), chain(14, j2=0.1)),
        "disorder_codes": ((12, 6, None, None), _disorder_terms(12)),
        "full_space": ((10, None, None, None), tfim_terms(10, fields=np.linspace(-1, 1, 10))),
        "full_space_k0": ((11, None, 0, 1), tfim_terms(11, periodic=True)),
        "split_limit_below": ((24, 12, 0, 1), chain(24)),
        "beyond_split": ((22, 11, 0, None), chain(22, delta=0.5)),
        "over_32_sites": ((34, 4, 0, 1), chain(34, delta=0.5)),
        "over_32_sites_complex": ((33, 4, 3, None), chain(33, delta=0.5)),
    }


@pytest.mark.parametrize("name", ["one_row", "two_rows", "31_rows", "k_pi_negative_parity", "parity_only", "complex_odd",
                                  "complex_divisors", "dm_k0", "dm_no_symmetry", "fixed_weight", "disorder_codes",
                                  "full_space", "full_space_k0", "split_limit_below", "beyond_split", "over_32_sites",
                                  "over_32_sites_complex"])
def test_tiles_against_row_lists(name):
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator
    (sites, up, momentum, parity), terms = _cases()[name]
    op = GpuOperator(GpuBasis(sites, up=up, momentum=momentum, parity=parity), terms, storage="packed")
    h = op.to_scipy()
    info = op.info()
    off = h.copy()
    off.setdiag(0)
    off.eliminate_zeros()
    assert info["nnz_offdiag"] == off.nnz
    rng = np.random.default_rng(8)
    size = abs(h).sum(axis=1).max()
    for cplx in ([False, True] if op.is_real else [True]):
        x = rng.standard_normal(op.dim) + (1j * rng.standard_normal(op.dim) if cplx else 0.0)
        want = h @ x if cplx else (h @ x).real
        for precision, tolerance in ((64, 1e-14), (32, 2e-6)):
            dtype = {(64, False): torch.float64, (32, False): torch.float32, (64, True): torch.complex128,
                     (32, True): torch.complex64}[precision, cplx]
            xd = torch.tensor(x, dtype=dtype, device="cuda")
            yd = torch.full_like(xd, float("nan"))
            op.apply_device(xd, yd, precision=precision, complex_vectors=cplx)
            error = np.linalg.norm(yd.cpu().numpy() - want)
            assert error <= tolerance * size * np.linalg.norm(x)


@pytest.mark.parametrize("sites,momentum", [(14, 0), (13, 4)])
def test_complex_vectors_off_their_own_alignment(sites, momentum):
    """Interleaved complex vectors that start between two elements' boundaries."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(sites, up=sites // 2, momentum=momentum), heisenberg_terms(sites))
    n = op.dim
    for precision, dtype in ((64, torch.float64), (32, torch.float32)):
        x = torch.randn(2 * n + 1, device="cuda", dtype=dtype)
        y = torch.zeros(2 * n + 1, device="cuda", dtype=dtype)
        aligned, got = torch.empty(2 * n, device="cuda", dtype=dtype), x[1:].clone()
        op.apply_device(got, aligned, precision=precision, complex_vectors=True)
        op.apply_device(x[1:], y[1:], precision=precision, complex_vectors=True)
        assert torch.equal(y[1:], aligned) and float(y[0]) == 0.0


def test_infinities_reach_only_their_neighbours():
    """Unused slots of a tile read nothing: an infinite entry of x shows in the rows that hold its column."""
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    op = GpuOperator(GpuBasis(14, up=7, momentum=0, parity=1), heisenberg_terms(14, delta=0.3))
    h = op.to_scipy()
    for column in (0, op.dim - 1):
        x = torch.ones(op.dim, device="cuda", dtype=torch.float64)
        x[column] = float("inf")
        y = torch.empty_like(x)
        op.apply_device(x, y)
        touched = np.asarray(h[:, [column]].todense()).ravel() != 0
        assert np.array_equal(~torch.isfinite(y).cpu().numpy(), touched)


def test_sixteen_columns_at_a_partial_tile():
    import torch
    from qmbed_b200 import GpuBasis, GpuOperator, heisenberg_terms
    for sites in (6, 13):
        op = GpuOperator(GpuBasis(sites, up=sites // 2, momentum=0), heisenberg_terms(sites, delta=0.4))
        orbit = np.sqrt(op.basis.states()[2].astype(float))[:, None]
        h = op.to_scipy().toarray().real
        for nb in (8, 16):
            z = torch.randn(op.dim, nb, device="cuda", dtype=torch.float64)
            out = torch.full_like(z, float("nan"))
            op.apply_block_device(z, out, nb, alpha=0.5, beta=0.25)
            zh = z.cpu().numpy()
            want = 0.5 * (h @ (orbit * zh)) / orbit + 0.25 * zh
            assert np.linalg.norm(out.cpu().numpy() - want) <= 1e-14 * np.abs(h).sum(axis=1).max() * np.linalg.norm(zh)


def test_explicit_rows_of_a_complex_operator_stay_available():
    """The scan takes complex operators whatever storage they were asked for."""
    from qmbed_b200 import GpuBasis, GpuOperator
    from qmbed_b200.scan import j1j2_component_terms, scan_lowest
    basis = GpuBasis(10, up=5, momentum=2)
    ops = [[GpuOperator(basis, t, storage="packed") for t in j1j2_component_terms(10) if t[0][0] != "zz"]]
    values, _, _ = scan_lowest(ops, np.array([[1.0, 0.25], [0.8, 0.1]]), eigenpairs=1)
    for p, c in enumerate(((1.0, 0.25), (0.8, 0.1))):
        h = sum(k * o.to_scipy().toarray() for k, o in zip(c, ops[0]))
        assert abs(values[0, p, 0] - np.linalg.eigvalsh(h)[0]) < 1e-9


def test_hermiticity_verdicts():
    """Accepted and refused as by the row expansion: conjugate pairs pass, a lone or unequal partner does not."""
    from qmbed_b200 import GpuBasis, GpuOperator, QmbedError
    basis = GpuBasis(8, up=4, momentum=0)
    bonds = [(i, (i + 1) % 8) for i in range(8)]
    GpuOperator(basis, [("+-", [(0.5, b) for b in bonds]), ("-+", [(0.5, b) for b in bonds])])
    GpuOperator(basis, [("+-", [(1j, b) for b in bonds]), ("-+", [(-1j, b) for b in bonds])])
    for bad in ([("+-", [(0.5, (0, 1))])], [("+-", [(0.5, b) for b in bonds]), ("-+", [(0.5 + 1e-9, b) for b in bonds])],
                [("zz", [(1j, b) for b in bonds])]):
        with pytest.raises(QmbedError):
            GpuOperator(basis, bad)
    # large couplings take the row expansion
    GpuOperator(basis, [("zz", [(1e6, b) for b in bonds]), ("xx", [(1e6, b) for b in bonds]),
                        ("yy", [(1e6, b) for b in bonds])])
