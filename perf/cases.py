"""Workloads of the engine, one per way a program uses it, each through its public entry points.

A case is a dict of plain values. ``listed()`` names the standing workloads,
``draw(rng)`` gives another one of the same ranges, ``prepare(case, seed)``
builds what a program holds before the call, ``run(state)`` is one pass, and
``exact(case, seed)`` is the same result in 64-bit arithmetic by plain torch
(its own sector enumeration, terms and solvers).

Kinds of case:

* ``hv``: y = H x on device vectors, stored rows or matrix-free; what a
  program with its own Krylov method calls in its loop.
* ``block``: the three-term block action on row-major blocks, the step of a
  block (Chebyshev) method.
* ``flip``: y = H x of a transverse-field Ising chain on the full space.
* ``chebyshev``: a quench of that chain, propagated on the device.
* ``assemble``: a new Hamiltonian on a sector that is already there (a scan
  over couplings), and its first application.
* ``eigsh``: the lowest eigenvalues of a sector.
* ``ftlm``: finite-temperature Lanczos over random vectors.
"""

import math

import numpy as np
import torch

from qmbed_b200.engine import GpuBasis, GpuOperator, heisenberg_terms, tfim_terms
from qmbed_b200.lanczos import ftlm_sample

BETAS = (0.1, 0.5, 1.0, 2.0, 4.0)


def listed():
    return [
        # cfg "plain, small": the periodic chain of 20 sites at k = 0; the launches of one application count
        {"name": "hv_packed_L20_f64", "kind": "hv", "sites": 20, "momentum": 0, "parity": 0, "j2": False,
         "storage": "packed", "precision": 64, "complex": False},
        # an ordinary to large Lanczos step in FP64 on assembled rows
        {"name": "hv_packed_L31_f64", "kind": "hv", "sites": 31, "momentum": 0, "parity": 1, "j2": False,
         "storage": "packed", "precision": 64, "complex": False},
        # one momentum sector of the J1-J2 scan (complex rows with explicit values)
        {"name": "hv_complex_L26_k3", "kind": "hv", "sites": 26, "momentum": 3, "parity": 0, "j2": True,
         "storage": "packed", "precision": 64, "complex": True},
        # single precision on the fly: the FP32 phase of a solve that stores no rows
        {"name": "hv_free_L30_f32", "kind": "hv", "sites": 30, "momentum": 0, "parity": 1, "j2": False,
         "storage": "matrix_free", "precision": 32, "complex": False},
        # J1-J2 in a complex momentum sector without stored rows: the general expansion
        {"name": "hv_free_complex_L25_k5", "kind": "hv", "sites": 25, "momentum": 5, "parity": 0, "j2": True,
         "storage": "matrix_free", "precision": 64, "complex": True},
        # the filter step of a block solve on a large sector (blocks beyond the L2)
        {"name": "block_packed_L32_f32", "kind": "block", "sites": 32, "momentum": 0, "parity": 1, "j2": False,
         "storage": "packed", "precision": 32, "nb": 8},
        # the quench Hamiltonian in complex64, one application beyond the L2
        {"name": "flip_L25_c64", "kind": "flip", "sites": 25, "precision": 32, "complex": True},
        # a quench of 22 sites in complex128 over four output times
        {"name": "chebyshev_L22_c128", "kind": "chebyshev", "sites": 22, "precision": 64, "steps": 4, "time": 1.0},
        # a new point of a coupling scan: assembly on a resident sector and the first application
        {"name": "assemble_L28", "kind": "assemble", "sites": 28, "momentum": 0, "parity": 1, "j2": False},
        # cfg "plain, small" as a whole call: four lowest to 1e-12, reference algorithm in FP64
        {"name": "eigsh_L20_f64", "kind": "eigsh", "sites": 20, "momentum": 0, "parity": 0, "mode": "fp64", "wanted": 4,
         "tolerance": 1e-12},
        # cfg "XXZ": six lowest of the 28-site sector, filtered
        {"name": "eigsh_L28_filtered", "kind": "eigsh", "sites": 28, "momentum": 0, "parity": 1, "mode": "filtered",
         "wanted": 6, "tolerance": 1e-10},
        # finite temperature: two random vectors of 100 steps each
        {"name": "ftlm_L28", "kind": "ftlm", "sites": 28, "momentum": 0, "parity": 1, "vectors": 2, "steps": 100},
    ]


def draw(rng):
    """One more case: sizes uniform in the number of sites, so in the logarithm of the dimension."""
    kind = rng.choice(["hv", "hv", "hv", "block", "flip", "chebyshev", "assemble", "eigsh", "ftlm"])
    if kind in ("flip", "chebyshev"):
        if kind == "flip":
            return {"kind": kind, "sites": rng.randint(9, 25), "precision": rng.choice([32, 64]),
                    "complex": rng.random() < 0.7}
        return {"kind": kind, "sites": rng.randint(9, 21), "precision": rng.choice([32, 64]),
                "steps": rng.randint(1, 5), "time": round(rng.uniform(0.2, 1.0), 3)}
    cplx = kind == "hv" and rng.random() < 0.5
    top = {"hv": 26 if cplx else 31, "block": 31, "assemble": 28, "eigsh": 24, "ftlm": 27}[kind]
    sites = rng.randint({"hv": 12, "block": 14, "assemble": 12, "eigsh": 15, "ftlm": 16}[kind], top)
    case = {"kind": kind, "sites": sites}
    if cplx:
        case.update(momentum=rng.randint(1, (sites - 1) // 2), parity=0)
    else:
        momentum = rng.choice([0, 0, sites // 2]) if sites % 2 == 0 else 0
        case.update(momentum=momentum, parity=rng.choice([1, 1, -1, 0]) if sites > 15 else 1)
        if sites > 30:
            case["parity"] = 1
    if kind == "hv":
        case.update(j2=rng.random() < 0.4 and sites < 31, storage=rng.choice(["packed", "matrix_free"]),
                    precision=rng.choice([32, 64]), complex=cplx or rng.random() < 0.2)
    elif kind == "block":
        case.update(j2=rng.random() < 0.3 and sites < 30, storage=rng.choice(["packed", "packed", "matrix_free"]),
                    precision=rng.choice([32, 64]), nb=rng.choice([8, 8, 16]) if sites < 31 else 8)
    elif kind == "assemble":
        case.update(j2=rng.random() < 0.4 and sites < 28)
    elif kind == "eigsh":
        case.update(mode=rng.choice(["fp64", "filtered"]), wanted=rng.randint(1, 4), tolerance=1e-10, momentum=0, parity=1)
    else:
        case.update(vectors=rng.randint(1, 4), steps=rng.randint(20, 100))
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _couplings(case, seed):
    """(Delta, J2) of a chain, or the fields of a quench, drawn as the scans draw them."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 17])
    if case["kind"] in ("flip", "chebyshev"):
        return rng.uniform(-2.0, 2.0, case["sites"])
    return float(rng.uniform(0.5, 1.5)), float(rng.uniform(0.1, 0.5)) if case.get("j2") else 0.0


def _dtype(case):
    real = torch.float64 if case["precision"] == 64 else torch.float32
    if not case.get("complex"):
        return real
    return torch.complex128 if case["precision"] == 64 else torch.complex64


def _dimension(case):
    """Sector dimension by the character formula (half filling)."""
    n, up, k, p = case["sites"], case["sites"] // 2, case["momentum"], case["parity"]
    total = 0.0
    for a in range(n):
        d = math.gcd(n, a) or n
        if up % (n // d) == 0:
            total += math.cos(2 * math.pi * k * a / n) * math.comb(d, up // (n // d))
    if p:
        for a in range(n):  # site i -> a - i
            ones = sum(1 for i in range(n) if (2 * i - a) % n == 0)
            pairs = (n - ones) // 2
            fixed = sum(math.comb(ones, f) * math.comb(pairs, (up - f) // 2)
                        for f in range(min(ones, up) + 1) if (up - f) % 2 == 0)
            total += p * (math.cos(math.pi * (a + 1)) if 2 * k == n else 1.0) * fixed
        total /= 2
    return max(1, round(total / n))


def _vector(case, seed, dim, columns=1):
    shape = (dim, columns) if columns > 1 else (dim,)
    x = torch.randn(shape, generator=_generator(seed), device="cuda", dtype=torch.float64 if not case.get("complex")
                    else torch.complex128)
    return (x / math.sqrt(dim)).to(_dtype(case))


def _basis(case):
    return GpuBasis(case["sites"], up=case["sites"] // 2, momentum=case["momentum"], parity=case["parity"] or None)


def _flip_state(case, seed):
    n = 1 << case["sites"]
    x = torch.randn(n, generator=_generator(seed), device="cuda", dtype=torch.complex128 if case.get("complex")
                    else torch.float64)
    return (x / torch.linalg.vector_norm(x)).to(_dtype(case))


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind in ("flip", "chebyshev"):
        fields = _couplings(case, seed)
        s["op"] = GpuOperator(GpuBasis(case["sites"], normalization="pauli_cartesian"),
                              tfim_terms(case["sites"], fields=fields), storage="matrix_free")
        if kind == "flip":
            s["x"] = _flip_state(case, seed)
            s["y"] = torch.empty_like(s["x"])
        else:
            s["x"] = _flip_state({**case, "precision": 64, "complex": True}, seed)
            s["y"] = torch.empty_like(s["x"])
            bound = 2.0 * (case["sites"] - 1) + float(np.abs(fields).sum()) + 1.0
            s["interval"] = (-bound, bound)
            s["times"] = [case["time"] * (t + 1) / case["steps"] for t in range(case["steps"])]
        return s
    delta, j2 = _couplings(case, seed)
    s["terms"] = heisenberg_terms(case["sites"], delta=delta, j2=j2)
    s["basis"] = _basis(case)
    if kind == "assemble":
        s["x"] = _vector({**case, "precision": 64}, seed, len(s["basis"]))
        s["y"] = torch.empty_like(s["x"])
        return s
    s["op"] = GpuOperator(s["basis"], s["terms"], storage=case.get("storage", "packed"))
    if kind in ("hv", "block"):
        s["x"] = _vector(case, seed, s["op"].dim, case.get("nb", 1))
        s["y"] = torch.empty_like(s["x"])
        if kind == "block":
            s["p"] = _vector(case, seed + 1, s["op"].dim, case["nb"])
    else:
        s["seed"] = int(seed) & 0xFFFF
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("hv", "flip"):
        s["op"].apply_device(s["x"], s["y"], precision=case["precision"], complex_vectors=case["complex"])
        return s["y"]
    if kind == "block":
        s["op"].apply_block_device(s["x"], s["y"], case["nb"], precision=case["precision"], alpha=1.0 / 16.0, beta=0.125,
                                   gamma=0.5, p=s["p"])
        return s["y"]
    if kind == "chebyshev":
        s["y"].copy_(s["x"])
        s["op"].chebyshev_evolve_device(s["y"], s["times"], *s["interval"], precision=case["precision"])
        return s["y"]
    if kind == "assemble":
        op = GpuOperator(s["basis"], s["terms"])
        op.apply_device(s["x"], s["y"])
        return s["y"]
    if kind == "eigsh":
        return s["op"].eigsh(case["wanted"], krylov_dimension=40, tolerance=case["tolerance"], seed=s["seed"],
                             mode=case["mode"]).eigenvalues
    log_partition, energy, _ = ftlm_sample(s["op"], case["vectors"], BETAS, case["steps"], seed=s["seed"])
    return [log_partition, energy]


def work(case):
    """Bytes of the vectors, and of the sector or the rows where the path reads them; two flops per entry and column
    (eight for complex vectors)."""
    kind, n = case["kind"], case["sites"]
    if kind in ("flip", "chebyshev"):
        size = 1 << n
        if kind == "flip":
            each = (8 if case["precision"] == 64 else 4) * (2 if case["complex"] else 1)
            return {"bytes": 2 * size * each, "flops": size * (n + 1) * (4 if case["complex"] else 2)}
        bound = 2.0 * (n - 1) + n + 1.0
        passes = case["steps"] * (bound * case["time"] / case["steps"] + 25)
        return {"bytes": passes * 4 * size * (16 if case["precision"] == 64 else 8), "flops": passes * size * (n + 7) * 4}
    up, dim = n // 2, _dimension(case)
    bonds = n * (2 if case.get("j2") else 1)
    entries = dim * bonds * 2.0 * up * (n - up) / (n * (n - 1.0))
    if kind in ("hv", "block"):
        columns = case.get("nb", 1)
        cplx = bool(case.get("complex"))
        each = (8 if case["precision"] == 64 else 4) * (2 if cplx else 1)
        # stored rows: one 4-byte word per entry and the diagonal; on the fly: the states
        rows = 4 * entries + 8 * dim if case["storage"] == "packed" else 10 * dim
        vectors = (3 if kind == "block" else 2) * dim * each * columns
        return {"bytes": rows + vectors, "flops": (entries + dim) * columns * (8 if cplx else 2)}
    if kind == "assemble":
        return {"bytes": 10 * dim + 4 * entries + 8 * dim + 16 * dim, "flops": 4 * entries}
    if kind == "eigsh":
        steps = 80
        return {"bytes": steps * (4 * entries + 24 * dim), "flops": steps * (2 * entries + 4 * 40 * dim)}
    steps = case["vectors"] * case["steps"]
    # every step reads the rows and twice the basis built so far (overlaps, then the subtraction)
    return {"bytes": steps * (4 * entries + 24 * dim + case["steps"] * 8 * dim),
            "flops": steps * (2 * entries + 2 * case["steps"] * dim)}


# ---------------------------------------------------------------------------
# The same results in 64 bits, by plain torch
# ---------------------------------------------------------------------------

def _popcount(v):
    v = v - ((v >> 1) & 0x5555555555555555)
    v = (v & 0x3333333333333333) + ((v >> 2) & 0x3333333333333333)
    v = (v + (v >> 4)) & 0x0F0F0F0F0F0F0F0F
    v = v + (v >> 8)
    v = v + (v >> 16)
    return (v + (v >> 32)) & 0x7F


def _rotate(v, s, n):
    s %= n
    mask = (1 << n) - 1
    return v if s == 0 else ((v << s) | (v >> (n - s))) & mask


def _reflect(v, n):
    out = torch.zeros_like(v)
    for i in range(n):
        out |= ((v >> i) & 1) << (n - 1 - i)
    return out


class _Sector:
    """Representatives (orbit minima, ascending) and orbit sizes of a half-filled momentum / parity sector."""

    def __init__(self, case):
        n = self.n = case["sites"]
        self.k, self.p = case["momentum"], case["parity"]
        up, chunk, kept = n // 2, 1 << 26, []
        for start in range(0, 1 << n, chunk):
            v = torch.arange(start, min(start + chunk, 1 << n), device="cuda", dtype=torch.int64)
            v = v[_popcount(v) == up]
            for s in range(1, n):
                if s <= 4 or s % 4 == 0 or s == n - 1:
                    v = v[_rotate(v, s, n) >= v]
            if self.p and v.numel():
                u = _reflect(v, n)
                for s in range(n):
                    if s % 4 == 0:
                        keep = _rotate(u, s, n) >= v
                        v, u = v[keep], u[keep]
            kept.append(v)
        v = torch.cat(kept)
        u = _reflect(v, n) if self.p else None
        minimum, total, images = torch.ones_like(v, dtype=torch.bool), torch.zeros(v.numel(), device="cuda", dtype=torch.float64), \
            torch.zeros_like(v)
        for s in range(n):
            angle = 2 * math.pi * self.k * s / n
            for w, sign in ((v, 1.0),) + (((u, float(self.p)),) if self.p else ()):
                r = _rotate(w, s, n)
                minimum &= r >= v
                same = r == v
                total += same * (sign * math.cos(angle))
                images += same
        keep = minimum & (total > 0.5)
        self.states, group = v[keep], n * (2 if self.p else 1)
        self.orbit = (group // images[keep]).double()
        self.dim = self.states.numel()

    def locate(self, t):
        """(row or -1, character) of each state's image."""
        best, shift = t.clone(), torch.zeros_like(t)
        refl = torch.zeros_like(t, dtype=torch.bool)
        for w, flag in ((t, False),) + (((_reflect(t, self.n), True),) if self.p else ()):
            for s in range(self.n):
                r = _rotate(w, s, self.n)
                less = r < best
                best = torch.where(less, r, best)
                shift = torch.where(less, torch.full_like(shift, s), shift)
                refl = torch.where(less, torch.full_like(refl, flag), refl)
        row = torch.searchsorted(self.states, best).clamp(max=self.dim - 1)
        found = self.states[row] == best
        if (2 * self.k) % self.n == 0:
            chi = torch.where((shift % 2 == 1) & (self.k != 0), -1.0, 1.0).double()
            chi = torch.where(refl & (self.p < 0), -chi, chi)
        else:
            angle = (2 * math.pi / self.n) * ((self.k * shift) % self.n).double()
            chi = torch.complex(torch.cos(angle), torch.sin(angle))
        return torch.where(found, row, torch.full_like(row, -1)), chi


def _bonds(case, seed):
    n = case["sites"]
    delta, j2 = _couplings(case, seed)
    out = [(i, (i + 1) % n, 1.0, delta) for i in range(n)]
    if j2:
        out += [(i, (i + 2) % n, j2, j2 * delta) for i in range(n)]
    return out


def _hop(sector, i, j):
    """(rows, columns, entries / J) of the exchange on one bond."""
    v = sector.states
    rows = torch.nonzero(((v >> i) ^ (v >> j)) & 1).flatten()
    out = []
    for part in rows.split(1 << 23):
        col, chi = sector.locate(v[part] ^ ((1 << i) | (1 << j)))
        ok = col >= 0
        part, col, chi = part[ok], col[ok], chi[ok]
        out.append((part, col, 0.5 * chi * torch.sqrt(sector.orbit[part] / sector.orbit[col])))
    return out


def _diagonal(sector, bonds):
    d = torch.zeros(sector.dim, device="cuda", dtype=torch.float64)
    for i, j, _, zz in bonds:
        d += (0.25 - 0.5 * (((sector.states >> i) ^ (sector.states >> j)) & 1).double()) * zz
    return d


def _apply(case, seed, x):
    """H x on a sector, bond by bond (nothing stored); x has rows of `columns` values."""
    sector = _Sector(case)
    bonds = _bonds(case, seed)
    block = x.reshape(sector.dim, -1)
    orbit = torch.sqrt(sector.orbit)[:, None]
    if case["kind"] == "block":  # the block action works on x / sqrt(orbit)
        block = block * orbit
    y = _diagonal(sector, bonds)[:, None] * block
    for i, j, exchange, _ in bonds:
        for rows, cols, entry in _hop(sector, i, j):
            y.index_add_(0, rows, (exchange * entry)[:, None] * block[cols])
    if case["kind"] == "block":
        y = y / orbit
    return y.reshape(x.shape)


def _matrix(case, seed):
    sector = _Sector(case)
    bonds = _bonds(case, seed)
    rows, cols, vals = [torch.arange(sector.dim, device="cuda")], [torch.arange(sector.dim, device="cuda")], \
        [_diagonal(sector, bonds)]
    for i, j, exchange, _ in bonds:
        for r, c, e in _hop(sector, i, j):
            rows.append(r)
            cols.append(c)
            vals.append(exchange * e)
    size = (sector.dim, sector.dim)
    return torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals), size).coalesce().to_sparse_csr()


def _lanczos(matrix, v, steps):
    """Fully reorthogonalised Lanczos: diagonal and off-diagonal of the projected matrix."""
    basis = torch.zeros(steps, v.numel(), device="cuda", dtype=torch.float64)
    alpha, beta = [], []
    v = v / torch.linalg.vector_norm(v)
    for m in range(steps):
        basis[m] = v
        w = matrix @ v
        alpha.append(float(v @ w))
        q = basis[:m + 1]
        for _ in range(2):
            w = w - q.T @ (q @ w)
        b = float(torch.linalg.vector_norm(w))
        if m + 1 == steps or b < 1e-12:
            break
        beta.append(b)
        v = w / b
    return np.array(alpha), np.array(beta[:len(alpha) - 1])


def _ritz(alpha, beta):
    return np.linalg.eigh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))


def _rademacher(n, seed, index):
    """The sampler's documented start vector: the top bit of a splitmix64 hash of (seed, index, row)."""
    def mix(x):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))
    with np.errstate(over="ignore"):
        key = np.uint64((seed * 0xD1B54A32D192ED03 + index * 0x8CB92BA72F3D8DD7 + 1) & 0xFFFFFFFFFFFFFFFF)
        bits = mix(key ^ mix(np.arange(n, dtype=np.uint64)))
    return torch.from_numpy(np.where(bits >> np.uint64(63), -1.0, 1.0)).cuda()


def _chain_action(case, fields, x):
    n = case["sites"]
    index = torch.arange(1 << n, device="cuda", dtype=torch.int64)
    z = [((index >> i) & 1).double() * 2.0 - 1.0 for i in range(n)]
    d = sum(float(fields[i]) * z[i] for i in range(n)) - sum(z[i] * z[i + 1] for i in range(n - 1))

    def act(v):
        y = d * v
        for i in range(n):
            y = y - v.reshape(-1, 2, 1 << i).flip(1).reshape(-1)
        return y
    return act


def exact(case, seed):
    kind = case["kind"]
    if kind in ("flip", "chebyshev"):
        fields = _couplings(case, seed)
        if kind == "flip":
            x = _flip_state(case, seed).to(torch.complex128 if case["complex"] else torch.float64)
            return _chain_action(case, fields, x)(x)
        v = _flip_state({**case, "precision": 64, "complex": True}, seed)
        act = _chain_action(case, fields, v)
        scale = 2.0 * case["sites"] + float(np.abs(fields).sum())
        pieces = max(1, math.ceil(scale * case["time"]))
        for _ in range(pieces):  # Taylor series of steps with |H| dt <= 1
            term, total = v, v
            for order in range(1, 24):
                term = act(term) * (-1j * case["time"] / (pieces * order))
                total = total + term
            v = total
        return v
    if kind in ("hv", "block", "assemble"):
        given = {**case, "precision": case.get("precision", 64)}
        dim = _dimension(case)
        x = _vector(given, seed, dim, case.get("nb", 1))
        wide = torch.complex128 if x.is_complex() or (2 * case["momentum"]) % case["sites"] else torch.float64
        y = _apply(case, seed, x.to(wide))
        if kind == "block":
            y = y / 16.0 + 0.125 * x.to(wide) + 0.5 * _vector(given, seed + 1, dim, case["nb"]).to(wide)
        return y
    matrix = _matrix(case, seed)
    dim = matrix.shape[0]
    if kind == "eigsh":
        if dim <= 2048:
            return torch.linalg.eigvalsh(matrix.to_dense())[:case["wanted"]].cpu().numpy()
        start = torch.randn(dim, generator=_generator(seed + 5), device="cuda", dtype=torch.float64)
        return _ritz(*_lanczos(matrix, start, min(dim, 320)))[0][:case["wanted"]]
    partition, energy = [], []
    for r in range(case["vectors"]):
        e, u = _ritz(*_lanczos(matrix, _rademacher(dim, int(seed) & 0xFFFF, r), min(dim, case["steps"])))
        weight = u[0] ** 2
        row = [weight * np.exp(-b * (e - e[0])) for b in BETAS]
        partition.append([math.log(dim) - b * e[0] + math.log(w.sum()) for b, w in zip(BETAS, row)])
        energy.append([float((w * e).sum() / w.sum()) for w in row])
    return [np.array(partition), np.array(energy)]
