"""Graph blockade sectors (el_table.cu) and the hop kernel against the oracle:
prefix and suffix flips, dots of one and many vectors, sites without a drive;
sectors of no, few, half and most bits set, A channels beside J."""
import numpy as np
import pytest

from oracle import ref
from energy_level_b200 import configs

pytestmark = pytest.mark.gpu

EPS = {"float64": 2.3e-16, "complex128": 4.6e-16, "float32": 6e-8, "complex64": 1.2e-7}


def _grid(rows, cols):
    n = rows * cols
    return n, [[i, i + 1] for i in range(n) if (i + 1) % cols] + [[i, i + cols] for i in range(n - cols)]


def _drive(n, seed, cplx):
    rng = np.random.default_rng(seed)
    om = rng.uniform(0.5, 2.0, n) + (1j * rng.uniform(-0.5, 0.5, n) if cplx else 0)
    om[rng.integers(0, n)] = 0.0
    return om, rng.uniform(-2, 2, n), rng


@pytest.mark.parametrize("rows,cols", [(2, 2), (3, 4), (4, 5)])
@pytest.mark.parametrize("dtype,cdrive", [("float32", False), ("float64", False), ("complex64", True),
                                          ("complex128", False), ("complex128", True)])
def test_grid_hv(ctx, rows, cols, dtype, cdrive):
    import torch
    from energy_level_b200.core import Basis, Hamiltonian
    n, edges = _grid(rows, cols)
    om, de, rng = _drive(n, n, cdrive)
    pairs = configs.pairs_from_positions([[6.0 * (i // cols), 6.0 * (i % cols), 0.0] for i in range(n)])
    b = Basis(ctx, n, kind="blockade", edges=edges)
    h = Hamiltonian(ctx, b, om, de, pairs)
    codes = ref.independent_states(n, edges, None)
    for nvec in (1, 2, 8, 64):
        x = rng.normal(size=(b.dim, nvec)) + (1j * rng.normal(size=(b.dim, nvec)) if dtype.startswith("complex") else 0)
        t = torch.as_tensor(x, dtype=getattr(torch, dtype), device=ctx.device)
        xs = t.cpu().numpy().astype(complex if dtype.startswith("complex") else float)
        want = ref.hv(n, codes, om if cdrive else om.real, de, pairs, xs)
        scale = max(np.abs(want).max(), np.abs(ref.diagonal(n, codes, de, pairs)).max() * np.abs(x).max())
        assert np.abs(h.hv(t).cpu().numpy() - want).max() <= 40 * EPS[dtype] * scale, nvec   # n + 2 roundings


@pytest.mark.parametrize("nvec,chunk", [(1, 1), (32, 32), (70, 64)])
@pytest.mark.parametrize("mode", ["direct", "doubling"])
def test_grid_moments(ctx, nvec, chunk, mode):
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    n, edges = _grid(3, 4)
    om, de, _ = _drive(n, 5, False)
    pairs = configs.pairs_from_positions([[6.0 * (i // 4), 6.0 * (i % 4), 0.0] for i in range(n)])
    b = Basis(ctx, n, kind="blockade", edges=edges)
    h = Hamiltonian(ctx, b, om, de, pairs)
    codes = ref.independent_states(n, edges, None)
    lo, hi = solvers.bounds(h)
    c, r = solvers.kpm_scale(lo, hi)
    probes = np.random.default_rng(2).choice([-1, 1], size=(nvec, b.dim))
    mu = solvers.kpm_moments(h, 16, nvec, c, r, dtype="float64", chunk=chunk, probes=probes, mode=mode)
    want = ref.kpm_moments(lambda v: ref.hv(n, codes, om.real, de, pairs, v), b.dim, 16, probes, c, r)
    assert np.abs(mu - np.asarray(want)).max() <= 1e-11


@pytest.mark.parametrize("n,k", [(9, 0), (9, 1), (12, 3), (12, 9), (13, 6), (20, 10)])
@pytest.mark.parametrize("dtype", ["float64", "complex128", "complex64"])
def test_hops_match_oracle(ctx, n, k, dtype):
    import torch
    from energy_level_b200.core import Basis, Hamiltonian
    rng = np.random.default_rng(n + k)
    cplx = dtype.startswith("complex")
    ex = [(i, j, complex(rng.normal(), rng.normal() if cplx else 0.0), 0.0)
          for i in range(n) for j in range(i + 1, n) if rng.random() < 0.8]
    b = Basis(ctx, n, kind="charge", k=k)
    de = rng.uniform(-1, 1, n)
    h = Hamiltonian(ctx, b, np.zeros(n), de, [], exchange=ex)
    codes = ref.number_sector_basis(n, k)
    x = rng.normal(size=b.dim) + (1j * rng.normal(size=b.dim) if cplx else 0)
    t = torch.as_tensor(x, dtype=getattr(torch, dtype), device=ctx.device)
    xs = t.cpu().numpy().astype(complex if cplx else float)
    want = ref.hv(n, codes, np.zeros(n), de, [], xs, exchange=ex)
    # at most 100 hops a row: their roundings against the row's largest value
    assert np.abs(h.hv(t).cpu().numpy() - want).max() <= 200 * EPS[dtype] * np.abs(want).max()


def test_full_basis_with_pair_creation(ctx):
    import torch
    from energy_level_b200.core import Basis, Hamiltonian
    n = 9
    rng = np.random.default_rng(3)
    ex = [(i, j, complex(rng.normal(), rng.normal()), complex(rng.normal(), rng.normal()))
          for i in range(n) for j in range(i + 1, n)]
    om = rng.uniform(0.5, 1.5, n) + 0.3j
    h = Hamiltonian(ctx, Basis(ctx, n), om, rng.uniform(-1, 1, n), [], exchange=ex)
    x = rng.normal(size=h.dim) + 1j * rng.normal(size=h.dim)
    want = ref.hv(n, None, om, h.delta, [], x, exchange=ex)
    got = h.hv(torch.as_tensor(x, device=ctx.device)).cpu().numpy()
    assert np.abs(got - want).max() <= 200 * EPS["complex128"] * np.abs(want).max()
