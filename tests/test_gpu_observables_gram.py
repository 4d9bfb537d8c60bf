"""Site and all-pair observables of one pass (el_observe.cu) against the
oracle: every basis kind, real and complex states, few and many pairs, either
order of a pair's sites, bases smaller than a stage of rows; and the
Gershgorin bounds behind the Chebyshev plan against a dense H."""
import numpy as np
import pytest

from oracle import ref
from energy_level_b200 import configs

pytestmark = pytest.mark.gpu

GRID = [[i, i + 1] for i in range(12) if (i + 1) % 4] + [[i, i + 4] for i in range(8)]
BASES = [("full", 3, None, None), ("full", 12, None, None), ("chain", 9, configs.chain_edges(9), None),
         ("chain", 17, configs.chain_edges(17), None), ("ring", 13, configs.ring_edges(13), None),
         ("grid", 12, GRID, None), ("charge", 11, None, 4)]


def _basis(ctx, kind, n, edges, k):
    from energy_level_b200.core import Basis
    if kind == "full":
        return Basis(ctx, n), np.arange(1 << n)
    if kind == "charge":
        return Basis(ctx, n, kind="charge", k=k), ref.number_sector_basis(n, k)
    return Basis(ctx, n, kind="blockade", edges=edges), ref.independent_states(n, edges, None)


@pytest.mark.parametrize("kind,n,edges,k", BASES)
@pytest.mark.parametrize("dtype", ["float64", "complex128", "complex64"])
def test_sites_and_pairs(ctx, kind, n, edges, k, dtype):
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Hamiltonian
    b, codes = _basis(ctx, kind, n, edges, k)
    h = Hamiltonian(ctx, b, np.ones(n), np.zeros(n), [])
    rng = np.random.default_rng(n)
    x = rng.normal(size=b.dim) + (1j * rng.normal(size=b.dim) if dtype.startswith("complex") else 0)
    x /= np.linalg.norm(x)
    t = torch.as_tensor(x, dtype=getattr(torch, dtype), device=ctx.device)
    v = t.cpu().numpy().astype(complex)
    bits = np.array([[(int(c) >> (n - 1 - i)) & 1 for c in codes] for i in range(n)])
    rank = {int(c): r for r, c in enumerate(codes)}
    p = np.abs(v) ** 2
    every = [(i, j) if (i + j) % 2 else (j, i) for i in range(n) for j in range(i + 1, n)]
    for pairs in ([], every[:3], every * (1 + 36 // len(every))):
        ob = solvers.spin_observables(h, t, pairs)
        sums = 40 * 2.3e-16            # FP64 sums of values below 1
        assert abs(ob["norm"] - p.sum()) <= sums
        assert np.abs(ob["n"] - bits @ p).max() <= sums
        sm = [sum(np.conj(v[r]) * v[rank[int(c) | 1 << (n - 1 - i)]] for r, c in enumerate(codes)
                  if not bits[i, r] and (int(c) | 1 << (n - 1 - i)) in rank) for i in range(n)]
        assert np.abs(ob["sm"] - sm).max() <= sums
        for q, (i, j) in list(enumerate(pairs))[::max(1, len(pairs) // 12)]:
            assert abs(ob["nn"][q] - (bits[i] * bits[j] * p).sum()) <= sums
            move = (1 << (n - 1 - i)) | (1 << (n - 1 - j))
            want = sum(np.conj(v[rank[int(c) ^ move]]) * v[r] for r, c in enumerate(codes)
                       if not bits[i, r] and bits[j, r] and (int(c) ^ move) in rank)
            assert abs(ob["xy"][q] - want) <= sums, (i, j)


@pytest.mark.parametrize("kind,n,edges,k", BASES)
def test_gershgorin_holds_the_spectrum(ctx, kind, n, edges, k):
    """A Chebyshev step is exact only while the bounds hold the spectrum."""
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Hamiltonian
    b, codes = _basis(ctx, kind, n, edges, k)
    rng = np.random.default_rng(n)
    om, de = rng.uniform(0.5, 2.0, n), rng.uniform(-9.0, 9.0, n)
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=6.0))
    h = Hamiltonian(ctx, b, om, de, pairs)
    H = ref.dense_h(n, codes, om, de, pairs)
    e, U = np.linalg.eigh(H)
    psi = rng.normal(size=b.dim) + 0j
    psi /= np.linalg.norm(psi)
    t = torch.as_tensor(psi, dtype=torch.complex128, device=ctx.device)
    solvers.cheb_step(h, t, 25.0, tol=1e-13)
    want = U @ (np.exp(-2j * np.pi * 1e-3 * 25.0 * e) * (U.conj().T @ psi))
    assert np.abs(t.cpu().numpy() - want).max() <= 1e-11
