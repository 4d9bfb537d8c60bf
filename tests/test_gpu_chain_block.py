"""Chain / ring sector H-apply (el_chain.cu) against the oracle at the sizes
where its tiling changes: the shortest sectors it takes, the first sizes with
several tiles, rows of 1 to 32 chunks, amplitudes missing on some sites."""
import numpy as np
import pytest

from oracle import ref
from energy_level_b200 import configs

pytestmark = pytest.mark.gpu

# errors: |row sum| terms add at most about n + 2 roundings of terms below the
# largest |H x|, with FP32 inputs exact: n eps < 40 eps of that scale
TOL = {"float64": 40 * 2.3e-16, "complex128": 80 * 2.3e-16, "float32": 40 * 6e-8, "complex64": 80 * 6e-8}


def _system(kind, n, seed, cplx):
    rng = np.random.default_rng(seed)
    om = rng.uniform(0.5, 2.0, n) + (1j * rng.uniform(-0.5, 0.5, n) if cplx else 0)
    om[rng.integers(0, n, 2)] = 0.0          # sites without a drive
    pos = configs.chain_positions(n, a=5.5, jitter=rng.uniform(-0.5, 0.5, n))
    pairs = configs.pairs_from_positions(pos)
    edges = configs.ring_edges(n) if kind == "ring" else configs.chain_edges(n)
    return om, rng.uniform(-2, 2, n), pairs, edges


@pytest.mark.parametrize("kind,n", [("chain", 6), ("chain", 7), ("chain", 8), ("chain", 11), ("chain", 17),
                                    ("chain", 22), ("ring", 9), ("ring", 10), ("ring", 13), ("ring", 19)])
@pytest.mark.parametrize("dtype,cdrive", [("float32", False), ("float64", False), ("complex64", False),
                                          ("complex64", True), ("complex128", True)])
def test_hv_edges(ctx, kind, n, dtype, cdrive):
    import torch
    from energy_level_b200.core import Basis, Hamiltonian
    om, de, pairs, edges = _system(kind, n, 5 + n, cdrive)
    b = Basis(ctx, n, kind="blockade", edges=edges)
    h = Hamiltonian(ctx, b, om, de, pairs)
    codes = ref.independent_states(n, edges, None)
    rng = np.random.default_rng(n)
    for nvec in (1, 2, 4, 8, 64):
        x = rng.normal(size=(b.dim, nvec))
        if dtype.startswith("complex"):
            x = x + 1j * rng.normal(size=(b.dim, nvec))
        tx = torch.as_tensor(x, dtype=getattr(torch, dtype), device=ctx.device)
        want = ref.hv(n, codes, om if cdrive else om.real, de, pairs, tx.cpu().numpy().astype(
            complex if dtype.startswith("complex") else float))
        got = h.hv(tx).cpu().numpy()
        # row scale: the diagonal's largest value times the largest entry
        scale = max(np.abs(want).max(), np.abs(ref.diagonal(n, codes, de, pairs)).max() * np.abs(x).max())
        assert np.abs(got - want).max() <= TOL[dtype] * scale, (nvec, np.abs(got - want).max() / scale)


@pytest.mark.parametrize("kind,n", [("chain", 15), ("ring", 14)])
@pytest.mark.parametrize("mode", ["direct", "doubling"])
@pytest.mark.parametrize("nvec,chunk", [(1, 1), (5, 4), (32, 32), (130, 128)])
def test_moments_with_block_dots(ctx, kind, n, mode, nvec, chunk):
    """The fused recurrence and its per-vector dot products (FP64 vectors)."""
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    om, de, pairs, edges = _system(kind, n, 31 + n, False)
    b = Basis(ctx, n, kind="blockade", edges=edges)
    h = Hamiltonian(ctx, b, om, de, pairs)
    codes = ref.independent_states(n, edges, None)
    probes = np.random.default_rng(2).choice([-1, 1], size=(nvec, b.dim))
    c, r = 30.0, 120.0        # the spectrum lies inside [c - r, c + r]
    num = 20
    mu = solvers.kpm_moments(h, num, nvec, c, r, dtype="float64", chunk=chunk, probes=probes, mode=mode)
    want = ref.kpm_moments(lambda v: ref.hv(n, codes, om.real, de, pairs, v), b.dim, num, probes, c, r)
    # moments are at most 1; the recurrence's error grows at most linearly in num
    assert np.abs(mu - np.asarray(want)).max() <= 1e-11


def test_bounds_and_evolution_on_a_ring(ctx):
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    n = 14
    om, de, pairs, edges = _system("ring", n, 9, True)
    b = Basis(ctx, n, kind="blockade", edges=edges)
    h = Hamiltonian(ctx, b, om, de, pairs)
    H = ref.dense_h(n, ref.independent_states(n, edges, None), om, de, pairs)
    e, U = np.linalg.eigh(H)
    lo, hi = solvers.bounds(h)
    assert abs(lo - e[0]) <= 1e-9 and abs(hi - e[-1]) <= 1e-9
    psi = np.random.default_rng(1).normal(size=b.dim) + 0j
    psi /= np.linalg.norm(psi)
    t = torch.as_tensor(psi, dtype=torch.complex128, device=ctx.device)
    solvers.cheb_step(h, t, 40.0, tol=1e-13)
    want = U @ (np.exp(-2j * np.pi * 1e-3 * 40.0 * e) * (U.conj().T @ psi))
    assert np.abs(t.cpu().numpy() - want).max() <= 1e-10
