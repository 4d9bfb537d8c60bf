"""Gram-Schmidt and update kernels behind the Lanczos drivers at the lengths
where their 16-byte pieces end (odd rows, one row more or less, unaligned
columns): with full reorthogonalisation the tridiagonal matrix of a short
Lanczos run equals that of the oracle's."""
import numpy as np
import pytest

from oracle import ref
from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 8, 11, 12, 13])     # 34, 55, 233, 377, 610 rows
@pytest.mark.parametrize("dtype,tol", [("float32", 2e-4), ("float64", 1e-10), ("complex64", 2e-4),
                                       ("complex128", 1e-10)])
def test_tridiagonal_matches_oracle(ctx, n, dtype, tol):
    from energy_level_b200 import spectrum
    from energy_level_b200.core import Basis, Hamiltonian
    rng = np.random.default_rng(n)
    edges = configs.chain_edges(n)
    om, de = rng.uniform(0.5, 2.0, n), rng.uniform(-2, 2, n)
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=7.0))
    h = Hamiltonian(ctx, Basis(ctx, n, kind="blockade", edges=edges), om, de, pairs)
    codes = ref.independent_states(n, edges, None)
    phi = rng.normal(size=h.dim) + (1j * rng.normal(size=h.dim) if dtype.startswith("complex") else 0)
    got = spectrum.lanczos(h, phi, 14, dtype=dtype)
    alphas, betas, _ = ref.lanczos_tridiag(lambda v: ref.hv(n, codes, om, de, pairs, v), phi, 14)
    # 14 steps of a well separated spectrum: rounding grows with the steps
    scale = np.abs(alphas).max()
    assert np.abs(got["alphas"] - alphas).max() <= tol * scale
    assert np.abs(got["betas"] - betas[:len(got["betas"])]).max() <= tol * scale


@pytest.mark.parametrize("n,reorth", [(9, "full"), (16, "partial"), (16, "none"), (18, "partial")])
def test_ground_pair_of_queued_steps(ctx, n, reorth):
    """The two lowest energies after queued steps, reorthogonalised or not."""
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    rng = np.random.default_rng(n)
    edges = configs.chain_edges(n)
    om, de = rng.uniform(0.5, 2.0, n), rng.uniform(-2, 2, n)
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=7.0))
    h = Hamiltonian(ctx, Basis(ctx, n, kind="blockade", edges=edges), om, de, pairs)
    H = ref.sparse_h(n, ref.independent_states(n, edges, None), om, de, pairs)
    import scipy.sparse.linalg as spla
    want = np.sort(spla.eigsh(H, k=2, which="SA", tol=1e-12)[0]) if n > 9 else np.linalg.eigvalsh(H.toarray())[:2]
    r = solvers.lanczos_ground(h, max_iter=200, tol=1e-9, reorth=reorth, return_vec=True)
    assert r["converged"]
    assert abs(r["evals"][0] - want[0]) <= 1e-9
    if reorth != "none":       # without it a converged value comes back as its own copy
        assert abs(r["evals"][1] - want[1]) <= 1e-8
    v = r["vec"].cpu().numpy()
    assert np.linalg.norm(H @ v - r["evals"][0] * v) <= 1e-8
