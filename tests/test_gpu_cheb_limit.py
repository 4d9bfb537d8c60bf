"""Chebyshev steps of a small full basis on both sides of the largest number of
terms that the one-launch step takes (1024), against the eigenvectors."""
import numpy as np
import pytest

from energy_level_b200 import configs
from oracle import ref

pytestmark = pytest.mark.gpu

CONV = 2.0 * np.pi * 1e-3


@pytest.mark.parametrize("tau,one_launch", [(2400.0, True), (4800.0, False)])
def test_long_step_matches_eigenvectors(ctx, tau, one_launch):
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    n = 8
    rng = np.random.default_rng(2)
    om, de = rng.uniform(0.5, 2.0, n), rng.uniform(-2.0, 2.0, n)
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=6.2))
    h = Hamiltonian(ctx, Basis(ctx, n), om, de, pairs)
    w, U = np.linalg.eigh(ref.dense_h(n, None, om, de, pairs))
    x = rng.normal(size=h.dim) + 1j * rng.normal(size=h.dim)
    x /= np.linalg.norm(x)
    psi = torch.as_tensor(x, dtype=torch.complex128, device=ctx.device)
    terms = solvers.cheb_step(h, psi, tau, tol=1e-13)
    assert (terms - 1 <= 1024) == one_launch and 400 < terms < 3000
    want = U @ (np.exp(-1j * CONV * tau * w) * (U.conj().T @ x))
    # phases of up to CONV tau max|w| (below 6e3) in FP64: 6e3 x 2.2e-16, and
    # as much per term for the recurrence's rounding
    assert np.linalg.norm(psi.cpu().numpy() - want) < 6e3 * 2.2e-16 * 10
