"""Chebyshev steps of small full bases in one launch (el_cheb_coop.cu) against
the Taylor propagator, which runs one launch per term: every tile shape (one
tile, several, 2 and 4 rows per thread), real and complex drives, sites
without a drive, steps of one term."""
import numpy as np
import pytest

from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 5, 9, 10, 11, 15, 16, 17, 18, 19])
@pytest.mark.parametrize("dtype,cdrive", [("complex128", False), ("complex128", True), ("complex64", False),
                                          ("complex64", True)])
def test_step_matches_taylor(ctx, n, dtype, cdrive):
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    rng = np.random.default_rng(n)
    om = rng.uniform(0.5, 2.0, n) + (1j * rng.uniform(-0.5, 0.5, n) if cdrive else 0)
    om[n // 2] = 0.0
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=6.5, jitter=rng.uniform(-0.3, 0.3, n)))
    h = Hamiltonian(ctx, Basis(ctx, n), om, rng.uniform(-2, 2, n), pairs)
    x = rng.normal(size=h.dim) + 1j * rng.normal(size=h.dim)
    x /= np.linalg.norm(x)
    a = torch.as_tensor(x, dtype=getattr(torch, dtype), device=ctx.device)
    b = torch.as_tensor(x, dtype=torch.complex128, device=ctx.device)
    # the largest step: a CONV tau near 40 periods of the expansion; the
    # smallest keep one and two terms
    for tau in (30.0, 1e-9, 1e-3, 4.0):
        solvers.cheb_step(h, a, tau, tol=1e-13 if dtype == "complex128" else 1e-7)
        solvers.taylor_step(h, b, tau, tol=1e-14)
    # complex128: rounding of about 100 terms; complex64: the diagonal's FP32
    # rounding (spread below 100 MHz) times CONV tau, and the terms'
    tol = 1e-12 if dtype == "complex128" else 2e-5
    assert float((a.to(torch.complex128) - b).norm()) <= tol
