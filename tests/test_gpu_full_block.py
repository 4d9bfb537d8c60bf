"""Full-basis H-apply (el_full.cu) against the oracle: the smallest bases its
tiles take, one and several tiles, rows of 1 to 32 chunks, missing amplitudes
and the fused dot products."""
import numpy as np
import pytest

from oracle import ref
from energy_level_b200 import configs

pytestmark = pytest.mark.gpu

# n + 2 roundings of terms below the scale (see the assertion), n <= 17
TOL = {"float64": 40 * 2.3e-16, "complex128": 80 * 2.3e-16, "float32": 40 * 6e-8, "complex64": 80 * 6e-8}


def _system(n, seed, cplx):
    rng = np.random.default_rng(seed)
    om = rng.uniform(0.5, 2.0, n) + (1j * rng.uniform(-0.5, 0.5, n) if cplx else 0)
    om[rng.integers(0, n, 2)] = 0.0          # sites without a drive
    pos = configs.chain_positions(n, a=5.5, jitter=rng.uniform(-0.5, 0.5, n))
    return om, rng.uniform(-2, 2, n), configs.pairs_from_positions(pos)


@pytest.mark.parametrize("n,nvecs", [(5, (2, 8)), (7, (2, 4, 64)), (10, (2, 16, 128)), (12, (2, 8)), (16, (1, 2)), (17, (1,))])
@pytest.mark.parametrize("dtype,cdrive", [("float32", False), ("float64", False), ("complex64", False),
                                          ("complex64", True), ("complex128", False), ("complex128", True)])
def test_hv_edges(ctx, n, nvecs, dtype, cdrive):
    import torch
    from energy_level_b200.core import Basis, Hamiltonian
    om, de, pairs = _system(n, 3 + n, cdrive)
    b = Basis(ctx, n)
    h = Hamiltonian(ctx, b, om, de, pairs)
    rng = np.random.default_rng(n)
    for nvec in nvecs:
        x = rng.normal(size=(b.dim, nvec))
        if dtype.startswith("complex"):
            x = x + 1j * rng.normal(size=(b.dim, nvec))
        tx = torch.as_tensor(x, dtype=getattr(torch, dtype), device=ctx.device)
        want = ref.hv(n, None, om if cdrive else om.real, de, pairs, tx.cpu().numpy().astype(
            complex if dtype.startswith("complex") else float))
        got = h.hv(tx).cpu().numpy()
        scale = max(np.abs(want).max(), np.abs(ref.diagonal(n, np.arange(b.dim), de, pairs)).max() * np.abs(x).max())
        assert np.abs(got - want).max() <= TOL[dtype] * scale, (nvec, np.abs(got - want).max() / scale)


@pytest.mark.parametrize("n,nvec,chunk", [(16, 2, 1), (11, 6, 8), (8, 64, 64)])
@pytest.mark.parametrize("mode", ["direct", "doubling"])
def test_moments_with_block_dots(ctx, n, nvec, chunk, mode):
    """The fused recurrence and its dot products (FP64 vectors, generic path)."""
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    om, de, pairs = _system(n, 17 + n, False)
    b = Basis(ctx, n)
    h = Hamiltonian(ctx, b, om, de, pairs)
    lo, hi = solvers.bounds(h)
    c, r = solvers.kpm_scale(lo, hi)
    probes = np.random.default_rng(2).choice([-1, 1], size=(nvec, b.dim))
    mu = solvers.kpm_moments(h, 16, nvec, c, r, dtype="float64", chunk=chunk, probes=probes, mode=mode, generic=True)
    want = ref.kpm_moments(lambda v: ref.hv(n, None, om.real, de, pairs, v), b.dim, 16, probes, c, r)
    # moments are at most 1; the recurrence's error grows at most linearly in num
    assert np.abs(mu - np.asarray(want)).max() <= 1e-11
