"""Batched Lanczos past the sizes at which its kernels change form: instances
whose vector does not fit the CTA's shared memory next to ones whose vector
does, and cooperative solves with 256 rows per CTA (two threads per row) and
with 512 and 1024 (one)."""
import numpy as np
import pytest

from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


def _codes(n, edges):
    adj = [0] * n
    for a, b in edges or []:
        adj[n - 1 - a] |= 1 << (n - 1 - b)
        adj[n - 1 - b] |= 1 << (n - 1 - a)
    c = np.zeros(1, np.int64)
    for k in range(n):
        c = np.concatenate([c, c[(c & adj[k]) == 0] | (1 << k)])
    return c


def _instance(n, edges, seed):
    rng = np.random.default_rng(seed)
    calib = configs.calib_from_positions(configs.chain_positions(n, a=5.5, jitter=rng.uniform(-0.2, 0.2, n)))
    return dict(calib=calib, Om=np.full(n, 2.0), delta=-2.0 * rng.uniform(0.0, 3.0, n), edges=edges)


def _lowest(inst):
    """E0 and gap by ARPACK on the explicit sparse H."""
    import scipy.sparse as sp
    from scipy.sparse.linalg import eigsh
    n = len(inst["Om"])
    codes = _codes(n, inst["edges"])
    bits = np.array([(codes >> (n - 1 - q)) & 1 for q in range(n)], float)
    d = inst["delta"] @ bits + sum(p["V"] * bits[p["i"]] * bits[p["j"]] for p in inst["calib"]["pairs"])
    H = sp.diags(d).tocsr()
    for k in range(n):
        w = codes ^ (1 << k)
        p = np.searchsorted(codes, w).clip(max=len(codes) - 1)
        ok = np.nonzero(codes[p] == w)[0]
        H = H + sp.csr_matrix((np.full(len(ok), 0.5 * inst["Om"][n - 1 - k]), (ok, p[ok])), shape=H.shape)
    e = np.sort(eigsh(H, k=2, which="SA", tol=1e-12, return_eigenvectors=False))
    return e[0], e[1] - e[0]


# FP64 room: about 27,000 rows with one CTA per SM, 13,000 with two
@pytest.mark.parametrize("threads,ctas", [(256, 1), (256, 2), (512, 1), (512, 2), (1024, 1)])
def test_instances_around_the_shared_memory_limit(ctx, threads, ctas):
    from energy_level_b200.batched import BatchedGroundStates
    insts = [_instance(12, configs.chain_edges(12), 1), _instance(21, configs.chain_edges(21), 2),
             _instance(14, None, 3), _instance(18, configs.ring_edges(18), 4)]
    b = BatchedGroundStates(insts, dtype="float64", max_iter=300, tol=1e-10)
    b.run(threads=threads, ctas_per_sm=ctas)
    r = b.results()
    b.close()
    assert r["converged"].all()
    for i, inst in enumerate(insts):
        e0, gap = _lowest(inst)
        # residual 1e-10 max(1, |theta|); ARPACK's, and rounding of about 1e-13 |E|
        assert abs(r["E0"][i] - e0) < 1e-9 * max(1.0, abs(e0))
        assert abs(r["gap"][i] - gap) < 1e-7


@pytest.mark.parametrize("n,m", [(19, 75), (20, 36), (22, 16)])    # 256, 512 and 1024 rows per CTA
def test_cooperative_solve_with_wide_ctas(ctx, n, m):
    from energy_level_b200.batched import BatchedGroundStates
    b = BatchedGroundStates([_instance(n, configs.chain_edges(n), n)], dtype="float64", max_iter=m, tol=1e-10)
    b.run_coop(seed=5)
    c = b.results()
    b.run(seed=5)
    r = b.results()
    b.close()
    # the same start vector and number of steps: the same Ritz values, up to what
    # two orders of FP64 rounding (1e-13 of the spectrum's 100 MHz a step) grow
    # to in a Krylov space; a row left out or read twice shows above 1e-3
    assert abs(c["E0"][0] - r["E0"][0]) < 1e-6
    assert abs(c["gap"][0] - r["gap"][0]) < 1e-6
