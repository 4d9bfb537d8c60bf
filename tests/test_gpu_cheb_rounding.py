"""Series of complex64 Chebyshev steps on small full bases against the same
recurrence restated in FP32 on the CPU, rounding by rounding.  The phase of a
state drifts with the error of the recurrence's coefficients and of the
diagonal, so a rounding more in either shows only after many steps, and not in
occupations at all."""
import numpy as np
import pytest

from energy_level_b200 import configs
from fp32_restated import chebyshev_plan, f4, fma

pytestmark = pytest.mark.gpu


def _sum_lanes(parts):
    return (parts[0] + parts[2]) + (parts[1] + parts[3]) if len(parts) == 4 else parts[0]


def _restated_step(x, n, V, up, delta, plan):
    """up, delta by bit.  Bits k, k + G, ... are summed in ascending order, the
    G sums in a butterfly."""
    a, b, M, c = plan
    G = 4 if n <= 16 else 1
    codes = np.arange(1 << n)
    ur, ui, cr, ci = up.real.astype(f4), up.imag.astype(f4), c.real.astype(f4), c.imag.astype(f4)
    sums = []
    for q in range(G):
        s = np.zeros(len(codes), f4)
        for k in range(q, n, G):
            s = np.where((codes >> k) & 1, s + delta[k].astype(f4), s)
        sums.append(s)
    d = _sum_lanes(sums) + V.astype(f4)
    xr, xi = x.real.copy(), x.imag.copy()
    acc = [(c[0] * x.astype(complex)).real.astype(f4), (c[0] * x.astype(complex)).imag.astype(f4)]
    zr = zi = f4(0)
    for m in range(1, M + 1):
        al, be = (f4(1.0 / a), f4(-b / a)) if m == 1 else (f4(2.0 / a), f4(-2.0 * b / a))
        pr, pi = [], []
        for q in range(G):
            hr, hi = np.zeros(len(codes), f4), np.zeros(len(codes), f4)
            for k in range(q, n, G):
                vr, vi = xr[codes ^ (1 << k)], xi[codes ^ (1 << k)]
                if up.imag.any():
                    w = np.where((codes >> k) & 1, ui[k], -ui[k])
                    hr = hr + fma(ur[k], vr, -(w * vi))
                    hi = hi + fma(ur[k], vi, w * vr)
                else:
                    hr, hi = fma(ur[k], vr, hr), fma(ur[k], vi, hi)
            pr.append(hr)
            pi.append(hi)
        yr = fma(al, fma(d, xr, _sum_lanes(pr)), be * xr) - zr
        yi = fma(al, fma(d, xi, _sum_lanes(pi)), be * xi) - zi
        acc[0] = acc[0] + fma(cr[m], yr, -(ci[m] * yi))
        acc[1] = acc[1] + fma(cr[m], yi, ci[m] * yr)
        zr, zi, xr, xi = xr, xi, yr, yi
    return (acc[0] + 1j * acc[1]).astype(np.complex64)


# one tile (one and two rows per thread), several tiles (1, 2 and 4 rows)
@pytest.mark.parametrize("n,steps", [(5, 12), (9, 12), (10, 12), (11, 12), (14, 4), (16, 2), (17, 2), (18, 1)])
@pytest.mark.parametrize("cdrive", [False, True])
def test_complex64_steps_round_as_stated(ctx, n, steps, cdrive):
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Hamiltonian
    rng = np.random.default_rng(n)
    om = rng.uniform(0.5, 2.0, n) + (1j * rng.uniform(-0.5, 0.5, n) if cdrive else 0)
    om[n // 2] = 0.0
    de = rng.uniform(-2.0, 2.0, n)
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=6.5, jitter=rng.uniform(-0.3, 0.3, n)))
    h = Hamiltonian(ctx, Basis(ctx, n), om, de, pairs)
    x = rng.normal(size=h.dim) + 1j * rng.normal(size=h.dim)
    x = (x / np.linalg.norm(x)).astype(np.complex64)
    codes = np.arange(h.dim)
    bits = np.array([(codes >> (n - 1 - q)) & 1 for q in range(n)], float)
    V = sum(v * bits[i] * bits[j] for i, j, v in pairs)
    up, diag = 0.5 * om[::-1].astype(complex), V + de @ bits
    plan = chebyshev_plan(diag.min() - np.abs(up).sum(), diag.max() + np.abs(up).sum(), 20.0)
    psi = torch.as_tensor(x, device=ctx.device)
    for _ in range(steps):
        solvers.cheb_step(h, psi, 20.0, tol=1e-7)
        x = _restated_step(x, n, V, up, de[::-1], plan)
    # every operation is stated: equal bit for bit
    assert np.array_equal(psi.cpu().numpy(), x)
