"""complex64 pulse gradient against the same recurrence restated in FP32 on the
CPU, rounding by rounding: forward terms t_m, accumulated states, lambda and
the reverse terms u_m, so that a change in how a row is rounded shows at once
and not only as digits lost over some hundred steps."""
import numpy as np
import pytest

from energy_level_b200 import configs
from fp32_restated import chebyshev_plan, f4, fma

pytestmark = pytest.mark.gpu

def _cmul(a, z, first=True):
    """a z with the roundings of a row: first picks which product of the
    imaginary part is the fused one."""
    re = fma(a[0], z[0], -(a[1] * z[1]))
    im = fma(a[0], z[1], a[1] * z[0]) if first else fma(a[1], z[0], a[0] * z[1])
    return re, im


def _plan(V, flips, occ, tau, om, de):
    R = 0.5 * abs(om) * flips
    d = V - de * occ
    a, b, M, c = chebyshev_plan((d - R).min(), (d + R).max(), tau)
    return a, b, M, c.real.astype(f4), c.imag.astype(f4)


def _restated(n, codes, V, occ, psi0, target, tau, om, de):
    dim, K = len(codes), len(tau)
    T = []
    for k in range(n):
        w = codes ^ (1 << k)
        p = np.searchsorted(codes, w).clip(max=dim - 1)
        T.append(np.where(codes[p] == w, p, dim))
    T = np.array(T)
    plans = [_plan(V, (T < dim).sum(0), occ, tau[k], om[k], de[k]) for k in range(K)]

    def flips(x):     # four lanes take every fourth bit and meet in a butterfly
        z = np.append(x, f4(0))
        lane = []
        for q in range(4):
            s = np.zeros(dim, f4)
            for k in range(q, n, 4):
                s = np.where(T[k] < dim, fma(f4(0.5), z[T[k]], s), s)
            lane.append(s)
        return (lane[0] + lane[2]) + (lane[1] + lane[3])

    def product(k, x, s, one):
        a, b = f4(plans[k][0]), f4(plans[k][1])
        al, be = (f4(1) / a, -b / a) if one else (f4(2) / a, f4(-2) * b / a)
        d = fma(f4(-de[k]), occ.astype(f4), V.astype(f4))
        return fma(be, x, al * fma(f4(om[k]), s, d * x))

    x = (psi0.real, psi0.imag)
    terms = []
    for k in range(K):
        _, _, M, cr, ci = plans[k]
        tl, z = [x], (f4(0), f4(0))
        for m in range(1, M + 1):
            y = tuple(product(k, x[q], flips(x[q]), m == 1) - z[q] for q in range(2))
            if m == 1:
                p = _cmul((cr[0], ci[0]), x, first=False)
                acc = (fma(-ci[1], y[1], fma(cr[1], y[0], p[0])), fma(ci[1], y[0], fma(cr[1], y[1], p[1])))
            else:
                p = _cmul((cr[m], ci[m]), y, first=False)
                acc = (acc[0] + p[0], acc[1] + p[1])
            z, x = x, y
            tl.append(y)
        terms.append(tl)
        x = acc
    psi = (x[0] + 1j * x[1]).astype(np.complex64)
    ov = np.vdot(target.astype(complex), psi.astype(complex))
    lam = _cmul((f4(ov.real), f4(ov.imag)), (target.real, target.imag), first=False)
    go, gd = np.zeros(K), np.zeros(K)
    for k in range(K - 1, -1, -1):
        a, _, M, cr, ci = plans[k]
        x, z = _cmul((cr[M], -ci[M]), lam), (f4(0), f4(0))
        for m in range(M - 1, -1, -1):
            s = (flips(x[0]), flips(x[1]))
            p = _cmul((cr[m], -ci[m]), lam)
            y = tuple(product(k, x[q], s[q], m == 0) - z[q] + p[q] for q in range(2))
            w = 2.0 / a * (1.0 if m == 0 else 2.0)
            for q in range(2):
                t = terms[k][m][q].astype(float)
                go[k] += w * np.sum(s[q].astype(float) * t)
                gd[k] -= w * np.sum(occ * x[q].astype(float) * t)
            z, x = x, y
        lam = x
    return abs(ov) ** 2, go, gd, psi


# the terms of the last pulse (a step of 3.6 us, more than 256 terms) are more than
# a step's coefficients in shared memory: rows in memory, not in registers
@pytest.mark.parametrize("n,tau", [(12, [10.0, 10.0, 10.0]), (9, [25.0, 0.0, 0.001, 8.0]), (10, [12.0, 3600.0])])
def test_complex64_gradient_rounds_as_stated(n, tau):
    import torch
    from energy_level_b200.adjoint import PulseProblem
    from oracle import ref
    edges = configs.ring_edges(n)
    calib = configs.calib_from_positions(configs.ring_positions(n))
    prob = PulseProblem(calib, "g" * n, target="g" * n, dtype="complex64",
                        plan=dict(projected=True, blockade_edges=edges, constraint=dict(kind="blockade")))
    codes = np.asarray(ref.independent_states(n, edges, None)).astype(np.int64)
    bits = np.array([(codes >> (n - 1 - q)) & 1 for q in range(n)], float)
    occ = bits.sum(0)
    V = sum(p["V"] * bits[p["i"]] * bits[p["j"]] for p in calib["pairs"])
    rng = np.random.default_rng(n)
    vec = lambda: (lambda v: (v / np.linalg.norm(v)).astype(np.complex64))(
        rng.normal(size=len(codes)) + 1j * rng.normal(size=len(codes)))
    psi0, target = vec(), vec()
    prob.psi0 = torch.as_tensor(psi0, device="cuda")
    prob.target = torch.as_tensor(target, device="cuda")
    om, de = rng.uniform(1.0, 3.0, len(tau)), rng.uniform(-4.0, 4.0, len(tau))
    F, go, gd, psi = prob.evaluate(np.array(tau), om, de, want_state=True)
    rF, rgo, rgd, rpsi = _restated(n, codes, V, occ, psi0, target, tau, om, de)
    # the FP32 vectors are equal bit for bit; what is left is the order of the
    # FP64 sums: at most dim x terms (322 x 400) additions of 1.1e-16
    assert np.array_equal(psi.cpu().numpy(), rpsi)
    tol = len(codes) * 400 * 1.2e-16
    assert abs(F - rF) <= tol
    assert np.abs(go - rgo).max() <= tol * max(1.0, np.abs(rgo).max())
    assert np.abs(gd - rgd).max() <= tol * max(1.0, np.abs(rgd).max())
