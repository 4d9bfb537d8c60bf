"""FP32 arithmetic restated on the CPU, rounding by rounding."""
import numpy as np

CONV = 2.0 * np.pi * 1e-3
f4 = np.float32


def fma(a, b, c):
    """a b + c of FP32 values, rounded once (formed in extended precision)."""
    return (np.asarray(a, np.longdouble) * np.asarray(b, np.longdouble) + np.asarray(c, np.longdouble)).astype(f4)


def chebyshev_plan(lo, hi, tau, tol=1e-7):
    """a, b, M and the coefficients of exp(-i CONV H tau) for a spectrum in [lo, hi]."""
    from scipy.special import jv
    a, b = max(0.5 * (hi - lo) * (1.0 + 1e-6), 1e-12), 0.5 * (hi + lo)
    x, phi = a * CONV * tau, b * CONV * tau
    mmax = int(x + 30.0 + 6.0 * np.cbrt(x + 1.0))
    J = jv(np.arange(mmax + 1), x)
    over = [m for m in range(1, mmax + 1) if 2.0 * abs(J[m]) > 0.25 * tol]
    M = min(over[-1] + 1, mmax) if over else 1
    m = np.arange(M + 1)
    return a, b, M, np.where(m == 0, 1.0, 2.0) * J[:M + 1] * np.array([1, -1j, -1, 1j])[m & 3] * np.exp(-1j * phi)
