"""Cooperative pulse gradient with its terms stored, row values in registers
and coefficients in shared memory, against the one-launch-per-term schedule:
steps of zero and of very different length, bases of a few rows, of one pass
of the grid and of several, and a diagonal objective."""
import numpy as np
import pytest

from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


def _problem(n, dtype, ring, observable):
    from energy_level_b200.adjoint import PulseProblem
    edges = configs.ring_edges(n) if ring else configs.chain_edges(n)
    calib = configs.calib_from_positions(configs.ring_positions(n) if ring else configs.chain_positions(n))
    plan = dict(projected=True, blockade_edges=edges, constraint=dict(kind="blockade"))
    kw = dict(target="rg" * (n // 2) + "g" * (n % 2))
    if observable:
        from oracle import ref
        codes = ref.independent_states(n, edges, None)
        kw = dict(observable=np.array([bin(int(c)).count("1") for c in codes], float))
    return PulseProblem(calib, "g" * n, plan=plan, dtype=dtype, **kw)


@pytest.mark.parametrize("n,ring", [(4, False), (9, True), (14, False), (20, True), (23, False)])
@pytest.mark.parametrize("observable", [False, True])
@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-11), ("complex64", 2e-5)])
def test_coop_matches_per_term_schedule(n, ring, observable, dtype, tol):
    prob = _problem(n, dtype, ring, observable)
    rng = np.random.default_rng(n)
    tau = np.array([0.0, 25.0, 0.001, 60.0, 0.0, 8.0, 0.0])   # one-term steps next to long ones
    om = rng.uniform(0.5, 3.0, len(tau))
    de = rng.uniform(-4.0, 4.0, len(tau))
    try:
        prob.set_schedule("coop")
        a = prob.evaluate(tau, om, de, want_state=True)
        b = prob.evaluate(tau, om, de)
        prob.set_schedule("stream")
        c = prob.evaluate(tau, om, de, want_state=True)
    finally:
        prob.set_schedule("auto")
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
    assert abs(a[0] - c[0]) <= tol * max(1.0, abs(c[0]))
    for x, y in ((a[1], c[1]), (a[2], c[2])):
        assert np.abs(x - y).max() <= tol * max(np.abs(y).max(), 1e-3)
    assert float((a[3] - c[3]).abs().max()) <= tol
