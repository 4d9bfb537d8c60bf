"""The start state and labels that the evolution forms without a host vector
equal the general forms (CPU)."""
import numpy as np

from energy_level_b200 import observables, state


def test_product_labels_equal_product_label():
    for n in (0, 1, 3, 6):
        assert observables.product_labels(n) == [observables.product_label(n, s) for s in range(1 << n)]


def test_basis_code_is_the_only_amplitude_of_state_vector():
    for spec in ("ggrg", None, [0, 1, "g", "r"], "|rgrg>", {"kind": "product", "amplitudes": ["g", "r", "g", [0, 1]]}):
        v = state.state_vector(spec, 4)
        c = state.basis_code(spec, 4)
        assert c is not None and v[c] == 1.0 and np.abs(v).sum() == 1.0
    for spec in (5, [[1, 1], 0, 0, 0], ("sup", ["gggg", "rrrr"]), "ground", np.eye(16)[3], [[0, 1j], 0, 0, 0]):
        assert state.basis_code(spec, 4) is None
