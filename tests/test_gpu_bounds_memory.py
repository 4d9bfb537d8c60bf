"""What spectral bounds hold on the device does not depend on the largest number
of steps that the caller allows."""
import numpy as np
import pytest

from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


def test_bounds_workspace_does_not_grow_with_max_iter():
    import torch
    from energy_level_b200 import solvers
    from energy_level_b200.core import Basis, Context, Hamiltonian
    n = 24
    pairs = configs.pairs_from_positions(configs.chain_positions(n, a=6.5))

    def held(max_iter):
        c = Context(0)
        try:
            h = Hamiltonian(c, Basis(c, n), np.full(n, 2.0), np.linspace(-1.0, 1.0, n), pairs)
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            e = solvers.bounds(h, max_iter=max_iter)
            torch.cuda.synchronize()
            return e, before - torch.cuda.mem_get_info()[0]
        finally:
            c.close()

    held(300)                      # kernels are loaded
    assert held(2**31 - 1) == held(300)
