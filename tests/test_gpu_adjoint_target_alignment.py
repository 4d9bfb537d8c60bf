"""The target state of a pulse gradient is read wherever it starts: a pointer
aligned to one real value, as a C caller may pass, gives the same results as
one aligned to a complex value."""
import numpy as np
import pytest

from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


class _Pointer:
    def __init__(self, buf, values):
        self.buf, self.values = buf, values      # the buffer stays alive

    def data_ptr(self):
        return self.buf.data_ptr() + self.values * self.buf.element_size()


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n", [9, 21])           # rows in registers, and in memory
def test_target_aligned_to_one_value(dtype, n):
    import torch
    from energy_level_b200.adjoint import PulseProblem
    plan = dict(projected=True, blockade_edges=configs.ring_edges(n), constraint=dict(kind="blockade"))
    prob = PulseProblem(configs.calib_from_positions(configs.ring_positions(n)), "g" * n,
                        target="rg" * (n // 2) + "g" * (n % 2), plan=plan, dtype=dtype)
    tau, om, de = np.full(5, 30.0), np.linspace(1.0, 2.0, 5), np.linspace(-3.0, 3.0, 5)
    a = prob.evaluate(tau, om, de)
    real = torch.view_as_real(prob.target).reshape(-1)
    buf = torch.zeros(real.numel() + 2, dtype=real.dtype, device=real.device)
    buf[1:-1] = real
    prob.target = _Pointer(buf, 1)
    assert prob.target.data_ptr() % (2 * buf.element_size()) != 0
    b = prob.evaluate(tau, om, de)
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
    prob.target = torch.view_as_complex(real.reshape(-1, 2))
