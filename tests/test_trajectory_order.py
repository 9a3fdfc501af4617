"""The storage order of a trajectory's particles on both sides of the size up to
which it is formed without asking whether it is needed."""
import numpy as np
import pytest
import torch

from morphompm_b200 import layout

DX, SHAPE = 1.0 / 32, (32, 30, 28)


@pytest.mark.parametrize("n", [1, 2, 1000, layout.ASK_ABOVE, layout.ASK_ABOVE + 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_order_is_the_cell_order(n, dtype):
    x = np.random.default_rng(n).uniform(-0.05, 1.05, size=(n, 3))
    t = torch.as_tensor(x).to(dtype)
    ref = layout.cell_order_host(t.double().numpy(), DX, SHAPE)
    order = layout.trajectory_order(t, DX, SHAPE)
    if n < 2:
        assert order is None
        return
    assert np.array_equal(order.numpy(), ref)
    # particles in cell order stay where they are
    again = layout.trajectory_order(t[order].contiguous(), DX, SHAPE)
    if n > layout.ASK_ABOVE:
        assert again is None
    else:
        assert np.array_equal(again.numpy(), np.arange(n))
