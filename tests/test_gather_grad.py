"""A slab that requires grad is refused where a gather would drop the gradient
silently (torch.index_select with out= refuses it too), and taken without grad."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


def test_gather_refuses_grad():
    from morphompm_b200.runtime import gather_columns
    src, order = torch.zeros(24, 5), torch.arange(5, dtype=torch.int32)
    with pytest.raises(RuntimeError, match="detach"):
        gather_columns(src.requires_grad_(True), order, torch.empty(24, 5))


@pytest.mark.gpu
def test_batch_load_refuses_grad():
    from morphompm_b200.batch import Batch, host_slab
    rng = np.random.default_rng(0)
    sc = [dict(x=rng.uniform(0.3, 0.7, size=(500, 3)), shape=(16, 16, 16), dx=1 / 16, dt=1e-4, model="nh", mu=400.0,
               lam=500.0, growth_A=0.1, ramp_steps=0, wall=2, phi=None)]
    slab = torch.as_tensor(host_slab(sc, np.float32))
    for device in ("cuda", "cpu"):
        b = Batch(sc, 2, dtype=torch.float32)
        assert b.order is not None
        s = slab.to(device, copy=True).requires_grad_(True)
        with pytest.raises(RuntimeError):
            b.load(s, non_blocking=False)
        with torch.no_grad():
            Batch(sc, 2, dtype=torch.float32).load(s, non_blocking=False)
