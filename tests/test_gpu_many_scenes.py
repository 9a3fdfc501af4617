"""More scenes than one launch of the per-scene sums takes (65535)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_scene_sums_of_many_scenes():
    from morphompm_b200 import _lib as L
    from morphompm_b200.runtime import Plan, ROW_F, SceneSpec
    sizes = np.random.default_rng(0).integers(0, 3, size=65535 + 70)
    sizes[65536] = 70000            # several chunks in the second launch
    specs = [SceneSpec(shape=(1, 1, 1), n=int(k), model=L.MODEL_NEOHOOKEAN, dx=0.1, dt=1e-4, damping=0.05, pmass=1.0,
                       vol0=1.0, mu=1.0, lam=1.0, growth_mode=1) for k in sizes]
    plan = Plan(specs, dtype=torch.float64)
    n = plan.n
    d = 1.0 + np.random.default_rng(1).random(n)
    slab = np.zeros((24, n))
    slab[15], slab[19], slab[23] = d, 1.0, 1.0
    s = torch.as_tensor(slab).cuda()
    loss = torch.full((len(sizes),), -1.0, dtype=torch.float64, device="cuda")
    off = np.concatenate([[0], np.cumsum(sizes)])
    ref = np.array([math.fsum(d[a:b]) for a, b in zip(off[:-1], off[1:])])
    for _ in range(2):
        plan.loss_detF(s.data_ptr() + ROW_F * n * 8, 1, n, loss)
        # sums of k values in [1, 2]: a rounding error of at most k eps per term
        assert np.all(np.abs(loss.cpu().numpy() - ref) <= 2.3e-16 * 2 * sizes * np.maximum(ref, 1.0))
