"""Per-scene sums over one, two and many chunks of slots, with empty and
one-particle scenes between them: the detF loss of states with known
determinants, twice (the chunk counters must return to zero)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sizes", [[1], [32768], [32769], [65537], [0, 5, 40000, 0, 1, 100000, 32768]])
def test_scene_sums(sizes):
    from morphompm_b200 import _lib as L
    from morphompm_b200.runtime import Plan, ROW_F, SceneSpec
    specs = [SceneSpec(shape=(8, 8, 8), n=k, model=L.MODEL_NEOHOOKEAN, dx=0.1, dt=1e-4, damping=0.05, pmass=1.0,
                       vol0=1.0, mu=1.0, lam=1.0, growth_mode=1) for k in sizes]
    plan = Plan(specs, dtype=torch.float64)
    n = plan.n
    d = 1.0 + np.random.default_rng(n).random(n)
    slab = np.zeros((24, n))
    slab[15], slab[19], slab[23] = d, 1.0, 1.0
    s = torch.as_tensor(slab).cuda()
    loss = torch.zeros(len(sizes), dtype=torch.float64, device="cuda")
    off = np.concatenate([[0], np.cumsum(sizes)])
    ref = np.array([d[a:b].sum() for a, b in zip(off[:-1], off[1:])])
    for _ in range(2):
        loss.fill_(-1.0)
        plan.loss_detF(s.data_ptr() + ROW_F * n * 8, 1, n, loss)
        # sums of k values in [1, 2]: a rounding error of at most k eps per term
        assert np.all(np.abs(loss.cpu().numpy() - ref) <= 2.3e-16 * 2 * np.array(sizes) * np.maximum(ref, 1.0))
