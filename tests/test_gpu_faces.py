"""A warp that holds a stencil at a face of the grid takes another node loop for
all its particles: the particles inside must not notice.  One cloud alone and
the same cloud with particles at the lower z face beside it, in the same (x, y)
columns (neighbours in the sorted order) but too far below to share a node:
states and gradients of the cloud agree bitwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("model", ["nh", "hencky", "hb"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("explicit_fg", [False, True])
def test_inner_particles_do_not_depend_on_neighbours(model, dtype, explicit_fg):
    from morphompm_b200.batch import host_slab, scene_spec_from_dict
    from morphompm_b200.runtime import Plan
    from morphompm_b200.trajectory import Rollout
    rng = np.random.default_rng(8)
    dx, shape = 1.0 / 16, (16, 15, 20)
    hb = dict(kappa=1e4, K=1.0, n=0.5, tau_y=10.0, m=100.0, eps=1e-4)
    n, m = 3000, 1500
    inner = rng.uniform([4, 4, 8], [11, 11, 14], size=(n, 3)) * dx
    face = rng.uniform([4, 4, 0.0], [11, 11, 1.3], size=(m, 3)) * dx
    dt = getattr(torch, dtype)
    vel = rng.standard_normal((3, n + m)) * 0.2
    g = 1.0 + 0.2 * rng.random(n + m)
    runs = []
    for x in (inner, np.concatenate([inner, face])):
        k = len(x)
        sc = dict(x=x, shape=shape, dx=dx, dt=2e-4, model=model, mu=400.0, lam=500.0, growth_A=0.15, hb=hb)
        plan = Plan([scene_spec_from_dict(sc, growth_mode=0 if explicit_fg else 1)], dtype=dt, device="cuda")
        Fg = None
        if explicit_fg:
            Fg = torch.zeros(9, k, dtype=dt, device="cuda")
            Fg[0::4] = torch.as_tensor(g[:k], dtype=dt).cuda()
        slab = host_slab([sc], np.dtype(dtype))
        slab[3:6] = vel[:, :k]
        ro = Rollout(plan, 4, advect=True, Fg=Fg)
        ro.run(torch.as_tensor(slab).cuda())
        torch.cuda.synchronize()
        runs.append((ro.final[:, :n].clone(), ro.bar0[:, :n].clone()))
    (f0, b0), (f1, b1) = runs
    assert torch.equal(f0, f1)
    assert torch.equal(b0, b1)
