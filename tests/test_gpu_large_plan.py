"""Plans with more particles than three CTAs of 256 on every SM hold, where the
emitting G2P is compiled for more warps: chained steps against independent
ones, and scenes of such a batch against the same scenes run alone (fewer
particles: the other form of G2P and the cluster sort).  Bitwise, as for small
plans."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HB = dict(kappa=1e4, K=1.0, n=0.5, tau_y=10.0, m=100.0, eps=1e-4)


def _scenes(models, sizes):
    rng = np.random.default_rng(23)
    out = []
    for i, (m, n) in enumerate(zip(models, sizes)):
        edge = 40
        out.append(dict(x=rng.uniform(0.15, 0.85, size=(n, 3)), shape=(edge,) * 3, dx=1.0 / edge, dt=2e-5, model=m,
                        mu=400.0, lam=500.0, growth_A=0.1 + 0.02 * i, ramp_steps=0, wall=2, hb=HB,
                        phi=np.linspace(0.5, 1.0, n) if i == 1 else None))
    return out


@pytest.mark.parametrize("model", ["nh", "hencky", "hb"])
def test_chained_steps_match_independent_steps(model, dtype="float32"):
    """FP32: in FP64 the prepass kernel, which independent steps take, and the
    kernels of one model may differ in a contraction on plans of any size."""
    from morphompm_b200.batch import host_slab, scene_spec_from_dict
    from morphompm_b200.runtime import Plan, slab_particles
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sc = _scenes([model], [768 * sms + 1000])
    plan = Plan([scene_spec_from_dict(s) for s in sc], dtype=getattr(torch, dtype), device="cuda")
    slab = host_slab(sc, np.dtype(dtype))
    slab[3:6] = np.random.default_rng(1).standard_normal((3, plan.n)) * 0.05 / 40 / 2e-5
    out = []
    for chain in (False, True):
        a = torch.as_tensor(slab).cuda()
        b = torch.empty_like(a)
        for t in range(4):
            plan.step_fwd(slab_particles(a), slab_particles(b), True, t, None, chained=chain and t > 0,
                          emit=chain and t < 3)
            a, b = b, a
        torch.cuda.synchronize()
        out.append(a)
    assert torch.equal(out[0], out[1])
    assert plan.status() & ~8 == 0


def _run(sc, dtype):
    from morphompm_b200.batch import Batch, host_slab
    b = Batch(sc, 4, dtype=getattr(torch, dtype))
    b.load(host_slab(sc, np.dtype(dtype)), non_blocking=False)
    b.run()
    torch.cuda.synchronize()
    return b


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_large_batch_equals_scenes_alone(dtype):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # runs of one model beyond the rule's line and, beside them, small ones
    sizes = [60000, 2000, 768 * sms + 500 - 60000, 50000, 70000, 700]
    sc = _scenes(["nh", "hencky", "nh", "hb", "hb", "hencky"], sizes)
    b = _run(sc, dtype)
    fin, bar0 = b.final_state(), b.initial_cotangents()
    off = np.concatenate([[0], np.cumsum(sizes)])
    for i, s in enumerate(sc):
        one = _run([s], dtype)
        assert torch.equal(fin[:, off[i]:off[i + 1]], one.final_state()), i
        assert torch.equal(bar0[:, off[i]:off[i + 1]], one.initial_cotangents()), i
        assert torch.equal(b.loss[i], one.loss[0]) and torch.equal(b.dloss_dg[i], one.dloss_dg[0]), i
