"""Particles per cell far from the usual eight: one step and its VJP against
the oracle with 1 to several hundred particles in each occupied cell, in and
out of cell order, with particles outside the grid and at its faces, and a
growth-law trajectory (isotropic growth in the kernels) against the oracle's."""
import numpy as np
import pytest

from oracle import mpm_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N, DX, DT = 16, 1.0 / 16, 2e-4
# relative to each output's largest value: 200 roundings a term, and up to 1e3
# times that where a gradient is a difference of node values that were divided
# by a lone particle's small node masses; in FP32 a fifth of it (the positions
# are exact in both)
TOL = {"float32": 0.2 * 2e5 * 1.2e-7, "float64": 2e5 * 2.3e-16}


def _models(name):
    from morphompm_b200 import constitutive as K
    from morphompm_b200.config import Material
    mat = Material(E=1e3, nu=0.3)
    if name == "hb":
        return K.HerschelBulkley(), O.Model(kind="hb")
    return {"nh": K.NeoHookean, "hencky": K.Hencky}[name](mat), O.Model.elastic(name, 1e3, 0.3)


def _cloud(counts, rng):
    """counts[i] particles in the i-th of some distinct cells of the inner box."""
    cells = np.stack(np.unravel_index(rng.permutation(8 ** 3)[:len(counts)], (8, 8, 8)), 1) + 4
    x = np.concatenate([(c + 0.5 + rng.uniform(0.05, 0.95, size=(k, 3))) * DX for c, k in zip(cells, counts)])
    return x


def _close(a, b, tol):
    a = a.double().cpu().numpy() if torch.is_tensor(a) else np.asarray(a)
    return np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))


@pytest.mark.parametrize("counts", [
    [1] * 200, [9] * 37, [10] * 11, [27] * 12, [96], [97], [96, 1, 97, 3] * 3, [400] * 3, [1] * 30 + [300] + [2] * 40,
], ids=lambda c: f"{len(c)}cells_{sum(c)}")
@pytest.mark.parametrize("name,dtype", [("nh", "float64"), ("hencky", "float64"), ("hb", "float32"),
                                        ("nh", "float32")])
@pytest.mark.parametrize("shuffled", [False, True])
def test_step_and_vjp_vs_oracle(counts, name, dtype, shuffled):
    from morphompm_b200 import transfer
    from morphompm_b200.config import Material, SimConfig
    from morphompm_b200.state import ParticleState
    rng = np.random.default_rng(sum(counts) + len(counts))
    x = _cloud(counts, rng)
    # particles at the faces and outside of the grid
    x = np.concatenate([x, [[0.01, 0.5, 0.5], [0.5, 0.998, 0.5], [1.4, 0.5, 0.5], [-0.4, 0.2, 0.1]]])
    if shuffled:
        x = x[rng.permutation(len(x))]
    n = len(x)
    dt = getattr(torch, dtype)
    r = lambda *s: rng.standard_normal((n,) + s)
    host = [x, 0.1 * r(3), 0.3 * r(3, 3), np.eye(3) + 0.02 * r(3, 3), 1.1 * np.eye(3) + 0.01 * r(3, 3)]
    dev = [torch.as_tensor(a, dtype=dt).cuda() for a in host]
    host = [a.double().cpu().numpy() for a in dev]
    bars = [torch.as_tensor(a, dtype=dt).cuda() for a in (r(3), r(3), r(3, 3), r(3, 3))] + \
           [torch.as_tensor(r(3, 3)).cuda()]
    hbars = [a.double().cpu().numpy() for a in bars]
    m, om = _models(name)
    cfg = SimConfig(N=N, dx=DX, dt=DT, sp=DX / 2, material=Material(E=1e3, nu=0.3))
    scene = O.scene_from_cfg(N, DX, DT, cfg.damping, DX / 2, cfg.material.density)
    ns, cache = transfer.step(ParticleState(*dev), m, cfg, advect=True)
    g = transfer.step_vjp(cache, *bars, advect=True)
    ons, oc = O.step(O.State(*host), om, scene, advect=True)
    og = O.step_vjp(oc, *hbars, advect=True)
    tol = 1e-8 if name == "hencky" else TOL[dtype]       # Hencky: the divided-difference switch
    for a, b in zip((ns.x, ns.v, ns.C, ns.F), (ons.x, ons.v, ons.C, ons.F)):
        assert _close(a, b, tol)
    for a, b in zip(g, og):
        assert _close(a, b, tol)


@pytest.mark.parametrize("name", ["nh", "hencky", "hb"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(12, 11, 4), (12, 10, 2)])
def test_growth_law_trajectory_at_the_faces(name, dtype, shape):
    """Three growth steps and their adjoint on a grid a few nodes thick: most
    stencils cross a face, and Fg = g I in every kernel."""
    from morphompm_b200.batch import Batch, host_slab
    rng = np.random.default_rng(shape[2])
    dx = 1.0 / 12
    npd = np.dtype(dtype)
    x = (rng.uniform(0.0, 1.0, size=(700, 3)) * np.array(shape) * dx).astype(npd).astype(np.float64)
    om = O.Model(kind="hb") if name == "hb" else O.Model(kind=name, mu=400.0, lam=500.0)
    hb = dict(kappa=om.kappa, K=om.K, n=om.n, tau_y=om.tau_y, m=om.m, eps=om.eps)
    b = Batch([dict(x=x, shape=shape, dx=dx, dt=DT, model=name, mu=400.0, lam=500.0, growth_A=0.2, hb=hb)], 3,
              dtype=getattr(torch, dtype), advect=True)
    b.load(host_slab([dict(x=x)], npd), non_blocking=False)
    b.run()
    torch.cuda.synchronize()
    sc = O.Scene(shape=shape, dx=dx, dt=DT, damping=0.05, pmass=(dx / 2) ** 3, vol0=(dx / 2) ** 3)
    gr = O.Growth(A=0.2)
    st, caches = O.rollout(O.State.rest(x), om, sc, 3, advect=True, growth=gr)
    z3, z33 = np.zeros((700, 3)), np.zeros((700, 3, 3))
    out = O.rollout_vjp(caches, z3, z3, z33, O.seed_detF(st.F), z33, advect=True, growth=gr)
    tol = 1e-8 if name == "hencky" and dtype == "float64" else TOL[dtype]
    fin, bar = b.final_state(), b.initial_cotangents()
    rows = lambda s, i, k: s[i:i + k].t().reshape((700,) + ((3,) if k == 3 else (3, 3)))
    for got, ref in ((rows(fin, 0, 3), st.x), (rows(fin, 3, 3), st.v), (rows(fin, 6, 9), st.C), (rows(fin, 15, 9), st.F),
                     (rows(bar, 0, 3), out[0]), (rows(bar, 3, 3), out[1]), (rows(bar, 6, 9), out[2]),
                     (rows(bar, 15, 9), out[3]), (b.loss, np.array([O.loss_detF(st.F)])),
                     (b.dloss_dg, np.array([out[5]]))):
        assert _close(got, ref, tol)


@pytest.mark.parametrize("name,dtype", [("nh", "float64"), ("hb", "float32")])
@pytest.mark.parametrize("shuffled", [False, True])
def test_many_sparse_cells_vs_oracle(name, dtype, shuffled):
    """Enough cells of one or two particles for the sums to take 32 cells a warp,
    with dense cells among them that such a warp's records do not fit."""
    from morphompm_b200 import transfer
    from morphompm_b200.config import Material, SimConfig
    from morphompm_b200.state import ParticleState
    rng = np.random.default_rng(5)
    edge, dx = 40, 1.0 / 40
    cells = rng.permutation(36 ** 3)[:34000]
    counts = np.ones(len(cells), int)
    counts[::50] = 2
    counts[[100, 101, 5000]] = (150, 97, 400)
    c = np.stack(np.unravel_index(np.repeat(cells, counts), (36, 36, 36)), 1) + 1
    x = (c + 0.5 + rng.uniform(0.05, 0.95, size=c.shape)) * dx
    if shuffled:
        x = x[rng.permutation(len(x))]
    n = len(x)
    assert n <= 2 * len(cells)
    dt = getattr(torch, dtype)
    r = lambda *s: rng.standard_normal((n,) + s)
    dev = [torch.as_tensor(a, dtype=dt).cuda() for a in
           (x, 0.1 * r(3), 0.3 * r(3, 3), np.eye(3) + 0.02 * r(3, 3), 1.1 * np.eye(3) + 0.01 * r(3, 3))]
    bars = [torch.as_tensor(a, dtype=dt).cuda() for a in (r(3), r(3), r(3, 3), r(3, 3))] + \
           [torch.as_tensor(r(3, 3)).cuda()]
    m, om = _models(name)
    cfg = SimConfig(N=edge, dx=dx, dt=DT, sp=dx / 2, material=Material(E=1e3, nu=0.3))
    scene = O.scene_from_cfg(edge, dx, DT, cfg.damping, dx / 2, cfg.material.density)
    ns, cache = transfer.step(ParticleState(*dev), m, cfg, advect=True)
    g = transfer.step_vjp(cache, *bars, advect=True)
    f64 = lambda ts: [a.double().cpu().numpy() for a in ts]
    ons, oc = O.step(O.State(*f64(dev)), om, scene, advect=True)
    og = O.step_vjp(oc, *f64(bars), advect=True)
    for a, b in zip((ns.x, ns.v, ns.C, ns.F, *g), (ons.x, ons.v, ons.C, ons.F, *og)):
        assert _close(a, b, TOL[dtype])
