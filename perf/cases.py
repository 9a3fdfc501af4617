"""Performance cases of the differentiable growth step, through the package's
public entry points:

  step       transfer.step and transfer.step_vjp on the caller's tensors
  gradient   autograd.rollout_loss and its backward (explicit growth)
  batch      batch.Batch: load a state, replay the captured forward + loss +
             adjoint trajectory, read the results (growth law)
  material   a model's stress and stress_vjp

Each case is one pass of one of them.  ``prepare`` makes the inputs and what a
program keeps (models, configs, the captured batch), ``run`` is the pass,
``work`` counts what it cannot do without, and ``exact`` is the same pass in
plain torch float64.
"""
import math

import numpy as np
import torch

DEV = "cuda"
DTYPES = {"float32": torch.float32, "float64": torch.float64}
MODELS = ("nh", "hencky", "hb")
HB = dict(kappa=1.0e4, K=1.0, n=0.5, tau_y=10.0, m=100.0, eps=1e-4)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one drop-in step and its VJP at the size of the unit tests: latency only
        dict(name="step_tiny_f64", kind="step", n=48, edge=8, model="hencky", dtype="float64", advect=True),
        # the drop-in step with positions frozen, as the reference's integrate.rollout does by default
        dict(name="step_cube_f64", kind="step", n=4096, edge=32, model="nh", dtype="float64", advect=False),
        # the drop-in step on a large odd-sized cloud, strided (n, 3, 3) fields, rate-dependent material
        dict(name="step_large_f32", kind="step", n=1000003, edge=128, model="hb", dtype="float32", advect=True),
        # the constitutive seam called by itself: large, with the 3x3 eigensolve
        dict(name="material_hencky_f32", kind="material", n=1048583, model="hencky", dtype="float32"),
        # a torch training loop over one trajectory: scalar growth, positions frozen, FP64
        dict(name="gradient_cube_f64", kind="gradient", n=4096, edge=32, model="nh", dtype="float64", steps=25,
             ckpt=0, loss="detF", per_particle=False, advect=False),
        # the same with a per-particle growth field, checkpointed, odd size, FP32
        dict(name="gradient_field_f32", kind="gradient", n=20011, edge=48, model="hencky", dtype="float32",
             steps=24, ckpt=6, loss="detF", per_particle=True, advect=True),
        # free-swell cube with the growth ramp (the first growth workload)
        dict(name="cube_f32", kind="batch", scenes=1, n_lo=4096, n_hi=4096, edge_lo=32, edge_hi=32, models="nh",
             dtype="float32", steps=40, ckpt=0, loss="detF", ramp=100, dt=2.5e-5, aspect=1, field="none"),
        # bilayer strip, Hencky, one end clamped, the top layer growing
        dict(name="bilayer_f32", kind="batch", scenes=1, n_lo=32768, n_hi=32768, edge_lo=32, edge_hi=32,
             models="hencky", dtype="float32", steps=40, ckpt=0, loss="detF", ramp=2000, dt=1.25e-5, aspect=8,
             field="layer"),
        # inverse problem: positions observed, checkpoints every 20 steps, FP64
        dict(name="inverse_f64", kind="batch", scenes=1, n_lo=32768, n_hi=32768, edge_lo=64, edge_hi=64,
             models="nh", dtype="float64", steps=40, ckpt=20, loss="mse", ramp=0, dt=1e-4, aspect=1, field="none"),
        # the headline workload: 256 uneven scenes of two materials (fewer steps)
        dict(name="batch_f32", kind="batch", scenes=256, n_lo=2048, n_hi=65536, edge_lo=32, edge_hi=64,
             models="nh+hencky", dtype="float32", steps=8, ckpt=0, loss="detF", ramp=0, dt=2e-5, aspect=1,
             field="none"),
        # a batch of the FP64 path
        dict(name="batch_f64", kind="batch", scenes=40, n_lo=2048, n_hi=65536, edge_lo=32, edge_hi=64,
             models="nh+hencky", dtype="float64", steps=8, ckpt=0, loss="detF", ramp=0, dt=2e-5, aspect=1,
             field="none"),
        # one large scene: a sheet of rate-dependent material, radial growth, sqrt(N) checkpoints
        dict(name="sheet_f32", kind="batch", scenes=1, n_lo=2097152, n_hi=2097152, edge_lo=256, edge_hi=256,
             models="hb", dtype="float32", steps=6, ckpt=3, loss="detF", ramp=0, dt=2.5e-6, aspect=-8,
             field="radial"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edge_for(rng, n, lo=16, hi=256):
    """A grid edge whose inner box holds a cube of n particles at 8 per cell."""
    c = math.ceil((n / 8.0) ** (1.0 / 3.0))
    low = max(lo, c + 6)
    return min(hi, low + rng.randrange(0, max(1, low // 2)))


def draw(rng):
    kind = rng.choice(["step", "gradient", "batch", "batch", "batch", "material"])
    dtype = rng.choice(["float32", "float64"])
    if kind == "material":
        return dict(kind=kind, n=_log(rng, 1000, 1500000), model=rng.choice(MODELS), dtype=dtype)
    if kind == "step":
        n = _log(rng, 27, 1000000)
        return dict(kind=kind, n=n, edge=_edge_for(rng, n, lo=8), model=rng.choice(MODELS), dtype=dtype,
                    advect=rng.random() < 0.7)
    if kind == "gradient":
        n = _log(rng, 500, 60000)
        steps = rng.randrange(4, 40)
        # mean squared distances in FP64 only: one small number, badly conditioned in FP32
        loss = "mse" if dtype == "float64" and rng.random() < 0.5 else "detF"
        return dict(kind=kind, n=n, edge=_edge_for(rng, n), model=rng.choice(["nh", "hencky"]), dtype=dtype,
                    steps=steps, ckpt=rng.choice([0, 0, max(1, math.isqrt(steps))]), loss=loss,
                    per_particle=rng.random() < 0.5, advect=loss == "mse" or rng.random() < 0.6)
    single = rng.random() < 0.6
    scenes = 1 if single else _log(rng, 2, 160)
    n_hi = _log(rng, 2048, 1000000) if single else 65536
    n_lo = n_hi if single else 2048
    total = n_hi if single else scenes * (n_hi - n_lo) / math.log(n_hi / n_lo)
    steps = max(4, min(40, int((2.0e7 if dtype == "float32" else 1.2e7) / total)))
    steps = max(4, steps - rng.randrange(0, 1 + steps // 3))
    edge = _edge_for(rng, n_hi, lo=32) if single else 64
    models = rng.choice(["nh", "hencky", "hb", "nh+hencky"]) if not single else rng.choice(MODELS)
    loss = "mse" if dtype == "float64" and rng.random() < 0.4 else "detF"
    return dict(kind=kind, scenes=scenes, n_lo=n_lo, n_hi=n_hi, edge_lo=edge if single else 32, edge_hi=edge,
                models=models, dtype=dtype, steps=steps, ckpt=rng.choice([0, max(1, math.isqrt(steps))]), loss=loss,
                ramp=rng.choice([0, 200]), dt=rng.choice([5e-6, 1e-5]), aspect=1,
                field=rng.choice(["none", "radial"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt * 7919 + 17) % (1 << 62))
    return g


def _positions(gen, n, lo, cells, dx):
    """n particles jittered in the 2x2x2 sub-cells of a box of cells, in cell order."""
    k = torch.arange(n, device=DEV)
    sub, c = k % 8, k // 8
    ci = torch.stack([c // (cells[1] * cells[2]), (c // cells[2]) % cells[1], c % cells[2]], 1) + \
        torch.tensor(lo, device=DEV)
    s = torch.stack([sub // 4, (sub // 2) % 2, sub % 2], 1)
    u = torch.rand(n, 3, generator=gen, device=DEV, dtype=torch.float64)
    return (2 * ci + s + u) * (dx / 2.0)


def _box(n, shape, aspect):
    """Cells of a box for n particles at 8 per cell, and its low corner: a
    cube (aspect 1), a strip `aspect` times as long in x, or a sheet with
    -aspect times the thickness as its sides."""
    m = n / 8.0
    if aspect == 1:
        c = [math.ceil(m ** (1.0 / 3.0) - 1e-9)] * 3
    elif aspect > 1:
        w = math.ceil((m / aspect) ** (1.0 / 3.0) - 1e-9)
        c = [math.ceil(m / (w * w)), w, w]
    else:
        t = math.ceil((m / (aspect * aspect)) ** (1.0 / 3.0) - 1e-9)
        side = math.ceil(math.sqrt(m / t) - 1e-9)
        c = [side, side, t]
    return c, [(s - k) // 2 for s, k in zip(shape, c)]


def _motion(gen, x, speed):
    """Velocity, affine velocity and deformation gradient of a cloud in
    motion: smooth fields of position and a little noise."""
    n = x.shape[0]
    mid = x.mean(0)
    size = (x.max(0).values - x.min(0).values).max().clamp_min(1e-9)
    y = (x - mid) / size
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.float64)
    v = speed * (y @ (torch.eye(3, device=DEV, dtype=torch.float64) + 0.3 * rnd(3, 3)).t()) + 0.05 * speed * rnd(n, 3)
    ph = y @ (4.0 * rnd(3, 9)) + 6.28 * torch.rand(9, generator=gen, device=DEV, dtype=torch.float64)
    wave = torch.sin(ph).reshape(n, 3, 3)
    eye = torch.eye(3, device=DEV, dtype=torch.float64)
    F = eye + 0.03 * wave + 0.004 * rnd(n, 3, 3)
    C = (speed / size) * (0.5 * torch.cos(ph).reshape(n, 3, 3) + 0.1 * rnd(n, 3, 3))
    return v, C, F


def _lame(E, nu):
    return E / (2.0 * (1.0 + nu)), E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))


def _single(case, seed):
    """Inputs of the single-scene cases, float64 values already rounded to the
    case's type."""
    gen = _gen(seed)
    n, edge = case["n"], case["edge"]
    dx = 0.1 if edge == 8 else 1.0 / edge
    cells, lo = _box(n, (edge,) * 3, 1)
    x = _positions(gen, n, lo, cells, dx)
    E, nu = 1.0e3, 0.3
    mu, lam = _lame(E, nu)
    d = dict(n=n, shape=(edge,) * 3, dx=dx, dt=1e-5, damping=0.05, density=1.0, sp=dx / 2, mu=mu, lam=lam, E=E, nu=nu)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.float64)
    eye = torch.eye(3, device=DEV, dtype=torch.float64).expand(n, 3, 3)
    if case["kind"] == "step":
        v, C, F = _motion(gen, x, 2.0)
        d["state"] = [x, v, C, F, 1.1 * eye + 0.01 * rnd(n, 3, 3)]
        d["bars"] = [rnd(n, 3), rnd(n, 3), 0.1 * rnd(n, 3, 3), rnd(n, 3, 3), rnd(n, 3, 3)]
    else:
        d["x0"] = x
        g = 1.02 + 0.08 * float(torch.rand((), generator=gen, device=DEV))
        d["growth"] = (g * eye + 0.02 * rnd(n, 3, 3)) if case["per_particle"] else torch.tensor(
            g, device=DEV, dtype=torch.float64)
        d["x_obs"] = x.mean(0) + 1.01 * (x - x.mean(0)) + 1e-3 * dx * rnd(n, 3)
    dt = DTYPES[case["dtype"]]
    for k in ("x0", "growth", "x_obs"):
        if k in d:
            d[k] = d[k].to(dt).contiguous()
    for k in ("state", "bars"):
        if k in d:
            d[k] = [a.to(dt).contiguous() for a in d[k]]
    if "bars" in d:
        d["bars"][4] = d["bars"][4].double()     # the growth cotangent is float64 throughout
    return d


def _material(case, seed):
    gen = _gen(seed)
    n, dt = case["n"], DTYPES[case["dtype"]]
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.float64)
    eye = torch.eye(3, device=DEV, dtype=torch.float64).expand(n, 3, 3)
    return [a.to(dt).contiguous() for a in (eye + 0.08 * rnd(n, 3, 3), 1.1 * eye + 0.02 * rnd(n, 3, 3),
                                            2.0 * rnd(n, 3, 3), rnd(n, 3, 3))]


def _model_obj(name, E=1.0e3, nu=0.3):
    from morphompm_b200 import constitutive as K
    from morphompm_b200.config import Material
    if name == "hb":
        return K.HerschelBulkley(**HB)
    return {"nh": K.NeoHookean, "hencky": K.Hencky}[name](Material(E=E, nu=nu, density=1.0))


def _batch_sizes(case):
    """Particles and grid edge of each scene: spread over the ranges, the same for every seed."""
    S = case["scenes"]
    ns, edges = [], []
    for s in range(S):
        q = ((s + 0.5) * 0.6180339887498949) % 1.0 if S > 1 else 0.0
        r = ((s + 0.5) * 0.7548776662466927) % 1.0 if S > 1 else 0.0
        n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** q))
        e = case["edge_lo"] + int(r * (case["edge_hi"] - case["edge_lo"] + 1))
        ns.append(n)
        edges.append(max(e, math.ceil((n / 8.0) ** (1 / 3)) + 6) if case["aspect"] == 1 else e)
    return ns, edges


def _batch(case, seed):
    """Scenes, the (24, n) state to load and the observation, in the caller's order."""
    gen = _gen(seed)
    ns, edges = _batch_sizes(case)
    host = np.random.default_rng(int(seed) % (1 << 31))
    names = case["models"].split("+")
    dt = DTYPES[case["dtype"]]
    scenes, slabs, obs = [], [], []
    for s, (n, edge) in enumerate(zip(ns, edges)):
        dx = 1.0 / edge
        shape = (3 * edge, edge, edge) if case["aspect"] > 1 else (edge,) * 3
        cells, lo = _box(n, shape, case["aspect"])
        x = _positions(gen, n, lo, cells, dx)
        v, C, F = _motion(gen, x, 3.0)
        E, nu = float(host.uniform(5e2, 5e3)), float(host.uniform(0.2, 0.45))
        g = float(host.uniform(1.02, 1.3))
        mu, lam = _lame(E, nu)
        xh = x.cpu().numpy()
        phi = None
        if case["field"] == "radial":
            c = xh.mean(0)
            phi = np.exp(-((xh[:, 0] - c[0]) ** 2 + (xh[:, 1] - c[1]) ** 2) / 0.05)
        elif case["field"] == "layer":
            phi = (xh[:, 1] >= xh[:, 1].mean()).astype(np.float64)
        d = dict(name="s%d" % s, x=xh, shape=shape, dx=dx, dt=case["dt"], damping=0.05, density=1.0,
                 model=names[s % len(names)], E=E, nu=nu, mu=mu, lam=lam, growth_A=g - 1.0, ramp_steps=case["ramp"],
                 phi=phi, wall=2, hb=dict(HB))
        if case["aspect"] > 1:
            d.update(wall=0, clamp_lo=(0, 0, 0), clamp_hi=(lo[0] + 2, edge, edge))
        scenes.append(d)
        slabs.append(torch.cat([x.t(), v.t(), C.reshape(n, 9).t(), F.reshape(n, 9).t()], 0))
        m = x.mean(0)
        obs.append(m + 1.01 * (x - m))
    slab = torch.cat(slabs, 1).to(dt).contiguous()
    x_obs = torch.cat(obs, 0).to(dt)
    return scenes, slab, x_obs


# ---------------------------------------------------------------------------
# preparation and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "material":
        return dict(kind=kind, model=_model_obj(case["model"]), arrays=_material(case, seed))
    if kind in ("step", "gradient"):
        from morphompm_b200.config import Material, SimConfig
        d = _single(case, seed)
        cfg = SimConfig(N=case["edge"], dx=d["dx"], dt=d["dt"], damping=d["damping"], sp=d["sp"],
                        material=Material(E=d["E"], nu=d["nu"], density=d["density"]))
        s = dict(kind=kind, model=_model_obj(case["model"], d["E"], d["nu"]), cfg=cfg, case=dict(case))
        if kind == "step":
            from morphompm_b200.state import ParticleState
            s.update(state=ParticleState(*d["state"]), bars=d["bars"])
        else:
            s.update(x0=d["x0"].requires_grad_(True), growth=d["growth"].requires_grad_(True), x_obs=d["x_obs"])
        return s
    from morphompm_b200.batch import Batch
    scenes, slab, x_obs = _batch(case, seed)
    b = Batch(scenes, case["steps"], dtype=DTYPES[case["dtype"]], ckpt_every=case["ckpt"] or None,
              loss=case["loss"], x_obs=x_obs.cpu().numpy() if case["loss"] == "mse" else None,
              slab_host=slab.cpu().numpy())
    b.load(slab)
    b.capture()
    return dict(kind=kind, batch=b, slab=slab)


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.load(state["slab"])
        b.replay()
        return dict(loss=b.loss, dloss_dg=b.dloss_dg, final=b.final_state(), bar0=b.initial_cotangents())
    if kind == "material":
        m, (F, Fg, C, tb) = state["model"], state["arrays"]
        return dict(tau=m.stress(F, Fg, C), bars=m.stress_vjp(F, Fg, C, tb))
    case = state["case"]
    if kind == "step":
        from morphompm_b200 import transfer
        new, cache = transfer.step(state["state"], state["model"], state["cfg"], advect=case["advect"])
        bars = transfer.step_vjp(cache, *state["bars"], advect=case["advect"])
        return dict(state=[new.x, new.v, new.C, new.F, new.Fg], bars=bars)
    from morphompm_b200 import autograd
    L = autograd.rollout_loss(state["x0"], state["growth"], state["model"], state["cfg"], case["steps"],
                              advect=case["advect"], loss=case["loss"],
                              x_obs=state["x_obs"] if case["loss"] == "mse" else None,
                              ckpt_every=case["ckpt"] or None)
    gx, gg = torch.autograd.grad(L, [state["x0"], state["growth"]])
    return dict(loss=L.detach(), x0=gx, growth=gg)


def work(case):
    """Bytes: each input once and each output once, and over a trajectory what
    one forward and one reverse step must move per particle (the state read
    and written; state, new C and cotangents read, cotangents written), with
    about 0.2 nodes per particle.  Operations: the 27-node stencil sums."""
    w = 4 if case["dtype"] == "float32" else 8
    if case["kind"] == "material":
        return {"bytes": float(case["n"] * w * (3 * 9 + 9 + 4 * 9 + 3 * 9)), "flops": float(case["n"] * 500)}
    if case["kind"] == "step":
        return {"bytes": float(case["n"] * (w * (33 + 33 + 33 + 9 + 24 + 24) + 8 * 18)),
                "flops": float(case["n"] * 27 * 90)}
    if case["kind"] == "gradient":
        n = case["n"]
    else:
        n = sum(_batch_sizes(case)[0])
    return {"bytes": float(n * case["steps"] * w * (57 + 99 + 6.4)), "flops": float(n * case["steps"] * 27 * 90)}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _mat_inv(A):
    a, b, c, d, e, f, g, h, i = (A[:, r, s] for r in range(3) for s in range(3))
    co = torch.stack([e * i - f * h, c * h - b * i, b * f - c * e, f * g - d * i, a * i - c * g, c * d - a * f,
                      d * h - e * g, b * g - a * h, a * e - b * d], 1).reshape(-1, 3, 3)
    return co / _det(A)[:, None, None]


def _det(A):
    return (A[:, 0, 0] * (A[:, 1, 1] * A[:, 2, 2] - A[:, 1, 2] * A[:, 2, 1])
            - A[:, 0, 1] * (A[:, 1, 0] * A[:, 2, 2] - A[:, 1, 2] * A[:, 2, 0])
            + A[:, 0, 2] * (A[:, 1, 0] * A[:, 2, 1] - A[:, 1, 1] * A[:, 2, 0]))


def _eig(S):
    """Eigenvalues (n, 3) and eigenvectors (columns, (n, 3, 3)) of symmetric
    3x3 matrices by Jacobi rotations."""
    A = [[S[:, i, j].clone() for j in range(3)] for i in range(3)]
    V = [[torch.full_like(S[:, 0, 0], 1.0 if i == j else 0.0) for j in range(3)] for i in range(3)]
    for _ in range(9):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = A[p][q]
            z = apq == 0
            th = (A[q][q] - A[p][p]) / (2.0 * torch.where(z, torch.ones_like(apq), apq))
            sg = torch.where(th < 0, -torch.ones_like(th), torch.ones_like(th))
            t = torch.where(z, torch.zeros_like(th), sg / (th.abs() + torch.sqrt(th * th + 1.0)))
            c = 1.0 / torch.sqrt(t * t + 1.0)
            s = t * c
            A[p][p], A[q][q] = A[p][p] - t * apq, A[q][q] + t * apq
            A[p][q] = A[q][p] = torch.zeros_like(apq)
            r = 3 - p - q
            arp, arq = A[r][p], A[r][q]
            A[r][p] = A[p][r] = c * arp - s * arq
            A[r][q] = A[q][r] = s * arp + c * arq
            for k in range(3):
                vp, vq = V[k][p], V[k][q]
                V[k][p], V[k][q] = c * vp - s * vq, s * vp + c * vq
    return (torch.stack([A[0][0], A[1][1], A[2][2]], 1),
            torch.stack([torch.stack(row, 1) for row in V], 1))


class _LogSym(torch.autograd.Function):
    """Logarithm of symmetric positive 3x3 matrices; its derivative by divided
    differences of the eigenvalues."""

    @staticmethod
    def forward(ctx, b):
        lam, V = _eig(b)
        ctx.save_for_backward(lam, V)
        return (V * torch.log(lam)[:, None, :]) @ V.transpose(1, 2)

    @staticmethod
    def backward(ctx, G):
        lam, V = ctx.saved_tensors
        bi, bj = lam[:, :, None], lam[:, None, :]
        d = (bi - bj) / bj
        L = torch.where(d == 0, 1.0 / bj, torch.log1p(d) / torch.where(d == 0, torch.ones_like(d), bj * d))
        G = 0.5 * (G + G.transpose(1, 2))
        return V @ ((V.transpose(1, 2) @ G @ V) * L) @ V.transpose(1, 2)


def _stress(kind, F, Fg, C, mu, lam):
    """Kirchhoff stress; kind: a model's name, or one index into MODELS per particle."""
    eye = torch.eye(3, device=F.device, dtype=F.dtype)
    if not isinstance(kind, str):
        tau = torch.zeros_like(F)
        for k, name in enumerate(MODELS):
            at = torch.nonzero(kind == k).reshape(-1)
            if at.numel():
                tau = tau.index_add(0, at, _stress(name, F[at], Fg[at], C[at], mu[at], lam[at]))
        return tau
    if kind == "hb":
        D = 0.5 * (C + C.transpose(1, 2))
        gd = torch.sqrt(2.0 * (D * D).sum((1, 2)) + HB["eps"] ** 2)
        eta = HB["K"] * gd ** (HB["n"] - 1.0) + HB["tau_y"] * (1.0 - torch.exp(-HB["m"] * gd)) / gd
        return HB["kappa"] * torch.log(_det(F) / _det(Fg))[:, None, None] * eye + 2.0 * eta[:, None, None] * D
    Fe = F @ _mat_inv(Fg)
    lnJ = torch.log(_det(Fe))[:, None, None]
    b = Fe @ Fe.transpose(1, 2)
    if kind == "nh":
        return mu.reshape(-1, 1, 1) * (b - eye) + lam.reshape(-1, 1, 1) * lnJ * eye
    return mu.reshape(-1, 1, 1) * _LogSym.apply(b) + lam.reshape(-1, 1, 1) * lnJ * eye


def _step(P, x, v, C, F, Fg, advect):
    """One growth step in float64.  P: per-particle scene constants and the
    grid (node offsets, free nodes)."""
    n = x.shape[0]
    dx, idx_, k4 = P["dx"][:, None], 1.0 / P["dx"][:, None], 4.0 / P["dx"] ** 2
    X = (x if advect else x.detach()) * idx_
    base = torch.floor(X.detach() - 0.5)
    fx = X - base
    w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2], 1)   # (n, 3, 3)
    w27 = (w[:, :, None, None, 0] * w[:, None, :, None, 1] * w[:, None, None, :, 2]).reshape(n, 27)
    o = torch.stack(torch.meshgrid(*[torch.arange(3, device=x.device)] * 3, indexing="ij"), -1).reshape(27, 3)
    dp = (o.to(x.dtype)[None] - fx[:, None, :]) * dx[:, None, :]
    node = base.long()[:, None, :] + o[None]
    shape = P["shape"][:, None, :]
    ok = ((node >= 0) & (node < shape)).all(2)
    at = P["node0"][:, None] + (node[..., 0] * shape[..., 1] + node[..., 1]) * shape[..., 2] + node[..., 2]
    at = torch.where(ok, at, torch.full_like(at, P["nodes"])).reshape(-1)
    tau = _stress(P["kind"], F, Fg, C, P["mu"], P["lam"])
    pm, vol = P["pmass"], P["pmass"] / P["density"]
    sk = (-k4 * vol * _det(Fg))[:, None, None] * tau
    A = pm[:, None, None] * C + P["dt"][:, None, None] * sk
    q = w27[..., None] * ((pm[:, None] * v)[:, None, :] + dp @ A.transpose(1, 2))
    zero = torch.zeros(P["nodes"] + 1, device=x.device, dtype=x.dtype)
    m = zero.index_add(0, at, (w27 * pm[:, None]).reshape(-1))
    mom = zero[:, None].expand(-1, 3).clone().index_add(0, at, q.reshape(-1, 3))
    act = (m.detach() > 1e-12) & P["free"]
    gv = torch.where(act[:, None], (1.0 - P["damping"]) * mom / torch.where(act, m, torch.ones_like(m))[:, None],
                     torch.zeros_like(mom))
    vi = gv[at].reshape(n, 27, 3) * w27[..., None]
    nv = vi.sum(1)
    nC = k4[:, None, None] * (vi.transpose(1, 2) @ dp)
    xn = x + P["dt"][:, None] * nv if advect else x.clone()
    Fn = F + P["dt"][:, None, None] * (nC @ F)
    return xn, nv, nC, Fn


def _grid(scenes):
    """Per-particle constants and the node table of scenes (dicts with n,
    shape, dx, dt, density, mu, lam, model, wall, clamp)."""
    rep = lambda f, dt=torch.float64: torch.repeat_interleave(
        torch.tensor([f(s) for s in scenes], device=DEV, dtype=dt), torch.tensor([s["n"] for s in scenes], device=DEV), 0)
    node0, total, free = [], 0, []
    for s in scenes:
        node0.append(total)
        total += int(np.prod(s["shape"]))
        k = torch.ones(tuple(s["shape"]), dtype=torch.bool, device=DEV)
        wall = s.get("wall", 0)
        if wall:
            k[:] = False
            k[wall:-wall, wall:-wall, wall:-wall] = True
        if s.get("clamp_hi"):
            (a, b, c), (d, e, f) = s["clamp_lo"], s["clamp_hi"]
            k[a:d, b:e, c:f] = False
        free.append(k.reshape(-1))
    for s, z in zip(scenes, node0):
        s["node0"] = z
    kinds = {s["model"] for s in scenes}
    return dict(dx=rep(lambda s: s["dx"]), dt=rep(lambda s: s["dt"]), pmass=rep(lambda s: s["density"] * (s["dx"] / 2) ** 3),
                density=rep(lambda s: s["density"]), mu=rep(lambda s: s["mu"]), lam=rep(lambda s: s["lam"]),
                kind=kinds.pop() if len(kinds) == 1 else rep(lambda s: MODELS.index(s["model"]), torch.long),
                shape=rep(lambda s: list(s["shape"]), torch.long), node0=rep(lambda s: s["node0"], torch.long),
                nodes=total, free=torch.cat(free + [torch.zeros(1, dtype=torch.bool, device=DEV)]), damping=0.05)


def _trajectory(P, state, growth, Fg_of, steps, advect, seed_of):
    """Forward, loss and the reverse sweep: returns the final state, the loss,
    the cotangents of the initial state and the gradient of `growth`."""
    states = [state]
    with torch.no_grad():
        for t in range(steps):
            states.append(_step(P, *states[-1], Fg_of(growth, t), advect))
    fin = [a.clone().requires_grad_(True) for a in states[-1]]
    loss = seed_of(fin)
    bars = [b if b is not None else torch.zeros_like(a)
            for a, b in zip(fin, torch.autograd.grad(loss.sum(), fin, allow_unused=True))]
    gg = torch.zeros_like(growth)
    for t in reversed(range(steps)):
        ins = [a.clone().requires_grad_(True) for a in states[t]]
        g = growth.clone().requires_grad_(True)
        out = _step(P, *ins, Fg_of(g, t), advect)
        got = torch.autograd.grad(out, ins + [g], bars, allow_unused=True)
        bars = [b if b is not None else torch.zeros_like(a) for a, b in zip(ins, got[:4])]
        if not advect:
            bars[0] = torch.zeros_like(bars[0])
        gg = gg + got[4]
    return states[-1], loss.detach(), bars, gg


def exact(case, seed):
    kind = case["kind"]
    if kind == "material":
        F, Fg, C, tb = (a.double() for a in _material(case, seed))
        mu, lam = _lame(1.0e3, 0.3)
        ins = [a.clone().requires_grad_(True) for a in (F, Fg, C)]
        one = torch.ones(F.shape[0], device=DEV, dtype=torch.float64)
        tau = _stress(case["model"], *ins, mu * one, lam * one)
        got = torch.autograd.grad(tau, ins, 0.5 * (tb + tb.transpose(1, 2)), allow_unused=True)
        return dict(tau=tau.detach(), bars=[g if g is not None else torch.zeros_like(F) for g in got])
    if kind in ("step", "gradient"):
        d = _single(case, seed)
        P = _grid([dict(n=case["n"], shape=d["shape"], dx=d["dx"], dt=d["dt"], density=d["density"], mu=d["mu"],
                        lam=d["lam"], model=case["model"])])
        advect = case["advect"]
        if kind == "step":
            ins = [a.double().clone().requires_grad_(True) for a in d["state"]]
            out = _step(P, *ins, advect)
            b = [a.double() for a in d["bars"]]
            got = list(torch.autograd.grad(out, ins, b[:4], allow_unused=True))
            got = [g if g is not None else torch.zeros_like(a) for g, a in zip(got, ins)]
            if not advect:
                got[0] = torch.zeros_like(got[0])
            got[4] = got[4] + b[4]
            return dict(state=[a.detach() for a in out] + [ins[4].detach()], bars=got)
        x0, growth = d["x0"].detach().double(), d["growth"].detach().double()
        n = case["n"]
        eye = torch.eye(3, device=DEV, dtype=torch.float64).expand(n, 3, 3)
        rest = [x0, torch.zeros_like(x0), torch.zeros_like(eye), eye.clone()]
        Fg_of = (lambda g, t: g) if case["per_particle"] else (lambda g, t: g * eye)
        xo = d["x_obs"].double()
        seed_of = (lambda s: _det(s[3]).sum()) if case["loss"] == "detF" else (lambda s: ((s[0] - xo) ** 2).sum() / n)
        _, L, bars, gg = _trajectory(P, rest, growth, Fg_of, case["steps"], advect, seed_of)
        return dict(loss=L, x0=bars[0], growth=gg)
    scenes, slab, x_obs = _batch(case, seed)
    ns = [s["x"].shape[0] for s in scenes]
    for s, n in zip(scenes, ns):
        s["n"] = n
    P = _grid(scenes)
    a = slab.double().t()
    n = a.shape[0]
    if n * case["steps"] > 6.0e7:
        return None
    state = [a[:, 0:3].contiguous(), a[:, 3:6].contiguous(), a[:, 6:15].reshape(n, 3, 3), a[:, 15:24].reshape(n, 3, 3)]
    sid = torch.repeat_interleave(torch.arange(len(ns), device=DEV), torch.tensor(ns, device=DEV))
    phi = torch.cat([torch.as_tensor(s["phi"], device=DEV) if s["phi"] is not None else
                     torch.ones(k, device=DEV, dtype=torch.float64) for s, k in zip(scenes, ns)])
    A = torch.tensor([s["growth_A"] for s in scenes], device=DEV, dtype=torch.float64)
    eye = torch.eye(3, device=DEV, dtype=torch.float64)
    ramp = lambda t: min(1.0, (t + 1) / case["ramp"]) if case["ramp"] > 0 else 1.0
    Fg_of = lambda g, t: (1.0 + g[sid] * ramp(t) * phi)[:, None, None] * eye
    per = lambda val: torch.zeros(len(ns), device=DEV, dtype=torch.float64).index_add(0, sid, val)
    xo = x_obs.double()
    cnt = torch.tensor(ns, device=DEV, dtype=torch.float64)
    seed_of = (lambda s: per(_det(s[3]))) if case["loss"] == "detF" else (lambda s: per(((s[0] - xo) ** 2).sum(1)) / cnt)
    fin, L, bars, gg = _trajectory(P, state, A, Fg_of, case["steps"], True, seed_of)
    flat = lambda s: torch.cat([s[0].t(), s[1].t(), s[2].reshape(n, 9).t(), s[3].reshape(n, 9).t()], 0)
    return dict(loss=L, dloss_dg=gg, final=flat(fin), bar0=flat(bars))
