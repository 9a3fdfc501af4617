"""Workload of tests/test_gpu_general_path.py: batches and chained steps on
their own grid (OWN) and on one padded until its plan takes the general sort,
segment and tile kernels (PADDED).  Run as a program with MORPHOMPM_CHECKED=1
it is the bounds-checked build's pass over those kernels:

    python tests/general_path_workload.py OUT.npz     (also writes the violation count)
"""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
for p in (os.path.dirname(HERE), HERE):
    if p not in sys.path:
        sys.path.insert(0, p)

OWN, PADDED = 24, 176
DX = 1.0 / OWN


def _scenes(edge):
    """One scene of each material, on `edge`^3 nodes; the first touches the
    grid's lower faces (there alone both grids end), one is empty and one a
    single particle."""
    rng = np.random.default_rng(17)
    hb = dict(kappa=1e4, K=1.0, n=0.5, tau_y=10.0, m=100.0, eps=1e-4)
    out = []
    for i, (n, model) in enumerate(((900, "nh"), (1700, "hencky"), (0, "nh"), (1, "hencky"), (2600, "hb"))):
        x = rng.uniform(0.0 if i == 0 else 5.0, 14.0, size=(n, 3)) * DX
        e = edge if i == 4 else OWN        # one scene with many tiles is enough
        out.append(dict(x=x, shape=(e,) * 3, dx=DX, dt=2e-5, model=model, mu=400.0, lam=500.0, growth_A=0.1 + 0.02 * i,
                        ramp_steps=0, wall=0, hb=hb))
    return out


def trajectory(dtype, ckpt, edge):
    import torch
    from morphompm_b200.batch import Batch, host_slab
    sc = _scenes(edge)
    npd = np.dtype(dtype)
    b = Batch(sc, 7, dtype=getattr(torch, dtype), ckpt_every=ckpt, material_grads=True)
    slab = host_slab(sc, npd)
    slab[3:6] = np.random.default_rng(4).standard_normal((3, b.n)) * 0.05 * DX / 2e-5     # some cells change each step
    b.load(slab, non_blocking=False)
    b.run()
    torch.cuda.synchronize()
    assert b.plan.status() & ~8 == 0       # particles leaving the grid only warn
    return {k: v.cpu().numpy() for k, v in (("loss", b.loss), ("dg", b.dloss_dg), ("dm", b.dloss_dmaterial),
                                            ("final", b.final_state()), ("bar0", b.initial_cotangents()))}


def steps(dtype, speed, edge, chain):
    """The state after five forward steps with velocities of `speed` cells per step."""
    import torch
    from morphompm_b200.batch import host_slab, scene_spec_from_dict
    from morphompm_b200.runtime import Plan, slab_particles
    sc = sorted(_scenes(edge), key=lambda s: s["model"])
    plan = Plan([scene_spec_from_dict(s) for s in sc], dtype=getattr(torch, dtype), device="cuda")
    slab = host_slab(sc, np.dtype(dtype))
    slab[3:6] = np.random.default_rng(6).standard_normal((3, plan.n)) * speed * DX / 2e-5
    a = torch.as_tensor(slab).cuda()
    b = torch.empty_like(a)
    tapes = [plan.new_tape() for _ in range(2)]
    for t in range(5):
        tape = tapes[(t - 1 if t == 4 else t) % 2]      # the last step overwrites the order it starts from
        plan.step_fwd(slab_particles(a), slab_particles(b), True, t, tape, chained=chain and t > 0,
                      emit=chain and t < 4)
        a, b = b, a
    torch.cuda.synchronize()
    return a


def run() -> dict:
    out = {}
    for dtype in ("float32", "float64"):
        for k, v in trajectory(dtype, 3, PADDED).items():
            out[f"{dtype}_{k}"] = v
        for speed in (0.01, 0.4):
            out[f"{dtype}_steps_{speed}"] = steps(dtype, speed, PADDED, True).cpu().numpy()
    return out


if __name__ == "__main__":
    from checked_workload import violations
    res = run()
    res["violations"] = np.array(violations())
    np.savez(sys.argv[1], **res)
