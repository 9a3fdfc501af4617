"""The batched stress and VJP at particle counts around a warp and a block, on
inputs that start off a 16-byte boundary, against the oracle in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from oracle import mpm_oracle as O


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 1000])
@pytest.mark.parametrize("name", ["nh", "hencky", "hb"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_stress_and_vjp_sizes(n, name, dtype):
    from morphompm_b200 import constitutive as K
    from morphompm_b200.config import Material
    mat = Material(E=1e3, nu=0.3)
    m = {"nh": K.NeoHookean, "hencky": K.Hencky}[name](mat) if name != "hb" else K.HerschelBulkley()
    om = O.Model.elastic(name, 1e3, 0.3) if name != "hb" else O.Model(kind="hb")
    rng = np.random.default_rng(n)
    dt = getattr(torch, dtype)
    arrs = [np.eye(3) + 0.1 * rng.standard_normal((n, 3, 3)), 1.1 * np.eye(3) + 0.02 * rng.standard_normal((n, 3, 3)),
            rng.standard_normal((n, 3, 3)), rng.standard_normal((n, 3, 3))]
    dev = []
    for a in arrs:
        buf = torch.zeros(9 * n + 1, dtype=dt, device="cuda")
        buf[1:] = torch.as_tensor(a.reshape(-1), dtype=dt)
        dev.append(buf[1:].view(n, 3, 3))
    F, Fg, C, tb = (a.double().cpu().numpy() for a in dev)
    tau = m.stress(*dev[:3])
    bars = m.stress_vjp(*dev)
    # 200 operations' rounding (FP64 Hencky VJP: the 1e-9 divided-difference switch)
    tol = 200 * (1.2e-7 if dtype == "float32" else 2.3e-16)
    if name == "hencky" and dtype == "float64":
        tol = 1e-8
    for got, ref in zip((tau, *bars), (O.stress(om, F, Fg, C), *O.stress_vjp(om, F, Fg, C, tb))):
        assert got.shape == (n, 3, 3)
        assert np.max(np.abs(got.double().cpu().numpy() - ref)) <= tol * max(1.0, np.max(np.abs(ref)))
