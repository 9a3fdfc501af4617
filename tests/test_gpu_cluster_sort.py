"""The sorted order, segment table and active-tile list that a forward step
records in its tape, against numpy, at the sizes where the one-launch cluster
sort changes shape (CTAs of the cluster, keys per thread) and just beyond it,
where the general kernels take over.  Integers: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _scene(n, shape, dx):
    from morphompm_b200 import _lib as L
    from morphompm_b200.runtime import SceneSpec
    return SceneSpec(shape=shape, n=n, model=L.MODEL_NEOHOOKEAN, dx=dx, dt=1e-4, damping=0.05, pmass=1e-3, vol0=1e-3,
                     mu=400.0, lam=500.0, growth_mode=1)


def _expected(x, shape, dx):
    """Local keys, and the node tiles (4 x 4 x 4) the inside stencils touch."""
    s = np.array(shape)
    base = np.floor(x * (1.0 / dx) - 0.5).astype(np.int64)
    inside = np.all((base >= -2) & (base < s), axis=1)
    c = base + 2
    key = np.where(inside, (c[:, 0] * (s[1] + 2) + c[:, 1]) * (s[2] + 2) + c[:, 2], np.prod(s + 2))
    nt = (s + 3) // 4
    lo, hi = np.maximum(base[inside], 0) // 4, np.minimum(base[inside] + 2, s - 1) // 4
    tiles = np.unique([(a * nt[1] + b) * nt[2] + d for l, h in np.unique(np.concatenate([lo, hi], 1), axis=0)
                       .reshape(-1, 2, 3) for a in range(l[0], h[0] + 1) for b in range(l[1], h[1] + 1)
                       for d in range(l[2], h[2] + 1)]).astype(np.int64)
    return key, int(np.prod(s + 2)), tiles, int(np.prod(nt))


@pytest.mark.parametrize("scenes", [
    [(1, 8)], [(33, 8)], [(1024, 8)], [(1025, 16)], [(4097, 32)], [(8193, 40)], [(16385, 24)], [(32769, 64)],
    [(65536, 128)], [(65537, 32)],
    [(700, 10), (0, 8), (1, 9), (9000, 33)],
])
@pytest.mark.parametrize("spread", ["inside", "one_cell", "leaving"])
def test_sorted_order_segments_and_tiles(scenes, spread):
    from morphompm_b200.runtime import Plan, slab_particles
    rng = np.random.default_rng(len(scenes) + sum(n for n, _ in scenes))
    xs, specs = [], []
    for n, edge in scenes:
        shape, dx = (edge, edge + 1, edge), 1.0 / edge
        if spread == "one_cell":
            x = (edge // 2 + 0.6 + 0.1 * rng.random((n, 3))) * dx
        else:
            lo, hi = (0.1, 0.9) if spread == "inside" else (-0.3, 1.3)
            x = rng.uniform(lo, hi, size=(n, 3))
        xs.append(x)
        specs.append(_scene(n, shape, dx))
    plan = Plan(specs, dtype=torch.float64)
    n = plan.n
    slab = np.zeros((24, n))
    slab[0:3] = np.concatenate(xs).T
    for i in range(3):
        slab[15 + 4 * i] = 1.0
    a = torch.as_tensor(slab).cuda()
    b = torch.empty_like(a)
    tape = plan.new_tape()
    plan.step_fwd(slab_particles(a), slab_particles(b), True, 0, tape)
    torch.cuda.synchronize()

    _check_tape(tape, n, xs, specs)


@pytest.mark.parametrize("scenes", [[(33, 8)], [(1024, 16)], [(4097, 32)], [(32769, 40)], [(65536, 64)],
                                    [(700, 10), (0, 8), (1, 9), (9000, 33)]])
@pytest.mark.parametrize("speed", [0.0, 0.0005, 0.008, 0.02, 0.5])
def test_chained_order(scenes, speed):
    """The order of chained steps, built from the previous step's order and the
    particles that changed cell: none, a few, around the merge's capacity of
    1024, and most of them (the passes)."""
    from morphompm_b200.runtime import Plan, ROW_V, slab_particles
    rng = np.random.default_rng(7)
    specs, x0 = [], []
    for n, edge in scenes:
        dx = 1.0 / edge
        specs.append(_scene(n, (edge, edge + 1, edge), dx))
        x0.append(rng.uniform(0.05, 0.95, size=(n, 3)))
    plan = Plan(specs, dtype=torch.float64)
    n = plan.n
    slab = np.zeros((24, n))
    slab[0:3] = np.concatenate(x0).T
    for i in range(3):
        slab[15 + 4 * i] = 1.0
    p = 0
    for (k, edge), sp in zip(scenes, specs):
        slab[ROW_V:ROW_V + 3, p:p + k] = rng.standard_normal((3, k)) * speed * sp.dx / sp.dt
        p += k
    a = torch.as_tensor(slab).cuda()
    b = torch.empty_like(a)
    tapes = [plan.new_tape() for _ in range(2)]
    for t in range(4):
        same = t == 3            # the last step overwrites the order it starts from
        tape = tapes[(t - 1 if same else t) % 2]
        x = a[0:3].cpu().numpy()
        plan.step_fwd(slab_particles(a), slab_particles(b), True, t, tape, chained=t > 0, emit=t < 3)
        torch.cuda.synchronize()
        off = np.concatenate([[0], np.cumsum([k for k, _ in scenes])])
        _check_tape(tape, n, [x[:, u:v].T for u, v in zip(off[:-1], off[1:])], specs)
        a, b = b, a


def _check_tape(tape, n, xs, specs):
    raw = tape.buf.cpu().numpy()[tape.ptr - tape.buf.data_ptr():]
    pad = lambda v: (v + 255) // 256 * 256
    at = lambda off, k: raw[off:off + 4 * k].view(np.int32).astype(np.int64)
    keys, cell0, tile0, tiles, outside = [], 0, 0, [], []
    for x, sp in zip(xs, specs):
        k, nc, t, nt = _expected(x, sp.shape, sp.dx)
        keys.append(k + cell0)
        outside.append(np.full(len(k), nc + cell0))
        tiles.append(t + tile0)
        cell0 += nc + 1
        tile0 += nt
    keys, tiles, outside = np.concatenate(keys), np.concatenate(tiles), np.concatenate(outside)
    order = np.argsort(keys, kind="stable")
    sk = keys[order]
    o = pad(4 * n)
    assert np.array_equal(at(0, n), sk)
    assert np.array_equal(at(o, n), order)
    start = np.flatnonzero((np.r_[True, sk[1:] != sk[:-1]]) & (sk < outside[order]))
    end = np.flatnonzero((np.r_[sk[1:] != sk[:-1], True]) & (sk < outside[order])) + 1
    nseg = int(at(4 * o, 1)[0])
    assert nseg == len(start)
    assert np.array_equal(at(2 * o, nseg), start) and np.array_equal(at(3 * o, nseg), end)
    nact = int(at(4 * o + 256 + pad(4 * tile0), 1)[0])
    assert nact == len(tiles)
    assert np.array_equal(at(4 * o + 256, nact), np.sort(tiles))
