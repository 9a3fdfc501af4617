"""The column gather of slabs (mpm_gather_columns) at sizes around a block and
a group of rows, and Batch.load from the forms a slab comes in: host, device,
another stride, the batch's own input.  Copies: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 24])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_gather_columns(rows, n, dtype):
    from morphompm_b200.runtime import gather_columns
    a = torch.randn(rows, n, dtype=dtype, device="cuda")
    order = torch.randperm(n, device="cuda").to(torch.int32)
    out = torch.full_like(a, 7.0)
    assert torch.equal(gather_columns(a, order, out), a[:, order.long()])


def test_gather_columns_refuses_bad_arguments():
    from morphompm_b200 import _lib as L
    lib = L.load()
    a = torch.zeros(2, 4, device="cuda")
    o = torch.zeros(4, dtype=torch.int32, device="cuda")
    b = torch.zeros_like(a)
    p = lambda t: t.data_ptr()
    for args in ((p(a), p(a), p(o), 2, 4, 4), (0, p(b), p(o), 2, 4, 4), (p(a), p(b), p(o), -1, 4, 4),
                 (p(a), p(b), p(o), 2, -1, 4), (p(a), p(b), p(o), 2, 4, 2)):
        assert lib.mpm_gather_columns(*args, None) == L.MPM_ERR_ARG
    assert lib.mpm_gather_columns(p(a), p(b), p(o), 2, 0, 4, None) == L.MPM_OK


@pytest.mark.parametrize("ckpt", [None, 1, 2])
def test_load_forms(ckpt):
    from morphompm_b200 import scenes
    from morphompm_b200.batch import Batch, host_slab
    sc = scenes.config4(seed=3, n_scenes=3, n_lo=300, n_hi=900)
    rng = np.random.default_rng(0)
    for s in sc:
        s["x"] = s["x"][rng.permutation(len(s["x"]))]
    b = Batch(sc, 5, ckpt_every=ckpt)
    assert b.order is not None
    slab = torch.as_tensor(host_slab(sc))
    b.load(slab, non_blocking=False)
    b.run()
    ref = (b.slab0.clone(), b.final_state(), b.initial_cotangents())
    assert torch.equal(ref[0], slab.cuda()[:, torch.as_tensor(b.order).cuda()])
    dev = slab.cuda()
    for src in (dev, dev.double(), dev.t().contiguous().t(), slab.numpy()):
        b.slab0.zero_()
        b.load(src, non_blocking=False)
        b.run()
        for x, y in zip(ref, (b.slab0, b.final_state(), b.initial_cotangents())):
            assert torch.equal(x, y)
    # the batch's own input as the source: permuted once more
    b.load(b.slab0)
    assert torch.equal(b.slab0, ref[0][:, torch.as_tensor(b.order).cuda()])
