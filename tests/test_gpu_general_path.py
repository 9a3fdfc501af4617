"""The general sort, segment, tile and re-sort kernels on small inputs.  A plan
of more than 65536 node tiles takes them whatever its particle count, so the
same particles on a grid that is only padded with empty nodes (176^3: 85184
tiles) run them, and on their own grid the one-launch cluster sort.  Positions,
spacing and the order of the cells are the same in both, hence every sum has
the same terms in the same order: results must agree bitwise."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import general_path_workload as W


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("ckpt", [None, 3, 1])
def test_padded_grid_gives_the_same_trajectory(dtype, ckpt):
    """Steps stored, checkpointed (two tapes in turn, segments recomputed) and
    checkpointed at every step."""
    ref = W.trajectory(dtype, ckpt, W.OWN)
    got = W.trajectory(dtype, ckpt, W.PADDED)
    assert set(ref) == set(got)
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("speed", [0.0, 0.01, 0.4])
def test_padded_grid_chained_steps(dtype, speed):
    """Independent steps, and chained ones (the incremental re-sort, from
    another tape and in place)."""
    for chain in (False, True):
        assert torch.equal(W.steps(dtype, speed, W.OWN, chain), W.steps(dtype, speed, W.PADDED, chain)), chain


def test_checked_build_on_the_general_path(tmp_path):
    """The bounds-checked build over these kernels: no index out of range, and
    bitwise the results of the release build."""
    from morphompm_b200 import build as B
    B.build(checked=True)
    out = tmp_path / "checked.npz"
    r = subprocess.run([sys.executable, os.path.abspath(W.__file__), str(out)],
                       env=dict(os.environ, MORPHOMPM_CHECKED="1"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    got = dict(np.load(out))
    rc, cnt, site, idx = (int(v) for v in got.pop("violations"))
    assert rc == 0, "the child did not load the checked library"
    assert cnt == 0, f"{cnt} out-of-range indices, first at site {site} index {idx}"
    ref = W.run()
    assert set(ref) == set(got)
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k
