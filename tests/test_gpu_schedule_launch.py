"""The launch knobs that change a grid or a block on their own: 64-thread
particle blocks and four times the node-gather blocks give bitwise the default
schedule's results, as the schedules of test_gpu_schedule.py do."""
import numpy as np
import pytest

from test_gpu_schedule import _run

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("tuning", [{"particle_block": 64}, {"scatter_ctas_per_sm": 4}])
def test_launch_knobs_are_bitwise_equal(dtype, tuning):
    from morphompm_b200 import scenes
    scn = scenes.config4(n_scenes=10, n_lo=512, n_hi=8192)
    ref, got = _run(scn, dtype, None), _run(scn, dtype, tuning)
    for a, b in zip(ref[:4], got[:4]):
        assert np.array_equal(a, b)
    assert got[4] == ref[4]
