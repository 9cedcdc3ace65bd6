"""SAD forward: volumes with an odd number of disparity groups, and of more than 256 disparities, up to the 512 that the call
accepts (two launches), against the oracle: bit-exact, whole and fractional
steps, ranges that start below zero, counts around the halves and their groups
of eight."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("C,H,W,lo,hi,step", [
    (5, 3, 300, 0, 255, 1.0), (5, 3, 300, 0, 256, 1.0), (17, 2, 600, 0, 263, 1.0), (3, 3, 130, -40, 260, 1.0),
    (16, 2, 520, 0, 510, 1.0), (4, 2, 530, 0, 511, 1.0), (6, 3, 200, 0, 135, 0.5), (6, 2, 90, -3, 252, 0.5)])
def test_more_than_256_disparities(C, H, W, lo, hi, step):
    from bpl_gb300 import ops
    g = np.random.default_rng(hi - lo)
    f0 = g.normal(size=(2, C, H, W)).astype(np.float32)
    f1 = g.normal(size=(2, C, H, W)).astype(np.float32)
    dev = torch.device("cuda:0")
    vol = ops.sad_forward(torch.from_numpy(f0).to(dev), torch.from_numpy(f1).to(dev), lo, hi, step)
    np.testing.assert_array_equal(vol.cpu().numpy(), oracle.sad_forward(f0, f1, lo, hi, step))


@pytest.mark.parametrize("D", [1, 8, 17, 24, 33, 40, 129, 250])
@pytest.mark.parametrize("step", [1.0, 0.5])
def test_odd_groups_of_disparities(D, step):
    """Blocks whose last warp is half without disparities."""
    from bpl_gb300 import ops
    g = np.random.default_rng(D)
    f0 = g.normal(size=(1, 21, 3, 150)).astype(np.float32)
    f1 = g.normal(size=(1, 21, 3, 150)).astype(np.float32)
    hi = int(D * step) - 1
    dev = torch.device("cuda:0")
    vol = ops.sad_forward(torch.from_numpy(f0).to(dev), torch.from_numpy(f1).to(dev), -1, hi, step)
    np.testing.assert_array_equal(vol.cpu().numpy(), oracle.sad_forward(f0, f1, -1, hi, step))


def test_513_disparities_are_refused():
    from bpl_gb300 import ops
    f = torch.zeros((1, 1, 1, 8), device="cuda:0")
    with pytest.raises(ops.BplError, match="at most 512"):
        ops.sad_forward(f, f, 0, 512)
