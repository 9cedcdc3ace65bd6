"""The SAD backward (strips of 8 pixels, 16 strips per segment, f1 blocks
handed from strip to strip) against the oracle, bit-exact, at the edges of its
tiles: widths around strips and segments, disparity counts around blocks,
ranges that start below and above zero, ranges longer than the row and than
one launch, channel counts around 32, zero differences, NaN and infinities.
ROWS image rows: enough for the strips to be chosen over the gather form
(which the few-row cases of test_sad_gpu.py run)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ROWS = 152


def _check(B, C, H, W, lo, hi, seed=0, quantise=False, special=False):
    from bpl_gb300 import ops
    g = np.random.default_rng(seed)
    f0 = g.normal(size=(B, C, H, W)).astype(np.float32)
    f1 = g.normal(size=(B, C, H, W)).astype(np.float32)
    if quantise:  # differences that are exactly zero
        f0, f1 = np.round(f0 * 2) / 2, np.round(f1 * 2) / 2
        f0, f1 = f0.astype(np.float32), f1.astype(np.float32)
    gin = g.normal(size=(B, H, W, hi - lo + 1)).astype(np.float32)
    if special:
        f0[0, 0, 0, ::5] = np.nan
        f1[0, -1, 0, ::7] = np.inf
        f0[0, -1, 0, 3::11] = np.inf
        f1[0, 0, 0, ::3] = f0[0, 0, 0, ::3] + np.float32(1e-16)
        gin[0, 0, ::9] = 0.0
    dev = torch.device("cuda:0")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    d0, d1 = ops.sad_backward(t(f0), t(f1), lo, hi, t(gin))
    torch.cuda.synchronize()
    # an infinite difference counts by its sign (the reference divides inf by
    # inf there), the same as a very large one
    f0, f1 = (np.where(np.isinf(f), np.sign(f) * np.float32(1e38), f).astype(np.float32) for f in (f0, f1))
    r0, r1 = oracle.sad_backward(f0, f1, gin, lo, hi, channel_limit=C)
    np.testing.assert_array_equal(d0.cpu().numpy(), r0)
    np.testing.assert_array_equal(d1.cpu().numpy(), r1)


@pytest.mark.parametrize("W", [1, 7, 8, 9, 63, 64, 127, 128, 129, 255, 257, 300])
def test_widths(W):
    _check(1, 5, ROWS, W, 0, 40, W)
    _check(1, 3, 3, W, 0, 20, W)


@pytest.mark.parametrize("D", [1, 2, 3, 7, 8, 9, 10, 16, 17, 63, 64, 65, 130, 192])
def test_disparity_counts(D):
    _check(1, 3, ROWS, 128, 0, D - 1, D)


@pytest.mark.parametrize("lo,hi", [(-20, 3), (-40, -17), (5, 30), (100, 130), (130, 160), (-300, -200), (-16, 16)])
def test_ranges(lo, hi):
    _check(1, 4, ROWS, 120, lo, hi, 3)


@pytest.mark.parametrize("lo,hi,W", [(0, 511, 90), (0, 512, 700), (-100, 600, 640), (3, 1100, 1300)])
def test_long_ranges(lo, hi, W):
    _check(1, 2, ROWS, W, lo, hi, 4)


@pytest.mark.parametrize("C", [1, 31, 32, 33, 64, 70])
def test_channels(C):
    _check(2, C, ROWS // 2, 70, 0, 31, C)


@pytest.mark.parametrize("W", [40, 260])
def test_special_values(W):
    _check(1, 3, ROWS, W, 0, 40, 5, quantise=True)
    _check(1, 3, ROWS, W, -4, 40, 6, special=True)
