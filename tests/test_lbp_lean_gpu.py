"""The FP32 stereo forward's hot loop (one straight-line block per step) against
the oracle where it can go wrong: label counts around the warp's slots, tap
blocks of 32 steps and their remainders, every window form it takes and the
ones it has to leave (ties, several labels below the candidate, zero, negative
and infinite weights), every argmin storage, both launch shapes.  Forward
parity is bitwise up to the host's exp/log (test_lbp_forward_gpu.py states it)."""
import numpy as np
import pytest

import cases
import oracle
from test_lbp_forward_gpu import assert_parity

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run(cost, jump, edge, msgs, delta, iters, dtype=torch.uint8):
    from bpl_gb300 import ops
    dev = torch.device("cuda:0")
    c, j, e, m = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (cost, jump, edge, msgs))
    for _ in range(iters):
        m, am, sc = ops.lbp_forward(0, c, j, e, m, delta, argmin_dtype=dtype)
    torch.cuda.synchronize()
    return m.cpu().numpy(), None if am is None else am.cpu().numpy().astype(np.float32), sc.cpu().numpy()


def _check(cost, jump, edge, msgs, delta, iters, dtype=torch.uint8):
    gpu = _run(cost, jump, edge, msgs, delta, iters, dtype)
    ref = oracle.lbp_forward(0, cost, jump, edge, msgs, delta, iters=iters)
    assert_parity((gpu[0], ref[1] if gpu[1] is None else gpu[1], gpu[2]), ref)


def _inputs(seed, B, H, W, L, taps="scalar", flat=False):
    g = cases.rng(seed)
    cost = cases.random_cost(g, B, H, W, L)
    if flat:  # most labels below the candidate
        cost = (cost * 0.01).astype(np.float32)
    jump = cases.stereo_taps(1, H, W, 0.1, 0.5) if taps == "scalar" else cases.random_taps8(g, 1, H, W)
    return cost, jump, cases.edge_weights(g, B, H, W), np.zeros((B, 4, H, W, L), np.float32)


@pytest.mark.parametrize("L", [1, 2, 16, 31, 32, 33, 48, 64, 65, 96, 112, 128, 129, 160, 192, 200, 224, 256])
@pytest.mark.parametrize("taps", ["scalar", "taps8"])
def test_label_counts(L, taps):
    _check(*_inputs(100 + L, 1, 6, 35, L, taps), 3, 2)


@pytest.mark.parametrize("W", [2, 3, 32, 33, 34, 64, 65, 66, 97])
def test_tap_blocks(W):
    _check(*_inputs(W, 1, 4, W, 48), 3, 2)
    cost, jump, edge, msgs = _inputs(W, 1, W, 4, 48)
    _check(cost, jump, edge, msgs, 3, 2)


@pytest.mark.parametrize("delta", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("taps", ["scalar", "taps8"])
def test_window_widths(delta, taps):
    _check(*_inputs(7 + delta, 1, 7, 40, 80, taps), delta, 2)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.float32, None])
@pytest.mark.parametrize("L", [96, 100, 70])
def test_argmin_storage(dtype, L):
    _check(*_inputs(3, 1, 6, 40, L), 3, 2, dtype)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("L", [32, 96, 192, 250])
def test_many_labels_below_the_candidate(L, flat):
    _check(*_inputs(11, 1, 8, 48, L, flat=flat), 3, 2)
    _check(*_inputs(12, 1, 8, 48, L, "taps8", flat=flat), 3, 1)


@pytest.mark.parametrize("L", [48, 192])
def test_mixed_forms(L):
    """Per pixel: offsets, weights that are zero or negative, a tap equal to or
    above L2, a non-zero own tap, exact ties, labels far above the rest."""
    g = cases.rng(5)
    cost, jump, edge, msgs = _inputs(5, 1, 9, 70, L)
    pick = g.integers(0, 10, size=edge.shape)
    edge = np.where(pick == 0, 0.0, np.where(pick == 1, -edge, edge)).astype(np.float32)
    off = g.integers(0, 6, size=jump[:, :, 0].shape)
    jump[:, :, 0] = np.where(off == 0, 1.5, 0.0)
    jump[:, :, 2] = np.where(off == 1, jump[:, :, 1], jump[:, :, 2])
    jump[:, :, 4] = np.where(off == 2, 0.75, jump[:, :, 4])
    jump[:, :, 3] = np.where(off == 3, 0.05, jump[:, :, 3])
    q = g.integers(0, 3, size=cost.shape[:3])
    cost = np.where((q == 0)[..., None], np.round(cost * 4) / 4, cost).astype(np.float32)
    cost[..., L // 3] += np.where(q == 1, 60.0, 0.0).astype(np.float32)
    _check(cost, jump, edge, msgs, 3, 2)


@pytest.mark.parametrize("L", [64, 192, 256])
def test_many_scanlines(L):
    """Enough scanlines for the one-warp blocks in both phases."""
    _check(*_inputs(21, 2, 330, 334, L)[:4], 3, 1)
