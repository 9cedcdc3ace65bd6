"""The FP32 stereo forward where steps of the hot loop's forms and of others
follow one another along a scanline: runs of one form of every length around the
32-step tap blocks, scanlines and blocks wholly of one form, against the
oracle."""
import numpy as np
import pytest

import cases
import oracle
from test_lbp_forward_gpu import _run_gpu, assert_parity

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _set(form, at, jump, edge):
    """Pixels `at` (H,W) of every direction to one form."""
    if form == "zero weight":
        edge[:, :, at] = 0.0
    elif form == "negative weight":
        edge[:, :, at] *= -1.0
    elif form == "offset":
        jump[:, :, 0, at] = 1.25
    elif form == "own tap":
        jump[:, :, 4, at] = 0.03125
    elif form == "wide":
        jump[:, :, 3, at] = jump[:, :, 5, at] * 1.5
    elif form == "narrow":
        jump[:, :, 2, at] = jump[:, :, 6, at] = jump[:, :, 1, at]


FORMS = ["lean", "wide", "zero weight", "narrow", "offset", "negative weight", "own tap"]


@pytest.mark.parametrize("L", [40, 96, 192])
@pytest.mark.parametrize("run", [1, 2, 31, 32, 33, 64, 200])
def test_runs_of_forms(L, run):
    g = cases.rng(L + run)
    H, W = 8, 141
    cost = cases.random_cost(g, 1, H, W, L)
    jump, edge = cases.random_taps8(g, 1, H, W), cases.edge_weights(g, 1, H, W)
    jump[:, :, 7] = jump[:, :, 1] = 0.5 + jump[:, :, 2:7].max(axis=2)
    which = (np.arange(W)[None, :] // run + np.arange(H)[:, None]) % len(FORMS)
    for k, form in enumerate(FORMS):
        _set(form, which == k, jump, edge)
    for c, j, e in ((cost, jump, edge), tuple(np.ascontiguousarray(np.swapaxes(a, -1 - (a is cost), -2 - (a is cost)))
                                             for a in (cost, jump, edge))):
        m = np.zeros((1, 4) + c.shape[1:], np.float32)
        ref = oracle.lbp_forward(0, c, j, e, m, 3, iters=2)
        assert_parity(_run_gpu(0, c, j, e, m, 3, 2), ref, f"runs of {run}")
