"""The semantic forwards with the full minimisation (lane = label, up to 32
labels) against the oracle: label counts around the groups of eight senders
and around multiples of 4 (pixel matrices by bulk or by 16-byte copies), single
rows and columns, widths around the ring and the 32-step weight blocks, tensors
off a 16-byte boundary, exact ties, values outside exp's fast range, every
argmin storage.  Bitwise up to the host's exp/log, as test_lbp_forward_gpu.py
states it."""
import numpy as np
import pytest

import cases
import oracle
from test_lbp_forward_gpu import assert_parity

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _shifted(a, shift):
    """A device copy that starts `shift` floats off its allocation."""
    flat = torch.zeros(a.size + 4, device="cuda:0")
    t = flat[shift:shift + a.size].view(a.shape)
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t


def _check(pixel, B, H, W, L, seed=0, q=None, shift=0, dtype=torch.uint8, scale=1.0, iters=2):
    from bpl_gb300 import ops
    g = cases.rng(seed)
    cost = (cases.random_cost(g, B, H, W, L, quantise=q) * scale).astype(np.float32)
    edge = cases.edge_weights(g, B, H, W, quantise=q)
    jump = cases.semantic_pixel_jump(g, H, W, L)[0] if pixel else cases.semantic_global_jump(g, L, quantise=q)[0]
    msgs = cases.random_messages(g, B, H, W, L, quantise=q)
    variant = 2 if pixel else 1
    c, j, e, m = (_shifted(a, shift) for a in (cost, jump, edge, msgs))
    for _ in range(iters):
        m, am, sc = ops.lbp_forward(variant, c, j, e, m, L, argmin_dtype=dtype)
    torch.cuda.synchronize()
    ref = oracle.lbp_forward(variant, cost, jump, edge, msgs, L, iters=iters)
    am = ref[1] if am is None else am.cpu().numpy().astype(np.float32)
    assert_parity((m.cpu().numpy(), am, sc.cpu().numpy()), ref)


@pytest.mark.parametrize("pixel", [False, True])
@pytest.mark.parametrize("L", [1, 2, 3, 4, 7, 8, 9, 12, 15, 16, 17, 19, 20, 23, 24, 25, 28, 31, 32])
def test_label_counts(pixel, L):
    _check(pixel, 1, 5, 9, L, seed=L)


@pytest.mark.parametrize("pixel", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 32, 33, 34, 65, 66])
def test_lengths(pixel, n):
    _check(pixel, 1, 2, n, 11, seed=n)
    _check(pixel, 1, n, 2, 12, seed=n)


@pytest.mark.parametrize("pixel", [False, True])
@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("L", [8, 19])
def test_off_boundary(pixel, shift, L):
    _check(pixel, 2 if not pixel else 1, 4, 10, L, seed=3, shift=shift)


@pytest.mark.parametrize("pixel", [False, True])
def test_ties_range_and_storage(pixel):
    _check(pixel, 1, 6, 12, 19, seed=4, q=4)
    _check(pixel, 1, 6, 12, 19, seed=5, scale=400.0)
    for dtype in (torch.int16, torch.float32, None):
        _check(pixel, 1, 4, 9, 19, seed=6, dtype=dtype)


def test_global_many_scanlines():
    _check(False, 3, 260, 262, 19, seed=7, iters=1)
