"""The FP16 stereo forward (labels in pairs, rows through a shared-memory ring or
registers two steps ahead) against its own arithmetic written out in numpy:
FP32 sums and minima, the stored row rounded to half, ties to the largest
label of the minimum of h and to the own, left, right window term.  Taps and
edge weights are multiples of 1/16, so their products are exact and the fused
multiply-adds round like separate additions: equality, not a tolerance.
Sizes: label counts around pairs and warps, widths around tap blocks and the
ring, both launch shapes, every argmin storage, tensors off a 16-byte
boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LEFT, RIGHT, UP, DOWN = 0, 1, 2, 3


def _emulate(cost, taps, edge, msgs, L):
    """One pass on (B,H,W,L) float32 copies of half values; taps (B,4,6,H,W)."""
    f = np.float32
    B, H, W, _ = cost.shape
    am = np.zeros(msgs.shape, np.float32)
    for d in (RIGHT, LEFT, DOWN, UP):
        e, hor = d ^ 1, d in (LEFT, RIGHT)
        n = W if hor else H
        line = (lambda t, i: t[:, :, i]) if hor else (lambda t, i: t[:, i])
        steps = [(i, i + 1) for i in range(n - 1)] if d in (RIGHT, DOWN) else [(i, i - 1) for i in range(n - 1, 0, -1)]
        for i, q in steps:
            parts = [line(msgs[:, k], i) for k in ((e, UP, DOWN) if hor else (RIGHT, LEFT, e))]
            h = line(cost, i)
            for p in parts:
                h = (h + p).astype(f)
            w = line(edge[:, d], i)[..., None]
            tp = [line(taps[:, d, k], i)[..., None] for k in range(6)]
            pm = h.min(-1, keepdims=True)
            arg_h = L - 1 - (h == pm)[..., ::-1].argmax(-1)[..., None]
            g = (tp[5] * w + pm).astype(f)
            inf = np.full(h.shape[:-1] + (1,), np.inf, f)
            # beating offsets: |jd| <= 1 when both its taps times w are below L2 w, the own label likewise
            own_ok = tp[3] * w < tp[5] * w
            side_ok = own_ok & (tp[2] * w < tp[5] * w) & (tp[4] * w < tp[5] * w)
            n0 = np.where(own_ok, (tp[3] * w + h).astype(f), np.inf)
            nl = np.where(side_ok, (tp[4] * w + np.concatenate([inf, h[..., :-1]], -1)).astype(f), np.inf)
            nr = np.where(side_ok, (tp[2] * w + np.concatenate([h[..., 1:], inf], -1)).astype(f), np.inf)
            t = np.arange(L)
            m, a = n0, np.broadcast_to(t, h.shape)
            a = np.where(nl < m, t - 1, a)
            m = np.minimum(m, nl)
            a = np.where(nr < m, t + 1, a)
            m = np.minimum(m, nr)
            win = m < g
            out = (np.where(win, m, g) - pm).astype(f).astype(np.float16).astype(f)
            line(msgs[:, e], q)[...] = out
            line(am[:, e], q)[...] = np.where(win, a, arg_h)
    return am


def _check(B, H, W, L, dtype=torch.uint8, shift=0, seed=0, iters=2, ties=True):
    from bpl_gb300 import ops
    g = np.random.default_rng(seed)
    Lp = ops.padded_labels(L)
    cost = -g.random((B, H, W, L)).astype(np.float16).astype(np.float32)
    if ties:  # exact ties of the minimum and of window terms
        cost = (np.round(cost * 8) / 8).astype(np.float32)
    edge = (g.integers(0, 33, size=(B, 4, H, W)) / 16).astype(np.float32)
    taps = np.zeros((B, 4, 6, H, W), np.float32)
    taps[:, :, 1] = taps[:, :, 5] = 0.5
    taps[:, :, 2] = taps[:, :, 4] = g.choice([0.125, 0.25, 0.5], size=(B, 4, H, W))
    dev = torch.device("cuda:0")

    def half(shape, values=None):
        flat = torch.zeros(int(np.prod(shape)) + 16, dtype=torch.float16, device=dev)
        t = flat[shift:shift + int(np.prod(shape))].view(shape)
        if values is not None:
            t[..., :L] = torch.from_numpy(values).to(dev)
        return t
    ch, mh = half((B, H, W, Lp), cost), half((B, 4, H, W, Lp))
    t, e = torch.from_numpy(taps).to(dev), torch.from_numpy(edge).to(dev)
    ref = np.zeros((B, 4, H, W, L), np.float32)
    for _ in range(iters):
        _, am, _ = ops.lbp_forward_f16(0, ch, t, e, mh, 3, L, argmin_dtype=dtype)
        ra = _emulate(cost, taps, edge, ref, L)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(mh[..., :L].float().cpu().numpy(), ref)
    assert not mh[..., L:].any()
    if dtype is not None:
        np.testing.assert_array_equal(am[..., :L].cpu().numpy().astype(np.float32), ra)


@pytest.mark.parametrize("L", [4, 7, 8, 9, 31, 33, 62, 63, 64, 65, 66, 100, 127, 128, 129, 191, 192, 193, 250, 256])
def test_label_counts(L):
    _check(1, 5, 37, L, seed=L)


@pytest.mark.parametrize("W", [2, 3, 4, 7, 8, 9, 31, 32, 33, 34, 65, 66])
def test_widths(W):
    _check(1, 3, W, 40, seed=W)
    _check(1, W, 3, 40, seed=W)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.float32, None])
@pytest.mark.parametrize("shift", [0, 1, 2, 8])
def test_storage_and_alignment(dtype, shift):
    _check(1, 4, 40, 70, dtype, shift, seed=3)


@pytest.mark.parametrize("L,shift", [(48, 0), (192, 0), (100, 1), (256, 0)])
def test_many_scanlines(L, shift):
    _check(4, 160, 170, L, shift=shift, seed=5, iters=1, ties=False)
