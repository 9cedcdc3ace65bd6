"""The FP16 stereo forward's steps outside the usual window, against the FP32
general arithmetic written out in numpy: beating ranges of two labels (8 taps)
and of none, offsets, windows wider than five labels, the full minimisation;
label counts around pairs and warps, both launch shapes, argmin stored and
not.  Taps and weights are multiples of 1/16 and costs of 1/64, so all sums are
exact and the stored halves equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LEFT, RIGHT, UP, DOWN = 0, 1, 2, 3


def _emulate(cost, taps, edge, msgs, delta):
    """One pass on (B,H,W,L) float32 copies of half values; the argmin where it is unique, else -1."""
    f = np.float32
    B, H, W, L = cost.shape
    Lv = taps.shape[2]
    am = np.zeros(msgs.shape, f)
    t = np.arange(L)
    for d in (RIGHT, LEFT, DOWN, UP):
        e, hor = d ^ 1, d in (LEFT, RIGHT)
        n = W if hor else H
        line = (lambda x, i: x[:, :, i]) if hor else (lambda x, i: x[:, i])
        for i, q in ([(i, i + 1) for i in range(n - 1)] if d in (RIGHT, DOWN) else [(i, i - 1) for i in range(n - 1, 0, -1)]):
            h = line(cost, i)
            for k in ((e, UP, DOWN) if hor else (RIGHT, LEFT, e)):
                h = (h + line(msgs[:, k], i)).astype(f)
            w = line(edge[:, d], i)[..., None, None]
            tp = line(np.moveaxis(taps[:, d], 1, -1), i)  # (B, n, Lv)
            idx = np.clip(Lv // 2 + t[:, None] - t[None, :], 1, Lv - 1)  # [t, s]
            term = (tp[..., idx] * w).astype(f) + h[..., None, :]
            lo = h.min(-1, keepdims=True)
            if delta < L:
                off = tp[..., 0][..., None]
                start = np.floor(np.abs(t - (delta - 1) + off - 1) + 0.5) * np.sign(t - (delta - 1) + off - 1)
                stop = np.floor(np.abs(t + delta + off + 1) + 0.5) * np.sign(t + delta + off + 1)
                inside = (t >= start.clip(0)[..., None]) & (t < stop[..., None])
                term = np.where(inside, term, np.inf).astype(f)
                cand = (tp[..., -1:] * w[..., 0] + lo).astype(f)
                m = np.minimum(term.min(-1), cand)
            else:
                m = term.min(-1)
            # where one sender alone gives the value
            ways = (term == m[..., None]).sum(-1)
            arg = term.argmin(-1).astype(f)
            if delta < L:
                arg = np.where(m < cand, np.where(ways == 1, arg, -1),
                               np.where((h == lo).sum(-1, keepdims=True) == 1, h.argmin(-1)[..., None], -1))
            else:
                arg = np.where(ways == 1, arg, -1)
            line(msgs[:, e], q)[...] = (m - lo).astype(np.float16).astype(f)
            line(am[:, e], q)[...] = arg
    return am


def _check(B, H, W, L, kind, delta, dtype=torch.uint8, shift=0):
    from bpl_gb300 import ops
    g = np.random.default_rng(L + delta + W)
    cost = (-g.integers(0, 256, size=(B, H, W, L)) / 64).astype(np.float32)
    edge = (g.integers(1, 9, size=(B, 4, H, W)) / 4).astype(np.float32)
    Lv = 8 if kind == "wide" else 6
    taps = np.zeros((B, 4, Lv, H, W), np.float32)
    taps[:, :, 1] = taps[:, :, Lv - 1] = 0.75
    c0 = Lv // 2
    taps[:, :, c0 - 1] = taps[:, :, c0 + 1] = 0.25
    if kind == "wide":
        taps[:, :, c0 - 2] = taps[:, :, c0 + 2] = 0.5
    elif kind == "own":   # neighbours at L2: no beating offset but the own label
        taps[:, :, c0 - 1] = taps[:, :, c0 + 1] = 0.75
    elif kind == "none":
        taps[:, :, c0 - 1:c0 + 2] = 0.75
    elif kind == "offset":
        taps[:, :, 0] = g.choice([-1.5, -0.25, 0.75, 2.0], size=(B, 4, H, W))
    dev = torch.device("cuda:0")
    Lp = ops.padded_labels(L)

    def half(shape, values=None):
        n = int(np.prod(shape))
        x = torch.zeros(n + 16, dtype=torch.float16, device=dev)[shift:shift + n].view(shape)
        if values is not None:
            x[..., :L] = torch.from_numpy(values).to(dev)
        return x
    c, m = half((B, H, W, Lp), cost), half((B, 4, H, W, Lp))
    _, am, _ = ops.lbp_forward_f16(0, c, torch.from_numpy(taps).to(dev), torch.from_numpy(edge).to(dev), m, delta, L,
                                   argmin_dtype=dtype)
    torch.cuda.synchronize()
    ref = np.zeros((B, 4, H, W, L), np.float32)
    ra = _emulate(cost, taps, edge, ref, delta)
    np.testing.assert_array_equal(m[..., :L].float().cpu().numpy(), ref)
    if dtype is not None:
        got = am[..., :L].cpu().numpy().astype(np.float32)
        assert np.array_equal(np.where(ra < 0, -1, got), ra) and got.min() >= 0 and got.max() < L


KINDS = [("wide", 3), ("wide", 2), ("own", 3), ("none", 3), ("offset", 3), ("usual", 7), ("usual", 300)]


@pytest.mark.parametrize("kind,delta", KINDS)
@pytest.mark.parametrize("L", [5, 8, 31, 33, 48, 64, 65, 100, 129, 193, 256])
def test_label_counts(kind, delta, L):
    _check(1, 3, 37, L, kind, delta)


@pytest.mark.parametrize("kind,delta", KINDS)
@pytest.mark.parametrize("dtype,shift", [(torch.int16, 0), (torch.float32, 1), (None, 0), (torch.uint8, 2)])
def test_storage(kind, delta, dtype, shift):
    _check(1, 4, 9, 70, kind, delta, dtype, shift)


@pytest.mark.parametrize("kind,delta", [("wide", 3), ("offset", 3), ("usual", 7)])
def test_many_scanlines(kind, delta):
    _check(4, 156, 158, 20, kind, delta)
