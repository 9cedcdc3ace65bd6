"""NaN costs in the LBP forwards.  A term that is NaN is skipped: it is neither
the minimum of h nor a window's minimum nor any argmin, as if its cost were
+inf; a pixel whose every label is NaN or infinite, or a weight that is, still gives
indices that are labels (the adjoint adds at them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _f16_inputs(B, H, W, L, seed):
    g = np.random.default_rng(seed)
    cost = -g.random((B, H, W, L)).astype(np.float16).astype(np.float32)
    edge = (g.integers(1, 33, size=(B, 4, H, W)) / 16).astype(np.float32)
    taps = np.zeros((B, 4, 6, H, W), np.float32)
    taps[:, :, 1] = taps[:, :, 5] = 0.5
    taps[:, :, 2] = taps[:, :, 4] = 0.125
    return g, cost, edge, taps


def _f16_run(cost, edge, taps, L, dtype, delta=3):
    from bpl_gb300 import ops
    dev = torch.device("cuda:0")
    B, H, W, _ = cost.shape
    c = torch.zeros((B, H, W, ops.padded_labels(L)), dtype=torch.float16, device=dev)
    c[..., :L] = torch.from_numpy(cost).to(dev)
    m = torch.zeros((B, 4, H, W, ops.padded_labels(L)), dtype=torch.float16, device=dev)
    t, e = torch.from_numpy(taps).to(dev), torch.from_numpy(edge).to(dev)
    _, am, _ = ops.lbp_forward_f16(0, c, t, e, m, delta, L, argmin_dtype=dtype)
    torch.cuda.synchronize()
    return m[..., :L].float().cpu().numpy(), am[..., :L].cpu().numpy().astype(np.float32)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.float32])
@pytest.mark.parametrize("L", [5, 40, 64, 130])
def test_f16_indices_of_nan_pixels_are_labels(dtype, L):
    _, cost, edge, taps = _f16_inputs(1, 7, 11, L, L)
    cost[0, 3, 4] = np.nan
    cost[0, 5, 7] = np.inf
    _, am = _f16_run(cost, edge, taps, L, dtype)
    assert am.min() >= 0 and am.max() < L


@pytest.mark.parametrize("kind", ["nan pixel", "inf pixel", "inf weight", "inf weights"])
@pytest.mark.parametrize("delta", [1, 3, 7])
@pytest.mark.parametrize("L", [5, 31, 32, 63, 70])
def test_f32_indices_are_labels(kind, delta, L):
    from bpl_gb300 import ops
    _, cost, edge, taps = _f16_inputs(1, 7, 11, L, L)
    if "pixel" in kind:
        cost[0, 3, 4] = np.nan if kind == "nan pixel" else np.inf
    elif kind == "inf weight":
        edge[0, :, 3, 4] = np.inf
    else:
        edge[:] = np.inf
    c, t, e = (torch.from_numpy(a).to("cuda:0") for a in (cost, taps, edge))
    m = torch.zeros((1, 4, 7, 11, L), device="cuda:0")
    _, am, _ = ops.lbp_forward(0, c, t, e, m, delta, argmin_dtype=torch.float32)
    am = am.cpu().numpy()
    assert am.min() >= 0 and am.max() < L


def _holes(g, cost):
    """One or two labels per pixel lost, beside the pixel's smallest cost and
    anywhere; the copy with +inf in their place."""
    B, H, W, L = cost.shape
    gap = np.zeros(cost.shape, bool)
    low = cost.argmin(-1)
    b, y, x = np.indices(low.shape)
    gap[b, y, x, np.clip(low + g.choice([-1, 1, 2], size=low.shape), 0, L - 1)] = True
    gap[b, y, x, g.integers(0, L, size=low.shape)] = True
    gap[b, y, x, low] = False
    gap &= g.random(low.shape)[..., None] < 0.5
    return np.where(gap, np.nan, cost).astype(np.float32), np.where(gap, np.inf, cost).astype(np.float32)


@pytest.mark.parametrize("L", [5, 33, 64, 130])
def test_f16_nan_terms_are_skipped(L):
    from test_f16_pairs_gpu import _emulate
    g, cost, edge, taps = _f16_inputs(2, 6, 9, L, 7 + L)
    nan, inf = _holes(g, cost)
    m, am = _f16_run(nan, edge, taps, L, torch.uint8)
    ref = np.zeros(m.shape, np.float32)
    with np.errstate(invalid="ignore"):
        ra = _emulate(inf, taps, edge, ref, L)
    np.testing.assert_array_equal(m, ref)
    np.testing.assert_array_equal(am, ra)


@pytest.mark.parametrize("form", ["lean", "own tap", "8 taps", "offset"])
@pytest.mark.parametrize("L", [5, 33, 96, 192])
def test_f32_nan_terms_are_skipped(form, L):
    """Steps of the hot loop and of the forms outside it alike."""
    import cases
    import oracle
    from test_lbp_forward_gpu import _run_gpu, assert_parity
    g, cost, edge, taps = _f16_inputs(2, 6, 40, L, 11 + L)
    if form == "own tap":
        taps[:, :, 3] = 0.03125
    elif form == "8 taps":
        taps = cases.random_taps8(g, 2, 6, 40)
    elif form == "offset":
        taps[:, :, 0] = 0.75
    nan, inf = _holes(g, (4.0 * cost).astype(np.float32))
    msgs = np.zeros((2, 4, 6, 40, L), np.float32)
    with np.errstate(invalid="ignore"):
        ref = oracle.lbp_forward(0, inf, taps, edge, msgs, 3)
    assert_parity(_run_gpu(0, nan, taps, edge, msgs, 3, 1), ref, form)
