"""The stereo layer with gradients off (no indices stored) gives the values of
the training forward, and a call under no_grad leaves nothing behind that a
later training step would see."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("L", [5, 48, 70])
def test_values_and_gradients(storage, L):
    from bpl_gb300.layers.stereo import MessagePassing
    dev = torch.device("cuda:0")
    g = cases.rng(L)
    B, H, W = 2, 9, 35
    prob = torch.from_numpy(cases.softmax_np(g.normal(0, 2, size=(B, H, W, L)).astype(np.float32))).to(dev)
    edge = torch.from_numpy(cases.edge_weights(g, B, H, W)).to(dev)
    up = torch.from_numpy(g.normal(size=(B, H, W, L)).astype(np.float32)).to(dev)
    mp = MessagePassing(dev, 2, L, 3, storage=storage)

    def start():
        return torch.zeros((B, 4, H, W, L), device=dev, requires_grad=True) if storage == "fp32" else None

    def train():
        p = prob.clone().requires_grad_(True)
        b, m = mp(p, edge, None, None, start())
        b.backward(up)
        return b.detach(), m.detach(), p.grad

    b0, m0, g0 = train()
    with torch.no_grad():
        b1, m1 = mp(prob, edge, None, None, start())
    b2, m2, g2 = train()
    assert torch.equal(b0, b1) and torch.equal(m0, m1) and not b1.requires_grad
    assert torch.equal(b0, b2) and torch.equal(m0, m2)
    assert float((g2 - g0).abs().max()) <= 1e-5 * float(g0.abs().max())


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (1, 33, 70)])
def test_scalar_taps_equal_the_packing(shape):
    from bpl_gb300 import ops
    dev = torch.device("cuda:0")
    N, H, W = shape
    L1, L2 = torch.tensor(0.125, device=dev), torch.tensor(2.5, device=dev)
    aff = torch.zeros((N, 4, 3, H, W), device=dev)
    aff[:, :, :2] = L1
    aff[:, :, 2] = L2
    assert torch.equal(ops.scalar_taps(L1, L2, N, H, W), ops.pack_taps(aff, torch.zeros((N, 4, H, W), device=dev)))
