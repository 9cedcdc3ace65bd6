"""GPU parity of the flow SAD forward where its row end and its channel loop
change form: warps wholly inside the image beside warps at its border, window
sizes around a warp's 16 displacements, channel counts around 8 and 32, rows
copied in bulk (width and offset multiples of 4) and not, and sums above the
reference's start value 9999999.  Bit-exact against the oracle."""
import numpy as np
import pytest

import cases
import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("C,H,W,sws,scale", [
    (1, 3, 64, 0, 1.0), (7, 5, 96, 3, 1.0), (8, 6, 100, 14, 1.0), (9, 6, 132, 15, 1.0), (31, 4, 64, 16, 1.0),
    (33, 5, 128, 24, 1.0), (40, 4, 97, 32, 1.0), (65, 3, 160, 8, 1.0), (32, 9, 192, 64, 1.0),
    (4, 6, 128, 16, 3e6), (16, 4, 132, 31, 1e6)])
def test_flow_forward_row_forms_bit_exact(C, H, W, sws, scale):
    from bpl_gb300 import ops
    g = cases.rng(900 + C + W + sws)
    f0 = (g.normal(0, 1, size=(2, C, H, W)) * scale).astype(np.float32)
    f1 = (g.normal(0, 1, size=(2, C, H, W)) * scale).astype(np.float32)
    f1[..., W // 2:] = f0[..., W // 2:]  # exact matches: zero sums and their ties
    dev = torch.device("cuda:0")
    outs = ops.flow_forward(torch.from_numpy(f0).to(dev), torch.from_numpy(f1).to(dev), sws)
    ref = oracle.flow_forward(f0, f1, sws)
    for nm, a, b in zip(("cv_u", "cv_v", "u_star", "v_star"), outs, ref):
        np.testing.assert_array_equal(a.cpu().numpy(), b, err_msg=nm)
