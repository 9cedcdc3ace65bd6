"""LBP forwards whose dynamic shared memory lies just below 48 KB, where the
kernel's static tables decide whether the launch needs the opt-in limit: each
as the first launch of its instantiation (a process of its own, since an
earlier larger launch would already have raised the limit), against the
oracle."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = {
    # name: (variant, B, H, W, L, taps, delta)
    "pixel_l24_truncated": (2, 1, 5, 9, 24, 0, 3),        # 4-warp blocks, 47744 bytes
    "pixel_l73_one_warp": (2, 1, 2, 612, 73, 0, 73),      # one-warp blocks, ring of 2: 46656
    "pixel_l74_one_warp": (2, 1, 2, 612, 74, 0, 74),      # 47808
    "stereo_l800_10_taps": (0, 1, 3, 9, 800, 10, 3),      # 46912
    "stereo_l800_11_taps": (0, 1, 3, 9, 800, 11, 3),      # 47936
    "stereo_l800_12_taps": (0, 1, 3, 9, 800, 12, 3),      # 49024
}


def _main(name):
    for p in ("bp-layers_gb300", "oracle", os.path.join("tests", "golden"), "tests"):
        sys.path.insert(0, os.path.join(ROOT, p))
    import numpy as np

    import cases
    import oracle
    from test_lbp_forward_gpu import _run_gpu, assert_parity
    variant, B, H, W, L, Lv, delta = CASES[name]
    g = cases.rng(len(name) + L)
    cost, edge = cases.random_cost(g, B, H, W, L), cases.edge_weights(g, B, H, W)
    if variant == 0:
        jump = np.sort(g.random((1, 4, Lv, H, W)), axis=2).astype(np.float32)
        jump[:, :, 0] = 0.0
    else:
        jump = cases.semantic_pixel_jump(g, H, W, L)[0]
    msgs = cases.random_messages(g, B, H, W, L)
    gpu = _run_gpu(variant, cost, jump, edge, msgs, delta, 1)
    assert_parity(gpu, oracle.lbp_forward(variant, cost, jump, edge, msgs, delta), name)


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_first_launch_near_the_default_limit(name):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), name], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


if __name__ == "__main__":
    _main(sys.argv[1])
