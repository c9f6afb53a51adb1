"""The order network's kernels at the sizes where their split changes: one and
32 vertices a graph; fewer graphs than SMs, one for each and for each of a
block's two groups, one more; nodes one below, at and above the 128 of a
weight-gradient block.  Against the CPU fp32 reference (tests/mpnn_ref.py) with
the tolerances of tests/test_gpu_mpnn.py, which state where they come from."""
import numpy as np
import pytest

import mpnn_ref as R
from fsig_gb300 import learn

pytestmark = pytest.mark.gpu

FWD_TOL, GRAD_TOL = 2e-2, 3e-2
SIZES = {"one": [1, 32], "127": [31, 32, 32, 32], "128": [32] * 4, "129": [32] * 4 + [1], "152": [6] * 152,
         "153": [5] * 153, "304": [4, 3] * 152, "305": [3, 4] * 152 + [32]}


@pytest.mark.parametrize("name", sorted(SIZES))
def test_forward_and_gradients(engine, name):
    import torch
    sizes = SIZES[name]
    rng = np.random.default_rng(len(sizes))
    goff = np.zeros(len(sizes) + 1, np.uint32)
    goff[1:] = np.cumsum(sizes)
    nbr = np.zeros(int(goff[-1]), np.uint32)
    for o, n in zip(goff, sizes):
        for i in range(1, n):
            for j in {int(rng.integers(0, i)), int(rng.integers(0, i))}:
                nbr[o + i] |= np.uint32(1 << j)
                nbr[o + j] |= np.uint32(1 << i)
    feat = rng.random((int(goff[-1]), 8)).astype(np.float32)
    tgt = rng.random(int(goff[-1])).astype(np.float32)
    p = learn.init_params(6)
    p[R.P_BIN:R.P_WS] = rng.normal(0, 0.1, R.H)
    p[R.P_B:R.P_WOUT] = rng.normal(0, 0.1, R.LAYERS * R.H)
    engine.mpnn_set_params(p)
    dev = engine.mpnn_forward(goff, feat, nbr)
    ref = R.forward(torch.tensor(p), goff, feat, nbr).numpy()
    assert np.abs(dev - ref).max() <= FWD_TOL * np.abs(ref).max()
    loss, g = engine.mpnn_train_step(goff, feat, nbr, tgt, lr=0.0)
    rloss, rg, _ = R.loss_and_grads(p, goff, feat, nbr, tgt)
    assert abs(loss - rloss) <= 1e-2 * rloss
    for block, sl in R.blocks():
        assert np.linalg.norm(g[sl] - rg[sl]) <= GRAD_TOL * max(np.linalg.norm(rg[sl]), 1e-12), block
