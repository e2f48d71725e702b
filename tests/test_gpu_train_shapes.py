"""Training steps whose coarsest level is no multiple of 8 pixels (batch x height / 8 x width / 8): the gradient of
the mean loss is that of eight copies of the batch, a shape whose levels are all whole groups of 8 pixels."""
import numpy as np
import pytest
import torch

from test_gpu_denoise import _feats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (1, 72, 72), (3, 40, 56), (1, 24, 136), (2, 8, 24)])
def test_gradients_are_those_of_eight_copies(rk, n, h, w):
    net = rk.Denoiser(8 * n * h * w, seed=4)
    rng = np.random.default_rng(n + h + w)
    net.set_params(np.concatenate([np.concatenate([
        rng.normal(0, np.sqrt(2.0 / (l["taps"] * (l["in_a"] + l["in_b"]))), l["out"] * l["taps"] * (l["in_a"] + l["in_b"])),
        rng.normal(0, 0.05, l["out"])]) for l in net.layers()]).astype(np.float32))
    f = _feats(n, h, w, 5)
    target = torch.full((n, h, w, 3), -10.0, device="cuda")
    loss = net.train_step(f, target, 0.0)
    got = net.gradients()
    want_loss = net.train_step(f.repeat(8, 1, 1, 1), target.repeat(8, 1, 1, 1), 0.0)
    want = net.gradients()
    assert loss == pytest.approx(want_loss, rel=1e-12)
    # a factor of 8 is exact in BF16, so the terms are equal and only the order of FP32 sums differs: at most 41,472
    # pixels, 16 an addition, 2^-23 each of a sum whose terms hardly cancel; a lost group of 8 pixels is 8 / 81 and more
    # of the coarsest levels' sums
    o = 0
    for l in net.layers():
        for size in (l["out"] * l["taps"] * (l["in_a"] + l["in_b"]), l["out"]):
            a, b = got[o:o + size].astype(np.float64), want[o:o + size].astype(np.float64)
            assert np.linalg.norm(b) > 0
            assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b), l
            o += size
