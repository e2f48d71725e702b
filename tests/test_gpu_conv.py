"""The staged-tile convolution kernels (conv.cu) at the sizes where they can go wrong: images smaller
than a tile and tiles cut by the image, one-plane inputs (8 channels, two taps per MMA step), layers
cut into column groups, the most channels that fit, channel counts that take the gathering GEMM, and
for the gradients every staging of the weight gradient: windows of 1 to 16 pixel groups, rows that
are no multiple of 8 pixels at the coarse levels, one-pixel levels."""
import pytest
import torch

from test_gpu_denoise import _feats, torch_unet
from test_gpu_gemm import _conv_ops, _conv_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,ca,cb,N,up", [(1, 1, 1, 8, 0, 16, False), (2, 17, 9, 8, 0, 32, False),
                                              (1, 16, 8, 16, 0, 3, False), (3, 15, 23, 32, 0, 32, False),
                                              (1, 18, 26, 96, 64, 64, True), (1, 33, 8, 96, 0, 96, False),
                                              (1, 6, 40, 64, 0, 160, False), (1, 20, 10, 224, 0, 16, False),
                                              (1, 9, 12, 24, 0, 32, False), (2, 2, 2, 8, 8, 48, True),
                                              (1, 300, 8, 48, 0, 48, False)])
def test_conv_edges(rk, n, h, w, ca, cb, N, up):
    xa, xb, wt = _conv_ops(n, h, w, ca, cb, N, up, 31 * h + 7 * w + N)
    c = torch.full((n * h * w, N), float("nan"), device="cuda")
    rk.conv3x3_bf16(xa, wt, c, xb=xb, up=up)
    # FP32 accumulation of BF16 products: |err| <= ~K * 2^-24 * sum|x||w|
    tol = 1e-5 * _conv_ref(xa, xb, wt, up, absolute=True) + 1e-6
    assert torch.all((c - _conv_ref(xa, xb, wt, up)).abs() <= tol)
    bias = torch.randn(N, device="cuda")
    d = torch.zeros(n * h * w, N, device="cuda", dtype=torch.bfloat16)
    rk.conv3x3_bf16(xa, wt, d, xb=xb, up=up, mode=rk.GEMM_STORE_BF16, bias=bias, relu=True)
    ref = (_conv_ref(xa, xb, wt, up) + bias).clamp_min(0)
    assert torch.all((d.float() - ref).abs() <= 2 ** -8 * ref.abs() + tol + 1e-6)  # one BF16 rounding more


# (n h / 8 w / 8 a multiple of 8); widths of the four levels: 48 24 12 6, 72 36 18 9, 8 4 2 1, 256 .. 32, 128 .. 16
@pytest.mark.parametrize("n,h,w", [(2, 32, 48), (1, 64, 72), (8, 8, 8), (1, 16, 256), (2, 40, 128)])
def test_gradients_of_every_staging(rk, n, h, w):
    net = rk.Denoiser(n * h * w, seed=3)
    import numpy as np
    rng = np.random.default_rng(h + w)
    net.set_params(np.concatenate([np.concatenate([
        rng.normal(0, np.sqrt(2.0 / (l["taps"] * (l["in_a"] + l["in_b"]))), l["out"] * l["taps"] * (l["in_a"] + l["in_b"])),
        rng.normal(0, 0.05, l["out"])]) for l in net.layers()]).astype(np.float32))
    f = _feats(n, h, w, 5)
    target = torch.rand(n, h, w, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    net.train_step(f, target, 0.0)
    got, o = net.gradients(), 0
    ref, ws = torch_unet(net.layers(), net.params(), f.float())
    (f.float()[..., 4:7] + ref - target).abs().mean().backward()
    for i, (w_, b_) in enumerate(ws):
        for g in (w_.grad.permute(0, 2, 3, 1).reshape(-1).cpu().numpy(), b_.grad.cpu().numpy()):
            mine = got[o:o + g.size]
            o += g.size
            # BF16 activations and gradients against FP32 ones, as in test_gradients_match_autograd
            assert np.linalg.norm(mine - g) <= 0.2 * np.linalg.norm(g) + 1e-6, (i, g.size)
