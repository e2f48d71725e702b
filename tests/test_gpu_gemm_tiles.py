"""The GEMM's tile widths (tile_width, gemm.cu): sizes whose rounds of tiles take 256, 224, 208, ... 64 columns,
with ragged last tiles in both directions, against the product in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(4096, 4096, 64), (128, 4096, 256), (128, 130, 72), (1, 257, 8), (1000, 3000, 200), (2048, 2048, 136),
                                   (3001, 4001, 64), (4096, 1000, 64), (700, 9001, 40), (129, 19456, 64), (130, 2433, 1000)])
@pytest.mark.parametrize("f32", [True, False])
def test_tile_widths(rk, m, n, k, f32):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    b = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    c = torch.full((m, n), float("nan"), dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    rk.gemm_bf16(a, b, c, mode=rk.GEMM_STORE_F32 if f32 else rk.GEMM_STORE_BF16)
    want = a.double() @ b.double().t()
    # products of bf16 are exact in FP32; k - 1 additions that round or truncate at 2^-23 of a partial sum
    tol = k * 2.0 ** -23 * (a.double().abs() @ b.double().abs().t())
    if not f32:
        tol = tol + 2.0 ** -8 * (want.abs() + tol)  # rounded to bf16
    assert bool(((c.double() - want).abs() <= tol).all())
