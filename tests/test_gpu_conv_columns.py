"""A convolution of more columns than conv_kernel's grid has column groups for (224 channels leave room for 16
columns per group: 65,535 groups): it takes the gathering GEMM."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16 * 65535, 16 * 65535 + 3])
def test_more_columns_than_groups(rk, N):
    x = torch.zeros(1, 1, 1, 224, device="cuda", dtype=torch.bfloat16)
    x[..., 0] = 1.0
    x[..., 223] = 2.0
    wt = torch.zeros(N, 9 * 224, device="cuda", dtype=torch.bfloat16)
    wt[:, 4 * 224] = (torch.arange(N, device="cuda") % 251).bfloat16()  # the centre tap
    wt[:, 4 * 224 + 223] = 1.0
    c = torch.full((1, N), -1.0, device="cuda")
    rk.conv3x3_bf16(x, wt, c)
    assert torch.equal(c[0], (torch.arange(N, device="cuda") % 251).float() + 2.0)
