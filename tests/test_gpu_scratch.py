"""The image passes' scratch is given back on request, by a program that has no simulation, batch or denoiser to
destroy, and calls after that take it again."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_scratch_is_released(rk):
    w, h = 8192, 7936  # a radius byte per bin: 62 MB
    bins = torch.full((h, w, 4), 4.0, device="cuda")  # int(1 / 4^0.4) = 0: every bin is copied
    out = torch.empty_like(bins)
    rk.density_estimate(bins, w, h, 1, 0, 0.4, out)  # (the first call also loads the kernels, which stay)
    torch.cuda.synchronize()
    rk.release_scratch()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        rk.density_estimate(bins, w, h, 1, 0, 0.4, out)
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] >= w * h  # held between calls
        rk.release_scratch()
        assert torch.cuda.mem_get_info()[0] >= before
    rk.density_estimate(bins, w, h, 1, 0, 0.4, out)
    assert torch.equal(out, bins)
    rk.release_scratch()
