"""The density-estimation sweep (image.cu) against an FP64 gather, where it can go wrong: grids smaller
than a tile or a warp, tiles cut by the grid, every row count per warp (by grid size), the largest
radius staged whole (12) and the smallest in bands (13), the largest that sweeps (56) and the first
that gathers (57), a minimum radius above the maximum, sparse rows (taken by source), dense rows
(taken by offset) and empty grids."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(bins, R, mn, curve):
    b = bins.double()
    a = b[..., 3]
    r = torch.zeros(a.shape, dtype=torch.int64, device=a.device)
    for k in range(1, R + 1):
        r += (a <= (R / k) ** (1.0 / float(np.float32(curve)))).long()
    r = torch.where(a > 0, r.clamp_min(mn), torch.full_like(r, -1))
    big, (h, w) = max(R, mn), a.shape
    out = torch.zeros_like(b)
    rr = torch.arange(big + 1, device=a.device, dtype=torch.float64)
    for dy in range(-min(big, h - 1), min(big, h - 1) + 1):
        for dx in range(-min(big, w - 1), min(big, w - 1) + 1):
            d2 = dx * dx + dy * dy
            if 4 * d2 > (2 * big + 1) ** 2:
                continue
            wt = (1 - d2 / (rr + 0.5) ** 2) * 0.63661977236 / rr.clamp_min(1) ** 2
            wt = torch.where(4 * d2 <= (2 * rr + 1) ** 2, wt, torch.zeros_like(wt))
            wt[0] = float(d2 == 0)
            wt = torch.cat([wt, wt.new_zeros(1)])
            ys, xs = slice(max(0, -dy), h - max(0, dy)), slice(max(0, -dx), w - max(0, dx))
            yd, xd = slice(max(0, dy), h + min(0, dy)), slice(max(0, dx), w + min(0, dx))
            out[yd, xd] += b[ys, xs] * wt[r[ys, xs]][..., None]
    return out


@pytest.mark.parametrize("w,h,R,mn,mean", [(1, 1, 9, 0, 2.0), (5, 40, 12, 0, 0.2), (33, 9, 13, 0, 1.0), (65, 33, 9, 0, 0.02),
                                           (130, 70, 0, 2, 5.0), (130, 70, 1, 0, 300.0), (97, 41, 56, 0, 0.01), (64, 32, 57, 0, 0.05),
                                           (200, 100, 6, 3, 20.0), (96, 64, 9, 0, 0.0), (1100, 530, 9, 0, 0.5),
                                           (3841, 1100, 4, 0, 3.0), (700, 300, 20, 0, 0.3)])
def test_density_matches_fp64(rk, w, h, R, mn, mean):
    g = torch.Generator(device="cuda").manual_seed(w + 31 * R)
    # half of the grid at the mean density, half at a twentieth of it, colours in (0, 1] per point
    rate = torch.full((h, w), mean, device="cuda")
    rate[:, w // 2:] *= 0.05
    hits = torch.poisson(rate, generator=g)
    bins = hits[..., None] * torch.cat([0.1 + 0.9 * torch.rand(h, w, 3, device="cuda", generator=g), torch.ones(h, w, 1, device="cuda")], -1)
    out = torch.full_like(bins, float("nan"))
    rk.density_estimate(bins.contiguous(), w, h, R, mn, 0.4, out)
    ref = _reference(bins, R, mn, 0.4)
    # non-negative terms, at most (2 max(R, mn) + 1)^2 FP32 additions and a rounded weight each: every
    # partial sum is at most the result, so the error is at most the count times 2^-24 of it
    n = (2 * max(R, mn) + 1) ** 2
    assert torch.all((out.double() - ref).abs() <= (n + 2) * 2.0 ** -24 * ref + 1e-30)
