"""Density estimation of bins whose colour or density is not finite: a bin reaches the outputs of its own
disc and no others, at every row count per warp, staged whole and in bands, and in the gather above the sweep's
radii.  Outside the discs the outputs are, bit for bit, those of the same grid with those colours at zero."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,R,mn", [(70, 45, 9, 0), (200, 100, 12, 0), (200, 100, 1, 0), (96, 64, 0, 2), (1100, 530, 9, 0),
                                      (3841, 1100, 4, 0), (200, 100, 13, 0), (700, 300, 20, 0), (3841, 1100, 17, 0),
                                      (97, 141, 56, 0), (150, 120, 57, 0)])
@pytest.mark.parametrize("mean", [0.05, 40.0])
def test_only_the_disc_is_touched(rk, w, h, R, mn, mean):
    g = torch.Generator(device="cuda").manual_seed(w + R)
    hits = torch.poisson(torch.full((h, w), mean, device="cuda"), generator=g)
    bins = hits[..., None] * torch.cat([0.1 + 0.9 * torch.rand(h, w, 3, device="cuda", generator=g), torch.ones(h, w, 1, device="cuda")], -1)
    bad = [(w // 2, h // 2, 0, math.inf, 1.0), (w // 3, h // 5, 1, math.nan, 3.0), (1, h - 2, 2, -math.inf, 2.0),
           (w - 1, 0, 0, math.nan, 50.0)]
    zero, covered = bins.clone(), torch.zeros(h, w, 4, dtype=torch.bool, device="cuda")
    ys, xs = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    for x, y, ch, value, a in bad:
        zero[y, x] = torch.tensor([0.0, 0.0, 0.0, a])
        bins[y, x] = zero[y, x]
        bins[y, x, ch] = value
        r = max(mn, min(R, int(R / a ** 0.4)))
        covered[..., ch] |= 4 * ((xs - x) ** 2 + (ys - y) ** 2) <= (2 * r + 1) ** 2
    # an infinite density: a disc of the smallest radius
    x, y = w // 4, h - 1
    bins[y, x] = torch.tensor([1.0, 1.0, 1.0, math.inf])
    zero[y, x] = torch.tensor([1.0, 1.0, 1.0, 1e30])
    covered[..., 3] |= 4 * ((xs - x) ** 2 + (ys - y) ** 2) <= (2 * mn + 1) ** 2
    out, ref = torch.zeros_like(bins), torch.zeros_like(bins)
    rk.density_estimate(bins, w, h, R, mn, 0.4, out)
    rk.density_estimate(zero, w, h, R, mn, 0.4, ref)
    assert bool((~torch.isfinite(out[covered])).all())
    assert bool((out[~covered] == ref[~covered]).all())
