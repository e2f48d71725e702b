"""The filter's staging (tonemap_filter_kernel): tiles of every size, bins stored by column modulo ss up to 8 and
plainly above, windows wider and narrower than a pixel's bins, images smaller than a tile; against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ss,ow,oh,radius,shape", [
    (1, 5, 3, 0.5, 0), (1, 33, 9, 3.0, 2), (2, 70, 19, 1.0, 0), (3, 31, 8, 1.0, 3), (4, 40, 17, 2.5, 0), (5, 65, 9, 0.4, 1),
    (8, 33, 10, 1.0, 0), (8, 12, 9, 2.4, 0), (9, 20, 9, 1.0, 0), (12, 9, 5, 1.7, 0), (12, 9, 5, 0.02, 1), (20, 4, 3, 1.0, 0), (31, 3, 2, 1.0, 3),
])
def test_filter_tiles_match_the_oracle(rk, orc, ss, ow, oh, radius, shape):
    w, h = ow * ss, oh * ss
    r = np.random.default_rng(ss * 100 + ow)
    a = r.poisson(r.exponential(20.0, (h, w))).astype(np.float32)
    bins = np.stack([a * r.uniform(0, 1, (h, w)), a * r.uniform(0, 1, (h, w)), a * r.uniform(0, 1, (h, w)), a], -1).astype(np.float32)
    b = torch.from_numpy(bins).cuda()
    img = torch.zeros(oh, ow, 4, device="cuda")
    rk.tonemap_filter(b, w, h, ss, radius, shape, 2.2, 4.0, 1.0, 0.05, out_f32=img)
    ref = orc.tonemap_filter(bins, ss, radius, shape, 2.2, 4.0, 1.0, 0.05)
    # sums of at most 64 + 64 products of terms >= 0, a log1p, two divisions and a power of a few ulp each, of values
    # up to 1 after the clamp: below 160 roundings of 2^-24 on either side
    assert np.allclose(img.cpu().numpy()[..., :3], np.asarray(ref)[..., :3], rtol=0, atol=2 * 160 * 2.0 ** -24)
