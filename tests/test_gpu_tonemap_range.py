"""The tonemap at vibrancy 1 over colours whose power overflows FP32 (gamma below 1) or is not defined: the
formula of tonemap.glsl:28-37 in FP32, where infinity times zero is NaN and NaN clamps to zero."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(bins, gamma, brightness, k2):
    f = np.float32
    c = bins.reshape(-1, 4)
    with np.errstate(all="ignore"):
        ls = f(0.5) * f(brightness) * np.log10(f(1) + c[:, 3:] * f(k2)).astype(f) / c[:, 3:]
        c = (c * ls).astype(f)
        ig = f(1) / f(gamma)
        gf = np.power(c[:, 3:], ig).astype(f) / c[:, 3:]
        v = np.power(c[:, :3], ig).astype(f) * f(0) + gf * c[:, :3]
    return np.nan_to_num(np.clip(np.nan_to_num(v, nan=0.0, posinf=np.inf, neginf=-np.inf), 0, 1)).reshape(bins.shape[0], bins.shape[1], 3)


@pytest.mark.parametrize("gamma", [0.05, 0.2, 0.9, 1.0, 2.2, 50.0])
def test_vibrancy_one_over_the_range(rk, gamma):
    colours = [0.0, -1.0, 1e-30, 0.01, 0.3, 2.0, 1e4, 1e12, 1e30, -1e30]
    bins = np.zeros((32, 64, 4), np.float32)
    for i in range(bins[..., 0].size):
        bins[i // 64, i % 64] = [colours[(i + q * (1 + i // 10)) % 10] for q in range(3)] + [1.0 + i % 7]
    b = torch.from_numpy(bins).cuda()
    want = _expected(bins, gamma, 4.0, 1.0)
    for f in (lambda o: rk.tonemap(b, 64, 32, 1, gamma, 4.0, 1.0, 1.0, out_f32=o),
              lambda o: rk.density_tonemap(b, 64, 32, 0, 0, 0.4, 1, gamma, 4.0, 1.0, 1.0, out_f32=o),
              lambda o: rk.tonemap_filter(b, 64, 32, 1, 0.3, rk.FILTER_BOX, gamma, 4.0, 1.0, 1.0, out_f32=o)):
        out = torch.full((32, 64, 4), -1.0, device="cuda")
        f(out)
        # the value before the clamp is a power of exponent up to 20 of a number with a few ulp of error: 20 * 8 ulp
        assert np.allclose(out.cpu().numpy()[..., :3], want, rtol=160 * 2.0 ** -24, atol=1e-30)
