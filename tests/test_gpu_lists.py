"""Draws through point lists (splat_list, range_step_kernel) on grids of 2^25 bins and more, against draws
straight into the planes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _square(rk, compiler, w, h, opacity, final=False, part=0.45):
    """Four half-size copies of a square, one per corner: points uniform over `part` of the frame to each side."""
    xs = [{"weight": 1, "color": k / 3, "color_speed": 0.5, "opacity": opacity[k], "vars": {"linear": 1},
           "coefs": (0.5, 0, 0, 0.5, 0.5 * (2 * (k & 1) - 1), 0.5 * (2 * (k >> 1) - 1))} for k in range(4)]
    g = {"size": (w, h), "center": (0.0, 0.0), "scale": part * min(w, h), "rotate": 7, "estimator": (9, 0, 0.4), "gamma": 2.2,
         "vibrancy": 1, "brightness": 4, "palette": [(i / 256.0, 1 - i / 256.0, 0.5) for i in range(256)], "xforms": xs}
    if final:
        g["final_xform"] = {"weight": 0, "color": 0.3, "color_speed": 0.2, "opacity": 0.75, "vars": {"linear": 1},
                            "coefs": (1, 0.1, -0.1, 1, 0, 0)}
    return rk.Flame.from_struct(compiler, g)


@pytest.mark.parametrize("genome,w,h,walkers,slots,passes,specialize", [
    ("unit", 8192, 4111, 155648, 1024, 24, 0),     # opacity 1; 17 ranges, the last one partial
    ("mixed", 8192, 4111, 155648, 1024, 24, 0),    # opacities 1 and others in one warp's ranges
    ("final", 8191, 4111, 155648, 2048, 24, -1),   # no point of opacity 1; the interpreter
    ("unit", 4096, 8192, 155648, 1024, 3, 0),      # exactly 2^25 bins; lists of a few points
    ("mixed", 8192, 4111, 622592, 4096, 256, 0),   # ranges of 2^20 bins
    ("small", 8192, 4111, 622592, 4096, 256, 0),   # one range, 2^24 points and more: counts apart from alpha; full lists
    ("contract", 8192, 4111, 155648, 1024, 40, 0),  # a dust of hot bins: the bins, then records
    ("random", 8192, 5000, 311296, 2048, 40, 0),   # uneven ranges
])
def test_lists_equal_direct_planes(rk, compiler, genome, w, h, walkers, slots, passes, specialize):
    if genome == "contract":
        f = rk.Flame.synthesize(compiler, rk.SYNTH_CONTRACT, 4, w, h)
    elif genome == "random":
        f = rk.Flame.synthesize(compiler, rk.SYNTH_RANDOM, 1, w, h, n_xforms=8, final_xform=True, force_parametric=True)
    else:
        f = _square(rk, compiler, w, h, {"unit": (1, 1, 1, 1)}.get(genome, (1, 0.5, 1, 0.25)), genome == "final",
                    0.02 if genome == "small" else 0.45)
    got = {}
    for layout in (rk.BINS_DIRECT, rk.BINS_AUTO):
        sim = rk.Sim(walkers, cta_slots=slots, seed=5, specialize=specialize)
        sim.set_bad_value_reset(True)
        sim.set_bin_layout(layout)
        sim.warmup(f, 9)
        bins = torch.zeros(h, w, 4, device="cuda")
        hits = torch.zeros(h, w, dtype=torch.int32, device="cuda")
        drawn = [sim.draw_to_bins(f, bins, hits, w, h, passes) for _ in range(3)]
        got[layout] = (bins, hits, drawn)
        sim.close()
    (b0, h0, d0), (b1, h1, d1) = got[rk.BINS_DIRECT], got[rk.BINS_AUTO]
    assert d0 == d1 and sum(d1) == int(h1.sum(dtype=torch.int64)) > 0
    assert torch.equal(h0, h1)
    # both are FP32 sums of the same n terms >= 0 in some order: each within n 2^-24 of the exact sum
    tol = 2.0 * (h0[..., None].double() + 4) * 2.0 ** -24 * torch.maximum(b0, b1).double()
    assert bool(((b0.double() - b1.double()).abs() <= tol).all())
