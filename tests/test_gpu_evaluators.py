"""The generated evaluator of a genome whose xforms share structures (one body per distinct structure) against
the interpreter: the same counts, whichever xforms are alike and wherever they stand."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = {  # a structure: variations and parameters, post transform
    "A": dict(vars={"linear": 0.6, "spherical": 0.2}),
    "B": dict(vars={"julian": 0.7, "pre_blur": 0.05}, params={"julian_power": 3, "julian_dist": 1}),
    "C": dict(vars={"sinusoidal": 0.8, "blur": 0.1}, post=(0.9, 0.1, -0.1, 0.9, 0.1, 0)),
    "D": dict(vars={"linear": 0.6, "spherical": 0.2}, post=(1, 0, 0, 1, 0.05, 0)),  # A with a post transform
}


@pytest.mark.parametrize("pattern,final", [("A", None), ("AAA", "C"), ("ABA", None), ("AAB", "A"), ("BAAB", "B"), ("ADCBADCB", "D"),
                                           ("A" * 20 + "B", None)])
def test_shared_bodies_equal_the_interpreter(rk, compiler, pattern, final):
    def xform(k, kind):
        t = 2.4 * k
        return dict({"weight": 0.2 + 0.1 * k, "color": k / len(pattern), "color_speed": 0.5, "opacity": 1.0 - 0.02 * k,
                     "coefs": (0.6 * np.cos(t), 0.6 * np.sin(t), -0.6 * np.sin(t), 0.6 * np.cos(t), 0.4 * np.cos(3 * t), 0.3 * np.sin(k))},
                    **KINDS[kind])
    pal = [(i / 256.0, 1 - i / 256.0, 0.5) for i in range(256)]
    g = {"size": (200, 150), "center": (0.0, 0.0), "scale": 60, "rotate": 0, "estimator": (9, 0, 0.4), "gamma": 2.2, "vibrancy": 1,
         "brightness": 4, "palette": pal, "xforms": [xform(k, c) for k, c in enumerate(pattern)]}
    if final:
        g["final_xform"] = dict(xform(1, final), weight=0)
    f = rk.Flame.from_struct(compiler, g)
    out = []
    for specialize in (1, -1):
        sim = rk.Sim(8192, seed=3, cta_slots=2048, specialize=specialize)
        sim.set_bad_value_reset(True)
        sim.warmup(f, 9)
        bins = torch.zeros(150, 200, 4, device="cuda")
        hits = torch.zeros(150, 200, dtype=torch.int32, device="cuda")
        drawn = sim.draw_to_bins(f, bins, hits, 200, 150, 60)
        out.append((hits.cpu().numpy(), drawn, bins.cpu().numpy().astype(np.float64)))
        sim.close()
    assert out[0][1] == out[1][1] > 0
    assert np.array_equal(out[0][0], out[1][0])
    n = np.maximum(out[0][0], 1)[..., None]  # the sums differ by their order of addition only
    assert np.all(np.abs(out[0][2] - out[1][2]) <= 2 * n * 2.0 ** -24 * np.maximum(out[0][2], out[1][2]) + 1e-30)
