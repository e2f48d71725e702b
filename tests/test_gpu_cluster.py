"""The cluster walker exchange (chaos_body.cuh, CLUSTER) against one CTA per mixing domain: the same
counts, drawn points, emitted points and xform ids on a nonlinear genome with the walker reset, a final
xform and RNG-drawing variations, at cluster sizes 8, 4 and 2 and 256 to 2048 slots per CTA (two per
thread), with several temporal samples, launches shorter than the pass count, and a tile splat."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(rk, f, walkers, slots, exchange, T, L, tile):
    sim = rk.Sim(walkers, temporal_samples=T, seed=11, cta_slots=slots, steps_per_launch=L)
    sim.set_bad_value_reset(True)
    sim.set_exchange(exchange)
    if tile:
        sim.set_splat(rk.SPLAT_TILE)
        sim.set_splat_tile(30, 20, 40, 30)
    sim.enable_xid_trace(8 + 80)
    sim.warmup(f, 7, 0.3 if T > 1 else 0.02)
    assert sim.specialized()
    bins = torch.zeros(96, 128, 4, device="cuda")
    hits = torch.zeros(96, 128, dtype=torch.int32, device="cuda")
    drawn = [sim.draw_to_bins(f, bins, hits, 128, 96, n) for n in (40, 33, 7)]
    out = hits.cpu().numpy(), drawn, sim.counters(), sim.read_xid_trace(88), bins.cpu().numpy()
    sim.close()
    return out


@pytest.mark.parametrize("walkers,slots,T,L,tile", [(4096, 4096, 1, 0, False), (8192, 2048, 1, 16, False), (32768, 1024, 4, 0, False),
                                                    (65536, 4096, 2, 0, True), (65536, 2048, 1, 0, False), (512, 512, 1, 0, False),
                                                    (131072, 4096, 1, 32, False), (262144, 4096, 1, 0, False), (61440, 1024, 1, 0, False)])
def test_cluster_exchange_equals_single_ctas(rk, compiler, walkers, slots, T, L, tile):
    f = rk.Flame.synthesize(compiler, rk.SYNTH_RANDOM, 5, 128, 96, n_xforms=5, final_xform=True, force_parametric=True)
    got = _run(rk, f, walkers, slots, rk.EXCHANGE_AUTO, T, L, tile)
    want = _run(rk, f, walkers, slots, rk.EXCHANGE_BARRIER, T, L, tile)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1] and got[2] == want[2]
    assert np.array_equal(got[3], want[3])
    # the colour sums differ by their order of addition only: at most count * 2^-24 of a sum of
    # non-negative terms on either side
    n = np.maximum(want[0], 1)[..., None]
    assert np.all(np.abs(got[4].astype(np.float64) - want[4]) <= 2 * n * 2.0 ** -24 * want[4] + 1e-30)
