"""Records and point lists hold device memory one in the other's place while a genome's first calls try both, and the
draws go on with the same counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_one_form_holds_memory(rk, compiler):
    w, h, passes = 8192, 4111, 100
    f = rk.Flame.synthesize(compiler, rk.SYNTH_CONTRACT, 4, w, h)  # a dust of hot bins
    got = {}
    for layout in (rk.BINS_AUTO, rk.BINS_DIRECT):
        sim = rk.Sim(311296, cta_slots=2048, seed=5)
        sim.set_bin_layout(layout)
        sim.warmup(f, 9)
        bins = torch.zeros(h, w, 4, device="cuda")
        hits = torch.zeros(h, w, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        free, drawn = [torch.cuda.mem_get_info()[0]], []
        for _ in range(5):
            drawn.append(sim.draw_to_bins(f, bins, hits, w, h, passes))
            free.append(torch.cuda.mem_get_info()[0])
        got[layout] = hits, drawn
        if layout == rk.BINS_AUTO:
            lists, records = 311296 * passes * 8 * 4, w * h * 32  # 1.0e9 and 1.1e9 bytes
            held = [free[0] - x for x in free[1:]]
            assert abs(held[0] - lists) < lists // 4  # the lists' scratch planes and heads besides
            assert abs(held[1] - records) < records // 8
            assert held[2] in held[:2] and held[2] == held[3] == held[4]
        sim.close()
    assert got[rk.BINS_AUTO][1] == got[rk.BINS_DIRECT][1]
    assert torch.equal(got[rk.BINS_AUTO][0], got[rk.BINS_DIRECT][0])
