"""What the device code must not rely on, read from its source: such faults need not show in a run of the code as
one compiler builds it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "refrakt_gb300", "csrc")


def _code(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_cluster_barriers_take_parted_warps():
    # the arrival and the wait follow lane-divergent code; PTX: .aligned is undefined unless the warp executes it together
    ops = re.findall(r"barrier\.cluster\.[\w.]+", _code("chaos_body.cuh"))
    assert len(ops) == 2 and not any("aligned" in o for o in ops)


def test_tensor_memory_reads_meet_first():
    # tcgen05.ld is .sync.aligned, and its callers store under conditions and wait in loops lane by lane
    body = re.search(r"void tmem_ld16\(.*?\n}", _code("umma.cuh"), re.S).group(0)
    assert 0 < body.find("__syncwarp()") < body.find("tcgen05.ld")
    # a warp that reads an accumulator gives up on its wait as a whole, or the others would wait for the lanes that left
    for name in ("gemm.cu", "conv.cu"):
        code = _code(name)
        assert "mbar_wait_warp(&" in code and not re.search(r"mbar_wait\(&(B\.)?acc_full", code)
