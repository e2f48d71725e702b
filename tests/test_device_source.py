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
