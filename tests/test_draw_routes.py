"""The routes of drawing calls on large bin grids (planes, records, point lists) and the memory they hold
(tests/cpp/draw_routes.cpp: the host code over a fake CUDA runtime; no GPU)."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "refrakt_gb300", "csrc")


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("routes") / "draw_routes")
    srcs = [os.path.join(ROOT, "tests", "cpp", "draw_routes.cpp")] + [os.path.join(CSRC, n + ".cpp") for n in
                                                                     ("genome", "parsers", "registry", "snippet_hashes")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", "/usr/local/cuda/include"] + srcs + ["-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scene", ["failed_call", "faster_form", "own_view", "memory", "captured"])
def test_routes(routes, scene):
    r = subprocess.run([routes, scene], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
