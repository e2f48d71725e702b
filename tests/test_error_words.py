"""A tensor-core kernel's bounded wait that runs out reaches the caller whose kernel it was (tests/cpp/error_words.cpp:
the host path over a fake CUDA runtime; no GPU)."""
import os
import subprocess

from conftest import ROOT


def test_waits_that_run_out_reach_their_caller(tmp_path):
    exe = str(tmp_path / "error_words")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "refrakt_gb300", "csrc"),
                    "-I", "/usr/local/cuda/include", os.path.join(ROOT, "tests", "cpp", "error_words.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
