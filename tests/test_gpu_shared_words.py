"""The interpreter's program words (SharedWords, variations.cuh) are reads of memory to the compiler: a kernel that
rewrites the program between two evaluations gets the new program's values, with the same arguments."""
import ctypes
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

SOURCE = """
#include <cuda_runtime.h>
#include "variations.cuh"
using namespace rfk;

// src: two programs of 64 words; out: word 3, the xform's colour and opacity, for each
__global__ void twice(const uint32_t* src, float* out) {
    __shared__ uint32_t s[64];
    const SharedWords w{(uint32_t)__cvta_generic_to_shared(s)};
    for (int k = 0; k < 2; k++) {
        __syncthreads();
        s[threadIdx.x] = src[64 * k + threadIdx.x];
        __syncthreads();
        const float word = w[X_COLOR];
        const XformOut o = eval_xform(w.a, 0.25f, 0.5f, 0.75f, false, Jsf{1, 2, 3, 4});
        if (threadIdx.x == 0) {
            out[3 * k] = word;
            out[3 * k + 1] = o.c;
            out[3 * k + 2] = o.op;
        }
    }
}
extern "C" __attribute__((visibility("default"))) int run_twice(const uint32_t* src, float* out) {
    twice<<<1, 64>>>(src, out);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
"""


def test_a_rewritten_program_is_read_again(rk, tmp_path):
    from refrakt_gb300 import nvbuild
    src, lib = tmp_path / "words.cu", tmp_path / "words.so"
    src.write_text(SOURCE)
    subprocess.run([nvbuild.NVCC] + nvbuild._flags() + ["-shared", "-o", str(lib), str(src)], check=True, capture_output=True)
    f = ctypes.CDLL(str(lib)).run_twice
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    x_color, x_cs, x_omcs, x_opacity = 16, 17, 18, 19  # program.h; no terms, no post transform
    prog = torch.zeros(2, 64, dtype=torch.float32, device="cuda")
    prog[0, x_color], prog[0, x_cs], prog[0, x_omcs], prog[0, x_opacity] = 0.5, 0.5, 0.5, 0.125
    prog[1, x_color], prog[1, x_cs], prog[1, x_omcs], prog[1, x_opacity] = 1.0, 0.25, 0.75, 0.5
    out = torch.full((6,), -1.0, device="cuda")
    torch.cuda.synchronize()
    assert f(prog.data_ptr(), out.data_ptr()) == 0
    assert out.tolist() == [0.5, 0.75 * 0.5 + 0.25, 0.125, 1.0, 0.75 * 0.75 + 0.25, 0.5]
