"""The weight gradients of single layers (conv_wgrad_kernel) against FP64 sums of the same BF16 products: windows of
every width with neighbours inside the row, in more than 16 planes (the 160-channel decoder layer), upsampled and
concatenated inputs, rows that are no multiple of 8 pixels, the 1x1 head, one and several splits.  All values are
positive, so a neighbour or a row end that is lost or taken twice shows."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

SHIM = """
#include "conv.h"
#include "error_word.h"
using namespace rfk;
extern "C" __attribute__((visibility("default"))) int layer_wgrad(const void* xa, uint32_t ca, int up, const void* xb, uint32_t cb,
    uint32_t n, uint32_t h, uint32_t w, uint32_t taps, void* dz, uint32_t cout, uint32_t ldz, float* gw) {
    ErrorWord word;
    if (!word.acquire()) return -1;
    WgradTask t{};
    t.conv.xa = static_cast<const __nv_bfloat16*>(xa);
    t.conv.xb = static_cast<const __nv_bfloat16*>(xb);
    t.conv.ca = ca;
    t.conv.cb = cb;
    t.conv.up = up;
    t.conv.n = n;
    t.conv.h = h;
    t.conv.w = w;
    t.conv.taps = taps;
    t.conv.dz = static_cast<__nv_bfloat16*>(dz);
    t.cout = cout;
    t.ldz = ldz;
    t.gw = gw;
    cudaError_t e = launch_conv_wgrad(&t, 1, nullptr, 0, nullptr, word.get(), nullptr);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return e != cudaSuccess ? (int)e : -word.take();
}
"""


@pytest.fixture(scope="module")
def layer_wgrad(rk, tmp_path_factory):
    from refrakt_gb300 import nvbuild
    d = tmp_path_factory.mktemp("wgrad")
    src, lib = d / "wgrad.cpp", d / "wgrad.so"
    src.write_text(SHIM)
    objs = [os.path.join(nvbuild.OBJ_DIR, o) for o in ("conv.cu.o", "error_word.cpp.o")]
    subprocess.run([nvbuild.NVCC] + nvbuild._flags() + ["-shared", "-o", str(lib), str(src)] + objs, check=True, capture_output=True)
    f = ctypes.CDLL(str(lib)).layer_wgrad
    p, u = ctypes.c_void_p, ctypes.c_uint32
    f.argtypes = [p, u, ctypes.c_int, p, u, u, u, u, u, p, u, u, p]
    return f


@pytest.mark.parametrize("n,h,w,ca,cb,cout,taps,up", [
    (2, 20, 24, 96, 64, 64, 9, True), (2, 20, 40, 96, 64, 64, 9, True), (1, 24, 48, 96, 64, 64, 9, True),
    (1, 24, 80, 96, 64, 64, 9, True), (1, 10, 64, 96, 64, 64, 9, True), (1, 16, 128, 160, 0, 64, 9, False), (1, 9, 24, 0, 160, 64, 9, False),
    (2, 16, 24, 64, 48, 48, 9, True), (1, 40, 56, 8, 0, 32, 9, False), (1, 24, 96, 32, 0, 32, 9, False), (3, 7, 8, 96, 0, 96, 9, False),
    (2, 12, 6, 96, 64, 64, 9, True), (2, 18, 18, 48, 0, 64, 9, False), (8, 1, 1, 64, 0, 96, 9, False), (1, 33, 9, 96, 0, 96, 9, False),
    (2, 128, 192, 32, 0, 32, 9, False), (1, 256, 256, 48, 32, 32, 9, True), (1, 16, 24, 32, 0, 3, 1, False), (2, 128, 256, 32, 0, 3, 1, False)])
def test_layer_weight_gradient(layer_wgrad, n, h, w, ca, cb, cout, taps, up):
    g = torch.Generator(device="cuda").manual_seed(n + 3 * h + 5 * w + ca)
    rand = lambda *s: (0.5 + torch.rand(*s, device="cuda", generator=g)).bfloat16()
    xa = rand(n, h // 2, w // 2, ca) if up else rand(n, h, w, ca) if ca else None
    xb = rand(n, h, w, cb) if cb else None
    if not ca:
        xa, ca, xb, cb = xb, cb, None, 0
    ldz = (cout + 7) // 8 * 8
    dz = torch.zeros(n, h, w, ldz, device="cuda", dtype=torch.bfloat16)
    dz[..., :cout] = rand(n, h, w, cout)
    C = ca + cb
    gw = torch.ones(cout, taps * C, device="cuda")
    ptr = lambda t: None if t is None else t.data_ptr()
    torch.cuda.synchronize()
    assert layer_wgrad(ptr(xa), ca, int(up), ptr(xb), cb, n, h, w, taps, ptr(dz), cout, ldz, ptr(gw)) == 0
    x = xa.double()
    if up:
        x = x.repeat_interleave(2, 1).repeat_interleave(2, 2)
    if cb:
        x = torch.cat([x, xb.double()], -1)
    side = 3 if taps == 9 else 1
    pad = torch.nn.functional.pad(x, (0, 0, side // 2, side // 2, side // 2, side // 2))
    z = dz[..., :cout].double().reshape(-1, cout).t()
    want = torch.stack([z @ pad[:, dy:dy + h, dx:dx + w].reshape(-1, C) for dy in range(side) for dx in range(side)], 1).reshape(cout, taps * C)
    # products of BF16 are exact in FP32; one addition a pixel, rounded or truncated at 2^-23 of a partial sum, and one a split
    tol = (n * h * w + 65) * 2.0 ** -23 * want
    assert bool(((gw.double() - 1 - want).abs() <= tol + 1e-5).all())
