"""The loss gradient in its two forms (eight channels a thread, one where the gradient is off 16-byte
alignment or the channels are no multiple of eight) and the bias gradient summed beside the weight
gradient on partial tiles."""
import ctypes as C

import numpy as np
import pytest

from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def lib():
    from importlib import import_module
    return import_module(fem.__name__ + ".solver")._Handle.get()


# the gradient is rounded to BF16 (2⁻⁹ of it), the loss summed in FP64 from FP32 differences
@pytest.mark.parametrize("nt,co,npix,offset", [(3, 16, 1, 0), (3, 16, 1000, 0), (3, 16, 1000, 1), (8, 24, 77, 0), (11, 32, 300, 0),
                                               (5, 12, 64, 0)])
def test_mse(nt, co, npix, offset):
    L, h = lib()
    g = torch.Generator(device="cuda").manual_seed(co + npix)
    out = torch.randn(npix, co, generator=g, device="cuda")
    tgt = torch.randn(npix, nt, generator=g, device="cuda")
    dy = torch.full((npix * co + offset,), 7.0, dtype=torch.bfloat16, device="cuda")[offset:]
    loss = C.c_double()
    p = lambda t: C.c_void_p(t.data_ptr())
    assert L.femb200_mse_loss_grad(h, p(out), p(tgt), nt, co, 0.25, p(dy), npix, C.byref(loss)) == 0
    d = (out[:, :nt] - tgt).double()
    want = torch.zeros(npix, co, dtype=torch.float64, device="cuda")
    want[:, :nt] = 0.5 * d
    assert float((dy.view(npix, co).double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    assert abs(loss.value - 0.25 * float((d * d).sum())) <= 1e-6 * loss.value


# FP32 sums of at most 5 000 BF16 values of both signs: 5 000 units in the last place of their magnitude
@pytest.mark.parametrize("ci,co", [(16, 16), (32, 16), (16, 32), (32, 32)])
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 5, 131), (1, 9, 513)])
def test_bias_gradient(ci, co, B, H, W):
    L, h = lib()
    g = torch.Generator(device="cuda").manual_seed(ci * co + W)
    x = torch.randn(B, H, W, ci, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(B, H, W, co, generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.zeros(co, 9 * ci + 8, device="cuda")
    db = torch.full((co,), 3.0, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    assert L.femb200_conv3x3_weight_grad(h, p(x), p(dy), p(dw), p(db), B, H, W, ci, co) == 0
    torch.cuda.synchronize()
    want = 3.0 + dy.double().reshape(-1, co).sum(0)
    mag = 3.0 + dy.double().abs().reshape(-1, co).sum(0)
    assert bool(((db.double() - want).abs() <= 5000 * 6e-8 * mag).all())
