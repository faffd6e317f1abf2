"""The tensor-core convolutions where every CTA takes many tiles: three halo stages and two accumulator
sets of the forward and data-gradient kernel, two stages and the accumulation over tiles of the
weight-gradient kernel come round several times, on tile counts that are no multiple of the grid.
Reference: the same sums in FP64 torch."""
import math

import pytest

from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
ws = fem.warmstart

ROWS, SEG = 4, 128      # a tile: output rows, pixels of a row
PER_SM = 2              # most CTAs an SM holds (their stages take 79.5 KB or more)


def shape(W, per_cta):
    """B, H of at least per_cta tiles for each of PER_SM CTAs an SM; a ragged last tile row, and a count
    that no grid of one or two CTAs an SM divides."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nseg = -(-W // SEG)
    B = 3
    rows = -(-(per_cta * PER_SM * sms + 7) // (B * nseg))
    while any((B * nseg * rows) % (k * sms) == 0 for k in (1, 2)):
        rows += 1
    return B, ROWS * rows - 1, B * nseg * rows, sms


def data(seed, *s):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)


def shifts(x):
    """x moved by each of the nine taps, zero outside the grid: (tap, B, H, W, c) in FP64."""
    B, H, W, c = x.shape
    p = torch.zeros(B, H + 2, W + 2, c, dtype=torch.float64, device="cuda")
    p[:, 1:-1, 1:-1] = x.double()
    for ky in range(3):
        for kx in range(3):
            yield 3 * ky + kx, p[:, ky:ky + H, kx:kx + W]


# seven tiles a CTA: stages (3) and accumulator sets (2) come round, both mbarriers pass two phases
@pytest.mark.parametrize("ci,co", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("W", [6, 133])
def test_forward(ci, co, mode, W):
    B, H, _, _ = shape(W, 7)
    x = data(ci + co + mode + W, B, H, W, ci)
    w = torch.zeros(co, 9 * ci + 8, device="cuda", dtype=torch.bfloat16)
    w[:, :9 * ci] = 0.2 * data(1 + ci, co, 9 * ci)
    b = 0.1 * data(2 + co, co).float() if mode != 2 else None
    mask = data(3 + co, B, H, W, co) if mode == 2 else None
    out = torch.full((B, H, W, co), 9.0, device="cuda", dtype=torch.float32 if mode == 1 else torch.bfloat16)
    lib, h = fem.solver._Handle.get()
    assert lib.femb200_conv3x3_forward(h, ws._p(x), ws._p(w), ws._p(b), ws._p(mask), ws._p(out), B, H, W, ci, co, mode) == 0
    torch.cuda.synchronize()
    want = 0.0
    for tap, s in shifts(x):
        want = want + s @ w[:, tap * ci:(tap + 1) * ci].double().T
    want = (want + b.double()).clamp(min=0) if mode == 0 else want + b.double() if mode == 1 else want * (mask > 0)
    # FP32 sums of 9·ci products (their rounding: below 300 units in the last place of their scale); BF16
    # outputs are rounded by half of 2⁻⁸ of themselves
    tol = 300 * 2.0 ** -24 if mode == 1 else 2.0 ** -8
    assert float((out.double() - want).abs().max()) <= tol * float(want.abs().max())


# five tiles a CTA: both stages and mbarriers pass two phases
@pytest.mark.parametrize("ci,co", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("W", [6, 133])
def test_weight_and_bias_gradient(ci, co, W):
    B, H, tiles, sms = shape(W, 5)
    x, dy = data(5 + ci + W, B, H, W, ci), data(6 + co + W, B, H, W, co)
    dw = torch.zeros(co, 9 * ci + 8, device="cuda")
    db = torch.full((co,), 2.0, device="cuda")
    lib, h = fem.solver._Handle.get()
    assert lib.femb200_conv3x3_weight_grad(h, ws._p(x), ws._p(dy), ws._p(dw), ws._p(db), B, H, W, ci, co) == 0
    torch.cuda.synchronize()
    d = dy.double().reshape(-1, co)
    # an accumulator takes 32 additions a tile over a CTA's tiles (one CTA an SM at least), then one of each
    # CTA: no more roundings of 2⁻²³ than additions
    steps = 32 * math.ceil(tiles / sms) + PER_SM * sms
    top = 0.0
    err = 0.0
    for tap, s in shifts(x):
        want = d.T @ s.reshape(-1, ci)
        top = max(top, float(want.abs().max()))
        err = max(err, float((dw[:, tap * ci:(tap + 1) * ci].double() - want).abs().max()))
    assert err <= steps * 2.0 ** -23 * top
    assert bool((dw[:, 9 * ci:] == 0).all())
    # a thread sums up to 4 rows · SEG pixels of its CTA's tiles; the sum's magnitude bounds every partial
    n = 4 * SEG * math.ceil(tiles / sms) + 64 * PER_SM * sms
    assert bool(((db.double() - 2.0 - d.sum(0)).abs() <= n * 2.0 ** -24 * d.abs().sum(0)).all())
    assert bool(((db.double() - 2.0 - d.sum(0)).abs() <= 0.01 * math.sqrt(len(d))).all())
